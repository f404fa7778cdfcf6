"""The copying form of the host-buffer calls and the server, which other hosts take
and TX_HOST_COPIES=1 asks for: the tests of host buffers and served levels in such
a process, and images whose bands of block rows are of different sizes."""
import os
import subprocess
import sys

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
ROOT = os.path.dirname(HERE)


def _run(args):
    r = subprocess.run([sys.executable] + args, cwd=ROOT, capture_output=True, text=True, timeout=600,
                       env=dict(os.environ, TX_HOST_COPIES="1"))
    assert r.returncode == 0, r.stdout[-4000:] + r.stderr[-4000:]


@pytest.mark.gpu
def test_host_buffers_and_served_levels(cuda, oracle):
    files = ("test_gpu_host_buffers.py", "test_gpu_served_mips.py", "test_gpu_host_pages.py")
    _run(["-m", "pytest", "-q", "-x", "-m", "gpu", "-p", "no:cacheprovider", "-k", "not device"] +
         [os.path.join(HERE, f) for f in files])


@pytest.mark.gpu
def test_bands(cuda, oracle):
    _run([os.path.abspath(__file__)])


def main():
    import texpresso_gb300 as tx
    from oracle import oracle
    from texpresso_gb300 import workloads

    # block rows: one band, whole bands of 32, one short of tapered bands, tapered
    for h, launches in ((31 * 4, 1), (64 * 4, 2), (99 * 4 - 1, 3), (100 * 4, 9), (231 * 4 + 2, 9)):
        for fmt in range(5):
            w = 61 if fmt % 2 else 64
            f, alg = tx.Format(fmt), (fmt + h) % 2
            img = workloads.ramp_texture(w, h, seed=h + fmt, alpha="ramp")
            out = np.full(f.compressed_size(w, h) + 16, 77, np.uint8)
            before = tx.kernel_launch_count()
            f.compress(img, w, h, tx.Params(algorithm=tx.Algorithm(alg)), out[:-16])
            assert tx.kernel_launch_count() - before == launches, (h, tx.kernel_launch_count() - before)
            ref = oracle.compress(fmt, img, w, h, oracle.make_params(alg))
            assert np.array_equal(out[:-16], ref) and (out[-16:] == 77).all(), (h, fmt)
            back = np.zeros((h, w, 4), np.uint8)
            f.decompress(ref, w, h, back)
            assert np.array_equal(back, oracle.decompress(fmt, ref, w, h).reshape(h, w, 4)), (h, fmt)


if __name__ == "__main__":
    sys.path.insert(0, ROOT)
    main()
