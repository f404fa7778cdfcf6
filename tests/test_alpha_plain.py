"""The alpha books of blocks without pixels of 0 or 255: the builder compiled for
the host against the general ones over every range, and on the GPU blocks whose
range or extremes decide between the two, against the oracle."""
import os
import shutil
import subprocess

import numpy as np
import pytest

from conftest import ROOT


def test_books_on_the_host(tmp_path):
    nvcc = shutil.which("nvcc") or "/usr/local/cuda/bin/nvcc"
    if not os.path.exists(nvcc):
        pytest.skip("nvcc not found")
    exe = str(tmp_path / "test_alpha_plain")
    subprocess.run([nvcc, "-std=c++17", "-O2", "-I", os.path.join(ROOT, "texpresso_gb300", "csrc"),
                    "-I", os.path.join(ROOT, "include"),
                    os.path.join(ROOT, "tests", "cpp", "test_alpha_plain.cu"), "-o", exe], check=True)
    r = subprocess.run([exe], capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


@pytest.mark.gpu
@pytest.mark.parametrize("fmt", [3, 4])
@pytest.mark.parametrize("lowest,highest", [(1, 254), (0, 254), (1, 255), (0, 255), (248, 254), (249, 254), (1, 8)])
def test_blocks(tx, cuda, oracle, fmt, lowest, highest):
    rng = np.random.default_rng(lowest * 256 + highest)
    w, h = 509, 132
    base = rng.integers(lowest, highest + 1, (-(-h // 4), -(-w // 4), 2))
    width = rng.integers(0, 14, base.shape)
    up = lambda a: np.repeat(np.repeat(a, 4, 0), 4, 1)[:h, :w]
    img = np.zeros((h, w, 4), np.uint8)
    img[..., :2] = np.clip(up(base) + rng.integers(0, 256, (h, w, 2)) % (up(width) + 1), lowest, highest)
    f = tx.Format(fmt)
    src = cuda.from_numpy(img).cuda()
    out = cuda.zeros(f.compressed_size(w, h), dtype=cuda.uint8, device="cuda")
    tx.compress_device(f, src.data_ptr(), w * 4, 4, w, h, tx.Params(), out.data_ptr(), out.numel(),
                       cuda.cuda.current_stream().cuda_stream)
    assert np.array_equal(out.cpu().numpy(), oracle.compress(fmt, img, w, h, oracle.make_params(1)))
