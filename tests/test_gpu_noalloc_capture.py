"""The allocation-free batch launch under stream capture: one call with one item
does all set-up, so the next may capture every kernel.  Runs in a process of its
own, where no other test has loaded a kernel."""
import ctypes
import os
import subprocess
import sys

import numpy as np
import pytest

ROOT = os.path.dirname(os.path.dirname(os.path.abspath(__file__)))


@pytest.mark.gpu
def test_first_call_then_capture(cuda, oracle):
    r = subprocess.run([sys.executable, os.path.abspath(__file__)], cwd=ROOT, capture_output=True, text=True, timeout=300)
    assert r.returncode == 0, r.stdout + r.stderr


def main():
    import torch
    import texpresso_gb300 as tx
    from oracle import oracle
    from texpresso_gb300 import workloads

    launch = tx.library().tx_batch_launch_noalloc
    launch.argtypes = [ctypes.POINTER(tx.BatchItem), ctypes.c_size_t, ctypes.c_void_p]
    w, h = 61, 34
    img = workloads.ramp_texture(w, h, seed=3, alpha="ramp")
    src = torch.from_numpy(img).cuda()
    items, outs = [], []
    for fmt in range(5):
        for alg in range(3):
            p = tx.Params(algorithm=tx.Algorithm(alg))
            out = torch.zeros(tx.Format(fmt).compressed_size(w, h), dtype=torch.uint8, device="cuda")
            items.append(tx.batch_item(fmt, src.data_ptr(), w * 4, w, h, p, out.data_ptr()))
            outs.append((fmt, alg, out))
    stream = torch.cuda.Stream()
    torch.cuda.synchronize()
    assert launch((tx.BatchItem * 1)(items[-1]), 1, stream.cuda_stream) == 0  # BC5
    torch.cuda.synchronize()
    graph = torch.cuda.CUDAGraph()
    with torch.cuda.graph(graph, stream=stream):
        assert launch((tx.BatchItem * len(items))(*items), len(items), stream.cuda_stream) == 0
    graph.replay()
    torch.cuda.synchronize()
    for fmt, alg, out in outs:
        ref = oracle.compress(fmt, img, w, h, oracle.make_params(alg))
        assert np.array_equal(out.cpu().numpy(), ref), (fmt, alg)


if __name__ == "__main__":
    sys.path.insert(0, ROOT)
    main()
