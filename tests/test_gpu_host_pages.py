"""Host-buffer calls on memory of other kinds: page-locked and device memory, and
outputs whose pages nothing has touched."""
import ctypes
import mmap

import numpy as np
import pytest

from texpresso_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", [0, 2, 4])
@pytest.mark.parametrize("where", ["pinned", "device", "untouched"])
def test_memory_kinds(tx, cuda, oracle, fmt, where):
    w, h = 700, 301
    f, p = tx.Format(fmt), tx.Params(algorithm=tx.Algorithm.RangeFit)
    img = workloads.ramp_texture(w, h, seed=fmt, alpha="ramp")
    size = f.compressed_size(w, h)

    def room(n, content=None):
        if where == "untouched" and content is None:
            m = mmap.mmap(-1, n)
            return m, ctypes.addressof(ctypes.c_char.from_buffer(m)), lambda: np.frombuffer(m, np.uint8)
        t = cuda.from_numpy(content.reshape(-1).copy()) if content is not None else cuda.zeros(n, dtype=cuda.uint8)
        t = t.cuda() if where == "device" else t.pin_memory()
        return t, t.data_ptr(), lambda: t.cpu().numpy()

    lib = tx.library()
    src, src_at, _ = room(img.size, img)
    out, out_at, out_bytes = room(size)
    cuda.cuda.synchronize()
    prm = p._c()
    assert lib.tx_compress(fmt, src_at, img.size, w, h, ctypes.byref(prm), out_at, size) == 0
    ref = oracle.compress(fmt, img, w, h, oracle.make_params(0))
    assert np.array_equal(out_bytes(), ref)
    back, back_at, back_bytes = room(img.size)
    cuda.cuda.synchronize()
    assert lib.tx_decompress(fmt, out_at, size, w, h, back_at, img.size) == 0
    assert np.array_equal(back_bytes(), oracle.decompress(fmt, ref, w, h).reshape(-1))
    del src, out, back
