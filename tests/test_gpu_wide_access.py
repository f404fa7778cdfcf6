"""Decoders with every alignment of images and rows: aligned
ones take 16-byte accesses, the others narrower ones, and the bytes are the
same.  Sizes sit at the edges of a block, of a quad of pixels and of a CTA."""
import numpy as np
import pytest

from texpresso_gb300 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("fmt", range(5))
@pytest.mark.parametrize("w,h", [(1, 1), (4, 4), (5, 9), (130, 7), (516, 12)])
@pytest.mark.parametrize("offset,pad", [(0, 0), (0, 16), (4, 4), (0, 4), (1, 3), (16, 1)])
def test_decode_alignments(tx, cuda, oracle, fmt, w, h, offset, pad):
    f = tx.Format(fmt)
    rng = np.random.default_rng(1000 * fmt + w)
    data = rng.integers(0, 256, f.compressed_size(w, h)).astype(np.uint8)  # any bytes are blocks
    ref = oracle.decompress(fmt, data, w, h).reshape(h, w * 4)
    pitch = w * 4 + pad
    src = cuda.from_numpy(data).cuda()
    out = cuda.full((offset + pitch * h + 16,), 77, dtype=cuda.uint8, device="cuda")
    tx.decompress_device(f, src.data_ptr(), data.size, w, h, out.data_ptr() + offset, pitch,
                         cuda.cuda.current_stream().cuda_stream)
    got = out.cpu().numpy()
    rows = got[offset:offset + pitch * h].reshape(h, pitch)
    assert np.array_equal(rows[:, :w * 4], ref)
    assert (rows[:, w * 4:] == 77).all() and (got[:offset] == 77).all() and (got[offset + pitch * h:] == 77).all()
