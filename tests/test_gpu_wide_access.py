"""Decoders and mip producer with every alignment of images and rows: aligned
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


@pytest.mark.parametrize("channels", [1, 2, 3, 4])
@pytest.mark.parametrize("offset,pad", [(0, 0), (0, 16), (4, 4), (1, 3)])
def test_mip_alignments(tx, cuda, channels, offset, pad):
    rng = np.random.default_rng(channels * 10 + offset)
    sizes = [(1, 1), (2, 1), (1, 5), (3, 3), (8, 2), (9, 7), (16, 16), (511, 5), (512, 6), (1030, 33)]
    sizes += [(int(a), int(b)) for a, b in rng.integers(1, 40, (290, 2))]  # more jobs than one launch takes
    jobs, keep = [], []
    for w, h in sizes:
        img = rng.integers(0, 256, (h, w, channels)).astype(np.uint8)
        dw, dh = max(1, w // 2), max(1, h // 2)
        sp, dp = w * channels + pad, dw * channels + pad
        src = np.zeros(offset + sp * h, np.uint8)
        np.lib.stride_tricks.as_strided(src[offset:], (h, w * channels), (sp, 1))[:] = img.reshape(h, -1)
        s = cuda.from_numpy(src).cuda()
        d = cuda.full((offset + dp * dh + 16,), 77, dtype=cuda.uint8, device="cuda")
        jobs.append((s.data_ptr() + offset, sp, w, h, channels, d.data_ptr() + offset, dp))
        keep.append((img, s, d, dw, dh, dp))
    tx.mip_batch_device(jobs, cuda.cuda.current_stream().cuda_stream)
    for img, _, d, dw, dh, dp in keep:
        got = d.cpu().numpy()
        rows = got[offset:offset + dp * dh].reshape(dh, dp)
        assert np.array_equal(rows[:, :dw * channels], workloads.mip_reference(img).reshape(dh, -1)), img.shape
        assert (rows[:, dw * channels:] == 77).all() and (got[offset + dp * dh:] == 77).all()
