"""Host buffers of every alignment, age and overlap: kernels read and write the
caller's memory where they can, and the bytes are those of the oracle.  Sizes
sit at the edges of a block and of a 16-byte row."""
import numpy as np
import pytest

from texpresso_gb300 import workloads

pytestmark = pytest.mark.gpu

PERCEPTUAL = (0.2126, 0.7152, 0.0722)


def _params(tx, oracle, alg, aw):
    return tx.Params(algorithm=tx.Algorithm(alg), weigh_colour_by_alpha=aw), oracle.make_params(alg, PERCEPTUAL, aw)


@pytest.mark.parametrize("fmt", range(5))
@pytest.mark.parametrize("w,h", [(1, 1), (4, 8), (13, 7), (130, 66)])
@pytest.mark.parametrize("src_off,dst_off", [(0, 0), (1, 8), (4, 16), (16, 1), (0, 4)])
def test_compress_and_decompress(tx, cuda, oracle, fmt, w, h, src_off, dst_off):
    f = tx.Format(fmt)
    alg = (w + fmt) % 3
    p, op = _params(tx, oracle, alg, bool(h % 2))
    room = np.zeros(src_off + w * h * 4, np.uint8)
    size = f.compressed_size(w, h)
    extra = f.block_size()  # a block past the image: no pixel is valid
    out = np.full(dst_off + size + extra + 32, 77, np.uint8)
    back = np.full(dst_off + w * h * 4 + 32, 77, np.uint8)
    for seed in (1, 2):  # the same buffers with other content
        img = workloads.ramp_texture(w, h, seed=seed, alpha="ramp")
        room[src_off:] = img.reshape(-1)
        f.compress(room[src_off:], w, h, p, out[dst_off:dst_off + size + extra])
        ref = oracle.compress(fmt, img, w, h, op)
        assert np.array_equal(out[dst_off:dst_off + size], ref)
        assert (out[:dst_off] == 77).all() and (out[dst_off + size + extra:] == 77).all()
        f.decompress(out[dst_off:dst_off + size], w, h, back[dst_off:dst_off + w * h * 4])
        assert np.array_equal(back[dst_off:dst_off + w * h * 4], oracle.decompress(fmt, ref, w, h).reshape(-1))
        assert (back[:dst_off] == 77).all() and (back[dst_off + w * h * 4:] == 77).all()


@pytest.mark.parametrize("fmt", range(5))
@pytest.mark.parametrize("where", [0, 8, 16, 4096])
def test_output_over_the_input(tx, cuda, oracle, fmt, where):
    f = tx.Format(fmt)
    w, h = 640, 333
    p, op = _params(tx, oracle, 0, False)
    img = workloads.ramp_texture(w, h, seed=5, alpha="ramp")
    size = f.compressed_size(w, h)
    room = img.reshape(-1).copy()
    f.compress(room, w, h, p, room[where:where + size])
    ref = oracle.compress(fmt, img, w, h, op)
    assert np.array_equal(room[where:where + size], ref)
    room = np.zeros(where + w * h * 4, np.uint8)
    room[where:where + size] = ref
    f.decompress(room[where:where + size], w, h, room[:w * h * 4])
    assert np.array_equal(room[:w * h * 4], oracle.decompress(fmt, ref, w, h).reshape(-1))


def test_untouched_and_read_only_memory(tx, cuda, oracle):
    f = tx.Format.Bc3
    w, h = 512, 260
    p, op = _params(tx, oracle, 0, False)
    img = workloads.ramp_texture(w, h, seed=9, alpha="ramp")
    ref = oracle.compress(2, img, w, h, op)
    for src in (bytes(img.reshape(-1)), img):
        out = np.empty(8 << 20, np.uint8)  # pages that nothing has touched
        f.compress(src, w, h, p, out[:ref.size])
        assert np.array_equal(out[:ref.size], ref)
    zero = np.zeros(4 * 1024 * 1024, np.uint8)  # untouched input: the zero page
    out = np.empty(f.compressed_size(1024, 1024), np.uint8)
    f.compress(zero, 1024, 1024, p, out)
    assert np.array_equal(out, oracle.compress(2, np.zeros((1024, 1024, 4), np.uint8), 1024, 1024, op))


@pytest.mark.parametrize("dst_off", [0, 8, 1])
def test_served_output_alignment(tx, cuda, oracle, dst_off):
    srv = tx.Server(memory_budget=256 << 20, step_blocks=4096, min_share=512)
    jobs = []
    for fmt in range(5):
        w, h = 37 + 60 * fmt, 90 - 15 * fmt
        img = workloads.ramp_texture(w, h, seed=fmt, alpha="ramp")
        out = np.full(dst_off + tx.chain_compressed_size(fmt, w, h, True) + 32, 77, np.uint8)
        p, op = _params(tx, oracle, fmt % 3, False)
        rid = srv.submit(img, w, h, tx.Format(fmt), p, out[dst_off:out.size - 32], mips=True)
        jobs.append((rid, fmt, img, out, op))
    for rid, fmt, img, out, op in jobs:
        assert srv.wait(rid, timeout_ms=60000)["status"] == 0
        at = dst_off
        while True:
            hh, ww = img.shape[:2]
            ref = oracle.compress(fmt, img, ww, hh, op)
            assert np.array_equal(out[at:at + ref.size], ref)
            at += ref.size
            if ww == 1 and hh == 1:
                break
            img = workloads.mip_reference(img)
        assert (out[:dst_off] == 77).all() and (out[at:] == 77).all()
    srv.close()
