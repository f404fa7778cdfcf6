"""Channel weights so small that products with them leave the normal f32 range, on
blocks whose colours differ in one channel or lie on a line: ClusterFit's bounds must
not exclude the reference's candidate.  The oracle's bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

WEIGHTS = [(0.0, 1e-42, 0.0), (1e-42, 0.0, 1e-42), (1e-42, 1e-42, 1e-42), (0.0, 0.0, 3e-39), (1e-33, 0.0, 0.0),
           (1e-24, 1e-24, 0.0), (1.0, 1e-42, 1e-30)]


def _image(seed, bw, bh):
    rng = np.random.default_rng(seed)
    img = np.empty((bh, bw, 4, 4, 4), np.uint8)
    for by in range(bh):
        for bx in range(bw):
            a, b, c = rng.integers(0, 256, (3, 3)), rng.integers(0, 256, 3), rng.integers(0, 3)
            t = rng.integers(0, 257, (4, 4, 1))
            if (bx + by) % 2:
                px = np.broadcast_to(b, (4, 4, 3)).copy()
                px[..., c] = rng.integers(0, 256, (4, 4))
                if bx % 3 == 0:
                    px[..., (c + 1) % 3] = 0
            else:
                px = (a[0] * t + a[1] * (256 - t)) // 256
            img[by, bx, :, :, :3] = px
            img[by, bx, :, :, 3] = rng.integers(128, 256, (4, 4))
    return np.ascontiguousarray(img.transpose(0, 2, 1, 3, 4).reshape(bh * 4, bw * 4, 4))


@pytest.mark.parametrize("weights", WEIGHTS)
@pytest.mark.parametrize("fmt", range(3))
@pytest.mark.parametrize("alg,aw", [(1, False), (2, False), (1, True)])
def test_bytes(tx, cuda, oracle, fmt, alg, aw, weights):
    img = _image(fmt * 10 + alg, 40, 30)
    h, w = img.shape[:2]
    f = tx.Format(fmt)
    src = cuda.from_numpy(img).cuda()
    out = cuda.zeros(f.compressed_size(w, h), dtype=cuda.uint8, device="cuda")
    p = tx.Params(algorithm=tx.Algorithm(alg), weights=weights, weigh_colour_by_alpha=aw)
    tx.compress_device(f, src.data_ptr(), w * 4, 4, w, h, p, out.data_ptr(), out.numel(),
                       cuda.cuda.current_stream().cuda_stream)
    ref = oracle.compress(fmt, img, w, h, oracle.make_params(alg, weights, aw))
    assert np.array_equal(out.cpu().numpy(), ref)
