"""RangeFit's nearest codes from positions on the line of codes, and its search
for pixels of one colour, against the oracle: blocks of few and many colours,
endpoints one grid step apart or the same, points near the middle between codes,
channel weights inside and outside the range the line decides, pixel masks."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# the last four have every point measured
WEIGHTS = [(0.2126, 0.7152, 0.0722), (0.0, 1.0, 0.0), (0.0, 0.0, 0.0), (-1.0, 0.5, 2.0), (1e-6, 1e6, 1.0),
           (1e-7, 1.0, 1.0), (2e6, 1.0, 1.0), (float("inf"), 1.0, 1.0), (float("nan"), 1.0, 1.0)]


def _blocks(seed):
    rng = np.random.default_rng(seed)
    out = []
    for n in range(1, 17):  # n colours at most
        pal = rng.integers(0, 256, (60, n, 3))
        pal[20:40] = rng.integers(0, 250, (20, 1, 3)) + rng.integers(0, 6, (20, n, 3))      # nearly one colour
        pal[40:] = np.linspace(0, 255, n)[None, :, None].astype(int) * np.ones((20, 1, 3), int)  # greys
        out.append(pal[np.arange(60)[:, None], rng.integers(0, n, (60, 16))])
    v = np.arange(240)
    ends = np.repeat(v[:, None, None] % 16 * 16, 16, 1) * np.ones((1, 1, 3), int)
    ends[:, 8:] += 8 + v[:, None, None] // 60  # about one grid step, in all channels
    out.append(np.clip(ends + rng.integers(-1, 2, ends.shape), 0, 255))
    rgb = np.concatenate(out)
    alpha = rng.integers(0, 256, rgb.shape[:2] + (1,))
    alpha[::3] = 255
    return np.concatenate([rgb, alpha], axis=2).astype(np.uint8).reshape(-1, 64)


@pytest.mark.parametrize("aw", [False, True])
@pytest.mark.parametrize("weights", WEIGHTS)
@pytest.mark.parametrize("fmt", [0, 1, 2])
def test_range_line(tx, cuda, oracle, fmt, weights, aw):
    blocks = _blocks(fmt)
    rng = np.random.default_rng(7)
    masks = rng.integers(0, 65536, len(blocks)).astype(np.uint32)
    masks[rng.random(len(blocks)) < 0.5] = 0xFFFF
    f = tx.Format(fmt)
    src, m = cuda.from_numpy(blocks).cuda(), cuda.from_numpy(masks.view(np.int32)).cuda()
    out = cuda.zeros(len(blocks) * f.block_size(), dtype=cuda.uint8, device="cuda")
    p = tx.Params(algorithm=tx.Algorithm.RangeFit, weights=weights, weigh_colour_by_alpha=aw)
    tx.compress_blocks_device(f, src.data_ptr(), m.data_ptr(), len(blocks), p, out.data_ptr(),
                              cuda.cuda.current_stream().cuda_stream)
    ref = oracle.compress_blocks(fmt, blocks, masks, oracle.make_params(0, weights, aw))
    got = out.cpu().numpy().reshape(len(blocks), -1)
    bad = np.flatnonzero((got != ref.reshape(got.shape)).any(axis=1))
    assert bad.size == 0, "%d blocks differ (first %d)" % (bad.size, bad[0])
