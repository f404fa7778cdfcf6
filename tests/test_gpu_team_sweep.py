"""The team form's compress4 sweep over every number of colours (up to five,
all candidates are evaluated; above, the bound leaves some out) and channel
weights at the ends of the bound's range, against the oracle: the same bytes."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

# ordinary, one channel, weights that count as zero in the bound, all of them
# such, the largest the bound takes, and larger ones
WEIGHTS = [(0.2126, 0.7152, 0.0722), (0.0, 1.0, 0.0), (8e-19, 1.0, 1e-25), (1e-22, 1e-22, 1e-20),
           (1.1e18, 2.0, 1e-18), (2e18, 1.0, 1.0)]


def _blocks(rng, colours, n):
    """n blocks of 16 pixels in `colours` colours: ramps, random ones, nearly one colour."""
    out = np.empty((n, 16, 4), np.uint8)
    for b in range(n):
        if b % 3 == 0:
            a, d = rng.integers(0, 256, 3), rng.integers(-8, 9, 3)
            pal = a + d * np.arange(colours)[:, None] + rng.integers(-2, 3, (colours, 3))
        elif b % 3 == 1:
            pal = rng.integers(0, 256, (colours, 3))
        else:
            pal = rng.integers(40, 200, 3) + rng.integers(-2, 3, (colours, 3))
        pal = np.unique(np.clip(pal, 0, 255), axis=0)
        idx = np.concatenate([np.arange(len(pal)), rng.integers(0, len(pal), 16 - len(pal))])
        out[b, :, :3] = pal[rng.permutation(idx)]
        out[b, :, 3] = rng.integers(128, 256, 16)
    return out.reshape(n, 64)


@pytest.mark.parametrize("weights", WEIGHTS)
@pytest.mark.parametrize("fmt,alg,aw", [(0, 1, False), (0, 2, True), (1, 2, False), (2, 1, False), (2, 1, True)])
def test_all_colour_counts(tx, cuda, oracle, fmt, alg, aw, weights):
    rng = np.random.default_rng(fmt * 10 + alg)
    blocks = np.concatenate([_blocks(rng, c, 60) for c in range(2, 17)])
    p = tx.Params(algorithm=tx.Algorithm(alg), weights=weights, weigh_colour_by_alpha=aw)
    f = tx.Format(fmt)
    src = cuda.from_numpy(blocks).cuda()
    out = cuda.zeros(len(blocks) * f.block_size(), dtype=cuda.uint8, device="cuda")
    tx.compress_blocks_device(f, src.data_ptr(), 0, len(blocks), p, out.data_ptr(), cuda.cuda.current_stream().cuda_stream)
    op = oracle.make_params(alg, weights, aw)
    # every block as a 4x4 image of its own
    ref = np.concatenate([oracle.compress(fmt, b.reshape(4, 4, 4), 4, 4, op) for b in blocks])
    assert np.array_equal(out.cpu().numpy(), ref)
