"""ClusterFit of BC2 / BC3 with one block per thread (tx_cluster_lanes.cu), which
large launches take: bit for bit the oracle's blocks, at the smallest launch
that takes it, at counts that are no multiple of a warp or a CTA, with more
than one wave of CTAs, with pixel masks and with rows that are not aligned.
The blocks mix the shapes that drive its paths: noisy ramps (bound alone),
nearly flat blocks (grid filter, ties on the 5:6:5 grid), few colours, none,
one colour, degenerate axes, alpha weights."""
import numpy as np
import pytest

from texpresso_gb300 import workloads

pytestmark = pytest.mark.gpu

PERCEPTUAL = (0.2126, 0.7152, 0.0722)


def mixed_blocks(n, seed):
    rng = np.random.default_rng(seed)
    base = rng.integers(0, 256, size=(4000, 1, 3))
    spread = rng.integers(0, 7, size=(4000, 1, 3))
    flat = np.clip(base + np.rint(rng.uniform(-1, 1, size=(4000, 16, 3)) * spread), 0, 255)
    flat = np.concatenate([flat, rng.integers(0, 256, size=(4000, 16, 1))], axis=2).astype(np.uint8).reshape(-1, 64)
    kinds = np.concatenate([workloads.random_blocks(2000, seed=seed + 1), workloads.grid_blocks(1000, seed=seed + 2), flat,
                            workloads.image_to_blocks(workloads.ramp_texture(256, 256, seed=seed + 3, alpha="ramp"))[0]])
    # runs of one kind, as in an image, and single blocks of any kind between them
    out = kinds[(np.arange(n) // 7 * 13 + np.arange(n) % 7) % len(kinds)]
    loose = rng.random(n) < 0.3
    out[loose] = kinds[rng.integers(0, len(kinds), int(loose.sum()))]
    return np.ascontiguousarray(out)


def wave(torch):
    return torch.cuda.get_device_properties(0).multi_processor_count * 512


def check(oracle, tx, torch, fmt, blocks, masks, weights, aw):
    b = torch.from_numpy(blocks).cuda()
    m = torch.from_numpy(masks.view(np.int32)).cuda() if masks is not None else None
    f = tx.Format(fmt)
    out = torch.zeros(blocks.shape[0] * f.block_size(), dtype=torch.uint8, device="cuda")
    p = tx.Params(algorithm=tx.Algorithm.ClusterFit, weights=weights, weigh_colour_by_alpha=aw)
    tx.compress_blocks_device(f, b.data_ptr(), m.data_ptr() if m is not None else 0, blocks.shape[0], p, out.data_ptr(),
                              torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    got = out.cpu().numpy().reshape(blocks.shape[0], -1)
    ref = oracle.compress_blocks(fmt, blocks, masks, oracle.make_params(1, weights, aw))
    diff = np.flatnonzero(np.any(got != ref, axis=1))
    assert diff.size == 0, "%d blocks differ (first %d)" % (diff.size, diff[0])


@pytest.mark.parametrize("aw", [False, True])
@pytest.mark.parametrize("weights", [PERCEPTUAL, (1.0, 1.0, 1.0), (0.0, 1.0, 0.0), (1e6, 1e-6, 3.0), (1e-6, 0.0, 2e-6)])
@pytest.mark.parametrize("fmt", [1, 2])
def test_weights(tx, cuda, oracle, fmt, weights, aw):
    n = -(-wave(cuda) * 21 // 25) + 1
    check(oracle, tx, cuda, fmt, mixed_blocks(n, 40 + fmt), None, weights, aw)


@pytest.mark.parametrize("waves,extra", [(0.8, 0), (0.84, 31), (1.0, 0), (2.0, -1), (2.6, 17)])
def test_counts_and_masks(tx, cuda, oracle, waves, extra):
    n = int(wave(cuda) * waves) + 1 + extra
    rng = np.random.default_rng(n)
    masks = rng.integers(0, 65536, n).astype(np.uint32)
    masks[rng.random(n) < 0.6] = 0xFFFF
    check(oracle, tx, cuda, 2, mixed_blocks(n, 60), masks, PERCEPTUAL, extra % 2 == 1)


def test_ragged_image(tx, cuda, oracle):
    blocks = mixed_blocks(256 * 280, 80)
    img = blocks.reshape(280, 256, 4, 4, 4).transpose(0, 2, 1, 3, 4).reshape(1120, 1024, 4)[:1117, :1021]
    img = np.ascontiguousarray(img)
    t = cuda.from_numpy(img).cuda()
    f = tx.Format.Bc3
    n = f.compressed_size(1021, 1117)
    assert n // 16 >= wave(cuda) * 21 // 25
    out = cuda.zeros(n, dtype=cuda.uint8, device="cuda")
    tx.compress_device(f, t.data_ptr(), 1021 * 4, 4, 1021, 1117, tx.Params(), out.data_ptr(), n,
                       cuda.cuda.current_stream().cuda_stream)
    cuda.cuda.synchronize()
    assert np.array_equal(out.cpu().numpy(), oracle.compress(2, img, 1021, 1117, oracle.make_params(1)))
