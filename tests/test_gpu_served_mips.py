"""Mip chains of served requests, several levels to a launch, against the oracle:
sizes at the edges of a 64x64 tile, one pixel wide or high, images of every
alignment in host memory, with and without levels."""
import numpy as np
import pytest

from texpresso_gb300 import workloads

pytestmark = pytest.mark.gpu

SIZES = [(1, 1), (1, 300), (300, 1), (2, 3), (63, 65), (64, 64), (65, 63), (128, 4), (129, 127), (260, 190), (1030, 67)]


@pytest.mark.parametrize("mips", [True, False])
@pytest.mark.parametrize("offset", [0, 1, 4, 16])
def test_levels(tx, cuda, oracle, offset, mips):
    srv = tx.Server(memory_budget=256 << 20, step_blocks=4096, min_share=512)
    p, op = tx.Params(algorithm=tx.Algorithm.RangeFit), oracle.make_params(0, (0.2126, 0.7152, 0.0722), False)
    jobs = []
    for w, h in SIZES:
        img = workloads.ramp_texture(w, h, seed=w + h, alpha="ramp")
        room = np.zeros(offset + img.size, np.uint8)
        room[offset:] = img.reshape(-1)
        out = np.zeros(tx.chain_compressed_size(0, w, h, mips), np.uint8)
        jobs.append((srv.submit(room[offset:], w, h, tx.Format.Bc1, p, out, mips=mips), img, room, out))
    for rid, img, _, out in jobs:
        assert srv.wait(rid, timeout_ms=60000)["status"] == 0
        at = 0
        while True:
            h, w = img.shape[:2]
            ref = oracle.compress(0, img, w, h, op)
            assert np.array_equal(out[at:at + ref.size], ref), (img.shape, at)
            at += ref.size
            if not mips or (w == 1 and h == 1):
                break
            img = workloads.mip_reference(img)
        assert at == out.size
    srv.close()
