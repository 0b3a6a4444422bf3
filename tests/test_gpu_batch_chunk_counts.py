"""Batch queries at the chunk counts where the prefix sums of the chunks' queue
counts move from the last block of pass 1 to a launch of their own, and at the
ends of the tiles of either, directly and through a graph that runs twice."""
import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import synth

pytestmark = pytest.mark.gpu

CHUNK = 256


@pytest.fixture(scope="module")
def case():
    import torch
    rng = np.random.default_rng(12)
    rings = [[synth.star_ring(-40.0 + 30 * k, 10.0 * k, 20 + 7 * k, 12.0, 0.3, rng)] for k in range(3)]
    P = [G.Polygon.from_rings(r) for r in rings]
    n = 9000 * CHUNK
    pts = np.concatenate([synth.near_edge_points(rings[k], n // 6, rng) if j else
                          rings[k][0].mean(0) + rng.uniform(-15, 15, (n // 6, 2))
                          for k in range(3) for j in range(2)])
    perm = rng.permutation(len(pts))
    d = torch.from_numpy(pts[perm]).cuda()
    want = []
    for p in P:
        lab = torch.zeros(len(pts), dtype=torch.uint8, device="cuda")
        G.Grid(p).classify().query_device(d.data_ptr(), len(pts), lab.data_ptr(), sync=True)
        want.append(lab)
    B = G.Batch(P, top_cells=[64] * 3)  # (small summaries: chunks as small as asked for)
    B.set_chunk(CHUNK)
    return B, d, want


@pytest.mark.parametrize("chunks", [1, 3, 255, 256, 257, 2046, 2047, 2048, 2049, 2050, 4097, 8191, 8192, 8193])
def test_chunk_counts(case, chunks):
    import torch
    B, d, want = case
    # three segments; the middle one takes what is left, its last chunk partial
    a, c = min(1, chunks - 1), chunks // 3
    sizes = [a * CHUNK, (chunks - a - c) * CHUNK - (100 if chunks > 3 else 0), c * CHUNK]
    off = np.concatenate([[0], np.cumsum(sizes)]).astype(np.int64)
    n = int(off[-1])
    assert n <= len(d)
    w = torch.cat([want[k][off[k]:off[k + 1]] for k in range(3)])
    lab = torch.zeros(n, dtype=torch.uint8, device="cuda")
    for prec in (G.QUERY_FP32_FILTER, G.QUERY_FP64_FILTER):
        lab.zero_()
        B.query_device(d.data_ptr(), off, lab.data_ptr(), prec, sync=True)
        assert torch.equal(lab, w)
        for _ in range(2):
            lab.zero_()
            B.query_device(d.data_ptr(), off, lab.data_ptr(), prec, graph=True)
            torch.cuda.synchronize()
            assert torch.equal(lab, w)
