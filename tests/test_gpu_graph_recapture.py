"""Graph queries with changing arguments, one behind the other on a busy
stream: the workspace of a replay that has not run yet is left alone."""
import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import synth

pytestmark = pytest.mark.gpu


def test_changing_offsets_without_waiting():
    import torch
    rng = np.random.default_rng(6)
    polys = synth.c3_polygons(12, seed=31, vmax=3000)
    B = G.Batch([G.Polygon.from_rings(r) for r, _c, _d in polys])
    sets = []
    for k in range(4):
        counts = rng.integers(0, 40000 if k % 2 else 4000, len(polys))
        off = np.concatenate([[0], np.cumsum(counts)]).astype(np.int64)
        pts = np.concatenate([synth.cap_points(c[0], c[1], 1.8 * d, n, rng) if n else np.zeros((0, 2))
                              for (_r, c, d), n in zip(polys, counts)])
        d_pts = torch.from_numpy(pts).cuda()
        want = torch.zeros(len(pts), dtype=torch.uint8, device="cuda")
        B.query_device(d_pts.data_ptr(), off, want.data_ptr(), sync=True)
        sets.append((off, d_pts, want, torch.zeros(len(pts), dtype=torch.uint8, device="cuda")))
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    for turn in range(3):
        for k, (off, d_pts, want, lab) in enumerate(sets):
            with torch.cuda.stream(side):
                lab.zero_()
                torch.cuda._sleep(20_000_000)
            if turn == 2:
                B.set_chunk(512 << k)
            B.query_device(d_pts.data_ptr(), off, lab.data_ptr(), stream=side.cuda_stream, graph=True)
        torch.cuda.synchronize()
        for off, d_pts, want, lab in sets:
            assert torch.equal(lab, want)
