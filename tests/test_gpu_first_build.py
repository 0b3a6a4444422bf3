"""The first index of a polygon, built right after its vertices were copied to
a device whose copy engines are busy, has the labels of every later one."""
import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import synth
from oracle import exact

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("edges", [300, 1200, 2500, 20000])
def test_first_build_while_copies_run(edges):
    import torch
    rng = np.random.default_rng(edges)
    host = torch.empty(64 << 20, dtype=torch.uint8).pin_memory()
    dev = torch.empty_like(host, device="cuda")
    side = torch.cuda.Stream()
    pts = synth.cap_points(10.0, 20.0, 8.0, 2000, rng)
    for k in range(6):
        rings = [synth.star_ring(10.0, 20.0, edges, 5.0, 0.3, rng)]
        P = G.Polygon.from_rings(rings)
        with torch.cuda.stream(side):
            dev.copy_(host, non_blocking=True)
        first = G.Grid(P, semantics=G.SEMANTICS_EXACT).classify().query(pts)
        side.synchronize()
        assert np.array_equal(first, G.Grid(P, semantics=G.SEMANTICS_EXACT).classify().query(pts)), k
        if k == 0:
            xyz, pe = P.export()
            assert np.array_equal(first, exact.ExactPolygon(xyz, pe, len(rings[0])).query_lonlat(pts))
