"""Index options with so few top cells that a cell is wider than a hemisphere:
every great circle comes near such a cell's center, whatever the cap's sine
says.  Labels against the exact oracle."""
import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import synth
from oracle import exact
from tests.test_gpu_level0_arcs import peninsula

pytestmark = pytest.mark.gpu


def _rings():
    rng = np.random.default_rng(23)
    out = [synth.star_ring(lon, lat, n, r, 0.3, rng) for lon, lat, n, r in
           [(10.0, 0.0, 40, 50.0), (120.0, 30.0, 300, 20.0), (-170.0, -40.0, 60, 35.0), (0.0, 85.0, 50, 20.0),
            (75.0, -10.0, 7, 60.0), (179.0, 5.0, 200, 3.0)]]
    for _ in range(12):  # an arm from a ring around a pole across the equator
        out.append(peninsula(10.0 * rng.integers(-18, 18), rng.uniform(3.0, 20.0), rng.random() < 0.5,
                             rng.uniform(-50.0, 30.0), 60, rng.uniform(80.0, 89.8)))
    for _ in range(24):  # long edges
        lon = np.sort(rng.uniform(-180.0, 180.0, rng.integers(4, 9)))
        out.append(np.stack([lon, rng.uniform(-70.0, 70.0, len(lon))], 1))
    return out


RINGS = _rings()


@pytest.mark.parametrize("top", [1, 2, 3, 4, 8, 30])
@pytest.mark.parametrize("leaf", [0, 1, 16])
def test_few_top_cells(top, leaf):
    rng = np.random.default_rng(24)
    for k, ring in enumerate(RINGS):
        P = G.Polygon.from_rings([ring])
        pts = np.concatenate([synth.uniform_points(3000, rng), synth.near_edge_points([ring], 300, rng), ring])
        xyz, pe = P.export()
        want = exact.ExactPolygon(xyz, pe, len(ring)).query_lonlat(pts)
        got = G.Grid(P, lattice_top=top, lattice_leaf=leaf).classify().query(pts)
        bad = np.nonzero(got != want)[0]
        assert len(bad) == 0, (k, len(bad), pts[bad[0]])
