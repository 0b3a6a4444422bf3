"""Level-0 labels where the cells are much wider than high: half of the
vertices within a degree of a pole, so cells are up to 64 times wider than
high, and row 0 at middle latitudes, where the great circle between two
neighbouring centers leaves both cells.  A meridional edge through a center
makes that cell's crossings uncertain in the plane, so the exact test decides
them.  Labels against the exact oracle, on every meridian and latitude."""
import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import synth
from oracle import exact

pytestmark = pytest.mark.gpu


def peninsula(lon, width, south=False, foot=45.0, n=297, lat=89.2):
    """A ring of n vertices around a pole and a peninsula from it down to
    `foot`, its west side along the meridian `lon`."""
    west = np.linspace(lon + width + 0.1, lon + 360.0, n)
    ring = np.stack([(west + 180.0) % 360.0 - 180.0, np.full(n, lat)], 1)
    ring[-1, 0] = lon
    ring = np.concatenate([ring, [[lon, foot + 0.004], [lon + width, foot]]])
    return ring * [1.0, -1.0] if south else ring


CASES = [peninsula(30.0, 9.6), peninsula(30.0, 9.6, south=True), peninsula(-110.0, 9.6), peninsula(90.0, 8.2),
         peninsula(-30.0, 12.3), peninsula(150.0, 9.1), peninsula(10.0, 9.6, foot=40.0), peninsula(-70.0, 9.9, foot=52.0),
         peninsula(30.0, 9.6, n=500), peninsula(-150.0, 7.0, foot=30.0), peninsula(-10.0, 9.6, n=900, lat=89.5)]


@pytest.mark.parametrize("case", range(len(CASES)))
def test_labels_of_wide_cells(case):
    ring = CASES[case]
    P = G.Polygon.from_rings([ring])
    rng = np.random.default_rng(case)
    s = np.sign(ring[0, 1])
    lo, la = np.meshgrid(np.arange(-179.5, 180.0, 3.0), s * np.concatenate([np.arange(20.0, 89.9, 1.3), [89.95]]))
    band = np.stack([rng.uniform(-180, 180, 4000), s * rng.uniform(ring[:, 1].__abs__().min() - 1.0, 90.0, 4000)], 1)
    pts = np.concatenate([np.stack([lo.ravel(), la.ravel()], 1), band, synth.uniform_points(3000, rng),
                          synth.near_edge_points([ring], 2000, rng)])
    xyz, pe = P.export()
    want = exact.ExactPolygon(xyz, pe, len(ring)).query_lonlat(pts)
    g = G.Grid(P, semantics=G.SEMANTICS_EXACT).classify()
    for prec in (G.QUERY_FP32_FILTER, G.QUERY_FP64_FILTER):
        got = g.query(pts, prec)
        bad = np.nonzero(got != want)[0]
        assert len(bad) == 0, (len(bad), len(pts), pts[bad[0]])
    off = np.array([0, len(pts), 2 * len(pts)], dtype=np.int64)
    import torch
    d = torch.from_numpy(np.concatenate([pts, pts])).cuda()
    lab = torch.zeros(2 * len(pts), dtype=torch.uint8, device="cuda")
    G.Batch([P, P]).query_device(d.data_ptr(), off, lab.data_ptr(), G.QUERY_FP32_FILTER, sync=True)
    assert np.array_equal(lab.cpu().numpy(), np.concatenate([want, want]))
