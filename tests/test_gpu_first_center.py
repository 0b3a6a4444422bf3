"""The first center's label where a polygon's first outer edges give no
reference point (no length, or other edges within a thousandth of their own
length), alone and in a group, against the exact oracle."""
import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import synth
from oracle import exact

pytestmark = pytest.mark.gpu


def late_comb(edges, side):
    """A comb of horizontal teeth: its closing edges, the first that serve,
    come last."""
    x = np.linspace(-side / 2, side / 2, edges)
    y = np.where(np.arange(edges) % 2, -side / 2, side / 2)
    ring = np.concatenate([np.stack([x, y], 1), [[1.02 * side / 2, -1.04 * side / 2], [-1.02 * side / 2, -1.04 * side / 2]]])
    return np.ascontiguousarray(ring[:, ::-1])


def repeated(ring, n):
    """The ring with n more copies of its first and of its last vertex (the
    first edges have no length, whichever way it is walked)."""
    return np.concatenate([np.repeat(ring[:1], n, 0), ring, np.repeat(ring[-1:], n, 0)])


def _rings():
    rng = np.random.default_rng(8)
    star = lambda n, lon, lat: synth.star_ring(lon, lat, n, 8.0, 0.2, rng)
    return [[late_comb(3000, 2.0)], [star(50, 20.0, 30.0)], [repeated(star(60, -100.0, -50.0), 1)],
            [repeated(star(90, 100.0, 60.0), 63)], [repeated(star(40, 170.0, -5.0), 64)], [star(9, 0.0, -80.0)],
            [repeated(star(300, 60.0, 10.0), 200), synth.star_ring(60.0, 10.0, 30, 1.0, 0.0, rng)],
            [late_comb(200, 2.0) + [120.0, 10.0]]]


def _points(rings, rng):
    c = rings[0].mean(0)
    return np.concatenate([c + rng.uniform(-9, 9, (1500, 2)) * [1.0, 0.8], synth.uniform_points(500, rng), rings[0][::7]])


def test_polygons_alone_and_in_a_group():
    import torch
    rings = _rings()
    rng = np.random.default_rng(9)
    P = [G.Polygon.from_rings(r) for r in rings]
    pts, want = [_points(r, rng) for r in rings], []
    for k, (p, r) in enumerate(zip(P, rings)):
        xyz, pe = p.export()
        want.append(exact.ExactPolygon(xyz, pe, len(r[0])).query_lonlat(pts[k]))
        assert np.array_equal(G.Grid(p).classify().query(pts[k]), want[k]), k
    off = np.concatenate([[0], np.cumsum([len(q) for q in pts])]).astype(np.int64)
    d = torch.from_numpy(np.concatenate(pts)).cuda()
    lab = torch.zeros(len(d), dtype=torch.uint8, device="cuda")
    G.Batch(P).query_device(d.data_ptr(), off, lab.data_ptr(), sync=True)
    assert np.array_equal(lab.cpu().numpy(), np.concatenate(want))


def test_no_edge_serves():
    """Two edges over one another: refused, and the library works on."""
    P = G.Polygon.from_rings([np.array([[0.0, 0.0], [10.0, 0.0], [0.0, 0.0], [10.0, 0.0]])])
    with pytest.raises(G.GahhgError) as e:
        G.Grid(P)
    assert "no outer-ring edge" in str(e.value)
    assert len(G.Grid(G.Polygon.from_rings([_rings()[1][0]])).classify().query([[0.0, 0.0]])) == 1


def test_many_edges_do_not_serve():
    """160,000 edges are tried: well under the 4 seconds of a trip for each
    (one block trying them in turn took 29)."""
    P = G.Polygon.from_rings([late_comb(160000, 2.0)])
    G.Grid(G.Polygon.from_rings([late_comb(100, 2.0)]))
    # (few cells, none divided: the rest of the build takes milliseconds)
    assert G.Grid(P, lattice_top=1000, lattice_leaf=60000).stats()["lattice_s"] < 2.0
