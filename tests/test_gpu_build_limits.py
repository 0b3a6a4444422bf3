"""Polygons whose edges fill an area: the refinement stops at its budget of
list entries, on level 0 too, and lists past 2^31 entries are refused."""
import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import _lib
from oracle import exact

pytestmark = pytest.mark.gpu


def comb(edges, side, upright=True):
    """A zigzag of `edges` edges, each from end to end of a square of `side`
    degrees around (0, 0), closed along one side of it.  The ring's first
    edge, from either end, lies outside the teeth."""
    h = side / 2
    x = np.linspace(-h, h, edges)
    y = np.where(np.arange(edges) % 2, -h, h)
    ring = np.concatenate([[[0.0, -1.04 * h], [-1.02 * h, -1.04 * h]], np.stack([x, y], 1), [[1.02 * h, -1.04 * h]]])
    return ring if upright else np.ascontiguousarray(ring[:, ::-1])


def test_level0_lists_past_the_budget_stay_leaves():
    """160,000 edges across 1,900 rows of cells: more than 2^28 entries on
    level 0, about 90 in a cell, none of which is divided."""
    ring = comb(160000, 60.0)
    P = G.Polygon.from_rings([ring])
    rng = np.random.default_rng(5)
    pts = np.concatenate([rng.uniform(-33.0, 33.0, (500, 2)), ring[rng.integers(0, len(ring), 50)]])
    xyz, pe = P.export()
    want = exact.ExactPolygon(xyz, pe, len(ring)).query_lonlat(pts)
    g = G.Grid(P, lattice_top=4_000_000).classify()
    # 20 bytes a record: those of level 0 alone (the next level has three times as many)
    assert 20 * 2 ** 28 < g.stats()["lattice_bytes"] < 50 * 2 ** 28
    for prec in (G.QUERY_FP32_FILTER, G.QUERY_FP64_FILTER):
        assert np.array_equal(g.query(pts, prec), want)


def test_lists_past_2_to_31_entries_are_refused():
    """180,000 edges across 13,000 columns of cells each."""
    P = G.Polygon.from_rings([comb(180000, 2.0, upright=False)])
    with pytest.raises(G.GahhgError) as e:
        G.Grid(P, lattice_top=200_000_000)
    assert e.value.status == _lib.ERR_CAPACITY and "list entries on level 0" in str(e.value)
    # the library works on
    Q = G.Polygon.from_rings([comb(100, 10.0)])
    assert set(G.Grid(Q).classify().query([[60.0, 60.0], [0.03, -5.05]])) == {1, 2}


@pytest.mark.parametrize("lat,spacing,n", [(45.0, 1e-7, 3000), (-88.8, 2e-6, 20000), (89.5, 1e-8, 2000)])
def test_vertices_closer_than_the_margin_of_the_cells(lat, spacing, n):
    """A border with n vertices `spacing` degrees apart: cells of any size list
    them all, and the refinement ends at its last level or its budgets."""
    s = np.sign(lat)
    w = n * spacing / np.cos(np.radians(lat))
    x = np.linspace(w, 0.0, n)
    y = lat - s * (1e-4 + 0.3 * spacing * (np.arange(n) % 2))
    ring = np.concatenate([[[0.0, lat], [w, lat - 0.1 * spacing]], np.stack([x, y], 1), [[-2.0, lat - s * 1.5]]])
    P = G.Polygon.from_rings([ring + [30.0, 0.0]])
    rng = np.random.default_rng(6)
    pts = np.concatenate([(ring + [30.0, 0.0])[rng.integers(0, len(ring), 200)] + rng.normal(size=(200, 2)) * spacing,
                          np.stack([30.0 + rng.uniform(-2.1, 0.1, 300), lat - s * rng.uniform(-0.1, 1.6, 300)], 1)])
    xyz, pe = P.export()
    want = exact.ExactPolygon(xyz, pe, len(ring)).query_lonlat(pts)
    g = G.Grid(P).classify()
    for prec in (G.QUERY_FP32_FILTER, G.QUERY_FP64_FILTER):
        assert np.array_equal(g.query(pts, prec), want)


@pytest.mark.parametrize("n", [2648, 9000])
def test_childrens_lists_past_the_budget(n):
    """Vertices 0.01 m apart on a small circle around a pole: a child lists most
    of its parent's edges at every size, 8 to 12 entries for one, so lists below
    the budget have children's of 2.1 and 2.3e9 entries.  The parents stay leaves."""
    x = np.linspace(150.0, 0.0, n)
    ring = np.concatenate([[[0.0, -87.85], [150.0, -88.1]], np.stack([x, np.full(n, -89.9999)], 1)]) + [20.0, 0.0]
    P = G.Polygon.from_rings([ring])
    rng = np.random.default_rng(7)
    pts = np.concatenate([np.stack([rng.uniform(-180, 180, 300), -90.0 + 10.0 ** rng.uniform(-5, -3.8, 300)], 1),
                          np.stack([rng.uniform(0, 190, 300), rng.uniform(-90.0, -87.0, 300)], 1),
                          ring[rng.integers(0, len(ring), 30)]])
    pts[:, 0] = (pts[:, 0] + 180.0) % 360.0 - 180.0
    xyz, pe = P.export()
    want = exact.ExactPolygon(xyz, pe, len(ring)).query_lonlat(pts)
    g = G.Grid(P).classify()
    assert 20 * 2 ** 26 < g.stats()["lattice_bytes"] < 100 * 2 ** 28
    for prec in (G.QUERY_FP32_FILTER, G.QUERY_FP64_FILTER):
        assert np.array_equal(g.query(pts, prec), want)
