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
