"""Queries at the sizes where a query kernel's rounds, grids and routes change,
and at coordinates its tables do not cover, against the reference's committed
labels and the exact oracle."""
import numpy as np
import pytest

import gahhg_b200 as G
from oracle import exact

pytestmark = pytest.mark.gpu

SIZES = (1, 31, 255, 256, 257, 1023, 1024, 1025, 4097)


@pytest.fixture(scope="module")
def na0(inputs, ref_outputs, tmp_path_factory):
    name = "various/NA0.txt"
    P = G.Polygon.from_file(inputs.polygon_file(name, tmp_path_factory.mktemp("na0")))
    return P, inputs.query("uniform"), ref_outputs.get("labels", name), len(inputs.rings_deg(name)[0])


@pytest.fixture(scope="module")
def na0_ref(na0):
    return G.Grid(na0[0], semantics=G.SEMANTICS_REFERENCE).classify()


@pytest.mark.parametrize("n", SIZES)
def test_reference_labels_of_the_first_points(na0, na0_ref, n):
    assert np.array_equal(na0_ref.query(na0[1][:n], G.QUERY_REFERENCE_FP64), na0[2][:n])


def test_reference_labels_of_many_points(na0, na0_ref):
    """More points than the grid has rounds, the last one partial."""
    k = 1 + 148 * 16 * 1024 // len(na0[1])
    got = na0_ref.query(np.tile(na0[1], (k + 1, 1))[:k * len(na0[1]) + 77], G.QUERY_REFERENCE_FP64)
    assert np.array_equal(got, np.tile(na0[2], k + 1)[:len(got)])


def test_reference_labels_off_the_table(na0, na0_ref):
    """Longitudes one turn away descend from level 0 and agree except within
    the tolerance of a border (2 pi is not twice the truncated pi)."""
    pts = na0[1][:20000].copy()
    want = na0[2][:20000]
    pts[:, 0] += np.where(np.arange(len(pts)) % 2, 360.0, -360.0)
    assert (na0_ref.query(pts, G.QUERY_REFERENCE_FP64) != want).mean() < 1e-3
    # the table's own borders
    for lon in (-180.0, 180.0):
        for lat in (-90.0, 90.0, 0.0):
            assert na0_ref.query([[lon, lat]], G.QUERY_REFERENCE_FP64)[0] in (1, 2)
