"""Queries at the sizes where a query kernel's rounds, grids and routes change,
and at coordinates its tables do not cover, against the reference's committed
labels and the exact oracle."""
import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import synth
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


# ---- exact labels: one launch up to 2^20 points, passes of their own above --

def _special(rings):
    """Points where a cell index, a ring of the summary or a descent can go
    wrong: domain ends, poles, the antimeridian, unusual coordinates, vertices."""
    v = np.concatenate(rings)
    lon = np.array([-540.0, -360.0, -180.0, np.nextafter(-180, 0), 0.0, np.nextafter(180, 0), 180.0, 360.0, 540.0, 541.0,
                    -900.5])
    lat = np.array([-270.0, -90.0, np.nextafter(-90, 0), 0.0, np.nextafter(90, 0), 90.0, 90.5, 170.0])
    ends = np.array([[x, y] for x in lon for y in lat])
    lo, hi = v.min(0), v.max(0)
    box = np.array([[x, y] for x in (lo[0], hi[0], lo[0] - 0.01, hi[0] + 0.01) for y in (lo[1], hi[1])])
    return np.concatenate([ends, box, v, v + [360.0, 0.0], v - [360.0, 0.0], 0.5 * (v + np.roll(v, 1, 0))])


def _polygon(kind):
    rng = np.random.default_rng(41)
    if kind == "sphere":
        return synth.c0_polygon()
    if kind == "antimeridian":
        return [synth.star_ring(179.5, -10.0, 700, 6.0, 0.2, rng), synth.star_ring(179.5, -10.0, 40, 0.8, 0.0, rng)]
    return [synth.star_ring(20.0, 86.0, 500, 9.0, 0.2, rng)]


@pytest.fixture(scope="module", params=["sphere", "antimeridian", "pole"])
def exact_case(request):
    rings = _polygon(request.param)
    P = G.Polygon.from_rings(rings)
    rng = np.random.default_rng(42)
    c = rings[0].mean(0)
    pts = np.concatenate([_special(rings), synth.uniform_points(3000, rng), synth.near_edge_points(rings, 3000, rng),
                          c + rng.uniform(-12, 12, (3000, 2)) * [1.0, 0.3]])
    pts = pts[rng.permutation(len(pts))]
    xyz, pe = P.export()
    want = exact.ExactPolygon(xyz, pe, len(rings[0])).query_lonlat(pts)
    return P, G.Grid(P, semantics=G.SEMANTICS_EXACT).classify(), rings, pts, want


@pytest.mark.parametrize("n", [1, 31, 33, 255, 257, 32768, 32769, (1 << 20) - 1, 1 << 20, (1 << 20) + 1,
                               (1 << 20) + 64 * 1024 + 97, 148 * 8 * 1024 * 2 + 130])
def test_exact_labels_of_the_first_points(exact_case, n):
    """Both filters, into labels at an odd address, from points on a 16-byte
    boundary that is not a 32-byte one."""
    import torch
    P, g, rings, pts, want = exact_case
    k = 1 + n // len(pts)
    want = np.tile(want, k)[:n]
    buf = torch.zeros((n + 1, 2), dtype=torch.float64, device="cuda")
    buf[1:] = torch.from_numpy(np.tile(pts, (k, 1))[:n])
    lab = torch.full((n + 2,), 7, dtype=torch.uint8, device="cuda")
    for prec in (G.QUERY_FP32_FILTER, G.QUERY_FP64_FILTER):
        g.query_device(buf.data_ptr() + 16, n, lab.data_ptr() + 1, prec, sync=True)
        got = lab.cpu().numpy()
        assert got[0] == 7 and got[-1] == 7
        bad = np.nonzero(got[1:-1] != want)[0]
        assert len(bad) == 0, (prec, len(bad), pts[bad[0] % len(pts)], got[1 + bad[0]], want[bad[0]])
        assert g.stats()["in_count"] == int((want == 2).sum())


@pytest.mark.parametrize("n", [5000, (1 << 20) + 5])
def test_all_points_undecided_by_the_first_tier(exact_case, n):
    """Points on vertices and edges only: more than tier 2's queue has room for."""
    import torch
    P, g, rings, pts, want = exact_case
    v = np.concatenate(rings)
    on = np.concatenate([v, 0.5 * (v + np.roll(v, 1, 0)), np.nextafter(v, 0.0)])
    xyz, pe = P.export()
    w = exact.ExactPolygon(xyz, pe, len(rings[0])).query_lonlat(on)
    k = 1 + n // len(on)
    d = torch.from_numpy(np.tile(on, (k, 1))[:n]).cuda()
    lab = torch.zeros(n, dtype=torch.uint8, device="cuda")
    for prec in (G.QUERY_FP32_FILTER, G.QUERY_FP64_FILTER):
        g.query_device(d.data_ptr(), n, lab.data_ptr(), prec, sync=True)
        assert np.array_equal(lab.cpu().numpy(), np.tile(w, k)[:n]), prec
    assert g.stats()["boundary_points"] > 0


@pytest.mark.parametrize("chunk", [256, 4096, 1 << 20])
def test_batch_chunks(exact_case, chunk):
    """A batch's tiles, chunk ends and summary ring, in every launch shape."""
    import torch
    P, g, rings, pts, want = exact_case
    off = np.array([0, len(pts), 2 * len(pts) - 77, 2 * len(pts) - 77, 3 * len(pts) - 77], dtype=np.int64)
    d = torch.from_numpy(np.concatenate([pts, pts[:-77], pts])).cuda()
    w = np.concatenate([want, want[:-77], want])
    B = G.Batch([P, P, P, P])
    B.set_chunk(chunk)
    lab = torch.zeros(len(w), dtype=torch.uint8, device="cuda")
    for shape in range(len(B.shapes())):
        B.set_shape(shape)
        for prec in (G.QUERY_FP32_FILTER, G.QUERY_FP64_FILTER):
            lab.zero_()
            B.query_device(d.data_ptr(), off, lab.data_ptr(), prec, sync=True)
            assert np.array_equal(lab.cpu().numpy(), w), (shape, prec)
