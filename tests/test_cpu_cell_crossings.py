"""What the index build's labels and lists rest on, against exact arithmetic
(gahhg_b200/csrc/cell_box.cuh and exact_pred.cuh, built for the host).

Every child's label and every level-0 parity is a count of crossings taken in
the plane at a cell's center: a crossing that the plane is certain of (or
certain that there is none) has to be the exact one, for edges through the
arc, through its ends, beside it by 1e-19 to 1e-2 of the cell's size, with an
end on it, short and long, at any latitude.  And a child lists every edge that
crosses an arc from its parent's center, or from its own, to a point of the
child, by the child's rectangle in the parent's plane.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

from oracle import exact
from tests.test_cpu_cell_box import _call, _unit, cells, crossing_edges

HERE = os.path.dirname(os.path.abspath(__file__))


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("cell") / "libcell_probe.so")
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                           os.path.join(os.path.dirname(HERE), "include"), "-o", out,
                           os.path.join(HERE, "native", "cell_probe.cpp")])
    return ctypes.CDLL(out)


def _crossings(probe, cfg):
    cfg = np.ascontiguousarray(cfg, dtype=np.float64)
    out = np.zeros((len(cfg), 2), dtype=np.int32)
    probe.center_crossings.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_void_p]
    probe.center_crossings(cfg.ctypes.data, len(cfg), out.ctypes.data)
    return out


def _near_arc(rng, R, q, size):
    """Edges whose line, or an end, passes a point of the great circle of
    arc(R, q) (in the arc, at its ends, beyond them) at 10^U[-19, -2] of the
    cell's size."""
    n = len(R)
    t = rng.uniform(-0.3, 1.3, (n, 1))
    t[rng.random(n) < 0.3] = rng.integers(0, 2)
    z = _unit((1 - t) * R + t * q)
    nrm = _unit(np.cross(R, q) + 1e-300)
    z = _unit(z + 10.0 ** rng.uniform(-19, -2, (n, 1)) * size[:, None] * rng.choice([-1.0, 1.0], (n, 1)) * nrm)
    d = rng.normal(size=(n, 3))
    along = rng.random(n) < 0.2  # nearly along the arc
    d[along] = (q - R)[along] + 1e-9 * rng.normal(size=(along.sum(), 3)) * size[along, None]
    d = _unit(d - np.sum(d * z, 1, keepdims=True) * z + 1e-300)
    la, lb = 10.0 ** rng.uniform(-9, -0.3, (2, n, 1))
    kind = rng.random(n)
    la[kind < 0.15] = 0.0  # the point is an end
    return _unit(z - np.tan(la) * d), _unit(z + np.tan(lb) * d)


@pytest.mark.parametrize("seed", [1, 2, 3, 4])
def test_certain_crossings_are_exact(probe, seed):
    rng = np.random.default_rng(seed)
    n = 40000
    lon, lat, hl, hp = cells(rng, n)
    u, v = rng.uniform(-1, 1, (2, n))
    snap = rng.random((2, n)) < 0.3
    u, v = np.where(snap[0], np.sign(u), u), np.where(snap[1], 0.0, v)
    vert = rng.random(n) < 0.3  # the border's middle above or below
    u, v = np.where(vert, 0.0, u), np.where(vert, np.where(rng.random(n) < 0.5, 1.0, -1.0), v)
    c, p = np.stack([lon, lat], 1), np.stack([lon + u * hl, lat + v * hp], 1)
    R, q = exact.vertex_xyz(c), exact.vertex_xyz(p)
    A, B = _near_arc(rng, R, q, np.maximum(hp, 1e-9) * np.pi / 180)
    # vertices on the center's meridian and on the border's, in degrees as polygons have them
    grid = rng.random(n) < 0.2
    A[grid] = exact.vertex_xyz(np.stack([lon, lat + 3 * hp * rng.uniform(-1, 1, n)], 1))[grid]
    B[grid] = exact.vertex_xyz(np.stack([np.where(rng.random(n) < 0.5, lon, lon + hl), lat - hp], 1))[grid]
    got = _crossings(probe, np.concatenate([c, p, A, B], 1))
    sure = (got[:, 0] >= 0) & (got[:, 0] < 2)
    assert np.array_equal(got[sure & (got[:, 1] >= 0), 0], got[sure & (got[:, 1] >= 0), 1])
    assert not np.any(sure & (got[:, 1] < 0))  # an end on an end of the arc is never certain
    assert sure.mean() > 0.3 and (got[sure, 0] == 1).mean() > 0.1
    mer = _call(probe.meridian_crossings, np.concatenate([c, p, A, B], 1)[vert])
    w = got[vert]
    sure = (mer >= 0) & (mer < 2) & (w[:, 1] >= 0)
    assert sure.mean() > 0.3 and np.array_equal(mer[sure], w[sure, 1])


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_edges_crossing_an_arc_to_a_childs_point_meet_its_rectangle(probe, seed):
    rng = np.random.default_rng(seed)
    n = 60000
    lon, lat, hl, hp = cells(rng, n)
    cx, cy = rng.integers(0, 4, (2, n)).astype(np.float64)
    u, v = rng.uniform(0, 1, (2, n))
    snap = rng.random((2, n)) < 0.4
    u, v = np.where(snap[0], np.round(u), u), np.where(snap[1], np.round(v), v)
    at = lambda a, b: exact.vertex_xyz(np.stack([lon + ((cx + a) * 0.5 - 1.0) * hl, lat + ((cy + b) * 0.5 - 1.0) * hp], 1))
    own = at(0.5, 0.5)
    # the child's own arcs, which its leaf or its children count along
    A, B = crossing_edges(rng, own, at(u, v))
    got = _call(probe.child_meets, np.concatenate([np.stack([lon, lat, hl, hp, cx, cy], 1), A, B], 1))
    assert not np.any(got == 0)
    assert (got == 1).mean() > 0.8


def test_childrens_rectangles_are_tight(probe):
    """Short edges at random over a cell: each child lists its sixteenth."""
    rng = np.random.default_rng(9)
    n = 100000
    h = 0.001 * 180.0 / np.pi
    lat = np.full(n, 35.0)
    lon = rng.uniform(-180, 180, n)
    hl = h / np.cos(lat * np.pi / 180)
    cx, cy = rng.integers(0, 4, (2, n)).astype(np.float64)
    u, v = rng.uniform(-1, 1, (2, n))
    A = exact.vertex_xyz(np.stack([lon + u * hl, lat + v * h], 1))
    B = _unit(A + 1e-7 * rng.normal(size=(n, 3)))
    got = _call(probe.child_meets, np.concatenate([np.stack([lon, lat, hl, np.full(n, h), cx, cy], 1), A, B], 1))
    assert 0.06 < (got == 1).mean() < 0.068
