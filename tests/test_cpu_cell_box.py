"""The cell rectangles that decide which edges a lattice cell lists
(gahhg_b200/csrc/cell_box.cuh, built for the host).

A query in a cell counts the listed edges that cross the arc from the cell's
center to it, so every edge that crosses such an arc must pass the rectangle
test, for cells of 1e-8 to 0.2 rad at any latitude (beside a pole too),
points anywhere in the cell and on its border, edges much shorter and much
longer than the cell.  The crossings are built, not searched: the edge runs
through a point of the arc.
"""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
RAD = 3.14159265 / 180.0


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    out = str(tmp_path_factory.mktemp("box") / "libbox_probe.so")
    subprocess.check_call(["g++", "-O2", "-ffp-contract=off", "-shared", "-fPIC", "-I",
                           os.path.join(os.path.dirname(HERE), "include"), "-o", out,
                           os.path.join(HERE, "native", "box_probe.cpp")])
    return ctypes.CDLL(out)


def _call(fn, cfg):
    cfg = np.ascontiguousarray(cfg, dtype=np.float64)
    out = np.zeros(len(cfg), dtype=np.int32)
    fn.argtypes = [ctypes.c_void_p, ctypes.c_long, ctypes.c_void_p]
    fn(cfg.ctypes.data, len(cfg), out.ctypes.data)
    return out


def _xyz(lon, lat):
    a, o = lat * RAD, lon * RAD
    return np.stack([np.cos(a) * np.sin(o), np.sin(a), np.cos(a) * np.cos(o)], -1)


def _unit(v):
    return v / np.linalg.norm(v, axis=-1, keepdims=True)


def cells(rng, n):
    """Centers and half sizes (degrees); a fifth of the cells touch a pole."""
    hp = 10.0 ** rng.uniform(-8, np.log10(0.12), n) / RAD
    hl = np.minimum(hp * 10.0 ** rng.uniform(-1, 1.8, n), 0.19 / RAD)
    lat = rng.uniform(-1, 1, n) * (90.0 - hp)
    pole = rng.random(n) < 0.2
    lat = np.where(pole, np.sign(lat) * (90.0 - hp), lat)
    return rng.uniform(-180, 180, n), lat, hl, hp


def crossing_edges(rng, R, q):
    """Edges through a point of arc(R, q): any direction, lengths 1e-9 to 0.5 rad on either side."""
    n = len(R)
    t = rng.uniform(0, 1, (n, 1))
    t[rng.random(n) < 0.3] = 1.0
    z = _unit((1 - t) * R + t * q)
    d = rng.normal(size=(n, 3))
    d = _unit(d - np.sum(d * z, 1, keepdims=True) * z)
    la, lb = 10.0 ** rng.uniform(-9, -0.3, (2, n, 1))
    return _unit(z - np.tan(la) * d), _unit(z + np.tan(lb) * d)


@pytest.mark.parametrize("seed", [1, 2, 3])
def test_edges_crossing_an_arc_in_the_cell_meet_its_rectangle(probe, seed):
    rng = np.random.default_rng(seed)
    n = 60000
    lon, lat, hl, hp = cells(rng, n)
    u, v = rng.uniform(-1, 1, (2, n))
    edge = rng.random((2, n)) < 0.4  # points on the sides and in the corners
    u, v = np.where(edge[0], np.sign(u), u), np.where(edge[1], np.sign(v), v)
    R, q = _xyz(lon, lat), _xyz(lon + u * hl, lat + v * hp)
    A, B = crossing_edges(rng, R, q)
    got = _call(probe.own_meets, np.concatenate([np.stack([lon, lat, hl, hp], 1), A, B], 1))
    assert not np.any(got == 0)
    assert (got == 1).mean() > 0.8


def test_rectangles_are_tight(probe):
    """Short edges at random near a cell: the share listed is the rectangle's
    area, not a cap's (five times the cell's)."""
    rng = np.random.default_rng(9)
    n = 100000
    h = 0.001 / RAD
    lat = np.full(n, 35.0)
    lon = rng.uniform(-180, 180, n)
    hl = h / np.cos(lat * RAD)
    u, v = rng.uniform(-2, 2, (2, n))
    z = _xyz(lon + u * hl, lat + v * h)
    A = z
    B = _unit(z + 1e-6 * rng.normal(size=(n, 3)))
    got = _call(probe.own_meets, np.concatenate([np.stack([lon, lat, hl, np.full(n, h)], 1), A, B], 1))
    assert np.all((got == 1)[(np.abs(u) <= 1) & (np.abs(v) <= 1)])
    assert 0.24 < (got == 1).mean() < 0.27  # 4 of 16 cell areas, and the rims
