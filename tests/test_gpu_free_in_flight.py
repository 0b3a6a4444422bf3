"""An index that is freed while queries without `sync` are still queued: they
complete with the right labels, although the next build takes its memory."""
import ctypes

import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import _lib, synth

pytestmark = pytest.mark.gpu

POINTS = 1_500_000


@pytest.fixture(scope="module")
def case():
    import torch
    rng = np.random.default_rng(3)
    rings = [synth.star_ring(20.0, 30.0, 60000, 25.0, 0.2, rng)]
    other = [synth.star_ring(-120.0, -20.0, 60000, 25.0, 0.3, rng)]
    pts = np.concatenate([synth.near_edge_points(rings, POINTS // 2, rng), synth.uniform_points(POINTS // 2, rng)])
    return rings, other, torch.from_numpy(pts[rng.permutation(POINTS)]).cuda()


def _delay(stream):
    """Keeps the stream busy for some tens of milliseconds."""
    import torch
    with torch.cuda.stream(stream):
        torch.cuda._sleep(100_000_000)


def _other_builds(other):
    return [G.Grid(G.Polygon.from_rings(other)) for _ in range(3)]


@pytest.mark.parametrize("kind,n", [("fp32", POINTS), ("fp64", POINTS), ("fp32", 5000), ("noalloc", 70000),
                                    ("reference", 100000)])
def test_grid(case, kind, n):
    import torch
    rings, other, d = case
    precision = {"fp64": G.QUERY_FP64_FILTER, "reference": G.QUERY_REFERENCE_FP64}.get(kind, G.QUERY_FP32_FILTER)
    semantics = G.SEMANTICS_REFERENCE if kind == "reference" else G.SEMANTICS_EXACT
    rings = [rings[0][::10]] if kind == "reference" else rings
    P = G.Polygon.from_rings(rings)
    want = torch.zeros(n, dtype=torch.uint8, device="cuda")
    lab = torch.zeros(n, dtype=torch.uint8, device="cuda")
    g = G.Grid(P, semantics=semantics).classify()
    g.query_device(d.data_ptr(), n, want.data_ptr(), precision, sync=True)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    _delay(side)
    if kind == "noalloc":
        _lib.check(_lib.lib().gahhg_query_device_noalloc(g._h, ctypes.c_void_p(d.data_ptr()), n,
                                                         ctypes.c_void_p(lab.data_ptr()), precision,
                                                         ctypes.c_void_p(side.cuda_stream)))
    else:
        g.query_device(d.data_ptr(), n, lab.data_ptr(), precision, stream=side.cuda_stream)
    del g
    keep = _other_builds(other)
    torch.cuda.synchronize()
    assert torch.equal(lab, want) and len(keep) == 3


@pytest.mark.parametrize("graph", [False, True])
def test_batch(case, graph):
    import torch
    rings, other, d = case
    off = np.array([0, POINTS // 2, POINTS], dtype=np.int64)
    P = [G.Polygon.from_rings(rings), G.Polygon.from_rings([rings[0][::7]])]
    want = torch.zeros(POINTS, dtype=torch.uint8, device="cuda")
    lab = torch.zeros(POINTS, dtype=torch.uint8, device="cuda")
    B = G.Batch(P)
    B.query_device(d.data_ptr(), off, want.data_ptr(), sync=True)
    side = torch.cuda.Stream()
    torch.cuda.synchronize()
    _delay(side)
    B.query_device(d.data_ptr(), off, lab.data_ptr(), stream=side.cuda_stream, graph=graph)
    del B
    keep = _other_builds(other) + [G.Batch([G.Polygon.from_rings(other)] * 2)]
    torch.cuda.synchronize()
    assert torch.equal(lab, want) and len(keep) == 4
