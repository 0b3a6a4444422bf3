"""Queries on host buffers of the sizes where their copies change: staged from
4 MB of points on, slots of 512 KB, chunks of 2^23 points; page-locked buffers
and calls that find the stage in use are copied directly."""
import threading

import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import synth

pytestmark = pytest.mark.gpu

MIN = (4 << 20) // 16  # points


@pytest.fixture(scope="module")
def case():
    import torch
    g = G.Grid(G.Polygon.from_rings(synth.c0_polygon()), semantics=G.SEMANTICS_EXACT).classify()
    pts = synth.uniform_points((1 << 23) + MIN + 3, np.random.default_rng(5))
    d = torch.from_numpy(pts).cuda()
    lab = torch.zeros(len(pts), dtype=torch.uint8, device="cuda")
    g.query_device(d.data_ptr(), len(pts), lab.data_ptr(), G.QUERY_FP32_FILTER, sync=True)
    return g, pts, lab.cpu().numpy()


@pytest.mark.parametrize("n", [1, MIN - 1, MIN, MIN + 1, 32768 * 12 * 2, 32768 * 25 + 1, 1 << 23, (1 << 23) + 1,
                               (1 << 23) + MIN + 3])
def test_sizes(case, n):
    g, pts, want = case
    # also points that start off a 16-byte boundary of the first slot
    for a in (0, min(1, len(pts) - n)):
        got = g.query(pts[a:a + n], G.QUERY_FP32_FILTER)
        assert np.array_equal(got, want[a:a + n])
        assert g.stats()["in_count"] == int((want[a:a + n] == 2).sum())


def test_page_locked(case):
    import torch
    g, pts, want = case
    n = 3 * MIN + 5
    pinned = torch.from_numpy(pts[:n]).pin_memory().numpy()
    assert np.array_equal(g.query(pinned, G.QUERY_FP64_FILTER), want[:n])


def test_threads(case):
    """Several grids queried at once: one of them at a time is staged."""
    g, pts, want = case
    grids = [g] + [G.Grid(G.Polygon.from_rings(synth.c0_polygon()), semantics=G.SEMANTICS_EXACT).classify()
                   for _ in range(3)]
    bad = []

    def work(k):
        for r in range(4):
            n = MIN + 100_003 * (k + r)
            if not np.array_equal(grids[k].query(pts[:n], G.QUERY_FP32_FILTER), want[:n]):
                bad.append((k, r))

    th = [threading.Thread(target=work, args=(k,)) for k in range(4)]
    for t in th:
        t.start()
    for t in th:
        t.join()
    assert not bad
