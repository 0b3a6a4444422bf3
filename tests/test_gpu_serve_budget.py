"""A budget that admitted a polygon's first build admits the same build again
when nothing else is resident: the working memory that the server learns from
a build does not turn it away."""
import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import _lib, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def polygon():
    rng = np.random.default_rng(4)
    ring, _ = synth.displaced_ring(15.0, 40.0, 20000, 25.0, base=64, amp_deg=2.0, rng=rng)
    return G.Polygon.from_rings([ring])


def _first_estimate(p):
    return 1.5 * 1024 * p.num_edges + 32 * p.num_edges  # before any build has been measured


@pytest.mark.parametrize("room", [1.01, 1.05, 1.09])
@pytest.mark.parametrize("lru", [True, False])
def test_builds_one_after_the_other(polygon, room, lru):
    srv = G.Server(slots=1, slot_points=1 << 16, hbm_budget=int(room * _first_estimate(polygon)), evict_lru=lru,
                   build_workers=1)
    pts = np.random.default_rng(5).uniform(-60, 60, (500, 2))
    want = G.Grid(polygon).classify().query(pts)
    for _ in range(5):
        pid, tk = srv.build(polygon)
        srv.wait(tk)
        assert srv.state(pid)[0] == _lib.POLY_READY
        tk, lab = srv.query(pid, pts)
        srv.wait(tk)
        assert np.array_equal(lab, want)
        if not lru:
            srv.evict(pid)
    st = srv.stats()
    assert st["builds_done"] == 5 and st["builds_failed"] == 0 and st["resident_bytes"] <= st["hbm_budget"]
    srv.close()


def test_working_memory_counts_beside_residents(polygon):
    """The largest budget that does not hold a resident polygon, a second
    index by its estimate and the second build's working memory refuses it."""
    srv = G.Server(slots=1, slot_points=1 << 16, hbm_budget=int(1.18 * _first_estimate(polygon)), evict_lru=False,
                   build_workers=1)
    a, tk = srv.build(polygon, pinned=True)
    srv.wait(tk)
    c, tk = srv.build(polygon)
    with pytest.raises(G.GahhgError) as e:
        srv.wait(tk)
    assert e.value.status == _lib.ERR_CAPACITY and srv.state(a)[0] == _lib.POLY_READY
    srv.evict(a)
    d, tk = srv.build(polygon)
    srv.wait(tk)
    assert srv.state(d)[0] == _lib.POLY_READY
    srv.close()
