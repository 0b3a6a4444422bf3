"""The pass-2 orders over pass 1's queue in parts: queues that are long enough
to be ordered and queues that stay in pass-1 order, parts of very different
lengths, empty ones, the ends of the parts and of the tiles."""
import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def case():
    import torch
    rng = np.random.default_rng(17)
    ring, _ = synth.displaced_ring(-60.0, 20.0, 150000, 40.0, base=64, amp_deg=4.0, rng=rng)
    g = G.Grid(G.Polygon.from_rings([ring])).classify()
    n = 3_000_007
    near = synth.device_c2_points([ring], n + 1, 18, "cuda")[:n]
    far = synth.device_points(n, 19, "cuda")
    return g, near, far


def _labels(g, d, n, prec, order):
    import torch
    lab = torch.full((n,), 9, dtype=torch.uint8, device="cuda")
    old = G.set_knob(G.KNOB_GROUPED_PASS2, order)
    try:
        g.query_device(d.data_ptr(), n, lab.data_ptr(), prec, sync=True)
    finally:
        G.set_knob(G.KNOB_GROUPED_PASS2, old)
    return lab, {k: g.stats()[k] for k in ("boundary_points", "esc_fp64", "esc_exact", "in_count")}


@pytest.mark.parametrize("mix", ["near", "far", "front", "back", "stripes"])
@pytest.mark.parametrize("n", [1 << 18, (1 << 20) + 1, 148 * 8 * 1024, 148 * 8 * 1024 + 1, 3_000_007])
def test_orders(case, mix, n):
    import torch
    g, near, far = case
    k = torch.arange(n, device="cuda")
    pick = {"near": k >= 0, "far": k < 0, "front": k < n // 3, "back": k >= n - n // 3,
            "stripes": (k // 65536) % 3 == 0}[mix]
    d = torch.where(pick[:, None], near[:n], far[:n]).contiguous()
    for prec in (G.QUERY_FP32_FILTER, G.QUERY_FP64_FILTER):
        want, st = _labels(g, d, n, prec, 0)
        assert int((want == 9).sum()) == 0
        for order in (1, 2, 3):
            got, s2 = _labels(g, d, n, prec, order)
            assert torch.equal(got, want) and s2 == st, (mix, n, prec, order)
