"""Device points that are not on a 16-byte boundary are refused by every entry
point before anything is launched."""
import ctypes

import numpy as np
import pytest

import gahhg_b200 as G
from gahhg_b200 import _lib, synth

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def polygon():
    return G.Polygon.from_rings([synth.star_ring(10.0, 20.0, 80, 20.0, 0.2, np.random.default_rng(2))])


def _refused(call):
    with pytest.raises(G.GahhgError) as e:
        call()
    assert e.value.status == _lib.ERR_ARG and "aligned" in str(e.value)


def test_points_off_a_16_byte_boundary(polygon):
    import torch
    n = 500
    buf = torch.zeros(2 * n + 2, dtype=torch.float64, device="cuda")
    lab = torch.full((n,), 7, dtype=torch.uint8, device="cuda")
    at, out = buf.data_ptr() + 8, lab.data_ptr()
    off = np.array([0, 200, n], dtype=np.int64)
    r = G.Grid(polygon, semantics=G.SEMANTICS_REFERENCE).classify()
    g = G.Grid(polygon).classify()
    B = G.Batch([polygon, polygon])
    for sync in (False, True):
        _refused(lambda: r.query_device(at, n, out, G.QUERY_REFERENCE_FP64, sync=sync))
        _refused(lambda: g.query_device(at, n, out, G.QUERY_REFERENCE_FP64, sync=sync))
        _refused(lambda: g.query_device(at, n, out, G.QUERY_AUTO, sync=sync))
        _refused(lambda: B.query_device(at, off, out, sync=sync))
    _refused(lambda: B.query_device(at, off, out, graph=True))
    torch.cuda.synchronize()
    assert bool((lab == 7).all())
    # nothing to read: nothing to refuse
    r.query_device(at, 0, out, G.QUERY_REFERENCE_FP64, sync=True)
    B.query_device(at, np.zeros(3, dtype=np.int64), out, sync=True)
    B.query_device(at, np.zeros(3, dtype=np.int64), out, graph=True)
    # aligned ones are answered
    want = r.query(np.zeros((n, 2)), G.QUERY_REFERENCE_FP64)
    r.query_device(buf.data_ptr(), n, out, G.QUERY_REFERENCE_FP64, sync=True)
    assert np.array_equal(lab.cpu().numpy(), want)
    lab.fill_(7)
    B.query_device(buf.data_ptr() + 16, off, out, graph=True)
    torch.cuda.synchronize()
    assert np.array_equal(lab.cpu().numpy(), g.query(np.zeros((n, 2))))
    _lib.check(_lib.lib().gahhg_query_device_noalloc(g._h, ctypes.c_void_p(buf.data_ptr()), n, ctypes.c_void_p(out),
                                                     G.QUERY_AUTO, None))
    torch.cuda.synchronize()
