"""Edges whose great circle rises above both ends by more than the margin of
the index's latitude range: a straight border beside a boundary of many short
edges (small cells), and small polygons beside a pole.  Points between the
ends' parallel and the great circle, against the exact oracle."""
import numpy as np
import pytest

import gahhg_b200 as G
from oracle import exact

pytestmark = pytest.mark.gpu


def border(lat, n, south):
    """A straight border of half a degree of arc on the poleward side, a zigzag of n vertices on the other."""
    w = 0.5 / np.cos(np.radians(lat))
    x = np.linspace(10.0 + w, 10.0, n)
    y = lat - 0.02 - 1e-4 * (np.arange(n) % 2)
    ring = np.concatenate([[[10.0, lat], [10.0 + w, lat]], np.stack([x, y], 1)])
    return ring * [1.0, -1.0] if south else ring


CASES = {"border%g%s" % (lat, "s" if s else "n"): (border(lat, 60000, s), 0)
         for lat in (30.0, 45.0, 60.0, 80.0, 88.0) for s in (False, True)}
CASES["pole"] = (np.array([[-140.29040683, -88.53180089], [-129.09686569, -88.60926148], [-134.73203957, -88.86888882],
                           [-145.91156275, -88.87028457], [-148.47874308, -88.64702504]]), 20000)


@pytest.mark.parametrize("name", sorted(CASES))
def test_points_between_the_ends_and_the_great_circle(name):
    ring, top = CASES[name]
    P = G.Polygon.from_rings([ring])
    rng = np.random.default_rng(3)
    lo, hi = ring.min(0), ring.max(0)
    s = np.sign(ring[0, 1])
    edge = ring[np.argsort(-s * ring[:, 1])[:2]]  # the two poleward vertices
    a, b = exact.vertex_xyz(edge)
    t = rng.uniform(0.02, 0.98, 1500)[:, None]
    z = (1 - t) * a + t * b
    z /= np.linalg.norm(z, axis=1, keepdims=True)
    lon, lat = np.degrees(np.arctan2(z[:, 0], z[:, 2])), np.degrees(np.arcsin(z[:, 1]))
    f = rng.uniform(-0.2, 1.3, 1500)  # from the ends' parallel to above the great circle
    base = s * np.minimum(np.abs(edge[:, 1]).max(), 90.0)
    pts = np.concatenate([np.stack([lon, np.clip(base + f * (lat - base), -90, 90)], 1),
                          rng.uniform(lo - 0.01, hi + 0.01, (500, 2))])
    pts[:, 1] = np.clip(pts[:, 1], -90, 90)
    xyz, pe = P.export()
    want = exact.ExactPolygon(xyz, pe, len(ring)).query_lonlat(pts)
    assert 0.2 < (want[:1500] == 2).mean() < 0.95
    g = G.Grid(P, lattice_top=top).classify()
    got = g.query(pts)
    bad = np.nonzero(got != want)[0]
    assert len(bad) == 0, (len(bad), pts[bad[0]], got[bad[0]], want[bad[0]])
