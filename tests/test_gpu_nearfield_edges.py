"""Near fields at the edges of the kernel's groups of 12 segments and 32
points, bit for bit against the oracle's sums where its points are not on a
segment, and with points on segment midpoints, E or H alone."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def acc():
    import nec_accel

    return nec_accel


@pytest.mark.parametrize("n,p", [(1, 1), (11, 31), (12, 32), (13, 33), (24, 64), (25, 65), (100, 200), (1, 97), (255, 5)])
def test_sums_match_the_oracle(acc, n, p):
    rng = np.random.default_rng(n * 1000 + p)
    segs = O.build_geometry(O.wires_array([(1, n, (0.0, 0.0, -3.0), (0.5, 0.1, 4.0), 1e-3)]))
    cur = rng.normal(size=n) + 1j * rng.normal(size=n)
    pts = rng.uniform(-8.0, 8.0, (p, 3))
    pts[:: max(p // 3, 1)] = segs["mid"][rng.integers(0, n, len(pts[:: max(p // 3, 1)]))]
    g = acc.gpu_segments_from(segs)
    e0, h0 = O.near_field(segs, cur, 14.2e6, pts)
    e, h = acc.near_field(g, cur, 14.2e6, pts)
    assert np.array_equal(e, e0) and np.array_equal(h, h0)
    assert np.array_equal(acc.near_field(g, cur, 14.2e6, pts, magnetic=False)[0], e)
    assert np.array_equal(acc.near_field(g, cur, 14.2e6, pts, electric=False)[1], h)
