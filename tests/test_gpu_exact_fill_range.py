"""The exact Z fill over its whole range of k R and R, bit for bit against
the oracle: scales from millimetres to thousands of kilometres, frequencies
from hertz to gigahertz, sizes around its 16 x 16 tiles."""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def acc():
    import nec_accel

    return nec_accel


@pytest.mark.parametrize("ground", [0, 1])
@pytest.mark.parametrize("n,scale,freq,rad", [
    (1, 1.0, 14.2e6, 1e-3), (15, 1.0, 14.2e6, 1e-3), (16, 1.0, 1e6, 1e-3), (17, 10.0, 30e6, 1e-3),
    (49, 20.0, 10e6, 5e-4), (200, 10.0, 100e6, 2e-3), (33, 1e-3, 3e9, 1e-6), (33, 1e6, 3e6, 1.0),
    (33, 1e-3, 1.0, 1e-6), (33, 10.0, 1e-300, 1e-3), (20, 1e-17, 1e6, 1e-19), (20, 1e16, 1e-10, 1.0),
    (20, 1e3, 1e14, 1e-3)])
def test_z_bit_identical_over_the_range(acc, n, scale, freq, rad, ground):
    rng = np.random.default_rng(n)
    segs = np.zeros(n, O.SEG_DTYPE)
    segs["mid"] = rng.uniform(-1, 1, (n, 3)) * scale
    d = rng.normal(size=(n, 3))
    segs["dir"] = d / np.linalg.norm(d, axis=1)[:, None]
    segs["dir"][::3] = [0.0, 0.0, 1.0]
    segs["mid"][::4, 0] = 0.0
    segs["length"], segs["radius"] = scale / 20 * rng.uniform(0.5, 1.5, n), rad
    z0 = O.assemble_z(segs, freq, ground)
    z1 = acc.fill_zmatrix(acc.zsegments_from(segs), freq, ground)
    far = np.isnan(z1.real) & ~np.isnan(z0.real)  # k R beyond the sin/cos restated for the device
    if freq < 1e14:
        assert not far.any()
    assert np.array_equal(z0.view(np.uint64)[~far.repeat(2, 1)], z1.view(np.uint64)[~far.repeat(2, 1)])
