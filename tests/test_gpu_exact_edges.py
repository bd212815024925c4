"""The plain form's kernels at the edges of their tiles, panels and pieces.

A random system of n segments on one wire (S = n + 1 unknowns, two free
ends) is solved from a given Z: normal equations, pivoted elimination and
substitution must equal the oracle's operations bit for bit (linear.rs:672-797,
:1321-1383) at sizes around every block width.
"""
import numpy as np
import pytest

from oracle import oracle as O

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def acc():
    import nec_accel

    return nec_accel


@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 14, 15, 16, 17, 30, 31, 32, 33, 47, 48, 63, 64, 65, 95, 96, 127, 128, 129,
                               159, 191, 255, 256, 257, 258, 273, 320, 385, 399, 514])
def test_solve_bit_identical_given_z(acc, n):
    rng = np.random.default_rng(n)
    z = rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))
    z[rng.integers(0, n, n), rng.integers(0, n, n)] = 0.0  # exact zeros keep their sign
    rhs = rng.normal(size=n) + 1j * rng.normal(size=n)
    cosv = np.cos(np.linspace(-1.5, 1.5, n))
    ends = np.array([[0, n - 1]])
    x0, p0 = O.solve_hallen(z, rhs, cosv, ends, [], [], [])
    x1, p1 = acc.solve_hallen(z, rhs, cosv, ends, [], return_pivots=True)
    assert np.array_equal(p0, p1)
    assert np.array_equal(x0.view(np.uint64), x1.view(np.uint64))
