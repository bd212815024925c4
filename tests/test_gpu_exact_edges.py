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


def test_panel_paths_agree_above_the_cluster_height(acc):
    """S = 3,360: the first panels outgrow a cluster of CTAs and go grid-wide
    (or, with grid_panels 0, one CTA from global memory); the rest are
    clusters.  Same bits either way."""
    import bench

    w, s, f = bench.mesh_workload(24)
    ant = acc.Antenna(acc.wires_array(w[:2240 // 2]), acc.sources_array([(3, 1, 1.0)]), [f], 1)
    got = []
    for grid in (1, 0):
        b = acc.HallenBatch([ant])
        assert b.units[0]["s"] > 3072
        b.schedule = {"grid_panels": grid}
        assert b.solve().status[0] == 0
        got.append(b.read_unit(0))
        b.close()
    assert np.array_equal(got[0][1], got[1][1])
    assert np.array_equal(got[0][0].view(np.uint64), got[1][0].view(np.uint64))


def test_near_ties_take_the_last_largest_pivot(acc):
    """Rows of equal and nearly equal magnitude in every column (a unitary
    DFT matrix times small perturbations): the pivots are the oracle's."""
    for n, eps in ((40, 0.0), (64, 1e-15), (300, 1e-14), (420, 3e-13)):
        k = np.arange(n)
        z = np.exp(-2j * np.pi * np.outer(k, k) / n)
        z = z * (1.0 + eps * np.random.default_rng(n).normal(size=(n, n)))
        rhs = np.exp(0.3j * k)
        cosv = np.cos(np.linspace(-1.0, 1.0, n))
        ends = np.array([[0, n - 1]])
        x0, p0 = O.solve_hallen(z, rhs, cosv, ends, [], [], [])
        x1, p1 = acc.solve_hallen(z, rhs, cosv, ends, [], return_pivots=True)
        assert np.array_equal(p0, p1)
        assert np.array_equal(x0.view(np.uint64), x1.view(np.uint64))


@pytest.mark.parametrize("n", [48, 96])
@pytest.mark.parametrize("scale", [1e-140, 1e-12, 1e70, 1e140])
def test_extreme_magnitudes(acc, n, scale):
    """Entries whose squares leave the range of the shared reciprocal: the
    general comparisons and divisions, bit for bit.  Where the elimination
    overflows to a column of NaNs the library reports it as singular."""
    rng = np.random.default_rng(n)
    z = (rng.normal(size=(n, n)) + 1j * rng.normal(size=(n, n))) * scale
    rhs = rng.normal(size=n) + 1j * rng.normal(size=n)
    cosv = np.cos(np.linspace(-1.5, 1.5, n))
    ends = np.array([[0, n - 1]])
    try:
        x0, p0 = O.solve_hallen(z, rhs, cosv, ends, [], [], [])
    except Exception:
        with pytest.raises(acc.AccelError):
            acc.solve_hallen(z, rhs, cosv, ends, [])
        return
    try:
        x1, p1 = acc.solve_hallen(z, rhs, cosv, ends, [], return_pivots=True)
    except acc.AccelError:
        assert np.isnan(x0).any()
        return
    assert np.array_equal(p0, p1)
    both = np.isnan(x0) & np.isnan(x1)  # a NaN's sign and payload are the hardware's
    assert np.array_equal(x0[~both].view(np.uint64), x1[~both].view(np.uint64))
