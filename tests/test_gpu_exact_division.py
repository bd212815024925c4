"""The plain form's square root and divisions on the device (sqrt_recip,
div_by, recip_rn, cp_div: shared reciprocals with a last correction) against
the IEEE operations, bit for bit.  The hard cases are built: square roots and
quotients whose exact value lies next to the middle of two doubles, roots
next to a double, and mantissas at both ends of the binade."""
from math import isqrt

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

SQRT, DIV_SQRT, RECIP, DIV, COMPLEX = 1, 2, 4, 8, 16


@pytest.fixture(scope="module")
def acc():
    import nec_accel

    nec_accel.default_context()
    return nec_accel


def _odd_root(v, bits):
    """r odd with r^2 = v (mod 2^bits), v = 1 (mod 8)."""
    r = 1
    for k in range(3, bits):
        if (r * r - v) >> k & 1:
            r += 1 << (k - 1)
    return r % (1 << bits)


def _sqrt_midpoints():
    """x whose root is (K + 1/2) 2^e less a little: x 2^t = K^2 + K - c, so the
    root's distance from the middle is about c / (2 K^2), relative."""
    x = []
    for t in (52, 53):
        m = t + 2
        for c in range(-400, 401, 2):
            r0 = _odd_root((4 * c + 1) % (1 << m), m)
            for r in (r0, -r0, r0 + (1 << (m - 1)), (1 << (m - 1)) - r0):
                k = ((r % (1 << m)) - 1) // 2  # K (K + 1) = c (mod 2^t)
                for top in range(0, 4):
                    kk = k + (top << t)
                    if not 1 << 52 <= kk < 1 << 53:
                        continue
                    q, rem = divmod(kk * kk + kk - c, 1 << t)
                    if rem == 0 and 1 << 52 <= q < 1 << 53:
                        x.append(float(q) * 2.0 ** t)
    return np.array(x) / 4.0 ** 52  # in [1, 4)


def _quotient_midpoints(rng, n):
    """(A, B) with A 2^54 = B M + c, M odd and of 54 bits: A / B lies next to
    the middle of two doubles, by c / (B M), relative."""
    a, b = [], []
    for _ in range(n):
        bb = int(rng.integers(1 << 51, 1 << 52)) * 2 + 1
        inv = pow(bb, -1, 1 << 54)
        for c in (1, -1, 3, -3, 5, -7, 33, -101):
            mm = -c * inv % (1 << 54)
            if mm < 1 << 53:
                continue
            q, rem = divmod(bb * mm + c, 1 << 54)
            if rem == 0 and 1 << 52 <= q < 1 << 53:
                a.append(float(q))
                b.append(float(bb))
    return np.array(a), np.array(b)


def _ends():
    """Mantissas at both ends of the binade, and just off squares."""
    m = np.concatenate([1.0 + np.arange(200) * 2.0 ** -52, 2.0 - np.arange(1, 200) * 2.0 ** -52])
    rng = np.random.default_rng(9)
    sq = (1.0 + rng.integers(1, 1 << 26, 20000) * 2.0 ** -26) ** 2
    return np.concatenate([m, 2.0 * m, sq, np.nextafter(sq, 0.0), np.nextafter(sq, 8.0)])


def _clean(acc, a, x):
    bad = acc.test_exact_division(a, x)
    k = np.flatnonzero(bad)
    assert len(k) == 0, (len(k), bad[k[0]], a[k[0]].hex(), x[k[0]].hex())


@pytest.mark.parametrize("exponent", [0, -50, 30, 49])
def test_roots_next_to_midpoints(acc, exponent):
    x = _sqrt_midpoints()
    assert len(x) > 400
    # the construction holds: the exact root lies within 2^-95 of a midpoint
    for v in x[:: len(x) // 50]:
        num, den = float(v).as_integer_ratio()
        s = 240
        root = isqrt((num << (2 * s)) // den)  # sqrt(v) 2^s
        lead = root.bit_length()
        frac = root & ((1 << (lead - 53)) - 1)
        half = 1 << (lead - 54)
        assert abs(frac - half) < 1 << (lead - 95)
    _clean(acc, np.cos(np.arange(len(x))), x * 4.0 ** exponent)


@pytest.mark.parametrize("scale", [0, -300, 300])
def test_quotients_next_to_midpoints(acc, scale):
    rng = np.random.default_rng(21)
    a, b = _quotient_midpoints(rng, 20000)
    assert len(a) > 40000
    a, b = a * 2.0 ** -52, b * 2.0 ** -52  # in [1, 2)
    _clean(acc, a * 2.0 ** scale, b * 2.0 ** (-scale // 2))
    # as quotients by a square root: the root of the rounded square is b
    x = b * b
    assert np.mean(np.sqrt(x) == b) > 0.99
    _clean(acc, -a, x)


def test_ends_of_the_binade(acc):
    v = _ends()
    rng = np.random.default_rng(5)
    for e in (0, -99, 50, 97):
        for f in (0, -200):
            _clean(acc, rng.permutation(v) * 2.0 ** f * np.where(np.arange(len(v)) % 2, 1.0, -1.0), v * 2.0 ** e)
    _clean(acc, np.where(np.arange(len(v)) % 2, 0.0, -0.0), v)


def test_random_over_the_guarded_range(acc):
    rng = np.random.default_rng(2)
    n = 1 << 22
    a = rng.uniform(-1.0, 1.0, n) * 10.0 ** rng.uniform(-100, 100, n)
    x = rng.uniform(0.5, 1.0, n) * 10.0 ** rng.uniform(-119, 119, n)
    _clean(acc, a, x)
    _clean(acc, rng.uniform(-1, 1, n), rng.uniform(1e-8, 1e4, n))
