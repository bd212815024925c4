"""sqrt(x) and a / sqrt(x) of the exact Z fill (fnec_math.cuh sqrt_recip,
div_by), built for the host, against the IEEE operations bit for bit."""
import ctypes
import os
import subprocess

import numpy as np
import pytest

HERE = os.path.dirname(os.path.abspath(__file__))
CSRC = os.path.join(os.path.dirname(HERE), "fnec-rust_b200", "csrc")


@pytest.fixture(scope="module")
def probe(tmp_path_factory):
    out = tmp_path_factory.mktemp("probe") / "exact_div.so"
    subprocess.run(["g++", "-O2", "-ffp-contract=off", "-fPIC", "-shared", "-I", CSRC,
                    os.path.join(HERE, "exact_div_probe.cpp"), "-o", str(out), "-lm"], check=True)
    L = ctypes.CDLL(str(out))
    P = ctypes.c_void_p
    L.probe_sqrt_div_mismatches.argtypes = [P, P, ctypes.c_long, P]
    L.probe_sqrt_div_mismatches.restype = ctypes.c_long
    L.probe_domain_count.argtypes = [P, ctypes.c_long]
    L.probe_domain_count.restype = ctypes.c_long
    return L


def _mantissa_edges():
    """x just off powers of four and off squares of short numbers, where the
    root lies next to a representable number or to the middle of two."""
    one = np.float64(1.0)
    m = [np.nextafter(one, 2), np.nextafter(one, 0), one, np.float64(2) - 2.0 ** -52, np.float64(4) - 2.0 ** -51]
    m += [np.float64(2) + k * 2.0 ** -51 for k in (1, 2, 3)] + [one + k * 2.0 ** -52 for k in (2, 3, 4, 5, 6, 7)]
    rng = np.random.default_rng(3)
    roots = 1.0 + rng.integers(1, 2 ** 26, 200_000) * 2.0 ** -26
    sq = roots * roots  # exact: 27-bit roots
    m = np.concatenate([np.array(m), sq, np.nextafter(sq, 0), np.nextafter(sq, 8)])
    return np.concatenate([m, m * 0.25, m * 2.0 ** 60, m * 2.0 ** -90, m * 0.5])


def test_sqrt_and_quotients_bit_identical_to_ieee(probe):
    rng = np.random.default_rng(17)
    x = np.concatenate([rng.uniform(1e-8, 1e4, 2_000_000), 10.0 ** rng.uniform(-30, 30, 2_000_000),
                        rng.uniform(1.0, 4.0, 2_000_000), _mantissa_edges()])
    a = rng.uniform(-1.0, 1.0, len(x))
    a[::5] *= 10.0 ** rng.uniform(-30, 0, len(a[::5]))
    a[::7] = 1.0
    a[::11] = -0.0
    assert probe.probe_domain_count(x.ctypes.data, len(x)) == len(x)
    bad = np.zeros(2)
    n = probe.probe_sqrt_div_mismatches(a.ctypes.data, x.ctypes.data, len(x), bad.ctypes.data)
    assert n == 0, [float.hex(v) for v in bad]


def test_domain_leaves_out_what_it_must(probe):
    x = np.array([0.0, -1.0, 2.0 ** -101, 2.0 ** 100, np.inf, -np.inf, np.nan, 5e-324])
    assert probe.probe_domain_count(x.ctypes.data, len(x)) == 0
