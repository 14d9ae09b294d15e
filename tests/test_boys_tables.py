"""The Boys tables the engine carries as module constants (csrc/gen_eri.py, boys_header)."""
import importlib.util
import os
import re

import numpy as np
import pytest
from scipy.special import gamma, gammainc

CSRC = os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "chronusq_public_b200", "csrc")


@pytest.fixture(scope="module")
def tables():
    spec = importlib.util.spec_from_file_location("gen_eri_for_boys", os.path.join(CSRC, "gen_eri.py"))
    g = importlib.util.module_from_spec(spec)
    spec.loader.exec_module(g)
    text = g.boys_header()

    def array(name):
        m = re.search(r"double %s\[(\d+)\] = \{([^}]*)\}" % name, text)
        v = np.array([float(x) for x in m.group(2).replace("\n", " ").split(",")])
        assert len(v) == int(m.group(1))
        return v
    return g, array("kBoysTable"), array("kBoysRows")


def _boys(n, T):
    """F_n(T) from the regularised lower incomplete gamma function (n + 1/2 > 0), T > 0."""
    return 0.5 * gamma(n + 0.5) * gammainc(n + 0.5, T) / T ** (n + 0.5)


@pytest.mark.parametrize("L", range(13))
def test_rows_are_taylor_coefficients(tables, L):
    """Rows on the points i / 8 (F_0's ten coefficients for L = 1, else F_L's nine and e^-T), then
    the far row: c_n = sqrt(pi)/2 (2n-1)!!/2^n."""
    g, _, rows = tables
    nt = g.BOYS_NTAYLOR
    off = sum((8 * t + 2) * (nt + 2) for t in g.BOYS_TMAX[:L])
    n = 8 * g.BOYS_TMAX[L] + 1
    row = rows[off:off + (n + 1) * (nt + 2)].reshape(n + 1, nt + 2)
    base, nc = (0, 10) if L == 1 else (L, nt + 1)
    T = np.arange(n) / 8.0                       # exact in binary
    fact = np.cumprod([1.0] + [float(k) for k in range(1, nc)])
    # scipy's incomplete gamma function is good to a few 1e-14 relative; F_n(0) = 1 / (2 n + 1)
    for k in range(nc):
        assert row[0, k] * fact[k] == pytest.approx(1.0 / (2 * (base + k) + 1), rel=1e-15)
        assert np.allclose(row[1:n, k] * fact[k], _boys(base + k, T[1:]), rtol=1e-12, atol=0)
    if L != 1:
        assert np.allclose(row[:n, nc], np.exp(-T), rtol=1e-15, atol=0)
    c = 0.5 * np.sqrt(np.pi)
    for k in range(base):
        c *= 0.5 * (2 * k + 1)
    far = np.zeros(nt + 2)
    far[0] = c
    if L == 1:
        far[1] = 0.5 * c
    assert np.allclose(row[n], far, rtol=4e-15, atol=0)


def test_table_is_the_boys_function(tables):
    g, table, _ = tables
    F = table[:g.BOYS_NT * g.BOYS_NORD].reshape(g.BOYS_NT, g.BOYS_NORD)
    T = 0.1 * np.arange(g.BOYS_NT)
    # T = i / 10 exactly: the double nearest 3.6 is off by enough to show in e^-T
    ex = np.exp(-np.arange(g.BOYS_NT, dtype=np.longdouble) / 10).astype(np.float64)
    assert np.allclose(table[g.BOYS_NT * g.BOYS_NORD:], ex, rtol=1e-15, atol=0)
    for n in (0, 8, 20, 31):
        assert F[0, n] == pytest.approx(1.0 / (2 * n + 1), rel=1e-15)
        assert np.allclose(F[1:, n], _boys(n, T[1:]), rtol=1e-12, atol=0)


@pytest.mark.parametrize("L", range(6))
def test_far_values_start_where_they_are_exact(tables, L):
    """From boys_tmax on, F_n = c_n T^(-n-1/2) holds to 1e-16 for n <= L (the far row's claim)."""
    g = tables[0]
    T = np.array([g.BOYS_TMAX[L], g.BOYS_TMAX[L] + 0.3, 60.0, 200.0])
    F, _ = g.boys_values(T[:3], L)
    c = 0.5 * np.sqrt(np.pi)
    for n in range(L + 1):
        far = c * T[:3] ** (-n - 0.5)
        # 1e-16 of truncation and the rounding of the power
        assert np.allclose(F[:, n].astype(np.float64), far, rtol=1e-15, atol=0)
        c *= 0.5 * (2 * n + 1)
