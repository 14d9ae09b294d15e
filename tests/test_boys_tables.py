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


@pytest.mark.parametrize("L", [0, 1, 5, 12])
def test_rows_are_taylor_coefficients(tables, L):
    g, table, rows = tables
    nt = g.BOYS_NTAYLOR
    row = rows.reshape(g.BOYS_MAXL + 1, g.BOYS_NT, nt + 2)[L]
    F = table[:g.BOYS_NT * g.BOYS_NORD].reshape(g.BOYS_NT, g.BOYS_NORD)
    T = 0.1 * np.arange(g.BOYS_NT)
    fact = np.cumprod([1.0] + [float(k) for k in range(1, nt + 1)])
    assert np.allclose(row[:, :nt + 1] * fact, F[:, L:L + nt + 1], rtol=1e-15, atol=0)
    # T = i / 10 exactly: the double nearest 3.6 is off by enough to show in e^-T
    ex = np.exp(-np.arange(g.BOYS_NT, dtype=np.longdouble) / 10).astype(np.float64)
    assert np.allclose(row[:, nt + 1], ex, rtol=1e-15, atol=0)
    assert np.allclose(table[g.BOYS_NT * g.BOYS_NORD:], ex, rtol=1e-15, atol=0)
    # scipy's incomplete gamma function is good to a few 1e-14 relative; F_n(0) = 1 / (2 n + 1)
    for k in (0, nt):
        assert F[0, L + k] == pytest.approx(1.0 / (2 * (L + k) + 1), rel=1e-15)
        assert np.allclose(F[1:, L + k], _boys(L + k, T[1:]), rtol=1e-12, atol=0)
