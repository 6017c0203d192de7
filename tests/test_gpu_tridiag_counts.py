"""The device's tridiagonal eigenvalues where counting could go wrong: one to a
few rows, decoupled rows, clusters, rows that differ by many orders of magnitude
and matrices of very large and small norm, against LAPACK at 1e-12 |T|."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _lowest(d, e, k):
    from ed_code_gb300 import _native as N

    m = len(d)
    d, e = np.ascontiguousarray(d, np.float64), np.ascontiguousarray(e, np.float64)
    out, vec, n = np.empty(k), np.empty((k, m)), C.c_int()
    N.check(N.lib().edg_tridiag_lowest(d.ctypes.data, e.ctypes.data, m, k, 0, out.ctypes.data, vec.ctypes.data,
                                       C.byref(n)))
    assert n.value == k
    return out


@pytest.mark.parametrize("m", [1, 2, 3, 4, 5, 6, 33, 300, 2000])
@pytest.mark.parametrize("kind", ["plain", "decoupled", "cluster", "graded", "large", "small"])
def test_lowest_values_match_lapack(cuda_device, m, kind):
    rng = np.random.default_rng(m)
    d, e = rng.standard_normal(m), np.abs(rng.standard_normal(m))
    if kind == "decoupled":
        e[::3] = 0.0
    elif kind == "cluster":
        d[:], e[:] = 1.0, 1e-9
    elif kind == "graded":
        d, e = d * np.logspace(0, -12, m), e * np.logspace(0, -12, m)
    elif kind == "large":
        d, e = d * 1e20, e * 1e20
    elif kind == "small":
        d, e = d * 1e-20, e * 1e-20
    e[0] = 0.0
    T = np.diag(d) + np.diag(e[1:], 1) + np.diag(e[1:], -1)
    k = min(m, 32)
    want = np.linalg.eigvalsh(T)[:k]
    got = _lowest(d, e, k)
    scale = np.abs(T).sum(axis=1).max()
    assert np.abs(got - want).max() <= 1e-12 * scale
