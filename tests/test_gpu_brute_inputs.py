"""The FP32 brute force (single pairs, long trajectories, no-allocation entry
point) on inputs where its error bound, lists or buckets come to an end: every
count equals the exact FP64 path's, so every value is equal, bit for bit."""
import ctypes

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _pair(gc, rows, k, path):
    """gc_ksg_pair on rows [6, T] as they are (the entry point takes any)."""
    rows = np.ascontiguousarray(rows)
    T = rows.shape[1]
    psi = np.zeros(T + 1)
    psi[1] = -0.57721566490153
    for n in range(1, T):
        psi[n + 1] = psi[n] + 1.0 / n
    mi = ctypes.c_double()
    o = gc._opts(path=path)
    gc._check(gc.lib().gc_ksg_pair(gc._dptr(rows), T, k, gc._dptr(psi), ctypes.byref(o), ctypes.byref(mi)))
    return mi.value


def _rows(kind, T, seed):
    rng = np.random.default_rng(seed)
    r = rng.standard_normal((6, T))
    r[3:] += 0.5 * r[:3]
    if kind == "both infinities":
        r[0, 3], r[0, T // 2] = np.inf, -np.inf
    elif kind == "one infinity":
        r[4, T // 3] = np.inf
    elif kind == "nan":
        r[1, [2, T // 2]] = np.nan
        r[:, T // 4] = np.nan
    elif kind == "beyond fp32":
        r[:3] *= 1e200
    elif kind == "one component beyond fp32":
        r[2] *= 5e38
    elif kind == "tiny":
        r *= 1e-200
    elif kind == "far from zero":
        r += 1e6
    return r


@pytest.mark.parametrize("kind", ["both infinities", "one infinity", "nan", "beyond fp32", "one component beyond fp32",
                                  "tiny", "far from zero"])
@pytest.mark.parametrize("T,k", [(60, 5), (700, 20), (2500, 9)])
def test_pair_rows_of_any_value(gc, T, k, kind):
    r = _rows(kind, T, T)
    a, b = _pair(gc, r, k, gc.PATH_AUTO), _pair(gc, r, k, gc.PATH_EXACT_FP64)
    assert a == b or (np.isnan(a) and np.isnan(b))
