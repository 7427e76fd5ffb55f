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


def _traj(kind, n, T, seed):
    from gmx_correlation_b200.synth import center, raw_positions
    rng = np.random.default_rng(seed)
    p = raw_positions(n, T, 12, 0.06, seed=seed, fp32=True)
    if kind == "far frame":
        p[:, T // 3] += 200.0
    elif kind == "far stretch":
        for a in range(n):
            p[a, (rng.integers(0, T) + np.arange(T // 3)) % T, a % 3] += 50.0
    elif kind == "scales":  # three scales a factor of 600 apart: two moves of the buckets
        p = p[:, :1] + (p - p[:, :1]) * rng.choice([1.0, 1.0 / 600, 1.0 / 360000], T)[None, :, None]
    elif kind == "two digits":  # coordinates stored to 0.01 nm
        p = np.round(p, 2)
    elif kind == "repeats":  # every frame many times
        p = p[:, np.arange(T) % 30]
    return center(p)[0]


KINDS = ["far frame", "far stretch", "scales", "two digits", "repeats"]


@pytest.mark.parametrize("kind", KINDS)
@pytest.mark.parametrize("T,k", [(300, 6), (2048, 50), (2049, 10), (5000, 60)])
def test_pair_equals_exact(gc, T, k, kind):
    X, psi, _ = gc.kraskov_prepare(_traj(kind, 2, T, T))
    assert _pair(gc, X, k, gc.PATH_AUTO) == _pair(gc, X, k, gc.PATH_EXACT_FP64)


@pytest.mark.parametrize("kind", KINDS)
def test_long_rows_equal_exact(gc, kind):
    x = _traj(kind, 3, 16500, 1)
    a, ax, ay = gc.kraskov_corrmatrix(x, 40, detail=True)
    b, bx, by = gc.kraskov_corrmatrix(x, 40, path=gc.PATH_EXACT_FP64, detail=True)
    np.testing.assert_array_equal(ax, bx)
    np.testing.assert_array_equal(ay, by)
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("kind", KINDS)
def test_no_alloc_equals_exact(gc, kind):
    torch = pytest.importorskip("torch")
    n, T, k = 12, 700, 15
    x = _traj(kind, n, T, 2)
    d_x = torch.from_numpy(x).cuda()
    d_out = torch.zeros(n * (n - 1) // 2, dtype=torch.float64, device="cuda")
    gc.ksg_pair_mi_noalloc(d_x.data_ptr(), n, T, k, d_out.data_ptr(), 0)
    torch.cuda.synchronize()
    want = gc.kraskov_corrmatrix(x, k, path=gc.PATH_EXACT_FP64)
    a1, a2 = np.tril_indices(n, -1)
    np.testing.assert_array_equal(d_out.cpu().numpy(), want[a1, a2])


def _ms(gc, x, k, path):
    torch = pytest.importorskip("torch")
    n, T = x.shape[0], x.shape[1]
    p = gc.KsgPlan(n, T, k, path=path)
    d_x = torch.from_numpy(x).cuda()
    d_out = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    ms = []
    for _ in range(4):
        p.run(d_x.data_ptr(), d_out.data_ptr())
        p.sync()
        ms.append(p.kernel_ms)
    p.close()
    return min(ms)


@pytest.mark.parametrize("kind", ["far frame", "two digits", "repeats"])
def test_never_slower_than_exact(gc, kind):
    """These inputs left nearly every query to the FP64 routine inside the
    brute-force kernel, which took longer than the exact kernel alone."""
    x = _traj(kind, 4, 17000, 4)
    assert _ms(gc, x, 50, gc.PATH_AUTO) < _ms(gc, x, 50, gc.PATH_EXACT_FP64)
