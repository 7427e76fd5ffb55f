"""The row walk and the FP32 brute force at the sizes where they can go wrong,
against the exact FP64 path: blocks of 32 atoms and their remainders, tiles of
the shortest and longest rows, the smallest and largest k, bucket windows far
apart, duplicated frames and exact ties; frames around the staged chunk and
the row sort's limit.  Both sides count the same neighbours and add the same
table entries in the same order, so every value is equal, bit for bit."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _traj(kind, n, T, seed):
    from gmx_correlation_b200.synth import synth_traj
    rng = np.random.default_rng(seed)
    x = synth_traj(n, T, 6, 0.08, seed=seed, fp32=True)
    if kind == "ties":  # a coarse lattice: many equal distances
        x = np.round(x * 40.0) / 40.0 + 0.0
    elif kind == "duplicates":  # a third of the frames repeat frame 0
        x[:, rng.choice(T, T // 3, replace=False)] = x[:, :1]
    elif kind == "tails":  # atoms with rare large excursions: k-th distances of very different size
        x[::3] *= 1.0 + 200.0 * (rng.random((len(x[::3]), T, 1)) < 4.0 / T)
    return x


@pytest.mark.parametrize("n,T,k,kind", [
    (24, 40, 1, "smooth"), (24, 40, 39, "smooth"), (31, 97, 5, "smooth"), (32, 129, 7, "ties"),
    (33, 128, 20, "smooth"), (64, 300, 10, "duplicates"), (65, 257, 12, "smooth"), (66, 500, 100, "tails"),
    (40, 1300, 254, "smooth"), (25, 2049, 60, "ties"), (24, 6040, 30, "smooth"), (24, 6060, 30, "smooth"),
    (97, 400, 4, "tails"),
])
def test_row_walk_equals_exact(gc, n, T, k, kind):
    x = _traj(kind, n, T, seed=n + T)
    a, ax, ay = gc.kraskov_corrmatrix(x, k, detail=True)
    b, bx, by = gc.kraskov_corrmatrix(x, k, path=gc.PATH_EXACT_FP64, detail=True)
    np.testing.assert_array_equal(ax, bx)
    np.testing.assert_array_equal(ay, by)
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n,T,k,lag,kind", [
    (24, 40, 1, 1, "smooth"), (25, 60, 38, 5, "smooth"), (32, 130, 6, 0, "ties"), (33, 200, 12, 3, "smooth"),
    (65, 150, 10, 1, "tails"), (40, 400, 9, 10, "duplicates"), (30, 1500, 100, 1, "smooth"),
    (24, 900, 255, 2, "smooth"), (24, 800, 254, 2, "smooth"), (24, 6000, 20, 1, "smooth"),
])
def test_te_rows_equal_exact(gc, n, T, k, lag, kind):
    x = _traj(kind, n, T, seed=n + T)
    np.testing.assert_array_equal(gc.te_matrix(x, k, lag), gc.te_matrix(x, k, lag, path=gc.PATH_EXACT_FP64))


@pytest.mark.parametrize("T,k,kind", [
    (20, 1, "smooth"), (33, 32, "smooth"), (500, 10, "ties"), (700, 40, "duplicates"), (2047, 100, "smooth"),
    (2048, 300, "smooth"), (2049, 6, "tails"), (4097, 50, "smooth"), (5000, 4999, "smooth"),
])
def test_single_pair_equals_exact(gc, T, k, kind):
    x = _traj(kind, 2, T, seed=T)
    X, psi, _ = gc.kraskov_prepare(x)
    assert gc.kraskov_wrap(X, psi, 1, 0, k) == gc.kraskov_corrmatrix(x, k, path=gc.PATH_EXACT_FP64)[1, 0]


@pytest.mark.parametrize("n,T,k,kind", [(3, 16386, 20, "smooth"), (4, 16500, 3, "tails"), (2, 17000, 900, "smooth"),
                                        (2, 16400, 15, "ties")])
def test_long_rows_equal_exact(gc, n, T, k, kind):
    x = _traj(kind, n, T, seed=n)
    a, ax, ay = gc.kraskov_corrmatrix(x, k, detail=True)
    b, bx, by = gc.kraskov_corrmatrix(x, k, path=gc.PATH_EXACT_FP64, detail=True)
    np.testing.assert_array_equal(ax, bx)
    np.testing.assert_array_equal(ay, by)
    np.testing.assert_array_equal(a, b)


def _sort_traj(kind, n, T, seed):
    rng = np.random.default_rng(seed)
    x = _traj("smooth", n, T, seed)
    if kind == "few_close":  # a dozen frames nearly equal: distances below the fine buckets, few
        x[:, 1:13] = x[:, :1] + 1e-5 * rng.standard_normal((n, 12, 3)).astype(np.float32)
    elif kind == "many_close":  # all frames nearly equal but for three far ones
        x = x[:, :1] + 1e-4 * (x - x[:, :1])
        x[:, [1, T // 2, T - 1]] += 50.0
    elif kind == "constant":  # one atom that never moves
        x[0] = x[0, :1]
    return x


@pytest.mark.parametrize("n,T,k,kind", [
    (3, 13, 12, "few_close"), (4, 256, 5, "few_close"), (25, 257, 9, "many_close"), (3, 300, 20, "constant"),
    (3, 513, 20, "smooth"), (24, 514, 11, "few_close"), (3, 1025, 40, "smooth"), (3, 1026, 25, "few_close"),
    (3, 2049, 30, "smooth"), (3, 2050, 30, "few_close"), (24, 2051, 12, "many_close"), (3, 4097, 8, "few_close"),
    (3, 4098, 40, "smooth"), (2, 8193, 100, "few_close"), (2, 8194, 20, "smooth"), (3, 9002, 15, "many_close"),
    (2, 16385, 6, "smooth"),
])
def test_rows_equal_exact(gc, n, T, k, kind):
    x = _sort_traj(kind, n, T, seed=n + T)
    a, ax, ay = gc.kraskov_corrmatrix(x, k, detail=True)
    b, bx, by = gc.kraskov_corrmatrix(x, k, path=gc.PATH_EXACT_FP64, detail=True)
    np.testing.assert_array_equal(ax, bx)
    np.testing.assert_array_equal(ay, by)
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("n,T,k,lag,kind", [
    (3, 14, 5, 1, "few_close"), (4, 259, 9, 2, "many_close"), (3, 300, 20, 3, "constant"), (25, 301, 7, 1, "few_close"),
    (3, 514, 20, 1, "smooth"), (24, 516, 11, 2, "few_close"), (3, 1026, 30, 1, "smooth"), (3, 1030, 30, 4, "smooth"),
    (24, 2052, 40, 1, "many_close"), (3, 2051, 25, 1, "few_close"), (3, 4100, 30, 2, "smooth"),
    (2, 8200, 50, 5, "few_close"), (2, 9001, 12, 1, "many_close"),
])
def test_te_fine_buckets_equal_exact(gc, n, T, k, lag, kind):
    x = _sort_traj(kind, n, T, seed=n + T)
    np.testing.assert_array_equal(gc.te_matrix(x, k, lag), gc.te_matrix(x, k, lag, path=gc.PATH_EXACT_FP64))
