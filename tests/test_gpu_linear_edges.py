"""Gaussian and copula MI at the edges of their kernels: tiles of 8 and 16 atoms
and the change between them (176 to 177 atoms), stages of 8 frames and their
remainders, the sort's sizes, ties; and input that is not finite.  Sums are in
the oracle's order; what is left is the rounding of logarithms and determinants
(the tolerance of the other tests of these estimators)."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _traj(n, T, seed, digits=None):
    from gmx_correlation_b200.synth import center, raw_positions
    p = raw_positions(n, T, 8, 0.06, seed=seed)
    return center(p if digits is None else np.round(p, digits))[0]


@pytest.mark.parametrize("n,T", [(2, 9), (7, 16), (8, 17), (9, 23), (15, 24), (16, 25), (17, 31), (33, 40), (64, 9),
                                 (176, 26), (177, 26), (177, 33), (192, 15), (193, 17), (209, 64)])
def test_gauss_tiles(gc, oracle, n, T):
    x = _traj(n, T, n + T)
    np.testing.assert_allclose(gc.gauss_corrmatrix(x), oracle.gauss_matrix(x), rtol=1e-12, atol=1e-14)


@pytest.mark.parametrize("n,T,digits", [(2, 9, None), (9, 32, None), (16, 63, 1), (17, 64, None), (5, 65, 1), (178, 66, None),
                                        (3, 129, 2), (4, 1024, None), (3, 1025, 1), (2, 2049, 2), (2, 16384, 2)])
def test_gcmi_sort_and_tiles(gc, oracle, n, T, digits):
    x = _traj(n, T, n + T, digits)
    np.testing.assert_allclose(gc.gcmi_corrmatrix(x), oracle.gcmi_matrix(x), rtol=1e-12, atol=1e-14)


@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
@pytest.mark.parametrize("n,T", [(3, 64), (4, 70), (20, 300), (2, 17000)])
def test_not_finite_is_an_error_and_leaves_nothing(gc, n, T, value):
    """+inf and nan sort among the padding of the copula's sort, whose entries
    have no place in the output."""
    x = _traj(n, T, 5)
    want = gc.gcmi_corrmatrix(x), gc.gauss_corrmatrix(x), gc.te_matrix(x[:2, :60], 4, 1)
    for atom, comp in ((0, 0), (n - 1, 2)):
        y = x.copy()
        y[atom, [1, T // 2, T - 1], comp] = value
        for call in (gc.gcmi_corrmatrix, gc.gauss_corrmatrix, lambda v: gc.gcmi_batch([x, v])):
            with pytest.raises(gc.GCError) as e:
                call(y)
            assert e.value.status == 5
    for a, b in zip(want, (gc.gcmi_corrmatrix(x), gc.gauss_corrmatrix(x), gc.te_matrix(x[:2, :60], 4, 1))):
        np.testing.assert_array_equal(a, b)
