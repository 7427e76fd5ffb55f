"""Paths that few shapes reach, against the exact FP64 path (equal counts, so equal
values, bit for bit): 32-bit counts, brute force on pair lists and shards, the walks
with one query per lane over whole matrices; and calls from several threads."""
import threading

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _traj(n, T, seed, **kw):
    from gmx_correlation_b200.synth import synth_traj
    return synth_traj(n, T, 8, 0.06, seed=seed, fp32=True, **kw)


def _equal(gc, x, k, **kw):
    a, ax, ay = gc.kraskov_corrmatrix(x, k, detail=True, **kw)
    b, bx, by = gc.kraskov_corrmatrix(x, k, detail=True, path=gc.PATH_EXACT_FP64, **kw)
    np.testing.assert_array_equal(ax, bx)
    np.testing.assert_array_equal(ay, by)
    np.testing.assert_array_equal(a, b)
    return ax, ay


@pytest.mark.parametrize("T", [65535, 65536, 65600])
def test_counts_above_16_bits(gc, T):
    """Around the change to two planes of 32-bit counts."""
    x = _traj(2, T, 1)
    _equal(gc, x, 20)
    X, psi, _ = gc.kraskov_prepare(x)
    assert gc.kraskov_wrap(X, psi, 1, 0, 20) == gc.kraskov_corrmatrix(x, 20, path=gc.PATH_EXACT_FP64)[1, 0]


def test_counts_reach_beyond_16_bits(gc):
    """A k of nearly every frame: counts of 65,536 and more in both planes."""
    x = _traj(2, 65700, 2)
    nx, ny = _equal(gc, x, 65690)
    assert max(nx.max(), ny.max()) > 65535


@pytest.mark.parametrize("kw", [{"pair_list": np.array([5, 0, 3])}, {"pairs": (2, 5)}, {"pairs": (5, 6)}])
def test_brute_force_on_lists_and_shards(gc, kw):
    _equal(gc, _traj(4, 16500, 3), 25, **kw)


@pytest.mark.parametrize("n,T,k", [(60, 700, 300), (26, 6100, 12)])
def test_lane_walk_over_a_whole_matrix(gc, n, T, k):
    """More than 24 pairs an atom under the walk with one query per lane (k or rows
    beyond the row walk): rows in single groups."""
    _equal(gc, _traj(n, T, 4), k)


@pytest.mark.parametrize("n,T,k,lag", [(30, 700, 300, 2), (28, 6200, 9, 1), (30, 3300, 40, 1)])
def test_te_lane_kernels_over_a_whole_matrix(gc, n, T, k, lag):
    """TE beyond the row walk (k, rows) and beyond the row count alone."""
    x = _traj(n, T, 5)
    np.testing.assert_array_equal(gc.te_matrix(x, k, lag), gc.te_matrix(x, k, lag, path=gc.PATH_EXACT_FP64))


def test_several_threads(gc):
    """Threads share the pools, the idle streams, the kept plans and the kernels'
    shared memory limits; sizes differ so that each would disturb another's."""
    jobs = []
    for T in (300, 2000, 700, 4000):
        X, psi, _ = gc.kraskov_prepare(_traj(2, T, T))
        jobs.append(lambda X=X, psi=psi: gc.kraskov_wrap(X, psi, 1, 0, 9))
    for n, T in ((30, 400), (30, 400), (25, 900), (6, 2500)):
        x = _traj(n, T, n + T)
        jobs += [lambda x=x: gc.te_matrix(x, 6, 1), lambda x=x: gc.kraskov_corrmatrix(x, 6),
                 lambda x=x: gc.gcmi_corrmatrix(x), lambda x=x: gc.gauss_corrmatrix(x)]
    want = [j() for j in jobs]
    wrong = []

    def work(first):
        for r in range(3):
            for i in range(len(jobs)):
                at = (first * 7 + i) % len(jobs)
                try:
                    if not np.array_equal(jobs[at](), want[at]):
                        wrong.append((first, at, "value"))
                except gc.GCError as e:
                    wrong.append((first, at, str(e)))

    threads = [threading.Thread(target=work, args=(t,)) for t in range(6)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not wrong, wrong[:5]
