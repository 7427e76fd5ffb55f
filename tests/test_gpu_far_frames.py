"""Trajectories with frames far off (a broken frame, a stretch in another
periodic image) or on very different scales: an atom's largest distance is
then hundreds of times a usual one.  The results equal the exact FP64 path's,
bit for bit, and the row sort's further levels cost about a level each."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _traj(kind, n, T, seed):
    from gmx_correlation_b200.synth import synth_traj
    rng = np.random.default_rng(seed)
    x = synth_traj(n, T, 6, 0.08, seed=seed, fp32=True)
    if kind == "frame":
        x[:, T // 3] += 200.0
    elif kind == "stretch":
        for a in range(n):
            at = rng.integers(0, T) + np.arange(rng.integers(T // 10, T // 2))
            x[a, at % T, rng.integers(0, 3)] += 50.0
    elif kind == "scales":  # three scales a factor of 600 apart, and repeated frames
        scale = rng.choice([1.0, 1.0 / 600, 1.0 / 360000], T)
        x *= scale[None, :, None]
        x[:, :: max(2, T // 50)] = x[:, :1]
    return x


# every shape of the row sort: 64, 128 (8 and 16 distances a thread), 256, 512 and 1024 threads
_SIZES = [(24, 100, 7), (4, 513, 9), (25, 600, 12), (30, 1500, 20), (4, 3000, 15), (3, 6000, 11), (2, 9000, 8)]


@pytest.mark.parametrize("kind", ["frame", "stretch", "scales"])
@pytest.mark.parametrize("n,T,k", _SIZES)
def test_ksg_equals_exact(gc, n, T, k, kind):
    x = _traj(kind, n, T, seed=n + T)
    a, ax, ay = gc.kraskov_corrmatrix(x, k, detail=True)
    b, bx, by = gc.kraskov_corrmatrix(x, k, path=gc.PATH_EXACT_FP64, detail=True)
    np.testing.assert_array_equal(ax, bx)
    np.testing.assert_array_equal(ay, by)
    np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("kind", ["frame", "stretch", "scales"])
@pytest.mark.parametrize("n,T,k", [(24, 102, 7), (4, 515, 9), (30, 1300, 20), (3, 3000, 15), (2, 6000, 11), (2, 9000, 8)])
def test_te_equals_exact(gc, n, T, k, kind):
    x = _traj(kind, n, T, seed=n + T)
    np.testing.assert_array_equal(gc.te_matrix(x, k, 2), gc.te_matrix(x, k, 2, path=gc.PATH_EXACT_FP64))


def _ms(gc, x, k, lag):
    torch = pytest.importorskip("torch")
    n, T = x.shape[0], x.shape[1]
    p = gc.KsgPlan(n, T, k) if lag is None else gc.TePlan(n, T, k, lag)
    d_x = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    d_out = torch.zeros(n * n, dtype=torch.float64, device="cuda")
    ms = []
    for _ in range(4):
        p.run(d_x.data_ptr(), d_out.data_ptr())
        p.sync()
        ms.append(p.kernel_ms)
    p.close()
    return min(ms)


@pytest.mark.parametrize("n,T,k,lag", [(50, 4999, 100, None), (16, 2000, 20, None), (12, 3000, 20, 1)])
def test_a_far_frame_costs_little_more(gc, n, T, k, lag):
    """One frame far off puts every other distance of a row 8 octaves below
    its largest: a second level of the sort.  Three times the kernels' time of
    the same trajectory without it leaves room for more than two whole sorts
    (a full sort of such rows took 5 to 9 times)."""
    assert _ms(gc, _traj("frame", n, T, 3), k, lag) < 3.0 * _ms(gc, _traj("smooth", n, T, 3), k, lag)


def _handoffs(gc, x, k, pair_list=None):
    torch = pytest.importorskip("torch")
    n, T = x.shape[0], x.shape[1]
    p = gc.KsgPlan(n, T, k, pair_list=pair_list)
    d_x = torch.from_numpy(np.ascontiguousarray(x)).cuda()
    d_out = torch.zeros(n * (n - 1) // 2, dtype=torch.float64, device="cuda")
    p.run(d_x.data_ptr(), d_out.data_ptr())
    p.sync()
    h = p.handoffs
    p.close()
    return h


@pytest.mark.parametrize("n,T,k", [(60, 2000, 100), (30, 3000, 10)])
def test_rows_for_many_pairs_hand_over_no_more(gc, n, T, k):
    """The walk of a row for 32 pairs at once settles the queries that the walk
    with one query per lane (pair lists) settles: both count into the same
    buckets up to a query's bracket.  They differ in how far behind it an
    overflow still counts (up to 16 entries here, one bucket there)."""
    x = _traj("stretch", n, T, seed=7)
    one = _handoffs(gc, x, k, pair_list=np.arange(n * (n - 1) // 2))
    assert _handoffs(gc, x, k) <= 1.05 * one + 50
