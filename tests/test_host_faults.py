"""The host code on a CUDA runtime without a GPU (fake_cudart.cpp): what a
call leaves behind when a runtime call in the middle of it fails, what it does
when device memory is short, and what it leaves set for other threads."""
import ctypes
import subprocess

import numpy as np
import pytest

from tests.conftest import ROOT

TESTS = ROOT / "tests"


@pytest.fixture(scope="module")
def fake(tmp_path_factory):
    """The package bound to the library's objects linked with the fake runtime."""
    import gmx_correlation_b200 as gc
    from gmx_correlation_b200 import build
    build.build()
    so = tmp_path_factory.mktemp("fake") / "libgmxcorr_fake.so"
    subprocess.run([build.CXX, "-std=c++17", "-O1", "-fPIC", "-shared", "-Wl,-Bsymbolic",
                    f"-I{build.CUDA_HOME / 'include'}", "-o", str(so), str(TESTS / "fake_cudart.cpp"),
                    *sorted(str(o) for o in build.BUILD.glob("*.o")), "-lpthread"], check=True)
    mp = pytest.MonkeyPatch()
    mp.setenv("GMXCORR_B200_LIB", str(so))
    mp.setattr(gc, "_lib", None)
    L = gc.lib()
    for f in ("fake_calls",):
        getattr(L, f).restype = ctypes.c_long
    for f in ("fake_live", "fake_peak"):
        getattr(L, f).restype = ctypes.c_size_t
    L.fake_reset.argtypes = [ctypes.c_long]
    L.fake_limit.argtypes = [ctypes.c_size_t]
    yield gc
    mp.undo()


def _x(n, T, seed=0):
    return np.random.default_rng(seed).standard_normal((n, T, 3))


def _plan(gc, make):
    """A plan's run on device buffers of its own stream, then its end without a sync."""
    p = make()
    buf = np.zeros(200000)
    try:
        p.run(buf.ctypes.data, buf.ctypes.data, None)
    finally:
        p.close()


def _milca(N, k):
    from gmx_correlation_b200.milca import milca
    return milca("mi_xnynK", np.random.default_rng(1).exponential(1.0, (4, N)), k, dimx=2, dimy=2)


CALLS = {
    "ksg": lambda gc: gc.kraskov_corrmatrix(_x(5, 60), 4),
    "ksg rows": lambda gc: gc.kraskov_corrmatrix(_x(30, 60), 4),
    "ksg shard": lambda gc: gc.kraskov_corrmatrix(_x(5, 60), 4, pairs=(1, 7)),
    "ksg long": lambda gc: gc.kraskov_corrmatrix(_x(2, 16400), 4),
    "ksg exact": lambda gc: gc.kraskov_corrmatrix(_x(5, 60), 4, path=gc.PATH_EXACT_FP64),
    "ksg plan": lambda gc: _plan(gc, lambda: gc.KsgPlan(6, 70, 4)),
    "te plan": lambda gc: _plan(gc, lambda: gc.TePlan(6, 70, 4, 1)),
    "pair": lambda gc: gc.kraskov_wrap(np.ones((6, 90)), np.ones(91), 1, 0, 4),
    "prepare": lambda gc: gc.kraskov_prepare(_x(3, 50)),
    "gauss": lambda gc: gc.gauss_corrmatrix(_x(4, 50)),
    "gcmi": lambda gc: gc.gcmi_corrmatrix(_x(4, 50)),
    "te": lambda gc: gc.te_matrix(_x(5, 70), 4, 1),
    "te rows": lambda gc: gc.te_matrix(_x(30, 70), 4, 1),
    "ksg batch": lambda gc: gc.ksg_batch([_x(5, 60), _x(3, 50)], 4),
    "te batch": lambda gc: gc.te_batch([_x(5, 60), _x(3, 50)], 4, 1),
    "gcmi batch": lambda gc: gc.gcmi_batch([_x(5, 60), _x(3, 50)]),
    "features": lambda gc: gc.screen_features(_x(4, 60), 4),
    "milca": lambda gc: _milca(60, 5),
}


@pytest.mark.parametrize("kept", [False, True])
@pytest.mark.parametrize("name", CALLS)
def test_failed_call_leaves_no_work_pending(fake, name, kept):
    """Whatever runtime call fails, the streams have drained when the call
    returns: its device blocks may be handed to the next call at once, and
    copies from the caller's arrays have ended.  kept: with the plan or graph
    of an earlier call of the shape."""
    L, call = fake.lib(), CALLS[name]

    def ready():
        fake.batch_release()
        fake.release_cache()
        if kept:
            call(fake)

    ready()
    L.fake_reset(0)
    call(fake)
    total = L.fake_calls()
    assert total > 3 and L.fake_bad() == 0
    for at in range(1, total + 1):
        ready()
        L.fake_reset(at)
        try:
            call(fake)
        except fake.GCError:
            pass
        where = f"{name}: runtime call {at} of {total} failed"
        assert L.fake_pending() == 0, f"{where}: work pending"
        assert L.fake_bad() == 0, f"{where}: a stream destroyed with work pending"
        call(fake)
    fake.batch_release()
    fake.release_cache()


def _screened(gc):
    from gmx_correlation_b200.screen import TrainedScreen
    m = TrainedScreen.load().model
    gc.ksg_screened(_x(12, 80), 4, m, sigma_max=float("inf"), margin=0.0)


@pytest.mark.parametrize("name", [*CALLS, "screened"])
def test_no_kernel_before_its_tables_are_there(fake, name):
    """Uploads by cudaMemcpy from pageable memory may still be on their way in the
    legacy stream when it returns; the library's own streams do not wait for it."""
    call = CALLS.get(name, _screened)
    for _ in range(2):  # a new plan, a kept one
        fake.lib().fake_reset(0)
        call(fake)
        assert fake.lib().fake_early() == 0
    fake.batch_release()
    fake.release_cache()


def test_shared_memory_limits_do_not_depend_on_the_call(fake):
    """A kernel's dynamic shared memory limit belongs to the function on its
    device: a value of one call's own could lower it between another thread's
    setting it and its launch."""
    fake.release_cache()
    for n, T, k in ((30, 200, 5), (30, 2500, 5), (5, 900, 300), (4, 7000, 6), (3, 12000, 6), (2, 16500, 9)):
        x = _x(n, T)
        fake.kraskov_corrmatrix(x, k)
        fake.te_matrix(x, k, 1)
        fake.gcmi_corrmatrix(x)
        fake.kraskov_wrap(np.ones((6, T)), np.ones(T + 1), 1, 0, k)
        if T <= 16384:
            fake.screen_features(x, k)
    for N, k in ((300, 250), (900, 800)):  # more than the default limit, and more again
        _milca(N, k)
    for T in (300, 2500, 900):
        fake.ksg_batch([_x(30, T), _x(5, T // 2)], 5)
        fake.te_batch([_x(30, T), _x(5, T // 2)], 5, 1)
    fake.batch_release()
    fake.release_cache()
    names = ctypes.create_string_buffer(4096)
    varying = fake.lib().fake_varying_limits(names, 4096)
    assert fake.lib().fake_limited() > 10
    assert varying == 0, names.value.decode()


@pytest.mark.parametrize("name", CALLS)
def test_kept_memory_makes_way(fake, name):
    """A call that fits in device memory runs also when what earlier calls left
    behind (a kept plan, pooled blocks) fills it: those are given up."""
    L, call = fake.lib(), CALLS[name]

    def fresh():
        fake.batch_release()
        fake.release_cache()

    fresh()
    L.fake_reset(0)
    base = L.fake_live()
    call(fake)
    need = L.fake_peak() - base
    fresh()
    fake.te_matrix(_x(60, 1500), 4, 1)
    filled = L.fake_live() - base
    assert filled > need
    L.fake_limit(base + filled)
    try:
        call(fake)
    finally:
        L.fake_limit(180 << 30)
        fresh()


def test_a_large_te_plan_is_not_kept_whole(fake):
    """gc_te_matrix keeps its plan for the next call of the shape, but not one of
    many GB: its blocks serve the next call, of whatever shape, from the pool."""
    L = fake.lib()
    fake.release_cache()
    fake.te_matrix(_x(247, 2000), 100, 1)
    first = L.fake_live()
    assert first > 8 << 30  # the sorted rows alone
    fake.te_matrix(_x(246, 2000), 100, 1)
    assert L.fake_live() < 1.2 * first
    fake.release_cache()
