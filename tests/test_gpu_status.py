"""A bounded wait of a product's tensor-core kernels that runs out is reported
by the call that returns the product's result and leaves the context usable:
calls that synchronise by themselves and whose last operation is a product
(solves, Chebyshev, Brownian dynamics, batches).  Of products queued on a
caller's stream the next call reports it, once.

The wait runs out on an mbarrier that nothing arrives at (stokes_gpu_test_
stall_waits), after `polls` of about 20 us: long enough that a call has queued
all of its products before the first one gives up."""
import ctypes as C
import time

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu

POLLS = 500


@pytest.fixture
def stall(lib):
    yield lambda polls=POLLS: lib.stokes_gpu_test_stall_waits(polls, 0)
    lib.stokes_gpu_test_stall_waits(0, 0)


def _system(version, n, precision, seed=11):
    from libstokes_gb300 import System
    from libstokes_gb300.workloads import rsa_positions
    pos, side = rsa_positions(n, 0.2, seed=seed)
    s = System(version, pos, (side,) * 3)
    s.set_precision(precision)
    return s, pos


def _d(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def _engine(lib, s, precision):
    from libstokes_gb300 import abi
    p = abi.BDParams(peclet=1.0, dt=1e-3, n_cheb=2, n_lanczos=20, cheb_eps=0.0, check_every=0,
                     lj_e=0.0, lj_r0=2.0, seed=3, precision=precision)
    h = C.c_void_p()
    abi.check(lib.stokes_gpu_bd_create(s.sp, C.byref(p), C.byref(h)))
    abi.check(lib.stokes_gpu_bd_set_bounds(h, _d(np.array([0.2, 4.0]))))
    return h


# F N = 600 in mixed precision: the tensor-core path (small systems have none)
@pytest.mark.parametrize("call", ["noise", "noise_error", "run", "step_noise", "solve", "chebyshev",
                                  "bounds"])
@pytest.mark.parametrize("precision,n", [(0, 100), (1, 600)])
def test_host_calls_report_their_own_wait(lib, stall, call, precision, n):
    from libstokes_gb300 import abi
    s, pos = _system(0, n, precision)
    h = _engine(lib, s, precision)
    rng = np.random.default_rng(2)
    x, z, err = rng.standard_normal(s.n), np.zeros(s.n), C.c_double()
    good = s.atimes(x)

    def make():
        if call == "noise":
            return lib.stokes_gpu_bd_noise(h, _d(x), _d(z), None)
        if call == "noise_error":
            return lib.stokes_gpu_bd_noise(h, _d(x), _d(z), C.byref(err))
        if call == "run":
            return lib.stokes_gpu_bd_run(h, 0.0, 1)
        if call == "step_noise":
            return lib.stokes_gpu_bd_step_noise(h, 0.0, _d(x))
        if call == "bounds":
            return lib.stokes_gpu_bd_estimate_bounds(h, None)
        if call == "solve":
            # any residual will do: the start vector's product is the only one
            it, res = C.c_int(), C.c_double()
            return lib.stokes_gpu_solve(s.sp, 0, _d(x), _d(z), 20, 200, 1e30, C.byref(it),
                                        C.byref(res))
        a = np.array([1.0, 0.1])
        lib.chebyshev_eval_atimes(2, _d(a), s.n, _d(x), _d(z), 0.2, 4.0,
                                  C.cast(lib.atimes_3all, C.c_void_p),
                                  C.cast(s.sp, C.c_void_p))
        return lib.stokes_gpu_last_error()

    lib.stokes_gpu_set_error_mode(1)
    assert make() == abi.STOKES_GPU_OK, lib.stokes_gpu_last_error_message()
    assert stall() == abi.STOKES_GPU_OK
    assert make() == abi.STOKES_GPU_ETIMEOUT
    assert b"ran out" in lib.stokes_gpu_last_error_message()
    lib.stokes_gpu_test_stall_waits(0, 0)
    # the failure is not reported again, and results are right again
    s.set_pos(pos)
    y = np.zeros(s.n)
    assert lib.stokes_gpu_atimes(s.sp, _d(x), _d(y)) == abi.STOKES_GPU_OK
    assert rel_l2(y, good) < 1e-12
    lib.stokes_gpu_bd_destroy(h)
    s.close()


def test_batch_creation_reports_its_wait(lib, stall):
    """FP64: creation makes one product of each system and records the rest."""
    from libstokes_gb300 import abi
    systems = [_system(v, 40 + 7 * v, 0, seed=20 + v)[0] for v in (0, 1)]
    arr = (C.POINTER(type(systems[0].s)) * 2)(*[s.sp for s in systems])
    h = C.c_void_p()
    assert stall(50) == abi.STOKES_GPU_OK
    assert lib.stokes_gpu_batch_create(arr, 2, 0, C.byref(h)) == abi.STOKES_GPU_ETIMEOUT
    lib.stokes_gpu_test_stall_waits(0, 0)
    h = C.c_void_p()
    assert lib.stokes_gpu_batch_create(arr, 2, 0, C.byref(h)) == abi.STOKES_GPU_OK
    n = sum(s.n for s in systems)
    x, y = np.random.default_rng(3).standard_normal(n), np.zeros(n)
    assert lib.stokes_gpu_batch_atimes(h, _d(x), _d(y)) == abi.STOKES_GPU_OK
    o = 0
    for s in systems:
        assert rel_l2(y[o:o + s.n], s.atimes(x[o:o + s.n])) < 1e-12
        o += s.n
    lib.stokes_gpu_batch_destroy(h)
    for s in systems:
        s.close()


@pytest.mark.parametrize("precision,n", [(0, 100), (1, 600)])
def test_queued_products_report_once(lib, stall, precision, n):
    """Products on a caller's stream: the next call reports the wait that ran
    out; those still queued behind it do not raise it a second time."""
    import torch
    from libstokes_gb300 import abi
    s, pos = _system(0, n, precision)
    x = torch.from_numpy(np.random.default_rng(4).standard_normal(s.n)).cuda()
    p = torch.from_numpy(pos).cuda()
    y, good = torch.zeros_like(x), torch.zeros_like(x)
    st = torch.cuda.Stream()
    torch.cuda.synchronize()

    def product(out):
        return lib.stokes_gpu_atimes_dev(s.sp, p.data_ptr(), x.data_ptr(), out.data_ptr(),
                                         C.c_void_p(st.cuda_stream))

    assert product(good) == abi.STOKES_GPU_OK
    st.synchronize()
    assert stall(4 * POLLS) == abi.STOKES_GPU_OK
    t0 = time.perf_counter()
    assert product(y) == abi.STOKES_GPU_OK
    st.synchronize()
    span = time.perf_counter() - t0                  # two waits that ran out
    assert product(y) == abi.STOKES_GPU_ETIMEOUT
    assert product(y) == abi.STOKES_GPU_OK
    assert product(y) == abi.STOKES_GPU_OK           # queued behind the first
    time.sleep(0.75 * span)                          # the first has raised the word
    assert product(y) == abi.STOKES_GPU_ETIMEOUT
    lib.stokes_gpu_test_stall_waits(0, 0)
    torch.cuda.synchronize()
    assert product(y) == abi.STOKES_GPU_OK
    st.synchronize()
    assert torch.equal(y, good)
    s.close()
