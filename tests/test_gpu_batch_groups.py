"""Mixed batches at the edges of the back-projection's groups of four particles
and of its tables in shared memory, against each system's FP64 product at the
mixed tolerance 1e-6."""
import ctypes as C

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _dp(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


def _product(lib, systems, x):
    arr = (C.POINTER(type(systems[0].s)) * len(systems))(*[s.sp for s in systems])
    h = C.c_void_p()
    assert lib.stokes_gpu_batch_create(arr, len(systems), 1, C.byref(h)) == 0
    y = np.zeros_like(x)
    assert lib.stokes_gpu_batch_atimes(h, _dp(x), _dp(y)) == 0, lib.stokes_gpu_last_error_message()
    lib.stokes_gpu_batch_destroy(h)
    return y


def _check(lib, shapes, rng):
    from libstokes_gb300 import System
    systems = []
    for version, n, box in shapes:
        m = int(np.ceil(n ** (1 / 3)))
        g = np.stack(np.meshgrid(*(np.arange(m),) * 3, indexing="ij"), -1).reshape(-1, 3)
        cell = np.asarray(box) / m
        systems.append(System(version, (g[:n] + 0.5) * cell + rng.uniform(-0.3, 0.3, (n, 3)), box))
    x = rng.standard_normal(sum(s.n for s in systems))
    y = _product(lib, systems, x)
    at = 0
    for s in systems:
        assert rel_l2(y[at:at + s.n], s.atimes(x[at:at + s.n])) < 1e-6
        at += s.n
        s.close()


def test_sizes_around_a_group(lib):
    rng = np.random.default_rng(3)
    _check(lib, [(n % 2, n, (12.0, 13.0, 11.0)) for n in (1, 2, 3, 4, 5, 7, 8, 9, 31, 33)], rng)


def test_table_too_long_for_shared_memory(lib, monkeypatch):
    """|m| up to about 190 along one side: the table rows are read from global
    memory."""
    monkeypatch.setenv("LIBSTOKES_GB300_BATCH_ETA", "6")
    rng = np.random.default_rng(4)
    _check(lib, [(1, 9, (10.0, 10.0, 1200.0)), (0, 6, (11.0, 10.0, 12.0))], rng)
