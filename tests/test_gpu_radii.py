"""Unequal radii in mixed precision, changed between products: the split
follows the largest radius, the rest only their own tables.  1e-6 against FP64
as for every mixed product."""
import ctypes as C
import time

import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _d(a):
    return a.ctypes.data_as(C.POINTER(C.c_double))


@pytest.mark.parametrize("version,n", [(0, 60), (0, 600), (1, 450), (2, 60), (2, 300)])
def test_products_follow_the_radii(lib, version, n):
    from libstokes_gb300 import FP64, MIXED, System
    from libstokes_gb300.workloads import rsa_positions
    rng = np.random.default_rng(n)
    pos, side = rsa_positions(n, 0.15, seed=n)
    s = System(version, pos, (side,) * 3)
    x = rng.standard_normal(s.n)
    first = 0.6 + 0.4 * rng.random(n)
    first[3] = 1.0
    second = first[::-1].copy()                  # the same largest radius
    third = 0.8 * first                          # another one: another split
    radii = [first, second, first, third, None, np.ones(n), second]
    for a in radii:
        s.set_radius(a)
        s.set_precision(FP64)
        ref = s.atimes(x)
        s.set_precision(MIXED)
        y = [s.atimes(x) for _ in range(3)]      # direct, recorded, replayed
        assert rel_l2(y[0], ref) < 1e-6
        assert np.array_equal(y[0], y[1]) and np.array_equal(y[0], y[2])
    s.close()


def test_new_radii_do_not_remake_the_split(lib):
    """F N = 600, where the split, its plan and tables take about 600 us and a
    product 50: a product with new radii stays below 6 products (16 times as long
    if the split is remade)."""
    from libstokes_gb300 import MIXED, System
    from libstokes_gb300.workloads import rsa_positions
    n = 600
    rng = np.random.default_rng(1)
    pos, side = rsa_positions(n, 0.15, seed=2)
    s = System(0, pos, (side,) * 3)
    s.set_precision(MIXED)
    x, y = rng.standard_normal(s.n), np.zeros(s.n)
    radii = 0.6 + 0.4 * rng.random((20, n))
    radii[:, 0] = 1.0

    def span(change):
        t = []
        for a in radii:
            if change:
                s.set_radius(a)
            t0 = time.perf_counter()
            assert lib.stokes_gpu_atimes(s.sp, _d(x), _d(y)) == 0
            t.append(time.perf_counter() - t0)
        return np.median(t)

    s.set_radius(radii[0])
    span(False)
    assert span(True) < 6 * span(False)
    s.close()
