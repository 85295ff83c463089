"""Large mixed systems in long and flat boxes, where the split of a cube of as
many particles would need more reciprocal vectors along an axis than the limit:
they take a smaller one.  1e-6 against FP64 as for every mixed product."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _positions(n, box, rng):
    """n points on a jittered grid of the box."""
    box = np.asarray(box)
    m = np.maximum(1, np.round(box * (n / box.prod()) ** (1 / 3))).astype(int)
    while m.prod() < n:
        m[np.argmax(box / m)] += 1
    g = np.stack(np.meshgrid(*[np.arange(k) for k in m], indexing="ij"), -1).reshape(-1, 3)
    cell = box / m
    p = (g[rng.permutation(len(g))[:n]] + 0.5) * cell
    return p + rng.uniform(-0.4, 0.4, p.shape) * np.maximum(cell - 2.0, 0.0)


@pytest.mark.parametrize("version,n,shape,shear", [
    (0, 20000, (3.0, 1.0, 1.0), 0), (0, 20000, (1.0, 2.7, 1.0), 1), (1, 17000, (1.0, 1.0, 3.1), 0),
    (2, 17000, (3.0, 1.0, 1.0), 0), (0, 12000, (10.0, 10.0, 1.0), 0), (2, 512, (8.0, 1.0, 1.0), 0)])
def test_long_and_flat_boxes(lib, version, n, shape, shear):
    from libstokes_gb300 import FP64, MIXED, System
    rng = np.random.default_rng(n + version)
    a = (n * 4.19 / 0.15 / np.prod(shape)) ** (1 / 3)
    box = tuple(a * q for q in shape)
    s = System(version, _positions(n, box, rng), box)
    x = rng.standard_normal(s.n)
    ref = s.atimes(x)
    if shear:
        # FP64 keeps the struct's split on a sheared box (minutes at this size):
        # a shift of a whole box length is the unsheared lattice
        s.set_misc(0.0, shear, box[0])
    s.set_precision(MIXED)
    assert rel_l2(s.atimes(x), ref) < 1e-6
    s.set_precision(FP64)
    s.close()


def test_boxes_beyond_every_split_are_refused(lib):
    from libstokes_gb300 import MIXED, System, abi
    rng = np.random.default_rng(1)
    box = (400.0, 40.0, 40.0)
    s = System(0, _positions(4096, box, rng), box)
    s.set_precision(MIXED)
    y = np.zeros(s.n)
    d = y.ctypes.data_as(abi._dp)
    assert lib.stokes_gpu_atimes(s.sp, d, d) == abi.STOKES_GPU_ETOOBIG
    s.close()
