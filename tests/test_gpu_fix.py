"""FP64 products of equal spheres with the reciprocal sum in fixed point on the
tensor cores: sizes at the edges of its tiles, ranges of the inputs, boxes,
non-finite inputs and the bounded waits, against the CPU oracle.

Tolerance 1e-12 (relative L2) as for every FP64 product: the fixed-point
operands carry 55 bits below the largest magnitude of their kind, so the sums
are off by about 2^-56 sqrt(terms), well below the truncation of the Ewald
sums (1e-12 in the cutoff rule)."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _positions(n, box, rng):
    """n points in the box with a minimum distance of 2 where n allows it."""
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*(np.arange(m),) * 3, indexing="ij"), -1).reshape(-1, 3)
    cell = np.asarray(box) / m
    p = (g[rng.permutation(len(g))[:n]] + 0.5) * cell
    return p + rng.uniform(-0.45, 0.45, p.shape) * np.maximum(cell - 2.0, 0.0)


def _both(version, pos, box, x):
    from libstokes_gb300 import System
    from oracle.oracle import Oracle
    s = System(version, pos, box)
    y = [s.atimes(x) for _ in range(3)]         # direct, recorded, replayed
    s.close()
    assert np.array_equal(y[0], y[1]) and np.array_equal(y[0], y[2])
    o = Oracle(version, pos, box)
    o.set_split(o.xi_by_tratio(1.0), 1e-12)
    return y[0], o.atimes(x)


# particles around the 32, 64 and 128 wide tiles; boxes from a few radii up
@pytest.mark.parametrize("version", [0, 1, 2])
@pytest.mark.parametrize("n,side", [(1, 7.0), (2, 9.0), (31, 10.5), (33, 13.0), (64, 14.0),
                                    (65, 17.0), (127, 16.0), (128, 22.0), (129, 17.5),
                                    (161, 19.0)])
def test_tile_edges(lib, version, n, side):
    rng = np.random.default_rng(100 * n + version)
    pos = _positions(n, (side,) * 3, rng)
    y, yo = _both(version, pos, (side,) * 3, rng.standard_normal((3, 6, 11)[version] * n))
    assert rel_l2(y, yo) < 1e-12


@pytest.mark.parametrize("version", [0, 2])
@pytest.mark.parametrize("box", [(14.0, 19.0, 27.0), (30.0, 12.0, 12.0), (11.0, 13.0, 31.0)])
def test_boxes_and_unwrapped_positions(lib, version, box):
    rng = np.random.default_rng(7)
    n = 70
    pos = _positions(n, box, rng)
    x = rng.standard_normal((3, 11)[version // 2] * n)
    y, yo = _both(version, pos, box, x)
    assert rel_l2(y, yo) < 1e-12
    # whole-box shifts of single particles leave the periodic sum as it is
    from libstokes_gb300 import System
    s = System(version, pos + np.asarray(box) * rng.integers(-3, 4, (n, 3)), box)
    assert rel_l2(s.atimes(x), yo) < 1e-12
    s.close()


@pytest.mark.parametrize("scale", [1e-250, 1e-30, 1.0, 1e30, 1e250])
def test_input_ranges(lib, scale):
    """Forces, torques and stresslets of very different sizes, some zero."""
    rng = np.random.default_rng(11)
    n, box = 90, (18.0,) * 3
    pos = _positions(n, box, rng)
    x = rng.standard_normal((n, 11))
    x[:, 3:6] *= 1e-6
    x[:, 6:] *= 1e4
    x[:, 2] = 0.0
    x[::3] = 0.0
    y, yo = _both(2, pos, box, x.ravel())
    ys, _ = _both(2, pos, box, x.ravel() * scale)
    assert rel_l2(y, yo) < 1e-12
    assert rel_l2(ys / scale, yo) < 1e-12
    z, _ = _both(2, pos, box, np.zeros(11 * n))
    assert np.array_equal(z, np.zeros(11 * n))


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite_vectors(lib, bad):
    """A torque T_y that is not finite reaches every velocity component it
    couples to, of every particle; U_y holds no T_y (U = T x e) and keeps its
    value; the next product is clean."""
    from libstokes_gb300 import System
    rng = np.random.default_rng(13)
    n, box = 40, (14.0,) * 3
    s = System(1, _positions(n, box, rng), box)
    x = rng.standard_normal(6 * n)
    y = s.atimes(x)
    xb = x.copy()
    xb[6 * 17 + 4] = bad
    yb = s.atimes(xb).reshape(n, 6)
    assert not np.isfinite(yb[:, [0, 2, 3, 4, 5]]).any()
    assert rel_l2(yb[:, 1], y.reshape(n, 6)[:, 1]) < 1e-12
    assert np.array_equal(s.atimes(x), y)
    s.close()


def test_device_positions_that_are_not_finite(lib):
    """Positions in device memory are not checked on the host: a non-finite
    one makes every velocity NaN."""
    import torch
    from libstokes_gb300 import System, check
    rng = np.random.default_rng(17)
    n, box = 40, (14.0,) * 3
    pos = _positions(n, box, rng)
    s = System(0, pos, box)
    x = torch.from_numpy(rng.standard_normal(3 * n)).cuda()
    y = torch.zeros(3 * n, dtype=torch.float64, device="cuda")
    pos[5, 1] = np.nan
    p = torch.from_numpy(pos).cuda()
    check(s.lib.stokes_gpu_atimes_dev(s.sp, p.data_ptr(), x.data_ptr(), y.data_ptr(), None))
    assert torch.isnan(y).all()
    s.close()


def test_changes_between_products(lib):
    """Positions, version-independent split and box changes reach the tables."""
    from libstokes_gb300 import System
    from oracle.oracle import Oracle
    rng = np.random.default_rng(19)
    n = 60
    pos = _positions(n, (15.0,) * 3, rng)
    s = System(2, pos, (15.0,) * 3)
    x = rng.standard_normal(11 * n)
    s.atimes(x)
    s.set_pos(pos * 1.2)
    s.lib.stokes_set_l(s.sp, 18.0, 18.0, 18.0)
    s.lib.stokes_set_xi(s.sp, s.lib.xi_by_tratio(s.sp, 1.0), 1e-12)
    o = Oracle(2, pos * 1.2, (18.0,) * 3)
    o.set_split(o.xi_by_tratio(1.0), 1e-12)
    assert rel_l2(s.atimes(x), o.atimes(x)) < 1e-12
    s.close()


def test_bounded_wait_is_reported(lib):
    from libstokes_gb300 import GPUError, System
    rng = np.random.default_rng(23)
    n, box = 50, (15.0,) * 3
    s = System(0, _positions(n, box, rng), box)
    x = rng.standard_normal(3 * n)
    y = s.atimes(x)
    assert lib.stokes_gpu_test_stall_waits(50, 0) == 0
    try:
        with pytest.raises(GPUError):
            s.atimes_checked(x)
    finally:
        lib.stokes_gpu_test_stall_waits(0, 0)
    assert np.array_equal(s.atimes(x), y)
    s.close()


@pytest.mark.parametrize("version,n,side", [(0, 2, 9.0), (1, 2, 9.0), (1, 64, 14.0), (2, 129, 19.5),
                                            (0, 513, 30.0), (2, 300, 26.0)])
def test_new_inputs_every_time(version, n, side):
    """The kernels of a product overlap their starts: each has to read what the
    ones before it wrote in this product, not what an earlier one left."""
    from libstokes_gb300 import System
    rng = np.random.default_rng(70 + n)
    box = (side, side, side)
    s, f = (System(version, _positions(n, box, rng), box) for _ in range(2))
    for _ in range(6):
        pos, x = _positions(n, box, rng), rng.standard_normal((3, 6, 11)[version] * n)
        s.set_pos(pos)
        f.set_pos(pos)
        assert rel_l2(s.atimes(x), f.atimes(x, notbl=True)) < 1e-12
    s.close()
    f.close()


def _fcc(n, side, rng):
    m = 1
    while 4 * m ** 3 < n:
        m += 1
    base = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]])
    g = np.stack(np.meshgrid(*(np.arange(m),) * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    sites = ((g + base) * side / m).reshape(-1, 3)
    return sites[rng.permutation(len(sites))[:n]] + rng.uniform(0, side, 3)


@pytest.mark.parametrize("version", [0, 1, 2])
@pytest.mark.parametrize("n,side", [(32, 8.9), (112, 11.1), (112, 13.0), (120, 11.2), (256, 18.0)])
def test_lattice_positions(lib, version, n, side):
    """Spheres on a lattice: many pairs exactly half a box apart, where both
    images count and rounding decides which one is the nearest."""
    from libstokes_gb300 import System
    rng = np.random.default_rng(n + version)
    box = (side, side, side)
    pos = _fcc(n, side, rng)
    s = System(version, pos, box)
    x = rng.standard_normal((3, 6, 11)[version] * n)
    assert rel_l2(s.atimes(x), s.atimes(x, notbl=True)) < 1e-12
    s.close()
