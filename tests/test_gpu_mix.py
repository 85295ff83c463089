"""Mixed product of equal spheres with the reciprocal sum in 24-bit fixed point
on the tensor cores, at the edges of its tiles and ranges, against the FP64
product of the same inputs.

Tolerance 1e-6 (relative L2), the mixed-path bar: operands are rounded at 2^-25
of the largest entry of their block of 128, and sums of up to 128 products are
exact, so rounding stays within a few 2^-24 of the sums, as in FP32."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu
TOL = 1e-6


@pytest.fixture(autouse=True, params=["tc", ""])
def path(request, monkeypatch):
    """The GEMMs at every size, and what the library takes by itself (small
    systems: the SIMT kernels at a split with lattice images)."""
    if request.param:
        monkeypatch.setenv("LIBSTOKES_GB300_KSPACE", request.param)
    else:
        monkeypatch.delenv("LIBSTOKES_GB300_KSPACE", raising=False)


def _positions(n, box, rng):
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*(np.arange(m),) * 3, indexing="ij"), -1).reshape(-1, 3)
    cell = np.asarray(box) / m
    p = (g[rng.permutation(len(g))[:n]] + 0.5) * cell
    return p + rng.uniform(-0.45, 0.45, p.shape) * np.maximum(cell - 2.0, 0.0)


def _both(version, pos, box, x, **misc):
    from libstokes_gb300 import FP64, MIXED, System
    out = []
    for prec in (FP64, MIXED):
        s = System(version, pos, box)
        if misc:
            s.set_misc(0.0, misc["mode"], misc["shift"])
        s.set_precision(prec)
        y = [s.atimes(x) for _ in range(3)]     # direct, recorded, replayed
        s.close()
        assert np.array_equal(y[0], y[1], equal_nan=True)
        assert np.array_equal(y[0], y[2], equal_nan=True)
        out.append(y[0])
    return out


# particles around the 64 and 128 wide tiles and their pairs
@pytest.mark.parametrize("version", [0, 1, 2])
@pytest.mark.parametrize("n,side", [(2, 9.0), (63, 14.0), (64, 16.0), (65, 15.0), (127, 18.0),
                                    (128, 17.0), (129, 19.5), (257, 22.0), (513, 30.0)])
def test_tile_edges(version, n, side):
    rng = np.random.default_rng(40 + n + version)
    box = (side, side, side)
    y64, ymx = _both(version, _positions(n, box, rng), box,
                     rng.standard_normal((3, 6, 11)[version] * n))
    assert rel_l2(ymx, y64) < TOL


# few functions on x and many on y or z, and the reverse: row sets and column
# tiles with remainders
@pytest.mark.parametrize("version", [0, 1, 2])
@pytest.mark.parametrize("box", [(8.0, 24.0, 15.0), (34.0, 9.0, 12.0), (13.0, 11.0, 40.0)])
def test_box_shapes(version, box):
    rng = np.random.default_rng(7 + version)
    pos = _positions(90, box, rng) + rng.integers(-3, 4, (90, 3)) * np.asarray(box)
    y64, ymx = _both(version, pos, box, rng.standard_normal((3, 6, 11)[version] * 90))
    assert rel_l2(ymx, y64) < TOL


@pytest.mark.parametrize("mode,shift", [(1, 2.7), (2, -5.1)])
def test_sheared_box(mode, shift):
    rng = np.random.default_rng(11)
    box = (18.0, 20.0, 22.0)
    y64, ymx = _both(2, _positions(150, box, rng), box, rng.standard_normal(11 * 150),
                     mode=mode, shift=shift)
    assert rel_l2(ymx, y64) < TOL


@pytest.mark.parametrize("scale", [1e-20, 1e20])
def test_scales(scale):
    """Each unit follows its block: the same digits at any magnitude."""
    rng = np.random.default_rng(12)
    box = (19.0, 19.0, 19.0)
    y64, ymx = _both(2, _positions(140, box, rng), box, scale * rng.standard_normal(11 * 140))
    assert rel_l2(ymx / scale, y64 / scale) < TOL


def test_small_block_keeps_its_digits():
    """The torques of one block of 128 particles a millionth of the others:
    rounding is per block and per component, so the result of the small block's
    torques alone still carries FP32's digits."""
    rng = np.random.default_rng(13)
    n, box = 256, (24.0, 24.0, 24.0)
    x = np.zeros((n, 6))
    x[:, :3] = 1e-6 * rng.standard_normal((n, 3))
    x[:128, 3:] = 1e-6 * rng.standard_normal((128, 3))
    y64, ymx = _both(1, _positions(n, box, rng), box, x.ravel())
    assert rel_l2(ymx, y64) < TOL


@pytest.mark.parametrize("bad", [np.nan, np.inf, -np.inf])
def test_non_finite(bad):
    rng = np.random.default_rng(14)
    box = (17.0, 17.0, 17.0)
    x = rng.standard_normal((130, 3))
    x[129, 1] = bad
    y64, ymx = _both(0, _positions(130, box, rng), box, x.ravel())
    assert np.isnan(ymx).all() == np.isnan(y64).all()
    assert not np.isfinite(ymx).any()


@pytest.mark.parametrize("version,n,side", [(0, 2, 9.0), (1, 2, 9.0), (1, 64, 14.0), (2, 129, 19.5),
                                            (0, 513, 30.0), (2, 900, 36.0)])
def test_new_inputs_every_time(version, n, side):
    """The kernels of a product overlap their starts: each has to read what the
    ones before it wrote in this product, not what an earlier one left."""
    from libstokes_gb300 import MIXED, System
    rng = np.random.default_rng(70 + n)
    box = (side, side, side)
    s, f = (System(version, _positions(n, box, rng), box) for _ in range(2))
    s.set_precision(MIXED)
    for _ in range(8):
        pos, x = _positions(n, box, rng), rng.standard_normal((3, 6, 11)[version] * n)
        s.set_pos(pos)
        f.set_pos(pos)
        assert rel_l2(s.atimes(x), f.atimes(x, notbl=True)) < TOL
    s.close()
    f.close()


# unequal radii: columns by power of the radius, around the tiles
@pytest.mark.parametrize("version", [0, 1, 2])
@pytest.mark.parametrize("n,side", [(63, 16.0), (129, 19.5), (513, 31.0)])
def test_unequal_radii(version, n, side):
    from libstokes_gb300 import MIXED, System
    rng = np.random.default_rng(90 + n + version)
    box = (side, 0.9 * side, 1.1 * side)
    radius = rng.uniform(0.4, 1.0, n)
    pos = _positions(n, box, rng)
    s, f = System(version, pos, box), System(version, pos, box)
    s.set_radius(radius)
    f.set_radius(radius)
    s.set_precision(MIXED)
    for _ in range(4):
        x = rng.standard_normal((3, 6, 11)[version] * n)
        assert rel_l2(s.atimes(x), f.atimes(x)) < TOL
    s.close()
    f.close()


@pytest.mark.parametrize("version,equal", [(0, True), (2, True), (1, False)])
def test_cells(version, equal, monkeypatch):
    """The cell list of the real space (here forced by a high split), whose
    sources, their vectors and radii come in cell order."""
    from libstokes_gb300 import MIXED, System
    monkeypatch.setenv("LIBSTOKES_GB300_MIXED_ETA", "17")
    rng = np.random.default_rng(95)
    n, box = 701, (38.0, 42.0, 40.0)
    pos, radius = _positions(n, box, rng), rng.uniform(0.5, 1.0, n)
    s, f = System(version, pos, box), System(version, pos, box)
    if not equal:
        s.set_radius(radius)
        f.set_radius(radius)
    s.set_precision(MIXED)
    for _ in range(3):
        x = rng.standard_normal((3, 6, 11)[version] * n)
        assert rel_l2(s.atimes(x), f.atimes(x)) < TOL
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
@pytest.mark.parametrize("n,side", [(32, 8.9), (112, 11.1), (256, 18.0), (530, 24.0)])
def test_lattice_positions(version, n, side):
    """Many pairs exactly half a box apart."""
    from libstokes_gb300 import MIXED, System
    rng = np.random.default_rng(n + version)
    box = (side, side, side)
    s = System(version, _fcc(n, side, rng), box)
    x = rng.standard_normal((3, 6, 11)[version] * n)
    y = s.atimes(x, notbl=True)
    s.set_precision(MIXED)
    assert rel_l2(s.atimes(x), y) < TOL
    s.close()
