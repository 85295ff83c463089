"""FP64 dense matrix of equal spheres with the reciprocal moments in fixed point
on the tensor cores: sizes at the edges of its 8 x 8 pair tiles and its chunks,
boxes, coincident and non-finite positions and the bounded waits.

Systems of fewer than 32 (F, FT) or 12 particles take the other builder.
Tolerance 1e-12 of the matrix norm, as for every FP64 builder; against the CPU
oracle where that is quick and against the FP64 builder over the cube list, which
keeps libstokes' split, for the larger ones."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _positions(n, box, rng):
    m = int(np.ceil(n ** (1 / 3)))
    g = np.stack(np.meshgrid(*(np.arange(m),) * 3, indexing="ij"), -1).reshape(-1, 3)
    cell = np.asarray(box) / m
    p = (g[rng.permutation(len(g))[:n]] + 0.5) * cell
    return p + rng.uniform(-0.45, 0.45, p.shape) * np.maximum(cell - 2.0, 0.0)


@pytest.mark.parametrize("version", [0, 1, 2])
@pytest.mark.parametrize("n,side", [(1, 8.0), (12, 9.0), (15, 10.0), (16, 11.0), (31, 12.0),
                                    (32, 13.0), (33, 12.0)])
def test_oracle(lib, version, n, side):
    from libstokes_gb300 import System
    from oracle.oracle import Oracle
    rng = np.random.default_rng(10 * n + version)
    box = (side, side, side)
    pos = _positions(n, box, rng)
    s = System(version, pos, box)
    o = Oracle(version, pos, box)
    o.set_split(o.xi_by_tratio(1.0), 1e-12)
    assert rel_l2(s.matrix(), o.matrix()) < 1e-12
    s.close()


# 201 particles: 351 tiles, two chunks; unequal sides
@pytest.mark.parametrize("version", [0, 1, 2])
@pytest.mark.parametrize("n,box", [(64, (17.0, 17.0, 17.0)), (45, (12.0, 22.0, 16.0)),
                                   (40, (26.0, 11.0, 13.0)), (201, (24.0, 27.0, 22.0))])
def test_cube_builder(lib, version, n, box):
    from libstokes_gb300 import System
    rng = np.random.default_rng(n + version)
    pos = _positions(n, box, rng)
    s = System(version, pos, box)
    m = s.matrix()
    assert rel_l2(m, s.matrix(notbl=True)) < 1e-12
    assert np.array_equal(m, s.matrix())
    # any periodic image of a particle does
    t = System(version, pos + rng.integers(-2, 3, (n, 3)) * np.asarray(box), box)
    assert rel_l2(t.matrix(), m) < 1e-12
    s.close()
    t.close()


@pytest.mark.parametrize("version", [0, 2])
def test_two_particles_at_one_place(lib, version):
    """libstokes leaves the zero separation out of the real space, so the
    result depends on its split; the builder's own split gives the same."""
    from libstokes_gb300 import System
    from oracle.oracle import Oracle
    rng = np.random.default_rng(5)
    box = (13.0, 13.0, 13.0)
    pos = _positions(40, box, rng)
    pos[6] = pos[2]
    s = System(version, pos, box)
    o = Oracle(version, pos, box)
    o.set_split(o.xi_by_tratio(1.0), 1e-12)
    assert rel_l2(s.matrix(), o.matrix()) < 1e-12
    s.close()


def test_position_that_is_not_finite(lib):
    """In device memory: the rows and columns of that particle are NaN."""
    import torch
    from libstokes_gb300 import System, check
    rng = np.random.default_rng(6)
    n, box = 35, (13.0, 13.0, 13.0)
    pos = _positions(n, box, rng)
    s = System(0, pos, box)
    ref = s.matrix()
    pos[5, 1] = np.nan
    p = torch.from_numpy(pos).cuda()
    m = torch.zeros(3 * n, 3 * n, dtype=torch.float64, device="cuda")
    check(s.lib.stokes_gpu_matrix_dev(s.sp, p.data_ptr(), m.data_ptr(), None))
    m = m.cpu().numpy()
    hit = np.zeros(3 * n, bool)
    hit[15:18] = True
    assert np.isnan(m[hit]).all() and np.isnan(m[:, hit]).all()
    assert np.array_equal(m[~hit][:, ~hit], ref[~hit][:, ~hit])
    s.close()


def test_bounded_waits(lib):
    from libstokes_gb300 import GPUError, System
    rng = np.random.default_rng(8)
    box = (14.0, 14.0, 14.0)
    s = System(1, _positions(40, box, rng), box)
    m = s.matrix()
    assert lib.stokes_gpu_test_stall_waits(50, 0) == 0
    try:
        with pytest.raises(GPUError):
            s.matrix()
    finally:
        lib.stokes_gpu_test_stall_waits(0, 0)
    assert np.array_equal(s.matrix(), m)
    s.close()


def test_count_of_reference_terms(lib):
    """The term count is that of the reference's split, also where the builder
    takes a split of its own."""
    import ctypes as C
    from libstokes_gb300 import System, check
    rng = np.random.default_rng(9)
    s = System(2, _positions(40, (14.0, 14.0, 14.0), rng), (14.0, 14.0, 14.0))
    counts = []
    for _ in range(2):
        p = C.c_longlong()
        check(lib.stokes_gpu_count_real_terms_dense(s.sp, C.byref(p)))
        counts.append(p.value)
        s.matrix()
    v = 4.0 / 3.0 * np.pi * s.s.rmax2 ** 1.5 / 14.0 ** 3
    assert counts[0] == counts[1] and 0.9 < counts[0] / (40 * 40 * v) < 1.1
    s.close()


def _fcc(n, side, rng):
    m = 1
    while 4 * m ** 3 < n:
        m += 1
    base = np.array([[0, 0, 0], [0, .5, .5], [.5, 0, .5], [.5, .5, 0]])
    g = np.stack(np.meshgrid(*(np.arange(m),) * 3, indexing="ij"), -1).reshape(-1, 1, 3)
    sites = ((g + base) * side / m).reshape(-1, 3)
    return sites[rng.permutation(len(sites))[:n]] + rng.uniform(0, side, 3)


@pytest.mark.parametrize("version", [0, 1, 2])
@pytest.mark.parametrize("n,side", [(32, 9.0), (112, 11.1), (112, 13.0), (120, 15.0)])
def test_lattice_positions(lib, version, n, side):
    """Many pairs exactly half a box apart."""
    from libstokes_gb300 import System
    rng = np.random.default_rng(n + version)
    s = System(version, _fcc(n, side, rng), (side, side, side))
    assert rel_l2(s.matrix(), s.matrix(notbl=True)) < 1e-12
    s.close()
