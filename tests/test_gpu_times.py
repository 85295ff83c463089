"""cpu1, cpu2 and cpu3 of a drop-in product (include/stokes_abi.h): the device
time of the whole product, of its real part and of the rest, cpu1 = cpu2 + cpu3,
for every call: a product launched directly, the one recorded into a graph and
its replays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("version,n", [(0, 64), (1, 129), (2, 300)])
def test_phase_times_of_fp64_products(lib, version, n):
    from libstokes_gb300 import System
    from libstokes_gb300.workloads import rsa_positions
    pos, side = rsa_positions(n, 0.2, seed=5)
    s = System(version, pos, (side,) * 3)
    x = np.random.default_rng(6).standard_normal(s.n)
    for call in range(8):
        s.atimes(x)
        total, part, rest = s.s.cpu1, s.s.cpu2, s.s.cpu3
        # the real part runs inside the product's span
        assert 0.0 < part <= total, (call, total, part)
        assert rest >= 0.0 and abs(part + rest - total) <= 1e-6 * total, (call, total, part, rest)
    s.close()


def test_replays_measure_their_own_real_part(lib):
    """The same vectors and box, so one recorded graph; the spheres on a
    lattice over the box, then the lattice shrunk to a quarter of its width.
    The pairs evaluated in FP64 lie within 5.5 / xi = 0.46 box widths: 40% of all
    pairs, then all of them (0.43 at most), so the real part takes more than 1.5
    times as long (it is bound by them; 2.5 times if by nothing else)."""
    from libstokes_gb300 import System
    n, side = 1000, 110.0
    g = np.arange(10) + 0.5
    pos = np.stack(np.meshgrid(g, g, g, indexing="ij"), -1).reshape(-1, 3) * (side / 10)
    s = System(2, pos, (side,) * 3)
    x = np.random.default_rng(8).standard_normal(s.n)

    def real():
        for _ in range(4):
            s.atimes(x)
        return s.s.cpu2

    wide = real()
    s.set_pos(0.25 * pos)
    narrow = real()
    assert narrow > 1.5 * wide, (wide, narrow)
    s.close()
