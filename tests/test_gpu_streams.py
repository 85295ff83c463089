"""Products queued on a caller's stream, with changes of the system between
them and no synchronisation: each product uses the tables of its own call.  New
tables wait for the products of their own system only."""
import ctypes as C

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def _system(version, n, precision):
    from libstokes_gb300 import System
    from libstokes_gb300.workloads import rsa_positions
    pos, side = rsa_positions(n, 0.1, seed=n + version)
    s = System(version, pos, (side,) * 3)
    s.set_precision(precision)
    return s, pos, side


def _change(lib, s, side, kind, k):
    """State k of the system."""
    if kind == "box":
        b = side * (1.0, 1.06, 1.13)[k]
        lib.stokes_set_l(s.sp, b, b, b)
        lib.stokes_set_xi(s.sp, lib.xi_by_tratio(s.sp, 1.0), 1e-12)
    elif kind == "shear":
        s.set_misc(0.0, 1, (0.1, 0.37, 0.73)[k] * side)
    else:
        s.set_misc((0.0, 1.02, 0.0)[k])


# F N = 300: the clamp (rmin) turns the tensor-core path on and off; N = 64 has
# lattice images at the split of small systems, N = 600 takes the tensor cores
@pytest.mark.parametrize("precision", [0, 1])
@pytest.mark.parametrize("version,n,kind", [(0, 64, "box"), (0, 64, "shear"), (0, 300, "box"),
                                            (0, 300, "rmin"), (1, 300, "shear"), (0, 600, "box"),
                                            (2, 300, "box"), (2, 300, "shear")])
def test_changes_between_queued_products(lib, precision, version, n, kind):
    import torch
    from libstokes_gb300 import check
    s, pos, side = _system(version, n, precision)
    rng = np.random.default_rng(5)
    x = torch.from_numpy(rng.standard_normal(s.n)).cuda()
    p = torch.from_numpy(pos).cuda()
    st = torch.cuda.Stream()
    order = [0, 1, 0, 2, 1, 0]

    def product(out):
        check(lib.stokes_gpu_atimes_dev(s.sp, p.data_ptr(), x.data_ptr(), out.data_ptr(),
                                        C.c_void_p(st.cuda_stream)))

    alone = []
    for k in order:
        _change(lib, s, side, kind, k)
        y = torch.zeros_like(x)
        torch.cuda.synchronize()
        product(y)
        torch.cuda.synchronize()
        alone.append(y)
    queued = [torch.zeros_like(x) for _ in order]
    torch.cuda.synchronize()
    with torch.cuda.stream(st):
        torch.cuda._sleep(20_000_000)            # about 10 ms ahead of the first product
    for k, y in zip(order, queued):
        _change(lib, s, side, kind, k)
        product(y)
    torch.cuda.synchronize()
    for k, (a, b) in enumerate(zip(alone, queued)):
        assert torch.equal(a, b), (k, order[k])
    assert not torch.equal(alone[0], alone[1])
    s.close()


@pytest.mark.parametrize("call", ["fp64", "mixed", "matrix"])
def test_new_tables_leave_other_streams_alone(lib, call):
    """A change of box while a long kernel of somebody else's runs: the call
    returns before that kernel ends."""
    import torch
    s, pos, side = _system(0, 600, int(call == "mixed"))
    x = np.random.default_rng(9).standard_normal(s.n)

    def change_and_call(k):
        # (from the largest box down: the buffers have their size)
        b = side * (1.0 - 1e-4 * k)
        lib.stokes_set_l(s.sp, b, b, b)
        lib.stokes_set_xi(s.sp, lib.xi_by_tratio(s.sp, 1.0), 1e-12)
        return s.matrix() if call == "matrix" else s.atimes(x)

    for k in range(4):
        change_and_call(k)
    other = torch.cuda.Stream()
    torch.cuda.synchronize()
    with torch.cuda.stream(other):
        torch.cuda._sleep(1_000_000_000)         # half a second
    change_and_call(4)
    running = not other.query()
    torch.cuda.synchronize()
    assert running
    s.close()
