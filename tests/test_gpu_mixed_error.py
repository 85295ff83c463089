"""Error of mixed products of some hundred unequal spheres against FP64: no
larger than that of the FP32 sums at the split before the tensor-core path, as
measured on these inputs (mean of five systems), plus 5% for the choice of five."""
import numpy as np
import pytest

from conftest import rel_l2

pytestmark = pytest.mark.gpu


def _mean_error(version, n, phi):
    from libstokes_gb300 import MIXED, System
    err = []
    for seed in range(5):
        rng = np.random.default_rng(seed)
        side = (n * 4.19 / phi) ** (1 / 3)
        m = int(round(n ** (1 / 3)))
        m += m ** 3 < n
        g = np.stack(np.meshgrid(*(np.arange(m),) * 3, indexing="ij"), -1).reshape(-1, 3)
        cell = side / m
        pos = (g[rng.permutation(len(g))[:n]] + 0.5) * cell
        pos += rng.uniform(-0.4, 0.4, pos.shape) * max(cell - 2.0, 0.0)
        s = System(version, pos, (side,) * 3)
        s.set_radius(rng.uniform(0.6, 1.0, n))
        x = rng.standard_normal(s.n)
        ref = s.atimes(x)
        s.set_precision(MIXED)
        err.append(rel_l2(s.atimes(x), ref))
        s.close()
    return float(np.mean(err))


@pytest.mark.parametrize("version,n,phi,before", [
    (0, 600, 0.05, 1.529e-7), (0, 600, 0.25, 1.959e-7), (1, 600, 0.05, 1.429e-7),
    (0, 100, 0.25, 1.428e-7), (0, 300, 0.05, 1.239e-7), (1, 300, 0.05, 1.155e-7),
    (1, 600, 0.25, 2.023e-7), (2, 300, 0.05, 1.164e-7), (2, 300, 0.25, 1.930e-7)])
def test_error_of_unequal_spheres(lib, version, n, phi, before):
    assert _mean_error(version, n, phi) <= 1.05 * before
