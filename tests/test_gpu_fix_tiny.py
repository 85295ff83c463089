"""FP64 products of equal spheres in boxes of about one radius, where the tuned
split is so short-ranged (xi > 5.2) that the pairs summed in FP32 would begin
below the radial table (s = r^2 < 1): wherever the table does not reach, pairs
take the closed forms.  No such system is physical; libstokes computes it.

Tolerance: the self, real and reciprocal parts grow with xi against their sum
(self: a 1 - xi / sqrt(pi) (6 - 40/3 xi^2), m 0.9 - xi^3 / sqrt(pi) (12 - 30.24
xi^2)), and each carries a few roundings of its largest term.  64 ulp of the
largest self coefficient on x, plus the cutoff rule's 1e-12 on that scale."""
import math
import os
import subprocess
import sys

import numpy as np
import pytest

from conftest import ROOT, rel_l2

pytestmark = pytest.mark.gpu


def _self(version, xi):
    f = xi / math.sqrt(math.pi)
    c = [abs(1.0 - f * (6.0 - 40.0 / 3.0 * xi * xi)), abs(0.75 - 10.0 * f * xi * xi),
         abs(0.9 - f * xi * xi * (12.0 - 30.24 * xi * xi))]
    return max(c[:version + 1])


def _tolerance(version, xi, x, y):
    scale = _self(version, xi) * np.linalg.norm(x) / np.linalg.norm(y)
    return max(1e-12, (64 * 2.0 ** -53 + 1e-12) * scale)


@pytest.mark.parametrize("version", [0, 1, 2])
@pytest.mark.parametrize("n,side", [(1, 1.05), (3, 1.05), (7, 1.05), (40, 1.1), (5, 1.2),
                                    (33, 1.6)])
def test_boxes_of_about_one_radius(lib, version, n, side):
    from libstokes_gb300 import System
    from oracle.oracle import Oracle
    rng = np.random.default_rng(10 * n + version)
    pos = rng.uniform(0.0, side, (n, 3))
    x = rng.standard_normal((3, 6, 11)[version] * n)
    s = System(version, pos, (side,) * 3)
    y = s.atimes(x)
    s.close()
    o = Oracle(version, pos, (side,) * 3)
    o.set_split(o.xi_by_tratio(1.0), 1e-12)
    yo = o.atimes(x)
    assert rel_l2(y, yo) < _tolerance(version, 6.0 / side, x, yo)


def test_short_ranged_split_with_overlapping_pairs(lib, tmp_path):
    """LIBSTOKES_GB300_FP64_ETA reaches such a split in an ordinary box (read
    once per process, hence a process of its own)."""
    from oracle.oracle import Oracle
    n, side, eta = 60, 6.5, 36.0
    rng = np.random.default_rng(3)
    pos = rng.uniform(0.0, side, (n, 3))
    x = rng.standard_normal(3 * n)
    out = tmp_path / "y.npy"
    code = ("import sys, numpy as np; sys.path.insert(0, %r)\n"
            "import libstokes_gb300 as L\n"
            "rng = np.random.default_rng(3)\n"
            "pos = rng.uniform(0.0, %r, (%d, 3)); x = rng.standard_normal(3 * %d)\n"
            "s = L.System(0, pos, (%r,) * 3); np.save(%r, s.atimes(x))\n"
            % (ROOT, side, n, n, side, str(out)))
    subprocess.run([sys.executable, "-c", code], check=True, timeout=300,
                   env=dict(os.environ, LIBSTOKES_GB300_FP64_ETA=str(eta)))
    o = Oracle(0, pos, (side,) * 3)
    o.set_split(o.xi_by_tratio(1.0), 1e-12)
    yo = o.atimes(x)
    assert rel_l2(np.load(out), yo) < _tolerance(0, eta / side, x, yo)
