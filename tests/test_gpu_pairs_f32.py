"""The FP32 form's two-substep passes where the small grids of test_gpu_pairs.py do not
reach (needs a B200): their wall shear, the sizes at which they are taken by default,
and the mass over hundreds of substeps on a full GPU."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available
from test_gpu_pairs import macros
from test_gpu_parity import params_for

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]

STRESS = slice(5, 8)  # stup, stdown, stress


def run(pkg, p, precision, pairs, steps, states=True):
    p.precision = getattr(pkg, precision)
    with pkg.Channel(p) as ch:
        ch.set_fine_pairs(pairs)
        ch.init_seeded(42, 0.05, 0.005)
        log = ch.step(steps)
        mu = (2.0 / ch.geom.omega_f - 1.0) / 6.0
        return log, mu, [ch.export_state(l) for l in range(3)] if states else None


def assert_wall_shear(a, b, mu):
    """A wall stress is mu times the density times plane means of u, weighted 2, 3 and 1.
    The first row is of the seeded state, the same in both: u is off by the rounding of
    its sums of deviations of at most 0.06, below 3e-8 a node, the weighted means by six
    times that.  In the others populations may differ by 5e-7, u by ten times that."""
    np.testing.assert_allclose(a[0, STRESS], b[0, STRESS], rtol=0, atol=mu * 1e-6)
    np.testing.assert_allclose(a[1:, STRESS], b[1:, STRESS], rtol=0, atol=mu * 3.5e-5)


GRIDS = [(31, 60, 5, 16, 2, "PSLIP"), (33, 7, 6, 9, 2, "PSLIP"), (8, 90, 6, 16, 2, "RSLIP"),
         (34, 9, 7, 8, 4, "RSLIP"), (64, 40, 6, 8, 4, "PSLIP"), (10, 5, 7, 6, 3, "PSLIP")]


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(str(v) for v in g[:5]))
def test_wall_shear_of_pairs(pkg, grid):
    p = params_for(pkg, macros(*grid), "const")
    pair, mu, _ = run(pkg, p, "FP32", 1, 5, states=False)
    single, _, _ = run(pkg, p, "FP32", 0, 5, states=False)
    double, _, _ = run(pkg, p, "FP64", 0, 5, states=False)
    assert_wall_shear(pair, single, mu)
    # against the FP64 form: the same seeded state but for one rounding of a deviation
    np.testing.assert_allclose(pair[0, STRESS], double[0, STRESS], rtol=0, atol=mu * 1e-6)


def test_pairs_by_default_on_a_large_channel(pkg):
    """195 MB of fine state at ratio 4: the default takes pairs, two passes a step; the
    single substeps' state and log, and the same bits when run again."""
    p = params_for(pkg, macros(100, 80, 7, 10, 4, "RSLIP"), "const")
    p.precision = pkg.FP32
    passes = {}
    for mode in (-1, 0):
        with pkg.Channel(p) as ch:
            ch.set_fine_pairs(mode)
            ch.init_seeded(42)
            ch.set_profiling(True)
            ch.step(2)
            passes[mode] = ch.kernel_times()["fine"][1] / 2
    assert passes == {-1: 2, 0: 4}
    pair, mu, a = run(pkg, p, "FP32", -1, 5)
    again, _, c = run(pkg, p, "FP32", -1, 5)
    single, _, b = run(pkg, p, "FP32", 0, 5)
    np.testing.assert_array_equal(pair, again)
    for x, y, z in zip(a, b, c):
        np.testing.assert_allclose(x, y, rtol=0, atol=5e-7)
        np.testing.assert_array_equal(x, z)
    np.testing.assert_allclose(pair[:, 2:5], single[:, 2:5], rtol=1e-5)
    assert_wall_shear(pair, single, mu)


@pytest.mark.parametrize("grid", [(128, 96, 30, 16, 2, "RSLIP"), (64, 48, 12, 16, 4, None)],
                         ids=lambda g: "x".join(str(v) for v in g[:5]))
def test_mass_of_pairs_over_400_substeps(pkg, grid):
    """A collision rounds each population of a node a few times, some 4e-9 of mass in
    all; without a bias the mean over 1.5e6 nodes and 400 substeps stays below 1e-10.  A
    bias of one part in 2^24 of u^2 = 2.5e-3 a substep would make 6e-8."""
    p = params_for(pkg, macros(*grid), "const")
    steps = 400 // grid[4]
    pair, _, _ = run(pkg, p, "FP32", 1, steps, states=False)
    single, _, _ = run(pkg, p, "FP32", 0, steps, states=False)
    np.testing.assert_allclose(pair[:, 3], single[:, 3], rtol=0, atol=2e-8)
