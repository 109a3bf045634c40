"""Statistics sampling observes a run and does not change it (needs a B200): a
channel that samples every few steps takes the steps of one that never does, bit for
bit, whether its fine substeps are taken one or two at a time, and the statistics do
not depend on that."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available
from test_gpu_pairs import macros
from test_gpu_parity import params_for

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]

GRIDS = [(33, 7, 6, 9, 2, "PSLIP"), (16, 60, 7, 8, 2, "RSLIP"), (12, 10, 7, 6, 3, "PSLIP"),
         (34, 9, 7, 8, 4, "RSLIP"), (9, 6, 7, 5, 3, None)]


@pytest.mark.parametrize("precision", ["FP64", "FP32"])
@pytest.mark.parametrize("mode", ["const", "cfr"])
@pytest.mark.parametrize("pairs", [0, 1])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(str(v) for v in g[:5]))
def test_sampling_leaves_the_run_alone(pkg, grid, pairs, mode, precision):
    p = params_for(pkg, macros(*grid), mode)
    p.precision = getattr(pkg, precision)
    out = []
    for every in (0, 3, 1):
        with pkg.Channel(p) as ch:
            ch.set_fine_pairs(pairs)
            ch.set_sampling(every)
            ch.init_seeded(9)
            log = ch.step(10)
            out.append([ch.export_state(l) for l in range(3)] + [ch.export_history(), log])
            assert ch.stats()[1] == (0 if every == 0 else -(-10 // every))
    for other in out[1:]:
        for a, b in zip(out[0], other):
            np.testing.assert_array_equal(a, b)


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(str(v) for v in g[:5]))
def test_statistics_of_pairs_are_those_of_single_substeps(pkg, grid):
    """Constant force, 64 bits: the same states, and samples that differ by the order of
    their sums: at most some twelve roundings of a density of 1, 3e-15."""
    p = params_for(pkg, macros(*grid), "const")
    out = []
    for pairs in (0, 1):
        with pkg.Channel(p) as ch:
            ch.set_fine_pairs(pairs)
            ch.set_sampling(2)
            ch.init_seeded(9)
            ch.step(9)
            out.append(ch.stats()[0])
    np.testing.assert_allclose(*out, rtol=0, atol=1e-14)


@pytest.mark.parametrize("every", [7, 20])
@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_sampled_groups_match_unsampled_single_steps(pkg, precision, every):
    """Pairs at ratio 2, runs of sampled and plain steps: groups issued as graphs against
    steps issued one by one without sampling."""
    p = params_for(pkg, macros(16, 6, 7, 6, 2, "PSLIP"), "cfr")
    p.precision = getattr(pkg, precision)
    out = []
    for sampled in (False, True):
        with pkg.Channel(p) as ch:
            ch.set_fine_pairs(1)
            ch.init_seeded(4)
            if sampled:
                ch.set_sampling(every)
                log = np.concatenate([ch.step(n) for n in (301, 1, 298)])
            else:
                log = np.concatenate([ch.step(1) for _ in range(600)])
            out.append([ch.export_state(l) for l in range(3)] + [ch.export_history(), log])
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
