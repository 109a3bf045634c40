"""Interface history in and out (needs a B200): what is imported is exported again,
in both forms and at sizes that leave a block partly empty, and a channel resumed
from a state and a history takes the same steps as the one they came from."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available
from test_gpu_pairs import macros
from test_gpu_parity import params_for

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]


@pytest.mark.parametrize("precision", ["FP64", "FP32"])
@pytest.mark.parametrize("grid", [(4, 4, 5, 4, 2, None), (9, 5, 7, 5, 2, "RSLIP"), (16, 16, 7, 6, 3, "PSLIP"),
                                  (65, 5, 6, 4, 2, None)], ids=lambda g: "x".join(str(v) for v in g[:5]))
def test_history_round_trip(pkg, grid, precision):
    p = params_for(pkg, macros(*grid), "const")
    p.precision = getattr(pkg, precision)
    with pkg.Channel(p) as a, pkg.Channel(p) as b:
        rng = np.random.default_rng(1)
        shape = a.export_history().shape
        h = rng.standard_normal(shape).astype(np.float32).astype(np.float64) * 0.125
        if precision == "FP32":  # densities 1 + (a float); 24 bits below 1 fit a double's 53
            h[..., 0] += 1.0
        a.import_history(h)
        np.testing.assert_array_equal(a.export_history(), h)

        a.init_seeded(5)
        a.step(4)
        b.init_seeded(6)
        b.step(1)
        for level in range(3):
            b.import_state(level, a.export_state(level))
        b.import_history(a.export_history())
        a.step(3)
        b.step(3)
        for level in range(3):
            np.testing.assert_array_equal(a.export_state(level), b.export_state(level))
        np.testing.assert_array_equal(a.export_history(), b.export_history())
