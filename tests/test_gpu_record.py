"""The plane-statistics record against its definition (needs a B200): two passes over
the exported state, every sum in the reference's order (statistics.c:48-300), on planes
of more nodes than the device sums at a time, in both forms, and with populations that
are not finite."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available
from test_gpu_pairs import macros
from test_gpu_parity import params_for

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]

EX = [0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, 1, -1, -1, 0, 0, 0, 0]
EY = [0, 0, 0, 1, -1, 0, 0, 1, 1, -1, -1, 0, 0, 0, 0, 1, 1, -1, -1]
EZ = [0, 0, 0, 0, 0, 1, -1, 0, 0, 0, 0, 1, -1, -1, 1, 1, -1, -1, 1]


def record(ch):
    """UAVG VAVG WAVG UTIN VTIN WTIN REYS DAVG DTIN of the exported state."""
    g = ch.geom
    out = np.zeros((9, g.nz_profile))

    def ordered(x):  # i outer, j inner, one add after another from zero
        return np.add.accumulate(np.concatenate([[0.0], x.ravel()]))[-1]

    levels = [(1, range(1, g.zdf), 0), (0, range(2, g.nzc - 2), g.zdf - 2), (2, range(g.zdf - 1), g.zdf + g.nzc - 4)]
    with np.errstate(all="ignore"):
        for level, ks, off in levels:
            s = ch.export_state(level)
            for k in ks:
                f = s[:, :, k, :]
                d, m = np.zeros(f.shape[:2]), [np.zeros(f.shape[:2]) for _ in range(3)]
                for a in range(19):
                    d = d + f[..., a]
                    for c, e in enumerate((EX, EY, EZ)):
                        m[c] = m[c] + float(e[a]) * f[..., a]
                n = float(f.shape[0] * f.shape[1])
                v = [x / d for x in m] + [d]
                mean = [ordered(x) / n for x in v]
                u, vv, w, dd = (x - y for x, y in zip(v, mean))
                sq = [ordered(x) / n for x in (u * u, vv * vv, w * w, u * w, dd * dd)]
                out[:, off + k] = mean[:3] + [np.sqrt(x) for x in sq[:3]] + [sq[3], mean[3], np.sqrt(sq[4])]
    return out


@pytest.mark.parametrize("precision", ["FP64", "FP32"])
@pytest.mark.parametrize("grid", [(36, 31, 7, 5, 2, "PSLIP"), (32, 16, 6, 4, 2, None), (19, 27, 7, 6, 3, "RSLIP"),
                                  (16, 33, 7, 8, 4, None)], ids=lambda g: "x".join(str(v) for v in g[:5]))
def test_record_is_its_definition_bit_for_bit(pkg, grid, precision):
    p = params_for(pkg, macros(*grid), "const")
    p.precision = getattr(pkg, precision)
    with pkg.Channel(p) as ch:
        ch.init_seeded(7)
        ch.step(3)
        np.testing.assert_array_equal(ch.plane_stats(), record(ch))


@pytest.mark.parametrize("precision", ["FP64", "FP32"])
@pytest.mark.parametrize("population", [0, 3, 5, 7, 15])
@pytest.mark.parametrize("value", [np.inf, -np.inf, np.nan])
def test_record_of_populations_that_are_not_finite(pkg, population, value, precision):
    """One population of a coarse, a lower and an upper node: its plane's record is not
    a number wherever the definition's is, and the other planes' are unchanged."""
    p = params_for(pkg, macros(9, 6, 7, 5, 2, "PSLIP"), "const")
    p.precision = getattr(pkg, precision)
    with pkg.Channel(p) as ch:
        ch.init_seeded(7)
        for level, k in ((0, 3), (1, 2), (2, 4)):
            s = ch.export_state(level)
            s[4, 3, k, population] = value
            ch.import_state(level, s)
        np.testing.assert_array_equal(ch.plane_stats(), record(ch))
