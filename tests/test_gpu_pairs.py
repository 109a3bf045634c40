"""Two fine substeps in one pass against the oracle (needs a B200): the same bits
as the oracle's single substeps, at the edges of the kernels' tiles (a tile is 30
columns, or 62 with two warps side by side), of the planes they hold and of the
runs along y, and where they fall back to single substeps."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available
from test_gpu_parity import assert_state, pair, params_for

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]


def macros(xdv, ydv, zdv, zds, gr, pattern=None, **kw):
    return dict(dict(Rebs=200.0, ub=0.0866034, xdv=xdv, ydv=ydv, zdv=zdv, zds=zds, gratio=gr, TSTR=0, TEND=1, CFL=2.0,
                     gyplussize=4, wyplussize=4, gxplussize=4, wxplussize=4, XDIM=1, YDIM=1, ITER=50, pattern=pattern),
                **kw)


GRIDS = [
    (4, 4, 5, 4, 2, None),        # narrower than a tile
    (15, 6, 7, 4, 2, "RSLIP"),    # one full tile of 30
    (16, 5, 7, 5, 2, "PSLIP"),    # two warps side by side, the second one nearly empty
    (31, 4, 6, 8, 2, "SSLIP"),    # one full tile of 62, 16 warps
    (32, 4, 6, 8, 2, "PSLIP"),    # two tiles of 32 and 32
    (33, 7, 6, 9, 2, "PSLIP"),    # three tiles of 22, nine planes
    (8, 90, 6, 16, 2, "RSLIP"),   # sixteen planes, runs of several rows
    (31, 60, 5, 16, 2, "PSLIP"),  # the same with three tiles
    (8, 4, 7, 8, 4, "PSLIP"),     # two passes a step
    (10, 5, 7, 6, 3, "PSLIP"),    # a pass of two and a single substep
    (7, 5, 7, 5, 3, "RSLIP"),     # an odd row: single substeps
    (8, 4, 6, 17, 2, "RSLIP"),    # more planes than the kernels hold: single substeps
]


@pytest.mark.parametrize("mode", ["const", "cfr"])
@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(str(v) for v in g[:5]))
def test_pairs_match_oracle(pkg, port, grid, mode):
    ch, p = pair(pkg, port, macros(*grid), mode)
    ch.set_fine_pairs(1)
    la = ch.step(5)
    lb = p.step(5)
    assert_state(ch, p, exact=(mode == "const"))
    # momentum, mass, flow rate (the force is ub - momentum), wall shear
    np.testing.assert_allclose(la[:, 2:5], lb[:, 1:4], rtol=1e-11, atol=1e-15)
    np.testing.assert_allclose(la[:, 5:8], lb[:, 4:7], rtol=1e-9, atol=1e-14)


@pytest.mark.parametrize("grid", GRIDS, ids=lambda g: "x".join(str(v) for v in g[:5]))
def test_fp32_pairs_match_single_substeps(pkg, grid):
    """The FP32 form's pairs against its single substeps: the same arithmetic in
    another grouping, five steps: within 5e-7 (a collision rounds a deviation of at
    most 0.03 a few times, some 1e-8; at most 20 substeps)."""
    m = macros(*grid)
    p = params_for(pkg, m, "const")
    p.precision = pkg.FP32
    out = []
    for mode in (0, 1):
        with pkg.Channel(p) as ch:
            ch.set_fine_pairs(mode)
            ch.init_seeded(42, 0.05, 0.005)
            log = ch.step(5)
            out.append(([ch.export_state(lvl) for lvl in range(3)], log))
    for a, b in zip(out[0][0], out[1][0]):
        np.testing.assert_allclose(a, b, rtol=0, atol=5e-7)
    # momentum, mass, flow rate: sums of the states compared above
    np.testing.assert_allclose(out[0][1][:, 2:5], out[1][1][:, 2:5], rtol=1e-5)


def test_pairs_and_single_substeps_mix(pkg, port):
    """Sampled steps (their first substep alone) between steps in pairs, ratio 4
    with the filtered transfer: the oracle's state, whatever was on before."""
    m = macros(8, 4, 7, 8, 4, "PSLIP", fltr=True)
    ch, p = pair(pkg, port, m, "const")
    ch.set_sampling(3)
    for mode in (1, 0, 1):
        ch.set_fine_pairs(mode)
        ch.step(4)
        p.step(4)
        assert_state(ch, p, exact=True)
    _, n = ch.stats()
    assert n == 4  # steps 0, 3, 6, 9


def test_pairs_match_single_substeps_on_a_full_gpu(pkg):
    """Sixteen planes, every SM busy, 40 substeps: the same bits as the single
    substeps (rows that copies bring in while others are read)."""
    kw = dict(xdv=128, ydv=128, zdv=51, zds=16, gratio=2, Rebs=3000.0, ub=0.0866034, CFL=0.1, pattern="RSLIP",
              gyplussize=24, wyplussize=8, forcing=pkg.FORCING_CONST, force_const=1e-5)
    states = []
    for mode in (0, 1):
        with pkg.Channel(pkg.make_params(**kw)) as ch:
            ch.set_fine_pairs(mode)
            ch.init_seeded(42, 0.05, 0.005)
            ch.step(20)
            states.append([ch.export_state(lvl) for lvl in range(3)])
    for a, b in zip(*states):
        np.testing.assert_array_equal(a, b)
