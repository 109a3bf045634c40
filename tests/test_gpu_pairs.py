"""Two fine substeps in one pass against the oracle (needs a B200): the same bits
as the oracle's single substeps, at the edges of the kernels' tiles (a tile is 30
columns, or 62 with two warps side by side), of the planes they hold and of the
runs along y, and where they fall back to single substeps."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available
from test_gpu_parity import assert_state, pair

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
