"""Groups of six steps issued as one recorded graph against the same steps issued
one by one (needs a B200): a call of a single step is never a group, and the kernels
are deterministic, so the states, the log rows and the statistics are equal bit for
bit."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import gpu_available
from test_gpu_pairs import macros
from test_gpu_parity import params_for

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]

FORMS = [
    # grid, precision, pairs mode, filtered injection, mode, sample every
    ((8, 5, 7, 5, 2, "PSLIP"), "FP64", 0, 0, "const", 0),
    ((8, 5, 7, 5, 2, "PSLIP"), "FP64", 1, 0, "cfr", 1),
    ((10, 5, 7, 6, 3, "PSLIP"), "FP64", -1, 0, "cfr", 7),
    ((8, 6, 7, 8, 4, "RSLIP"), "FP64", 1, 1, "cfr", 20),
    ((9, 5, 7, 5, 2, "RSLIP"), "FP32", 0, 0, "cfr", 13),
    ((8, 6, 7, 8, 4, "PSLIP"), "FP32", 1, 0, "const", 1),
]


@pytest.mark.parametrize("form", FORMS, ids=lambda f: "x".join(str(v) for v in f[0][:5]) + f"-{f[1]}-{f[5]}")
def test_groups_match_single_steps(pkg, form):
    import torch

    grid, precision, pairs, fltr, mode, every = form
    p = params_for(pkg, macros(*grid), mode)
    p.precision = getattr(pkg, precision)
    p.fltr = fltr
    # groups from every one of the six start states; the longest call exceeds the log's
    # rows of one chunk, and a group is recorded when it has been due several times
    calls = [5, 6, 61, 1, 131, 7, 1103, 200, 3, 118]
    out, stream = [], torch.cuda.Stream()
    for single in (True, False):
        with pkg.Channel(p) as ch:
            ch.set_fine_pairs(pairs)
            ch.set_sampling(every)
            ch.init_seeded(3)
            log = []
            for q, n in enumerate(calls):
                if not single and q == 4:
                    ch.set_stream(stream.cuda_stream)
                if not single and q == 8:
                    ch.set_stream(None)
                for _ in range(n if single else 1):
                    log.append(ch.step(1 if single else n))
            state = [ch.export_state(l) for l in range(3)] + [ch.export_history(), np.concatenate(log)]
            if every:
                acc, samples = ch.stats()
                state += [acc, np.array(samples), ch.plane_stats()]
            out.append(state)
    for a, b in zip(*out):
        np.testing.assert_array_equal(a, b)
