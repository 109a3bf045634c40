"""The channel driver's host code on a stand-in for the CUDA runtime (no GPU): what the
calls return where the device reports a failure or memory runs out, and what is
launched.  Each test runs its statements in a child process with fake_cudart.c
preloaded; `rt` there is the stand-in, `channel` makes a channel."""
from __future__ import annotations

import os
import subprocess
import sys
import textwrap

import pytest

from conftest import PKG_NAME, ROOT

PRELUDE = f"""
import ctypes, importlib
import numpy as np
rt = ctypes.CDLL(None)
rt.fake_limit.argtypes = [ctypes.c_size_t]
rt.fake_used.restype = ctypes.c_size_t
for f in ("fake_launches", "fake_graph_launches", "fake_instantiated"):
    getattr(rt, f).restype = ctypes.c_long
pkg = importlib.import_module("{PKG_NAME}")
def params(xdv, ydv, zdv, zds, gr, precision="FP64", **kw):
    return pkg.make_params(xdv=xdv, ydv=ydv, zdv=zdv, zds=zds, gratio=gr, Rebs=200.0, CFL=2.0, pattern=None,
                           precision=getattr(pkg, precision), forcing=pkg.FORCING_CONST, force_const=1e-5, **kw)
def channel(*a, **kw):
    return pkg.Channel(params(*a, **kw))
def error(call):
    try:
        call()
    except pkg.DnsError as e:
        return e
    return None
"""


@pytest.fixture(scope="session")
def fake(tmp_path_factory):
    so = tmp_path_factory.mktemp("fake") / "fake_cudart.so"
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", "-Wall", "-Werror", str(ROOT / "tests" / "fake_cudart.c"), "-o",
                    str(so)], check=True)

    def run(code):
        r = subprocess.run([sys.executable, "-c", PRELUDE + textwrap.dedent(code)], cwd=ROOT, capture_output=True,
                           text=True, timeout=300, env=dict(os.environ, LD_PRELOAD=str(so)))
        assert r.returncode == 0, r.stderr[-3000:]

    return run


@pytest.mark.parametrize("precision", ["FP64", "FP32"])
def test_a_wait_that_ran_out_is_an_error_of_its_own(fake, precision):
    """A two-substep pass that gave up sets a word that stays set: the step's row has a
    NaN wall stress and dns_step says what happened, in that call and in later ones."""
    fake(f"""
    with channel(8, 5, 7, 5, 2, precision="{precision}") as ch:
        ch.set_fine_pairs(1)
        ch.step(4)
        assert rt.fake_launches(b"fine_pair") == 4
        rt.fake_lost(1)
        for _ in range(2):
            e = error(lambda: ch.step(1))
            assert e is not None and e.code == pkg.DNS_ECUDA and "wait" in str(e), e
            rt.fake_lost(0)
    """)


def test_a_nan_wall_stress_without_it_stays_what_it_was(fake):
    fake("""
    with channel(8, 5, 7, 5, 2) as ch:
        rt.fake_stress(ctypes.c_double(float("inf")))
        assert error(lambda: ch.step(2)) is None
        rt.fake_stress(ctypes.c_double(float("nan")))
        e = error(lambda: ch.step(2))
        assert e is not None and e.code == pkg.DNS_ENAN and "NaN" in str(e), e
    """)


# planes between the substeps, and (FP64) rho and u there: what only pairs need
PAIR_BYTES = "(gr // 2) * (gr * x) * (gr * y) * (2 * 19 * 4 if precision == 'FP32' else (2 * 19 + 2 * 4) * 8)"


@pytest.mark.parametrize("form", [("FP64", 128, 128, 51, 16, 2), ("FP64", 64, 48, 20, 16, 4), ("FP32", 96, 80, 20, 10, 4)])
def test_a_channel_that_fits_without_pairs_is_created(fake, form):
    """Sizes that take two substeps a pass by default: where memory lacks for their
    planes alone the channel takes its substeps one at a time, and it is refused only
    where it does not fit at all."""
    precision, *grid = form
    fake(f"""
    precision, (x, y, z, s, gr) = "{precision}", {tuple(grid)}
    need = {PAIR_BYTES}
    g = pkg.geometry(params(x, y, z, s, gr, precision))
    with channel(x, y, z, s, gr, precision) as ch:
        used = rt.fake_used()
        assert used >= g.device_bytes - 4096
        ch.step(2)
        assert rt.fake_launches(b"fine_pair") > 0
    pairs = rt.fake_launches(b"fine_pair")
    for short in (1, need):
        rt.fake_limit(used - short)
        with channel(x, y, z, s, gr, precision) as ch:
            ch.step(2)
            assert rt.fake_launches(b"fine_pair") == pairs
            e = error(lambda: ch.set_fine_pairs(1))
            assert e is not None and e.code == pkg.DNS_ENOMEM
            ch.step(2)
            rt.fake_limit(1 << 36)
            ch.set_fine_pairs(-1)
            ch.step(2)
            assert rt.fake_launches(b"fine_pair") > pairs
            pairs = rt.fake_launches(b"fine_pair")
        assert rt.fake_used() == 0
    rt.fake_limit(used - need - 8192)
    e = error(lambda: channel(x, y, z, s, gr, precision))
    assert e is not None and e.code == pkg.DNS_ENOMEM
    assert rt.fake_used() == 0
    """)


def test_pairs_make_room_for_a_call_that_needs_memory(fake):
    fake(f"""
    precision, (x, y, z, s, gr) = "FP32", (16, 16, 7, 8, 4)
    need = {PAIR_BYTES}
    with channel(x, y, z, s, gr, precision) as ch:
        ch.set_fine_pairs(1)
        ch.step(60)
        stage = 19 * (gr * x) * (gr * y) * (s + 1) * 8
        rt.fake_limit(rt.fake_used() + stage - need)
        ch.export_state(1)
        pairs = rt.fake_launches(b"fine_pair")
        assert pairs > 0
        ch.step(60)
        assert rt.fake_launches(b"fine_pair") == pairs
    with channel(x, y, z, s, gr, precision) as ch:
        ch.set_fine_pairs(1)
        rt.fake_limit(rt.fake_used() + stage - need - 1)
        e = error(lambda: ch.export_state(1))
        assert e is not None and e.code == pkg.DNS_ENOMEM
    """)


def test_steps_go_on_one_by_one_where_a_graph_cannot_be_launched(fake):
    fake("""
    with channel(8, 5, 7, 5, 2) as ch:
        for _ in range(12):
            ch.step(6)
        assert rt.fake_graph_launches() > 0
        rt.fake_fail_graph_launch(ctypes.c_long(1))
        n = rt.fake_launches(b"finalize2")
        for _ in range(3):
            ch.step(6)
        assert rt.fake_launches(b"finalize2") == n + 18
    """)


@pytest.mark.parametrize("pairs", [0, 1])
def test_groups_of_every_start_state_get_their_graph(fake, pairs):
    """Groups start from any of the two coarse buffers, the two fine ones and the three
    history slots, sampled or not; steps that change which of them go together (a state
    seeded again after an odd number of passes) find a place for their graphs too."""
    fake(f"""
    def groups(ch):
        for sampling in (0, 1):
            ch.set_sampling(sampling)
            for start in range(6):
                n = rt.fake_graph_launches()
                for _ in range(9):
                    ch.step(6)
                assert rt.fake_graph_launches() > n, (sampling, start)
                ch.step(1)
    with channel(8, 5, 7, 5, 2) as ch:
        ch.set_fine_pairs({1 - pairs})
        ch.step(1)
        ch.set_fine_pairs({pairs})
        ch.step(1)
        groups(ch)
        ch.init_seeded(1)
        groups(ch)
        groups(ch)
        assert rt.fake_instantiated() <= 24
    """)
