"""A step whose two-substep pass gave up is reported (needs a B200).  Nothing gives up
here: the word that such a pass sets is set from the host (a preloaded cudaMalloc tells
where it lies: the third of the 256-byte block that a channel allocates), and
the device's finalize and dns_step do the rest."""
from __future__ import annotations

import os
import subprocess
import sys

import pytest

from conftest import PKG_NAME, ROOT, gpu_available

pytestmark = [pytest.mark.gpu, pytest.mark.skipif(not gpu_available(), reason="no CUDA device")]

HOOK = r"""
#define _GNU_SOURCE
#include <dlfcn.h>
#include <stddef.h>
static void *block;
void *counter_block(void) { return block; }
int cudaMalloc(void **p, size_t n) {
  int (*real)(void **, size_t) = (int (*)(void **, size_t))dlsym(dlopen("libcudart.so.12", RTLD_LAZY), "cudaMalloc");
  int e = real(p, n);
  if (!e && n == 256) block = *p;
  return e;
}
"""

CHILD = f"""
import ctypes, importlib, sys
import numpy as np
pkg = importlib.import_module("{PKG_NAME}")
x, y, z, s, gr = map(int, sys.argv[1].split("x"))
p = pkg.make_params(xdv=x, ydv=y, zdv=z, zds=s, gratio=gr, Rebs=200.0, CFL=2.0, pattern="PSLIP", gyplussize=4,
                    wyplussize=4, gxplussize=4, wxplussize=4, precision=getattr(pkg, sys.argv[2]),
                    forcing=pkg.FORCING_CONST, force_const=1e-5)
rt = ctypes.CDLL(None)
rt.counter_block.restype = ctypes.c_void_p
cuda = ctypes.CDLL("libcudart.so.12")
with pkg.Channel(p) as ch:
    at = rt.counter_block()
    ch.init_seeded(3)
    ch.step(7)
    word = ctypes.c_uint(1)
    assert cuda.cudaMemcpy(ctypes.c_void_p(at + 8), ctypes.byref(word), 4, 1) == 0
    for n in (1, 70):
        try:
            ch.step(n)
        except pkg.DnsError as e:
            assert e.code == pkg.DNS_ECUDA and "wait" in str(e), e
        else:
            raise AssertionError("not reported")
"""


@pytest.mark.parametrize("precision", ["FP64", "FP32"])
@pytest.mark.parametrize("grid", ["8x5x7x5x2", "96x64x40x8x3"])  # finalize in one block and in 64
def test_a_pass_that_gave_up_is_reported(tmp_path, grid, precision):
    src, so = tmp_path / "hook.c", tmp_path / "hook.so"
    src.write_text(HOOK)
    subprocess.run(["gcc", "-shared", "-fPIC", "-O1", str(src), "-o", str(so), "-ldl"], check=True)
    r = subprocess.run([sys.executable, "-c", CHILD, grid, precision], cwd=ROOT, capture_output=True, text=True,
                       timeout=120, env=dict(os.environ, LD_PRELOAD=str(so)))
    assert r.returncode == 0, r.stderr[-3000:]
