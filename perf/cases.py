"""Performance cases of the grid-embedded channel solver.

Each case is one piece of work that a program using this library has it do,
through the public entry points (``Channel``, ``Batch``): coarse steps of a
channel with the log and the state or the statistics that the program reads
afterwards, a resumed run, the plane-statistics record and the energy budget of
a snapshot, and batches of channels advanced together.

Paths
  run      ``Channel.step(n)``, then what the program keeps: the state of all
           three levels (read into pinned buffers that the program owns), or, for
           a statistics run, the profiles of ``Channel.stats()``.
  resume   a run resumed from a state in host memory: import the levels and the
           interface history, step, read the state back.
  record   the plane-statistics record (``turb-fld``) of the current state, which
           ``dns_run`` writes every unit time.
  budget   the turbulence statistics and kinetic-energy budget of the current state.
  batch    ``Batch.run(n)`` on resident channels of uneven size, then the log and
           the statistics of every one, as the request loop reads them.

FP32 forms compute and store single-precision numbers; the interface hands them
out as doubles, and they are returned here as float32, the type they have.

``exact`` advances the same states in 64 bits with plain torch.
"""
from __future__ import annotations

import ctypes
import importlib
import math

import numpy as np
import torch

UB = 0.0866034
UC, AMP = 0.05, 0.005  # seeded start: laminar profile of this centre velocity + noise
PATTERNS = {"none": None, "ridges": "RSLIP", "posts": "PSLIP", "spanwise": "SSLIP"}


def _pkg():
    return importlib.import_module("dns-solvers-with-grid-embedding_b200")


# ------------------------------------------------------------------ the cases
def _height(c):
    """Fine-unit channel height NZs - 2."""
    return 2 * (c["zds"] + 1) + c["gr"] * (c["zdv"] - 4) + c["gr"] - 1 - 2


def _tau_re(c, tau=0.52):
    """Bulk Reynolds number that gives the fine relaxation time tau."""
    return 3.0 * UB * _height(c) / (tau - 0.5)


def _channel(path, precision, xdv, ydv, zdv, zds, gr, steps, pattern="none", gas=4, solid=4, reb=0.0, sample=0,
             filtered=False):
    c = dict(path=path, precision=precision, xdv=xdv, ydv=ydv, zdv=zdv, zds=zds, gr=gr, steps=steps, pattern=pattern,
             gas=gas, solid=solid, sample=sample, filtered=filtered)
    c["reb"] = float(reb) if reb else _tau_re(c)
    return c


def listed():
    def named(name, c):
        return dict(c, name=name)

    return [
        # the test suite's odd ridged channel: a call that is launches and latency only
        named("f64 tiny odd ridges", _channel("run", "fp64", 12, 6, 9, 6, 2, 10, "ridges", 6, 6, reb=200.0)),
        # the plain channel of the parity tests, resumed from a state in host memory
        named("f64 small resumed", _channel("resume", "fp64", 64, 64, 27, 8, 2, 200)),
        # the production channel of bench.py
        named("f64 production", _channel("run", "fp64", 256, 128, 83, 16, 2, 200, reb=5533.0)),
        # the superhydrophobic channel with posts: the largest single channel
        named("f64 posts large", _channel("run", "fp64", 384, 192, 115, 16, 2, 150, "posts", 16, 16, reb=13585.0)),
        # the reference's default grid ratio and fine extent, with the filtered transfer
        named("f64 ratio 4 filtered", _channel("run", "fp64", 96, 48, 55, 10, 4, 60, "ridges", 56, 8, filtered=True)),
        # ratio 3 on odd extents, statistics sampled every step as the long statistics runs do
        named("f64 ratio 3 sampled", _channel("run", "fp64", 75, 45, 31, 7, 3, 60, "spanwise", 9, 6, sample=1)),
        # the production channel as a single-precision statistics run
        named("f32 production", _channel("run", "fp32", 256, 128, 83, 16, 2, 320, reb=5533.0, sample=20)),
        # single precision on extents that are not a multiple of four
        named("f32 odd", _channel("run", "fp32", 131, 77, 45, 12, 2, 200, "ridges", 11, 11)),
        # the record dns_run writes every unit time, on the production channel
        named("record production", _channel("record", "fp64", 256, 128, 83, 16, 2, 20, reb=5533.0)),
        # the budget of a snapshot of the production channel
        named("budget production", _channel("budget", "fp64", 256, 128, 83, 16, 2, 20, reb=5533.0)),
        # a lightly loaded request loop: a few small channels, one group of steps
        dict(name="batch of 4", path="batch", count=4, mix=2, largest=128, steps=32),
        # the batched workload of bench.py: 96 channels of uneven size
        dict(name="batch of 96", path="batch", count=96, mix=4, largest=256, steps=32),
    ]


def draw(rng):
    def logint(lo, hi):
        return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))

    path = rng.choice(["run", "run", "run", "run", "resume", "record", "budget", "batch", "batch"])
    if path == "batch":
        return dict(path="batch", count=logint(1, 96), mix=rng.randrange(1 << 20), largest=rng.choice([64, 128, 192, 256]),
                    steps=32)
    gr = 2 if path == "budget" else rng.choice([2, 2, 2, 3, 4])
    xdv, ydv, zdv = logint(12, 320), logint(8, 160), logint(9, 110)
    zds = rng.randint(max(6, gr + 2), 16)
    precision = "fp64" if path in ("record", "budget") else rng.choice(["fp64", "fp64", "fp32"])
    pattern = rng.choice(sorted(PATTERNS))
    filtered = gr == 4 and zds >= 7 and rng.random() < 0.5
    gas, solid = rng.randint(4, 24), rng.randint(4, 24)
    sample = rng.choice([0, 0, 1, 20]) if path == "run" else 0
    while True:
        c = _channel(path, precision, xdv, ydv, zdv, zds, gr, 1, pattern, gas, solid, sample=sample, filtered=filtered)
        if _updates(c) <= 26_000_000:
            break
        xdv, ydv = max(12, xdv * 3 // 4), max(8, ydv * 3 // 4)
    # enough steps that the step loop is what counts, a fifth of a second at most
    c["steps"] = 20 if path in ("record", "budget") else max(10, min(200, int(2.2e9 / _updates(c))))
    return c


# ------------------------------------------------------------------ sizes
def _updates(c):
    """Node updates of one coarse step."""
    return c["xdv"] * c["ydv"] * c["zdv"] + 2 * c["gr"] * (c["gr"] * c["xdv"]) * (c["gr"] * c["ydv"]) * c["zds"]


def _nodes(c):
    """Nodes of the exported state (fine blocks with their wall plane)."""
    return c["xdv"] * c["ydv"] * c["zdv"] + 2 * (c["gr"] * c["xdv"]) * (c["gr"] * c["ydv"]) * (c["zds"] + 1)


def _channels(case):
    """The channels of a batch: grids, walls and Reynolds numbers of the batched workload's ranges."""
    r = np.random.default_rng(case["mix"])
    out = []
    for _ in range(case["count"]):
        nx = int(r.choice([n for n in (64, 128, 192, 256) if n <= case["largest"]]))
        ny, nz = int(r.choice((32, 48, 64))), int(r.choice((64, 96, 128)))
        pattern = str(r.choice(["ridges", "posts"]))
        pitch = int(r.choice((16, 24, 32)))
        gas = int(round(pitch * float(r.uniform(0.5, 0.9))))
        # at most this many wall units per fine cell, and Dean's correlation for the bulk Reynolds number
        retau = min(float(r.uniform(180.0, 395.0)), {32: 1.75, 48: 2.5, 64: 2.75}[ny] * (2 * ny - 1) / 2.0)
        zds = ny // 4
        out.append(_channel("run", "fp32", nx, nz, ny - zds + 3, zds, 2, case["steps"], pattern, gas, pitch - gas,
                            reb=2.0 * (retau / 0.175) ** (8.0 / 7.0), sample=20))
    return out


def work(case):
    if case["path"] == "batch":
        per = [work(c) for c in _channels(case)]
        return {"bytes": sum(w["bytes"] for w in per), "flops": sum(w["flops"] for w in per)}
    esz = 8 if case["precision"] == "fp64" else 4
    nodes = _nodes(case)
    if case["path"] == "record":  # the populations once; moments and their squares
        return {"bytes": 19 * 8.0 * nodes, "flops": 60.0 * nodes}
    if case["path"] == "budget":  # the populations once; moments, gradients and 44 products
        return {"bytes": 19 * 8.0 * nodes, "flops": 260.0 * nodes}
    # per coarse step every level's state is read once and written once; 270
    # operations a node update; then what the program reads back
    flops = 270.0 * _updates(case) * case["steps"]
    bytes_ = 2 * 19.0 * esz * nodes * case["steps"]
    if case["path"] == "resume":
        bytes_ += 2 * 19 * (8 + esz) * nodes
    elif case["path"] == "run" and not case["sample"]:
        bytes_ += 19 * (8 + esz) * nodes
    return {"bytes": bytes_, "flops": flops}


# ------------------------------------------------------------------ the calls
def _params(pkg, c):
    return pkg.make_params(
        xdv=c["xdv"], ydv=c["ydv"], zdv=c["zdv"], zds=c["zds"], gratio=c["gr"], Rebs=c["reb"], ub=UB, CFL=0.1,
        pattern=PATTERNS[c["pattern"]], gyplussize=c["gas"], wyplussize=c["solid"], gxplussize=c["gas"],
        wxplussize=c["solid"], forcing=pkg.FORCING_CFR, fltr=int(c["filtered"]), TSTR=0,
        precision=pkg.FP64 if c["precision"] == "fp64" else pkg.FP32)


def _level_shapes(c):
    nxf, nyf, zdf = c["gr"] * c["xdv"], c["gr"] * c["ydv"], c["zds"] + 1
    return [(c["xdv"], c["ydv"], c["zdv"], 19), (nxf, nyf, zdf, 19), (nxf, nyf, zdf, 19)]


def prepare(case, seed):
    pkg = _pkg()
    if case["path"] == "batch":
        b = pkg.Batch()
        ids = [b.add(_params(pkg, c), steps=1 << 40, seed=seed * 1000 + q, uc=UC, amp=AMP, sample_every=c["sample"])
               for q, c in enumerate(_channels(case))]
        return {"case": case, "batch": b, "ids": ids, "done": 0}
    ch = pkg.Channel(_params(pkg, case))
    ch.init_seeded(seed, UC, AMP)
    s = {"case": case, "ch": ch, "pkg": pkg}
    if case["path"] in ("record", "budget"):
        ch.step(case["steps"], log=False)
        return s
    ch.set_sampling(case["sample"])
    if case["path"] == "resume" or not case["sample"]:
        s["host"] = [torch.empty(sh, dtype=torch.float64, pin_memory=True) for sh in _level_shapes(case)]
        if case["precision"] == "fp32":
            s["host32"] = [torch.empty(sh, dtype=torch.float32) for sh in _level_shapes(case)]
    if case["path"] == "resume":
        s["start"] = [torch.empty(sh, dtype=torch.float64, pin_memory=True) for sh in _level_shapes(case)]
        for level, t in enumerate(s["start"]):
            _export(pkg, ch, level, t)
        s["history"] = ch.export_history()
    return s


def _export(pkg, ch, level, t):
    pkg._check(pkg.lib().dns_export_state(ch.h, level, ctypes.c_void_p(t.data_ptr())), "dns_export_state")


def run(state):
    case = state["case"]
    if case["path"] == "batch":
        b, first, n = state["batch"], state["done"], case["steps"]
        b.run(n)
        state["done"] += n
        return {"log": np.concatenate([b.log(i, first, n) for i in state["ids"]]).astype(np.float32),
                "stats": np.concatenate([b.stats(i)[0] for i in state["ids"]], axis=1).astype(np.float32)}
    ch = state["ch"]
    if case["path"] == "record":
        return {"record": ch.plane_stats()}
    if case["path"] == "budget":
        p = ch.tke_budget()
        return {"turb_fld": p[:19], "vort_fluc": p[19:22], "ke_budget": p[22:]}
    pkg = state["pkg"]
    if case["path"] == "resume":
        for level, t in enumerate(state["start"]):
            pkg._check(pkg.lib().dns_import_state(ch.h, level, ctypes.c_void_p(t.data_ptr())), "dns_import_state")
        ch.import_history(state["history"])
    log = ch.step(case["steps"])
    if case["path"] == "resume":
        log = log[:, 1:]  # the time stamps count on from call to call
    kind = np.float64 if case["precision"] == "fp64" else np.float32
    if case["sample"]:
        stats, n = ch.stats()
        return {"log": log.astype(kind), "stats": stats.astype(kind), "samples": n}
    for level, t in enumerate(state["host"]):
        _export(pkg, ch, level, t)
    if case["precision"] == "fp32":
        state["out"] = [a.copy_(b) for a, b in zip(state["host32"], state["host"])]
    else:
        state["out"] = state["host"]
    return {"log": log.astype(kind), "coarse": state["out"][0], "lower": state["out"][1], "upper": state["out"][2]}


# ------------------------------------------------------------------ the same in 64 bits, plain torch
_E = np.array([(0, 0, 0), (1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (1, 1, 0), (-1, 1, 0),
               (-1, -1, 0), (1, -1, 0), (1, 0, 1), (1, 0, -1), (-1, 0, -1), (-1, 0, 1), (0, 1, 1), (0, 1, -1),
               (0, -1, -1), (0, -1, 1)])
_W = [1 / 3] + [1 / 18] * 6 + [1 / 36] * 12
_OPP = [int(np.flatnonzero((_E == -e).all(1))[0]) for e in _E]
_MIR = [int(np.flatnonzero((_E == e * (1, 1, -1)).all(1))[0]) for e in _E]


def _moments(f):
    rho = f.sum(0)
    u = [sum(int(e[c]) * f[a] for a, e in enumerate(_E) if e[c]) / rho for c in range(3)]
    return rho, u


def _feq(a, rho, u, usq):
    eu = sum(int(_E[a][c]) * u[c] for c in range(3) if _E[a][c])
    return _W[a] * rho * (1 + 3 * eu + 4.5 * eu * eu - 1.5 * usq)


def _collide(f, om, g):
    rho, u = _moments(f)
    usq = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
    out = torch.empty_like(f)
    for a in range(19):
        force = int(_E[a][0]) * (1 / 6 if a <= 6 else 1 / 12) * g
        out[a] = f[a] - om * (f[a] - _feq(a, rho, u, usq)) + force * rho
    return out, rho, u


def _shift(t, e):
    """Stream one plane set [.., y, x] by (e_x, e_y), periodic."""
    return torch.roll(t, (int(e[1]), int(e[0])), (-2, -1)) if e[0] or e[1] else t


def _philox(ctr, key):
    def mul(a, m):  # 32 x 32 -> (high, low) in int64
        lo = (a & 0xFFFF) * m
        hi = (a >> 16) * m + (lo >> 16)
        return hi >> 16, ((hi & 0xFFFF) << 16) | (lo & 0xFFFF)

    c, k = list(ctr), list(key)
    for r in range(10):
        if r:
            k = [(k[0] + 0x9E3779B9) & 0xFFFFFFFF, (k[1] + 0xBB67AE85) & 0xFFFFFFFF]
        h0, l0 = mul(c[0], 0xD2511F53)
        h1, l1 = mul(c[2], 0xCD9E8D57)
        c = [h1 ^ c[1] ^ k[0], l1, h0 ^ c[3] ^ k[1], l0]
    return c


class _Exact:
    """The channel in 64 bits: levels [19, z, y, x]; fine blocks without their wall plane."""

    def __init__(self, c, seed):
        self.c, self.dev = c, "cuda" if torch.cuda.is_available() else "cpu"
        gr, zds, zdc = c["gr"], c["zds"], c["zdv"]
        self.nx, self.ny, self.nxf, self.nyf = c["xdv"], c["ydv"], gr * c["xdv"], gr * c["ydv"]
        self.zdf, self.H = zds + 1, _height(c)
        self.om_f = 1 / (3 / c["reb"] * UB * self.H + 0.5)
        self.om_c = 1 / (3 / c["reb"] * UB * self.H / gr + 0.5)
        kc = torch.arange(zdc, device=self.dev)
        kl, ku = torch.arange(1, zds + 1, device=self.dev), torch.arange(zds, device=self.dev)
        z = [(self.zdf - 1.5) + gr * (kc.double() - 1.0), kl.double() - 0.5,
             (self.zdf - 1.5) + gr * (zdc - 3.0) + ku.double()]
        self.lv, us = [], []
        for level, (k, zz, nx, ny) in enumerate(((kc, z[0], self.nx, self.ny), (kl, z[1], self.nxf, self.nyf),
                                                 (ku, z[2], self.nxf, self.nyf))):
            u = self._seeded(k, zz, ny, nx, level, seed)
            usq = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
            one = torch.ones_like(u[0])
            self.lv.append(torch.stack([_feq(a, one, u, usq) for a in range(19)]))
            us.append(u)
        self.hist = []
        for k in (1, zdc - 2):
            h = torch.zeros(23, self.ny, self.nx, dtype=torch.float64, device=self.dev)
            h[0] = 1
            for q in range(3):
                h[1 + q] = us[0][q][k]
            self.hist.append([h, h, h])
        flag = torch.ones(self.nyf, self.nxf, dtype=torch.bool, device=self.dev)  # solid
        pat, period = c["pattern"], c["gas"] + c["solid"]

        def slip(n):
            s = torch.zeros(n, dtype=torch.bool, device=self.dev)
            for j in range(c["solid"] // 2, n, period):
                s[j:j + c["gas"]] = True
            return s

        if pat in ("ridges", "posts"):
            flag &= ~slip(self.nyf)[:, None]
        if pat in ("spanwise", "posts"):
            flag &= ~slip(self.nxf)[None, :]
        self.solid = flag
        self.step_no, self.sums = 0, []
        self._flow()

    def _seeded(self, k, z, ny, nx, level, seed):
        n = (len(k), ny, nx)
        i = torch.arange(nx, device=self.dev).expand(n)
        j = torch.arange(ny, device=self.dev)[:, None].expand(n)
        kk = k[:, None, None].expand(n)
        r = _philox([i, j, kk, torch.full(n, level, device=self.dev)], [seed & 0xFFFFFFFF, seed >> 32])
        u = [AMP * (2 * ((x.double() + 0.5) / 4294967296.0) - 1) for x in r[:3]]
        zeta = z / self.H
        u[0] = u[0] + (4 * UC * zeta * (1 - zeta))[:, None, None]
        return u

    def _flow(self):
        """Momentum and mass of the state with their quadrature weights; the next step's force."""
        gr, zdf = self.c["gr"], self.zdf
        wc = torch.full((self.c["zdv"],), float(gr ** 3), device=self.dev, dtype=torch.float64)
        wc[0] = wc[-1] = 0.5 * gr ** 3
        kl, ku = range(1, zdf), range(zdf - 1)
        wl = torch.tensor([1.0 if k < zdf - gr else 0.0 for k in kl], device=self.dev, dtype=torch.float64)
        wu = torch.tensor([0.0 if k < gr else 0.5 if k == gr else 1.0 for k in ku], device=self.dev,
                          dtype=torch.float64)
        norm = float(self.nxf) * self.nyf * self.H
        mom = den = 0.0
        for f, w in zip(self.lv, (wc, wl, wu)):
            planes = f.sum((2, 3))
            mx = sum(int(e[0]) * planes[a] for a, e in enumerate(_E) if e[0])
            mom, den = mom + float((mx * w).sum()), den + float((planes.sum(0) * w).sum())
        self.mom, self.den = mom / norm, den / norm
        self.force = UB - self.mom

    def _fine(self, f, post, upper):
        """Streaming of one fine block; the interface plane of the result is left to the transfer."""
        zds = self.c["zds"]
        out = torch.empty_like(f)
        wall = zds - 1 if upper else 0
        iface = 0 if upper else zds - 1
        for b in range(19):
            e = _E[b]
            s = _shift(post[b], e)
            if e[2] == 0:
                out[b] = s
            elif e[2] > 0:
                out[b, 1:] = s[:-1]
            else:
                out[b, :-1] = s[1:]
            if e[2] == (-1 if upper else 1):  # leaves the wall: bounced back or reflected
                both = self.solid & _shift(self.solid, e)
                out[b, wall] = torch.where(both, post[_OPP[b]][wall], _shift(post[_MIR[b]][wall], e))
        return out, iface

    def _transfer(self, hist, tau):
        gr = self.c["gr"]
        n, p, pp = hist
        t = tau
        h = (2 * t ** 3 - 3 * t ** 2 + 1, t ** 3 - 2 * t ** 2 + t, -2 * t ** 3 + 3 * t ** 2, t ** 3 - t ** 2)
        v = h[0] * p + h[1] * (n - pp) * 0.5 + h[2] * n + h[3] * (3 * n - 4 * p + pp) * 0.5

        def diff(q, d):
            return 2 / 3 * (torch.roll(q, -1, d) - torch.roll(q, 1, d)) - 1 / 12 * (
                torch.roll(q, -2, d) - torch.roll(q, 2, d))

        dx, dy = diff(v, -1), diff(v, -2)
        dxy = diff(dy, -1)

        def basis(t):
            return ((2 * t ** 3 - 3 * t ** 2 + 1, t ** 3 - 2 * t ** 2 + t), (-2 * t ** 3 + 3 * t ** 2, t ** 3 - t ** 2))

        out = torch.empty(23, self.ny, gr, self.nx, gr, dtype=torch.float64, device=self.dev)
        for ii in range(gr):
            for jj in range(gr):
                bx, by = basis(ii / gr), basis(jj / gr)
                s = 0
                for a in range(2):
                    for b in range(2):
                        def at(q):
                            return torch.roll(q, (-b, -a), (-2, -1))
                        s = s + bx[a][0] * by[b][0] * at(v) + bx[a][1] * by[b][0] * at(dx) + \
                            bx[a][0] * by[b][1] * at(dy) + bx[a][1] * by[b][1] * at(dxy)
                out[:, :, jj, :, ii] = s
        m = out.reshape(23, self.nyf, self.nxf)
        u = [m[1], m[2], m[3]]
        usq = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        fac = self.om_c / (gr * self.om_f)
        return torch.stack([_feq(a, m[0], u, usq) + fac * m[4 + a] for a in range(19)])

    def _inject(self, f, k):
        """Coarse boundary plane from fine plane index k of block f."""
        gr, fac = self.c["gr"], self.c["gr"] * self.om_f / self.om_c
        if self.c["filtered"]:
            tr = {-2: 0.5, -1: 1.0, 0: 1.0, 1: 1.0, 2: 0.5}
            neq = 0
            for kk in tr:
                g = f[:, k + kk]
                rho, u = _moments(g)
                usq = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
                q = torch.stack([g[a] - _feq(a, rho, u, usq) for a in range(19)])
                for ii in tr:
                    for jj in tr:
                        neq = neq + tr[ii] * tr[jj] * tr[kk] / gr ** 3 * torch.roll(q, (-jj, -ii), (-2, -1))
            neq = neq[:, ::gr, ::gr]
            g = f[:, k, ::gr, ::gr]
            rho, u = _moments(g)
            u = [rho * x for x in u]  # the filtered transfer's equilibrium takes the momentum
            usq = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
            return torch.stack([_feq(a, rho, u, usq) + fac * neq[a] for a in range(19)])
        g = f[:, k, ::gr, ::gr]
        rho, u = _moments(g)
        usq = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
        eq = torch.stack([_feq(a, rho, u, usq) for a in range(19)])
        return eq + fac * (g - eq)

    def _profile_planes(self):
        """(index, [rho, u, v, w] of one plane) of the composite profile."""
        zdf, zdc = self.zdf, self.c["zdv"]
        mac = []
        for f in self.lv:
            rho, u = _moments(f)
            mac.append([rho] + u)
        for k in range(1, zdf):
            yield k, [q[k - 1] for q in mac[1]]
        for k in range(2, zdc - 2):
            yield zdf - 2 + k, [q[k] for q in mac[0]]
        for k in range(zdf - 1):
            yield zdf + zdc - 4 + k, [q[k] for q in mac[2]]

    def sample(self):
        rows = np.zeros((2 * self.zdf + self.c["zdv"] - 4, 9))
        for p, (rho, u, v, w) in self._profile_planes():
            m = [q.mean() for q in (u, v, w, rho)]
            du, dv, dw, dr = (q - x for q, x in zip((u, v, w, rho), m))
            rows[p] = torch.stack(m + [(du * du).mean(), (dv * dv).mean(), (dw * dw).mean(), (du * dw).mean(),
                                       (dr * dr).mean()]).cpu().numpy()
        self.sums.append(rows)

    def step(self):
        c, gr, zdf, zdc = self.c, self.c["gr"], self.zdf, self.c["zdv"]
        if c["sample"] and self.step_no % c["sample"] == 0:
            self.sample()
        row = {"force": self.force, "momentum": self.mom, "denst": self.den}
        post, _, _ = _collide(self.lv[0], self.om_c, self.force)
        new = torch.empty_like(post)
        for a in range(19):
            e = _E[a]
            new[a, 1:-1] = _shift(post[a], e)[1 - int(e[2]):zdc - 1 - int(e[2])]
        for w, k in enumerate((1, zdc - 2)):
            f = new[:, k]
            rho, u = _moments(f)
            usq = u[0] ** 2 + u[1] ** 2 + u[2] ** 2
            lev = torch.stack([rho] + u + [f[a] - _feq(a, rho, u, usq) for a in range(19)])
            self.hist[w] = [lev, self.hist[w][0], self.hist[w][1]]
        fine = [self.lv[1], self.lv[2]]
        for s in range(1, gr + 1):
            for w in range(2):
                post, rho, u = _collide(fine[w], self.om_f, self.force / gr)
                if s == 1:
                    k = (0, 1, 2) if w == 0 else (zdf - 2, zdf - 3, zdf - 4)
                    m = [float(u[0][q].mean()) for q in k]
                    visc = (2 / self.om_f - 1) / 6
                    r = float(rho[0 if w == 0 else zdf - 4].mean())
                    row["stdown" if w == 0 else "stup"] = (-2 * m[0] + 3 * m[1] - m[2]) * visc * r
                fine[w], iface = self._fine(fine[w], post, w == 1)
                fine[w][:, iface] = self._transfer(self.hist[w], s / gr)
        new[:, 0] = self._inject(fine[0], zdf - 2 - gr)
        new[:, -1] = self._inject(fine[1], gr)
        self.lv = [new] + fine
        dt = gr / (0.5 * self.H / 0.1)
        log = [dt * self.step_no, row["force"], row["momentum"], row["denst"],
               row["momentum"] * self.nyf * self.H / row["denst"], row["stup"], row["stdown"],
               0.5 * (row["stup"] + row["stdown"]), row["force"] * self.H / (2 * gr)]
        self.step_no += 1
        self._flow()
        return log

    def export(self):
        """The levels as [x, y, z, 19]; wall planes hold zeros after a seeded start."""
        out = []
        for level, f in enumerate(self.lv):
            a = f.permute(3, 2, 1, 0)
            if level:
                zero = torch.zeros_like(a[:, :, :1])
                a = torch.cat([zero, a] if level == 1 else [a, zero], 2)
            out.append(a.contiguous().cpu())
        return out

    def stats(self):
        NZ, zdf, zdc, gr = 2 * self.zdf + self.c["zdv"] - 4, self.zdf, self.c["zdv"], self.c["gr"]
        z = np.zeros(NZ)
        z[1:zdf] = np.arange(1, zdf) - 0.5
        z[zdf:zdf + zdc - 4] = gr * (np.arange(2, zdc - 2) - 1.0) + (zdf - 1.5)
        z[zdf + zdc - 4:NZ - 1] = np.arange(zdf - 1) + gr * (zdc - 3.0) + zdf - 1.5
        z[NZ - 1] = 2 * zdf + gr * (zdc - 4) + gr - 3
        s = np.stack(self.sums)  # samples, planes, 9
        out = np.zeros((14, NZ))
        out[0] = z / self.H
        m, q = s[..., :4], s[..., 4:]
        out[1:5] = m.mean(0).T
        out[5:10] = q.mean(0).T
        d = m - m.mean(0)
        for r, (i, j, k) in enumerate(((0, 0, 0), (1, 1, 1), (2, 2, 2), (0, 2, 3))):
            out[10 + r] = q[..., k].mean(0) + (d[..., i] * d[..., j]).mean(0)
        return out

    def record(self):
        out = np.zeros((9, 2 * self.zdf + self.c["zdv"] - 4))
        self.sums = []
        self.sample()
        r = self.sums[0].T
        out[0:3], out[3:6], out[6], out[7], out[8] = r[0:3], np.sqrt(r[4:7]), r[7], r[3], np.sqrt(r[8])
        return out

    def turb_fld(self):
        """Means, rms, shear stress, skewness and flatness of the composite profile (pressure = rho / 3)."""
        out = np.zeros((19, 2 * self.zdf + self.c["zdv"] - 4))
        for p, (rho, u, v, w) in self._profile_planes():
            pr = rho / 3
            m = [q.mean() for q in (u, v, w, pr)]
            du, dv, dw, dp = (q - x for q, x in zip((u, v, w, pr), m))
            su, sv, sw, sp = ((q * q).mean().sqrt() for q in (du, dv, dw, dp))
            r = [m[0], m[1], m[2], su, sv, sw, (du * dw).mean(), m[3], sp, (du ** 3).mean() / su ** 3,
                 (dv ** 3).mean() / sv ** 3, (dw ** 3).mean() / sw ** 3, (du ** 3 * dw ** 3).mean() / (su * sw) ** 3,
                 (dp ** 3).mean() / sp ** 3, (du ** 4).mean() / su ** 4, (dv ** 4).mean() / sv ** 4,
                 (dw ** 4).mean() / sw ** 4, (du ** 4 * dw ** 4).mean() / (su * sw) ** 4, (dp ** 4).mean() / sp ** 4]
            out[:, p] = torch.stack(r).cpu().numpy()
        return out


def _seconds(c):
    """About what one step of _Exact takes, times the steps."""
    return c["steps"] * (0.02 + 3e-9 * _updates(c))


def exact(case, seed):
    if case["path"] == "batch":
        chans = _channels(case)
        if sum(_seconds(c) for c in chans) > 18:
            return None
        logs, stats = [], []
        for q, c in enumerate(chans):
            x = _Exact(c, seed * 1000 + q)
            logs += [x.step() for _ in range(c["steps"])]
            stats.append(x.stats())
        return {"log": np.array(logs), "stats": np.concatenate(stats, axis=1)}
    if _seconds(case) > 18:
        return None
    x = _Exact(case, seed)
    log = np.array([x.step() for _ in range(case["steps"])])
    if case["path"] == "record":
        return {"record": x.record()}
    if case["path"] == "budget":  # the gradient profiles have no plain counterpart here
        return {"turb_fld": x.turb_fld(), "vort_fluc": None, "ke_budget": None}
    if case["path"] == "resume":
        log = log[:, 1:]
    if case["sample"]:
        return {"log": log, "stats": x.stats(), "samples": None}
    lv = x.export()
    return {"log": log, "coarse": lv[0], "lower": lv[1], "upper": lv[2]}
