"""The work users of oercel_b200 have it do, as timed cases.

Every case goes through the package's public entry points: oercel_b200.Engine,
oercel_b200.autograd, oercel_b200.cells, and the C ABI of include/dpd.h with
torch CUDA tensors as the device-memory carrier.  Kinds of case:

  run       one box advanced by a chunk of steps between two outputs, then its
            state read into device tensors (the loop of the command-line front
            end): chemistry off or the lipid chemistry, reference or benchmark
            physics, Philox or mix13 noise
  ensemble  many boxes of uneven size in one engine (a parameter sweep)
  catalyst  the reference's catalyst chemistry with branched lipids
  forces    one force evaluation of a given configuration (custom loops)
  vjp       the vector-Jacobian product of one force evaluation
  fit       one differentiated window with its gradient through
            oercel_b200.autograd (an optimizer iteration), continuing from the
            engine's state or from a start state whose gradient is wanted too
  analysis  the measures of a configuration between steps: observables with the
            virial, tail clusters, membrane aggregates, pair distances
  cells     cell detection in a snapshot on the host
"""
from __future__ import annotations

import math
import os
import sys

import numpy as np
import torch

sys.path.insert(0, os.path.join(os.path.dirname(os.path.dirname(os.path.abspath(__file__))), "welcome-youtube_b200"))
import oercel_b200 as ob  # noqa: E402
from oercel_b200 import _capi, autograd, cells, workloads  # noqa: E402

NEIGHBOURS = math.pi / 2.0  # half the cutoff disk: pairs per bead and unit density


# ---------------------------------------------------------------- the cases

def listed():
    return [
        # the reference engine's own small box (L = 32, 4,096 beads), a stats interval of 100 steps
        dict(name="run_4k", kind="run", L=32.0, rho=4.0, physics="bench", chem="off", noise="philox", steps=100),
        # an ordinary box of the reference's default physics (chains of four with angle terms), stirred, with the
        # temperature cycle, the reference's pair hash and an odd side; a stats row every step
        dict(name="run_31k_stirred", kind="run", L=101.7, rho=3.0, physics="reference", chem="off", noise="mix13",
             steps=100),
        # the 1,048,576-bead box with the lipid chemistry every step
        dict(name="run_1M_lipid", kind="run", L=512.0, rho=4.0, physics="bench", chem="lipid", noise="philox",
             steps=20),
        # the ensemble: 256 replicas of 2,048 to 65,536 beads, perturbed repulsions and rates
        dict(name="ensemble_256", kind="ensemble", replicas=256, nmin=2048, nmax=65536, steps=20),
        # the catalyst chemistry of the big-soup experiment on a quarter of its box, two checks
        dict(name="catalyst_197k", kind="catalyst", L=256.0, steps=20),
        # one force evaluation of a given configuration
        dict(name="forces_262k", kind="forces", L=256.0, rho=4.0),
        # one force VJP of a given configuration
        dict(name="vjp_66k", kind="vjp", L=128.0, rho=4.0),
        # the differentiated fit's box (16,384 beads), 200-step window, checkpoints every 20 steps, the gradient
        # truncated at 20 steps
        dict(name="fit_16k", kind="fit", L=64.0, replicas=1, steps=200, ckpt=20, last=50, horizon=20, state=False),
        # the gradient with respect to the start state too, through a short window
        dict(name="fit_4k_state", kind="fit", L=32.0, replicas=1, steps=20, ckpt=10, last=5, horizon=0, state=True),
        # the batched fit: 24 boxes of 65,536 beads, a 250-step window, checkpoints every 25 steps
        dict(name="fit_24x66k", kind="fit", L=128.0, replicas=24, steps=250, ckpt=25, last=50, horizon=20,
             state=False),
        # the measures of a large configuration between steps
        dict(name="analysis_786k", kind="analysis", L=512.0, rho=3.0),
        # cell detection in a snapshot of 49 vesicles in water
        dict(name="cells_L252", kind="cells", side=7),
    ]


def _log(rng, lo, hi):
    return math.exp(rng.uniform(math.log(lo), math.log(hi)))


def _side(rng, lo, hi, rho):
    """a box side for a bead count spread over the logarithm of lo..hi: whole or odd"""
    L = math.sqrt(_log(rng, lo, hi) / rho)
    return float(round(L)) if rng.random() < 0.3 else round(L, 3)


def draw(rng):
    kind = rng.choice(["run", "run", "run", "ensemble", "catalyst", "forces", "vjp", "fit", "fit", "analysis", "cells"])
    if kind == "run":
        rho = rng.choice([3.0, 4.0])
        L = _side(rng, 2000, 1_000_000, rho)
        n = rho * L * L
        return dict(kind=kind, L=L, rho=rho, physics=rng.choice(["bench", "bench", "reference"]),
                    chem=rng.choice(["off", "lipid"]), noise=rng.choice(["philox", "philox", "mix13"]),
                    steps=int(max(10, min(150, _log(rng, 10, 150), 2e7 / n))))
    if kind == "ensemble":
        r = int(_log(rng, 4, 256))
        return dict(kind=kind, replicas=r, nmin=2048, nmax=int(_log(rng, 4096, 65536)), steps=rng.randint(5, 20))
    if kind == "catalyst":
        return dict(kind=kind, L=_side(rng, 20_000, 700_000, 3.0), steps=10 * rng.randint(1, 3))
    if kind in ("forces", "vjp"):
        rho = rng.choice([3.0, 4.0])
        return dict(kind=kind, L=_side(rng, 2000, 262_000 if kind == "forces" else 140_000, rho), rho=rho)
    if kind == "fit":
        if rng.random() < 0.4:
            steps = rng.randint(5, 20)
            return dict(kind=kind, L=_side(rng, 2000, 16_000, 4.0), replicas=1, steps=steps, ckpt=rng.randint(5, 20),
                        last=rng.randint(1, 5), horizon=0, state=True)
        steps = rng.randint(60, 200)
        return dict(kind=kind, L=_side(rng, 4000, 60_000, 4.0), replicas=int(_log(rng, 1, 16)), steps=steps,
                    ckpt=rng.randint(10, 40), last=rng.randint(20, 50), horizon=20, state=False)
    if kind == "analysis":
        return dict(kind=kind, L=_side(rng, 10_000, 786_000, 3.0), rho=3.0)
    return dict(kind=kind, side=rng.randint(2, 7))


# ---------------------------------------------------------------- inputs made by torch alone

def _config(case, seed):
    """A liquid of H-T-T lipids (15 % of the beads), precursors (5 %) and water at density rho, as dense as a run's own:
    the beads sit on a jittered lattice, a lipid on three neighbouring sites, in a random order of bead numbers; float32
    positions in [0, L), unit normal velocities, types, links in bead order, all on the GPU, from the seed alone."""
    L = float(np.float32(case["L"]))
    n = int(round(case["rho"] * case["L"] * case["L"]))
    g = torch.Generator(device="cuda").manual_seed(seed)

    def normal(*s):
        return torch.randn(*s, generator=g, device="cuda", dtype=torch.float32)

    m = math.isqrt(n - 1) + 1
    site = torch.arange(n, device="cuda")
    p = torch.stack([site // m, site % m], 1).float() * (L / m) + normal(n, 2) * (0.2 * L / m)
    p = torch.remainder(p.double(), L).float()
    p[p >= L] = 0.0
    v = normal(n, 2)
    v = v - v.mean(0)
    blocks = torch.randperm(n // 3, generator=g, device="cuda")[:int(0.15 * n) // 3]
    part = torch.full((n,), -1, device="cuda")  # place in the lipid, -1 none
    for k in range(3):
        part[3 * blocks + k] = k
    t = torch.where(part < 0, 0, torch.where(part == 0, 1, 2))
    free = torch.nonzero(part < 0)[:, 0]
    t[free[torch.randperm(len(free), generator=g, device="cuda")[:int(0.05 * n)]]] = 3
    bead = torch.randperm(n, generator=g, device="cuda")  # bead number of each site
    at = torch.argsort(bead)                              # site of each bead
    prev = torch.where(part > 0, bead[(site - 1).clamp(min=0)], -1)
    nxt = torch.where((part >= 0) & (part < 2), bead[(site + 1).clamp(max=n - 1)], -1)
    cot = normal(n, 2)
    c = dict(x=p[at, 0], y=p[at, 1], vx=v[:, 0], vy=v[:, 1], type=t[at].to(torch.uint8), prev=prev[at].int(),
             next=nxt[at].int(), gx=cot[:, 0], gy=cot[:, 1])
    return {k: a.contiguous() for k, a in c.items()}


def _load(eng, c):
    """a configuration in device tensors into replica 0"""
    torch.cuda.synchronize()
    _capi.check(eng.lib.dpd_set_state(eng.h, 0, *[_capi.ptr(c[k]) for k in ("x", "y", "vx", "vy", "type")], None,
                                      _capi.ptr(c["prev"]), _capi.ptr(c["next"])))


FIELDS = ("x", "y", "vhx", "vhy", "vtx", "vty", "fx", "fy", "type", "gid", "prev", "next")


def _buffers(n):
    """device tensors for the state of n beads"""
    b = {k: torch.zeros(n, dtype=torch.float32, device="cuda") for k in FIELDS[:8]}
    b["type"] = torch.zeros(n, dtype=torch.uint8, device="cuda")
    b.update({k: torch.zeros(n, dtype=torch.int32, device="cuda") for k in FIELDS[9:]})
    return b


def _read(eng, r, buf, at=0, fields=FIELDS):
    """replica r's state into the tensors of buf from bead `at` on (fields left out are not read)"""
    p = [buf[k].data_ptr() + at * buf[k].element_size() if k in fields else None for k in FIELDS]
    _capi.check(eng.lib.dpd_get_state(eng.h, r, *p))


# ---------------------------------------------------------------- prepare

def _params(case, seed):
    if case.get("physics") == "reference":  # the reference's defaults, stirred, with a temperature cycle
        kv = dict(L=case["L"], rho=case["rho"], f_Ka=0, warmup=200, stir_A=0.02, stir_n=2, kT_amp=0.1, kT_period=50)
    else:
        kv = dict(workloads.PHYSICS, L=case["L"], rho=case.get("rho", 4.0))
    kv.update(seed=seed, noise=case.get("noise", "philox"))
    kv.update(workloads.CHEMISTRY if case.get("chem") == "lipid" else dict(chem=0))
    return ob.Params(**kv)


def _started(params, steps, n_beads=None):
    """an engine on the soups of params, past their hot start"""
    eng = ob.Engine(params, n_beads)
    for r in range(eng.nrep):
        eng.load_soup(r)
    eng.prime()
    eng.step(steps)
    return eng


class _Log:
    """pinned host memory for the events and stats rows a driver reads as the run goes on"""

    def __init__(self, eng, rows):
        rec = ob.Engine.EVENT_DTYPE
        self.events = torch.zeros((1 << 16) * rec.itemsize, dtype=torch.uint8, pin_memory=True).numpy().view(rec)
        self.count = torch.zeros(1, dtype=torch.int32, pin_memory=True).numpy()
        self.ring = None
        if rows:
            self.ring = torch.zeros(rows, 16, dtype=torch.int64, pin_memory=True).numpy().view(np.uint64)
            eng.stats_ring(0, self.ring)


def prepare(case, seed):
    kind = case["kind"]
    if kind == "run":
        eng = _started(_params(case, seed), 240 if case["physics"] == "reference" else 40)
        return dict(kind=kind, eng=eng, steps=case["steps"], log=_Log(eng, case["steps"]), chem=case["chem"],
                    buf=_buffers(eng.n_beads[0]))
    if kind == "ensemble":
        reps = workloads.config3(case["replicas"], nmin=case["nmin"], nmax=case["nmax"])
        for b, (p, _) in enumerate(reps):
            p.set("seed", str(1000 * seed + b))
        eng = _started([p for p, _ in reps], 20, [n for _, n in reps])
        return dict(kind=kind, eng=eng, steps=case["steps"], log=_Log(eng, 0), buf=_buffers(sum(eng.n_beads)))
    if kind == "catalyst":
        eng = _started(workloads.catalyst_plan(seed=seed, L=case["L"]), 40)
        return dict(kind=kind, eng=eng, steps=case["steps"], log=_Log(eng, 0), buf=_buffers(eng.n_beads[0]))
    if kind == "forces" or kind == "vjp":
        eng = ob.Engine(_params(case, seed))
        c = _config(case, seed)
        _load(eng, c)
        eng.build_cells()
        buf = _buffers(eng.n_beads[0])
        _read(eng, 0, buf)
        torch.cuda.synchronize()
        s = dict(kind=kind, eng=eng, buf=buf)
        if kind == "vjp":
            at = buf["gid"].long()
            s.update(g=(c["gx"][at], c["gy"][at]), out=[torch.empty_like(c["gx"]) for _ in range(4)],
                     grad=torch.zeros(_capi.NGRAD, dtype=torch.float64, device="cuda"),
                     stream=torch.cuda.ExternalStream(eng.stream()))
            torch.cuda.synchronize()
        return s
    if kind == "fit":
        rng = np.random.default_rng(seed)
        ps = [_params(dict(L=case["L"]), 1000 * seed + r) for r in range(case["replicas"])]
        for p in ps:
            p.set("f_lip", repr(float(rng.uniform(0.1, 0.3))))
        eng = _started(ps, 60)
        nb = 64
        spec = ob.Engine.rdf_spec(nbin=nb, rmax=2.0, sigma=0.05, last_steps=case["last"], horizon=case["horizon"])
        r = (np.arange(nb) + 0.5) * 2.0 / nb
        cfg = autograd.WindowConfig(eng, case["steps"], spec, 1.0 - np.exp(-(r / 0.6) ** 2), ckpt=case["ckpt"])
        a0, g0, k0 = autograd.engine_values(eng)
        leaf = [v.float().requires_grad_() for v in (a0[:4, :4].contiguous(), g0, k0)]
        s = dict(kind=kind, cfg=cfg, leaf=leaf, start=[])
        if case["state"]:
            st = eng.state(0)
            for k in (("x", "y"), ("vhx", "vhy"), ("vtx", "vty")):
                v = np.empty((eng.n_beads[0], 2), np.float32)
                v[st["gid"].astype(np.int64)] = np.stack([st[k[0]], st[k[1]]], 1)
                s["start"].append(torch.from_numpy(v).requires_grad_())
        return s
    if kind == "analysis":
        kv = dict(L=case["L"], rho=case["rho"], seed=seed, f_Ka=0, f_lip=0.25, warmup=200, chem=0)
        eng = _started(ob.Params(**kv), 300)
        return dict(kind=kind, eng=eng)
    return dict(kind=kind, snap=_vesicles(case["side"], seed))


def _vesicles(side, seed):
    """A snapshot of side x side vesicles (closed bilayers of H-T-T-T lipids, radii 5 to 12, every fifth with a smaller
    one inside) at jittered places in water with nutrients, catalysts and free lipids, on the host."""
    rng = np.random.default_rng(seed)
    pitch, L = 36.0, 36.0 * side
    rings = []
    for k in range(side * side):
        c = np.array([k // side, k % side]) * pitch + rng.uniform(-3.0, 3.0, 2)
        r = 5.0 + 7.0 * (0.618 * k % 1.0)
        rings.append((c, r))
        if r > 10.5:
            rings.append((c, 4.8))
    pos, lip = [], 0
    for c, r in rings:
        for s in (1.0, -1.0):
            rr = r + 1.65 * s
            k = max(int(2.0 * math.pi * rr / 0.62), 6)
            a = rng.uniform(0.0, 2.0 * math.pi) + 2.0 * math.pi * np.arange(k) / k
            u = np.stack([np.cos(a), np.sin(a)], 1)
            pos.append(np.stack([c + (rr - 0.5 * s * q) * u for q in range(4)], 1).reshape(-1, 2))
            lip += k
    free = 10 * side * side
    u = rng.normal(size=(free, 2))
    u /= np.linalg.norm(u, axis=1)[:, None]
    c = rng.uniform(0.0, L, (free, 2))
    pos.append(np.stack([c + 0.5 * q * u for q in range(4)], 1).reshape(-1, 2))
    lip += free
    w = rng.uniform(0.0, L, (int(3.6 * L * L), 2))
    keep = np.ones(len(w), bool)
    for c, r in rings:
        d = np.abs(w - c)
        d = np.minimum(d % L, L - d % L)
        keep &= np.abs(np.hypot(d[:, 0], d[:, 1]) - r) >= 1.95
    w = w[keep][:int(2.7 * L * L)]
    p = np.concatenate(pos + [w])
    p[:4 * lip] += rng.normal(0.0, 0.05, (4 * lip, 2))
    p = (p % L).astype(np.float32)
    p[p >= np.float32(L)] = 0.0
    t = np.concatenate([np.tile(np.array([1, 2, 2, 2], np.uint8), lip),
                        rng.choice(np.array([0, 3, 4, 5, 6], np.uint8), len(w), p=[0.92, 0.05, 0.01, 0.01, 0.01])])
    i = np.arange(4 * lip).reshape(-1, 4)
    b = np.stack([i[:, :3].ravel(), i[:, 1:].ravel()], 1).astype(np.int64)
    return cells.Snapshot(0, 0.0, L, p[:, 0].astype(np.float64), p[:, 1].astype(np.float64), t, b)


# ---------------------------------------------------------------- run

def run(s):
    kind = s["kind"]
    if kind == "run":
        eng, log = s["eng"], s["log"]
        eng.step_async(s["steps"])
        if s["chem"] == "lipid":
            eng.events_async(log.events, log.count)
        eng.sync()
        _read(eng, 0, s["buf"])
        row = eng.stats_decode(0, log.ring[eng.step_no % len(log.ring)])
        return dict(s["buf"], T=row["T"], px=row["px"], py=row["py"], maxbond=row["maxbond"],
                    n_chains=row["n_chains"], counts=row["counts"])
    if kind in ("ensemble", "catalyst"):
        eng, log = s["eng"], s["log"]
        eng.step_async(s["steps"])
        eng.events_async(log.events, log.count)
        eng.sync()
        at = 0
        for r, n in enumerate(eng.n_beads):
            _read(eng, r, s["buf"], at)
            at += n
        return s["buf"]
    if kind == "forces":
        s["eng"].forces(7)
        _read(s["eng"], 0, s["buf"], fields=("fx", "fy", "gid"))
        return {k: s["buf"][k] for k in ("fx", "fy", "gid")}
    if kind == "vjp":
        eng = s["eng"]
        _capi.check(eng.lib.dpd_force_vjp(eng.h, 0, 7, *[_capi.ptr(v) for v in s["g"]], *[_capi.ptr(v) for v in s["out"]],
                                          _capi.ptr(s["grad"])))
        with torch.cuda.stream(s["stream"]):  # the parameters' gradient in their own precision
            grad = s["grad"].float()
        return dict(xbar_x=s["out"][0], xbar_y=s["out"][1], vbar_x=s["out"][2], vbar_y=s["out"][3], grad=grad)
    if kind == "fit":
        for v in s["leaf"] + s["start"]:
            v.grad = None
        loss = autograd.window_loss(s["cfg"], *s["leaf"], *s["start"])
        loss.sum().backward()
        return dict(loss=loss.detach(), grad=[v.grad for v in s["leaf"]], start_grad=[v.grad for v in s["start"]])
    if kind == "analysis":
        eng = s["eng"]
        o = eng.observables(0)
        g = eng.aggregates(0, labels=True)
        return dict(obs=o, tails=eng.type_clusters(0, 2, 1.0), agg=g, rdf=eng.pair_hist(0, -1, -1, 3.0, 30),
                    rdf_tails=eng.pair_hist(0, 2, 2, 3.0, 30))
    d = cells.detect(s["snap"])
    keys = ("x", "y", "area", "n_lipids", "n_N", "n_W", "agg", "inner_heads", "outer_heads", "aspect", "solidity",
            "extent", "exposure")
    return dict(cells=np.array([[float(c[k]) for k in keys] for c in d["cells"]]).reshape(-1, len(keys)),
                label=d["label"], bead_cell=d["bead_cell"], mol=d["mol"], bead_agg=d["bead_agg"], summary=d["summary"])


# ---------------------------------------------------------------- work

def work(case):
    """Bytes: each pass over the beads (a step, a force evaluation) reads its state once (positions, velocities, types,
    links: 36 bytes) and writes it once; flops: the pairs inside the cutoff (60 operations each, 150 with
    their derivative) and 40 a bead."""
    kind = case["kind"]
    if kind == "cells":
        n = 3.4 * (36.0 * case["side"]) ** 2
        return dict(bytes=40.0 * n, flops=60.0 * n)
    rho = case.get("rho", 3.0 if kind == "catalyst" else 4.0)
    if kind == "ensemble":
        n = case["replicas"] * (case["nmax"] - case["nmin"]) / math.log(case["nmax"] / case["nmin"])
    else:
        n = rho * case["L"] ** 2 * case.get("replicas", 1)
    pair = NEIGHBOURS * rho
    if kind in ("run", "ensemble", "catalyst"):
        return dict(bytes=(case["steps"] * 72.0 + 45.0) * n, flops=case["steps"] * n * (60.0 * pair + 40.0))
    if kind == "forces":
        return dict(bytes=40.0 * n, flops=n * (60.0 * pair + 40.0))
    if kind == "vjp":
        return dict(bytes=52.0 * n, flops=n * (150.0 * pair + 40.0))
    if kind == "fit":
        back = case["steps"] if not case["horizon"] else min(case["steps"], case["last"] + case["horizon"])
        return dict(bytes=n * 72.0 * (case["steps"] + 2.0 * back),
                    flops=n * ((60.0 * pair + 40.0) * (case["steps"] + back) + 190.0 * pair * back))
    return dict(bytes=90.0 * n, flops=n * 9.0 * pair * 20.0)  # analysis


# ---------------------------------------------------------------- exact values in 64 bits

def _philox(c0, c1, c2, c3, k0, k1):
    """Philox4x32-10 (Salmon, Moraes, Dror, Shaw, SC'11), first output word, on int64 tensors of 32-bit values"""
    m = 0xFFFFFFFF

    def mul(a, b):  # 32 x 32 -> (high, low) with no 64-bit overflow
        ah, al, bh, bl = a >> 16, a & 0xFFFF, b >> 16, b & 0xFFFF
        t = al * bl
        u = ah * bl + (t >> 16)
        v = al * bh + (u & 0xFFFF)
        return ah * bh + (u >> 16) + (v >> 16), ((v & 0xFFFF) << 16) | (t & 0xFFFF)

    for r in range(10):
        h0, l0 = mul(c0, 0xD2511F53)
        h1, l1 = mul(c2, 0xCD9E8D57)
        c0, c1, c2, c3 = (h1 ^ c1 ^ k0) & m, l1, (h0 ^ c3 ^ k1) & m, l0
        k0, k1 = (k0 + 0x9E3779B9) & m, (k1 + 0xBB67AE85) & m
    return c0


def _pairs(x, y, L):
    """all pairs i < j closer than 1 (minimum image), from strips of one cutoff width"""
    ns = int(L)
    strip = torch.clamp((x * (ns / L)).long(), max=ns - 1)
    order = torch.argsort(strip, stable=True)
    at = torch.searchsorted(strip[order].contiguous(), torch.arange(ns + 1, device=x.device))
    at = at.tolist()
    ii, jj = [], []
    for c in range(ns):
        a = order[at[c]:at[c + 1]]
        d = (c + 1) % ns
        b = torch.cat([a, order[at[d]:at[d + 1]]])
        dx, dy = x[a][:, None] - x[b][None], y[a][:, None] - y[b][None]
        dx, dy = dx - L * torch.round(dx / L), dy - L * torch.round(dy / L)
        r2 = dx * dx + dy * dy
        hit = (r2 < 1.0) & (r2 > 1e-24)
        na = len(a)
        hit[:, :na] &= torch.ones(na, na, dtype=torch.bool, device=x.device).triu(1)
        p, q = torch.nonzero(hit, as_tuple=True)
        ii.append(a[p])
        jj.append(b[q])
    i, j = torch.cat(ii), torch.cat(jj)
    return torch.minimum(i, j), torch.maximum(i, j)


def exact(case, seed):
    kind = case["kind"]
    if kind not in ("forces", "vjp"):
        return None  # whole runs and windows: chaotic trajectories; the analyses give counts
    c = _config(case, seed)
    L = float(np.float32(case["L"]))
    x, y, vx, vy = (c[k].double() for k in ("x", "y", "vx", "vy"))
    n = len(x)
    i, j = _pairs(x, y, L)
    q = workloads.PHYSICS
    a = torch.full((8, 8), 25.0, dtype=torch.float64, device="cuda")
    for k, (s, t) in dict(a_W_H=(0, 1), a_W_T=(0, 2), a_H_T=(1, 2), a_W_P=(0, 3), a_H_P=(1, 3), a_P_T=(3, 2)).items():
        a[s, t] = a[t, s] = q[k]
    z = torch.zeros_like(i)
    u = _philox(i, j, z + 7, z, torch.full_like(i, seed & 0xFFFFFFFF), torch.full_like(i, seed >> 32))
    u = torch.where(u >= 1 << 31, u - (1 << 32), u)
    theta = u.double() * (math.sqrt(12.0) / 2.0 ** 32)
    X = torch.stack([x, y], 1)
    V = torch.stack([vx, vy], 1)
    up = torch.triu(a).requires_grad_()
    gam = torch.tensor(float(q["gamma"]), dtype=torch.float64, device="cuda", requires_grad=True)
    kb = torch.tensor(float(q["k_bond"]), dtype=torch.float64, device="cuda", requires_grad=True)
    if kind == "vjp":
        X.requires_grad_()
        V.requires_grad_()
    t = c["type"].long()
    ti, tj = torch.minimum(t[i], t[j]), torch.maximum(t[i], t[j])

    def image(d):
        return d - L * torch.round(d.detach() / L)

    d = image(X[i] - X[j])
    r = d.square().sum(1).sqrt()
    w = 1.0 - r
    rv = (d * (V[i] - V[j])).sum(1) / r
    sdt = torch.sqrt(2.0 * gam * q["kT"]) / math.sqrt(q["dt"])
    fm = w * (up[ti, tj] - gam * w * rv + sdt * theta) / r
    F = torch.zeros_like(X).index_add(0, i, fm[:, None] * d).index_add(0, j, -fm[:, None] * d)
    m = torch.nonzero(c["next"] >= 0)[:, 0]
    o = c["next"][m].long()
    b = image(X[o] - X[m])
    rb = b.square().sum(1).sqrt()
    fb = (kb * (1.0 - q["r0"] / rb))[:, None] * b
    F = F.index_add(0, m, fb).index_add(0, o, -fb)
    nc = int(L)
    cx, cy = (torch.clamp((v * (nc / L)).long(), 0, nc - 1) for v in (x, y))
    slot = torch.argsort(cx * nc + cy, stable=True)
    if kind == "forces":
        F = F.detach()[slot]
        return dict(fx=F[:, 0], fy=F[:, 1], gid=None)
    G = torch.stack([c["gx"], c["gy"]], 1).double()
    gx, gv, ga, gg, gk = torch.autograd.grad((F * G).sum(), [X, V, up, gam, kb])
    return dict(xbar_x=gx[slot, 0], xbar_y=gx[slot, 1], vbar_x=gv[slot, 0], vbar_y=gv[slot, 1],
                grad=torch.cat([ga.reshape(-1), gg[None], gk[None]]))
