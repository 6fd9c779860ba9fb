"""The force VJP over the box sizes its kernel splits differently (eight, four
and two lanes a bead), on three-cell and odd boxes, crowded cells (lists past
their capacity) and all eight types: against torch autograd of an all-pairs
FP64 model of the same forces, noise included."""
import ctypes as C

import numpy as np
import pytest

import oracle as O
import oercel_b200 as ob
from gpu_util import engine_with, links_from_next, oracle_params, params

pytestmark = pytest.mark.gpu


def box(L, n, types, seed, crowd):
    """beads on jittered lattices (no pair so close that FP32 decides), the first
    third in one corner when crowded; chains of three neighbouring sites"""
    rng = np.random.default_rng(seed)

    def lattice(k, side):
        m = int(np.ceil(np.sqrt(k)))
        i = np.arange(k)
        return (np.stack([i // m, i % m]) + 0.5 + rng.uniform(-0.25, 0.25, (2, k))) * (side / m)

    k = n // 3 if crowd else 0
    x, y = np.concatenate([lattice(k, 1.3), lattice(n - k, L)], 1) if k else lattice(n, L)
    nxt = np.full(n, -1, np.int32)
    for q in range(0, n // 10 * 3, 6):
        nxt[q], nxt[q + 1] = q + 1, q + 2
    f = lambda v: np.where(v.astype(np.float32) >= np.float32(L), 0, v).astype(np.float32)
    return f(x), f(y), rng.normal(size=(2, n)).astype(np.float32), rng.choice(types, n), nxt


def theta(p, step, gi, gj):
    """the oracle's noise of each pair"""
    op, f = oracle_params(p), O.lib().ora_theta
    return np.array([f(C.byref(op), step, int(a), int(b)) for a, b in zip(gi, gj)])


@pytest.mark.parametrize("L,n,types,crowd", [
    (3.0, 40, (0, 1, 2, 3), False), (7.3, 220, range(8), False), (9.0, 300, (0, 2), True),
    (60.3, 14500, (0, 1, 2, 3), False), (100.0, 40100, (0, 1, 2, 3, 5), False)])
def test_vjp_equals_autograd(cuda_ok, L, n, types, crowd):
    import torch
    p = params(L=L, seed=5, noise="philox")
    Lf = float(np.float32(L))
    x, y, v, t, nxt = box(Lf, n, np.array(list(types), np.uint8), 11, crowd)
    e = engine_with(p, x, y, v[0], v[1], t, *links_from_next(nxt))
    e.build_cells()
    s = e.state(0)
    step = 3
    rng = np.random.default_rng(1)
    g = rng.normal(size=(2, n)).astype(np.float32)
    got = e.force_vjp(0, step, g[0], g[1])
    D = lambda a: torch.tensor(np.asarray(a, np.float64), device="cuda")
    X = D(np.stack([s["x"], s["y"]], 1)).requires_grad_()
    V = D(np.stack([s["vtx"], s["vty"]], 1)).requires_grad_()
    A = D(np.array(p.a)).requires_grad_()
    gam, kb = D(p.gamma).requires_grad_(), D(p.k_bond).requires_grad_()
    image = lambda d: d - Lf * torch.round(d.detach() / Lf)
    ii, jj = [], []  # all pairs inside the cutoff, in blocks of rows
    with torch.no_grad():
        for a in range(0, n, 2048):
            d = image(X[a:a + 2048, None] - X[None])
            r2 = d.square().sum(2)
            i, j = torch.nonzero((r2 < 1.0) & (r2 > 1e-24), as_tuple=True)
            m = i + a < j
            ii.append(i[m] + a)
            jj.append(j[m])
    i, j = torch.cat(ii), torch.cat(jj)
    gid = s["gid"].astype(np.uint32)
    hi, hj = i.cpu().numpy(), j.cpu().numpy()
    th = D(theta(p, step, gid[hi], gid[hj]))
    T = torch.tensor(s["type"].astype(np.int64), device="cuda")
    lo, up = torch.minimum(T[i], T[j]), torch.maximum(T[i], T[j])
    d = image(X[i] - X[j])
    r = d.square().sum(1).sqrt()
    w = 1 - r
    rv = (d * (V[i] - V[j])).sum(1) / r
    sdt = torch.sqrt(2 * gam * p.kT) / p.dt ** 0.5
    fm = w * (A[lo, up] - gam * w * rv + sdt * th) / r
    F = torch.zeros_like(X).index_add(0, i, fm[:, None] * d).index_add(0, j, -fm[:, None] * d)
    m = torch.tensor(np.nonzero(s["next"] >= 0)[0], device="cuda")
    o = torch.tensor(s["next"][s["next"] >= 0].astype(np.int64), device="cuda")
    b = image(X[o] - X[m])
    rb = b.square().sum(1).sqrt()
    fb = (kb * (1 - p.r0 / rb))[:, None] * b
    F = F.index_add(0, m, fb).index_add(0, o, -fb)
    want = torch.autograd.grad((F * D(g.T)).sum(), [X, V, A, gam, kb])
    # a bead sums a dozen FP32 terms of up to its largest size: 2e-5 of the largest sum
    for q, w_ in ((0, want[0]), (2, want[1])):
        w_ = w_.cpu().numpy()
        for c in range(2):
            assert np.abs(got[q + c] - w_[:, c]).max() < 2e-5 * np.abs(w_[:, c]).max()
    # the parameters' sums: FP32 terms (a few roundings each, 6e-8) added in FP64, so 1e-6 of the terms' sizes
    with torch.no_grad():
        G = D(g.T)
        cd = ((G[i] - G[j]) * d).sum(1) / r
        sa = float((cd * w).abs().sum())
        sg = float((cd * w * (w * rv).abs()).abs().sum() + (cd * w * sdt * th / (2 * gam)).abs().sum())
        sk = float(((G[m] - G[o]) * b).sum(1).abs().sum())
    assert np.abs(got[4][:64].reshape(8, 8) - np.triu(want[2].cpu().numpy())).max() < 1e-6 * sa
    assert abs(got[4][64] - float(want[3])) < 1e-6 * sg
    assert abs(got[4][65] - float(want[4])) < 1e-6 * sk
