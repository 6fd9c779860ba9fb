"""The template forces of branched lipids where a chunk of 256 slots holds from
one first bead to 256 (the kernel takes 32 molecules at a time) and for the
shortest and longest molecules, against the oracle in FP64."""
import numpy as np
import pytest

import oracle as O
import oercel_b200 as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("arch,nT,tie,nmol", [
    ("y", 1, 0, 1),       # 3 beads, one molecule
    ("y", 1, 0, 33),      # one past a round
    ("y", 2, 1, 300),     # a chunk of first beads only, and more of them in the next
    ("bola", 6, 0, 64),   # 15 beads, whole rounds
    ("pi", 7, 2, 47),     # 16 beads, rungs
])
def test_molecules_per_chunk(cuda_ok, arch, nT, tie, nmol):
    L = 14.0
    p = ob.Params(L=L, lip_arch=arch, lip_nT=nT, lip_tie=tie, k_angle=5.0, k_head=3.0, cos_head=-0.5, f_Ka=0)
    t = p.template()
    ml = t.mlen
    n = nmol * ml + 5  # and five beads in no molecule
    rng = np.random.default_rng(nmol)
    ang = rng.uniform(0, 2 * np.pi, (nmol, 1))
    px, py = np.array(t.px[:ml]), np.array(t.py[:ml])
    bx = rng.uniform(0, L, (nmol, 1)) + np.cos(ang) * px - np.sin(ang) * py + rng.uniform(-0.1, 0.1, (nmol, ml))
    by = rng.uniform(0, L, (nmol, 1)) + np.sin(ang) * px + np.cos(ang) * py + rng.uniform(-0.1, 0.1, (nmol, ml))
    # slots: every molecule's first bead, then the other beads in a random order, the free ones among them
    slot = np.empty((nmol, ml), np.int64)
    slot[:, 0] = np.arange(nmol)
    rest = nmol + rng.permutation(n - nmol)
    slot[:, 1:] = rest[:nmol * (ml - 1)].reshape(nmol, ml - 1)
    x, y = (rng.uniform(0, L, n).astype(np.float32) for _ in range(2))
    x[slot], y[slot] = np.mod(bx, L), np.mod(by, L)
    top = np.nextafter(np.float32(L), np.float32(0))
    x, y = np.minimum(x, top), np.minimum(y, top)
    nxt, prev = np.full(n, -1, np.int32), np.full(n, -1, np.int32)
    nxt[slot[:, :-1]], prev[slot[:, 1:]] = slot[:, 1:], slot[:, :-1]
    typ = np.zeros(n, np.uint8)
    typ[slot[:, :t.nH]], typ[slot[:, t.nH:]] = 1, 2
    e = ob.Engine(p, n_beads=n)
    z = np.zeros(n, np.float32)
    e.set_state(0, x, y, z, z, typ, np.arange(n, dtype=np.uint32), prev, nxt)
    fx, fy, mb = e.bond_forces(0)
    op = O.params(L, np.full((8, 8), 25.0), k_bond=p.k_bond, r0=p.r0)
    fields = {k: list(getattr(t, k)[:m]) for k, m in (("bi", t.nb), ("bj", t.nb), ("br0", t.nb), ("ai", t.na),
                                                       ("aj", t.na), ("ak", t.na), ("akind", t.na), ("aK", t.na),
                                                       ("ac0", t.na))}
    ox, oy, omb = O.mol_forces(op, O.mol(dict(fields, mlen=ml, nb=t.nb, na=t.na)),
                               dict(x=x, y=y, next=nxt))
    scale = np.abs(np.stack([ox, oy])).max()
    assert np.abs(fx - ox).max() <= 1e-5 * scale and np.abs(fy - oy).max() <= 1e-5 * scale
    assert mb == pytest.approx(omb, rel=1e-6)
    assert fx.astype(np.float64).sum() == 0.0 and fy.astype(np.float64).sum() == 0.0
