"""The sort from bins (k_binfix) against the placement sort over the sizes and
densities where its rules change: one kernel or two, cells of the last scan
block, rows of 4, 8, 16 and 32 beads, cells past their row, several replicas,
and the density where bins end.  Cell starts, order and a run must be the same
as with the two-pass scan and placement (sort_mode 0)."""
import numpy as np
import pytest

import oercel_b200 as ob
from gpu_util import params

pytestmark = pytest.mark.gpu
KEYS = ("x", "y", "vhx", "vhy", "vtx", "vty", "fx", "fy", "type", "gid", "prev", "next")


def crowd(L, rho, seed, spots):
    """a soup with `spots` cells of about 12, 20, 40 and 300 beads"""
    p = params(L=L, rho=rho, seed=seed)
    s = ob.soup_for(p)
    rng = np.random.default_rng(seed)
    n, at = len(s["x"]), 0
    free = np.nonzero((s["prev"] < 0) & (s["next"] < 0))[0]
    for k, m in zip(range(spots), (12, 20, 40, 300)):
        i = free[at:at + m]
        at += m
        c = rng.integers(0, int(L), 2)
        s["x"][i] = np.float32(c[0] + rng.uniform(0.02, 0.98, len(i)))
        s["y"][i] = np.float32(c[1] + rng.uniform(0.02, 0.98, len(i)))
    return p, s, n


def engine(ps, ss, mode):
    e = ob.Engine(ps, [len(s["x"]) for s in ss])
    e.set_tuning(sort_mode=mode)
    for r, s in enumerate(ss):
        e.set_state(r, s["x"], s["y"], s["vx"], s["vy"], s["type"], None, s["prev"], s["next"])
    return e


@pytest.mark.parametrize("L,rho,spots,reps", [
    (3.0, 4, 0, 1), (5.5, 9, 2, 3), (17.0, 4, 4, 2), (32.0, 10, 4, 1), (32.0, 10.2, 2, 1), (181.0, 3, 4, 1),
    (182.4, 3, 4, 1), (60.0, 4, 3, 10), (443.0, 3, 1, 1), (444.0, 3, 0, 1)])
def test_bins_equal_placement(cuda_ok, L, rho, spots, reps):
    ps, ss = zip(*[crowd(L + 0.3 * r, rho, 3 + r, spots)[:2] for r in range(reps)])
    a, b = engine(list(ps), list(ss), 2), engine(list(ps), list(ss), 0)
    for e in (a, b):
        e.build_cells()
    for r in range(reps):
        assert np.array_equal(a.cells(r), b.cells(r))
        u, v = a.state(r), b.state(r)
        for k in KEYS:
            assert np.array_equal(u[k], v[k]), (r, k)
    if spots < 3:  # (three hundred beads in a cell: forces past the fixed-point range)
        for e in (a, b):
            e.prime()
            e.step(1)
            e.step(6)
        for r in range(reps):
            u, v = a.state(r), b.state(r)
            for k in KEYS:
                assert np.array_equal(u[k], v[k]), (r, k)
            assert np.array_equal(a.cells(r), b.cells(r))
    # switching the mode between steps keeps the run
    if reps == 1 and spots < 3:
        a.set_tuning(sort_mode=1)
        a.step(2)
        a.set_tuning(sort_mode=2)
        a.step(3)
        b.step(5)
        u, v = a.state(0), b.state(0)
        for k in KEYS:
            assert np.array_equal(u[k], v[k]), k
