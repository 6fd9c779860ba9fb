"""Condensed states: the same beads in a part of their box, at densities where
most cells hold more beads than their row of bins.  The sort from bins must give
the order of the placement sort, and not cost a multiple of it."""
import numpy as np
import pytest

import oercel_b200 as ob
from gpu_util import params

pytestmark = pytest.mark.gpu
KEYS = ("x", "y", "vhx", "vhy", "vtx", "vty", "fx", "fy", "gid")


def condensed(L, rho, local, mode=None, seed=3):
    """water at density `local` in a corner of an otherwise empty box; a small step keeps it there"""
    p = params(L=L, rho=rho, seed=seed, dt=0.001)
    rng = np.random.default_rng(seed)
    n = int(rho * L * L)
    x, y = (rng.uniform(0, L * (rho / local) ** 0.5, (2, n)) + 1.3).astype(np.float32) % np.float32(L)
    z = np.zeros(n, np.float32)
    e = ob.Engine(p, n_beads=n)
    if mode is not None:
        e.set_tuning(sort_mode=mode)
    e.set_state(0, x, y, z, z, z.astype(np.uint8), None, None, None)
    e.prime()
    return e


@pytest.mark.parametrize("L,rho,local", [(30.0, 4.0, 60.0), (190.0, 1.0, 40.0), (440.0, 4.0, 30.0)])
def test_bins_on_condensed_states(cuda_ok, L, rho, local):
    a, b = condensed(L, rho, local, 2), condensed(L, rho, local, 0)
    for e in (a, b):
        e.step(1)
        e.step(4)
    assert np.array_equal(a.cells(0), b.cells(0)) and np.diff(a.cells(0)).max() > 32
    u, v = a.state(0), b.state(0)
    for k in KEYS:
        assert np.array_equal(u[k], v[k]), k
    ms = [min(sum(e.profile_step()[:4]) for _ in range(5)) for e in (a, b)]
    assert ms[0] < 2.0 * ms[1], ms


@pytest.mark.parametrize("noise", ["philox", "mix13"])
@pytest.mark.parametrize("side,at,m", [
    (6.0, 5.0, 1600),    # a tile in parts
    (3.0, 11.0, 2200),   # parts of a row of cells
    (1.5, 9.3, 1500),    # cells that do not fit with their halos
    (5.0, -2.5, 1600),   # across both edges of the box
])
@pytest.mark.parametrize("shape", [(14, 14, 256), (6, 22, 256), (22, 6, 256), (1, 3, 256), (20, 20, 512)])
def test_crowded_tiles_in_parts(cuda_ok, shape, side, at, m, noise):
    """the same forces and next cells as a thread per bead gives"""
    L = 24.0
    p = params(L=L, seed=9, noise=noise)
    s = ob.soup_for(p)
    rng = np.random.default_rng(0)
    free = np.nonzero(s["prev"] + s["next"] == -2)[0][:m]
    for k in ("x", "y"):
        v = (at + rng.uniform(0.0, side, len(free))) % L
        s[k][free] = np.where(v.astype(np.float32) >= L, 0, v).astype(np.float32)
    runs = []
    for fk in (1, 0):
        e = ob.Engine(p)
        e.set_state(0, s["x"], s["y"], 0 * s["vx"], 0 * s["vy"], s["type"], None, s["prev"], s["next"])
        e.set_tuning(force_kernel=fk, **(dict(tile_w=shape[0], tile_h=shape[1], tile_threads=shape[2]) if fk == 0 else {}))
        e.build_cells()
        e.forces(5)
        runs.append(e.state())
    for k in ("fx", "fy"):
        assert np.array_equal(runs[0][k], runs[1][k])


def test_crowded_tiles_cost_no_multiple(cuda_ok):
    """density 6 in a corner of a box of mean density 2: its default tiles are too large for that, 8 x 16 are not"""
    e = condensed(440.0, 2.0, 6.0)
    own = min(e.profile_step()[-1] for _ in range(5))
    e.set_tuning(tile_w=8, tile_h=16)
    small = min(e.profile_step()[-1] for _ in range(5))
    assert own < 3.0 * small, (own, small)
