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
