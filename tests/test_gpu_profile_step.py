"""dpd_profile_step is a real step in every form of the cell sort: the same
state as dpd_step's, on a box of each form, one past the cells that block
prefixes hold included (there sort_mode 2 is the scan in two passes)."""
import numpy as np
import pytest

import oercel_b200 as ob
from gpu_util import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,n,mode,sort", [
    (40.0, 6400, 0, 4), (40.0, 6400, 1, 3), (40.0, 6400, 2, 1), (190.0, 90000, 2, 2), (40.0, 20000, 2, 3),
    (2049.0, 20000, 2, 4)])
def test_profiled_steps_are_steps(cuda_ok, L, n, mode, sort):
    rng = np.random.default_rng(7)
    x, y = rng.uniform(0, L, (2, n)).astype(np.float32) % np.float32(L)
    vx, vy = rng.normal(size=(2, n)).astype(np.float32)
    p = params(L=L, seed=3)
    got = []
    for profiled in (True, False):
        e = ob.Engine(p, n_beads=n)
        e.set_tuning(sort_mode=mode)
        e.set_state(0, x, y, vx, vy, rng.integers(0, 1, n).astype(np.uint8), None, None, None)
        e.prime()
        for _ in range(3):
            if profiled:
                ms = e.profile_step()
                assert (np.asarray(ms[:4]) > 0.0).sum() >= sort
            else:
                e.step(1)
        assert e.kernels_per_step()[0] == sort + 2
        got.append((e.state(0), e.cells(0), e.step_no))
    (s, c, k), (t, d, m) = got
    assert k == m and np.array_equal(c, d)
    for q in s:
        assert np.array_equal(s[q], t[q]), q
