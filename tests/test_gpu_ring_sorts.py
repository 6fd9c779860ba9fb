"""The stats ring over the kernels that collect its rows (the sort from bins in
one kernel and in two, the prefix sort's fix-up, a kernel of its own before the
other sorts, the end of a call), with stirring, whose sums the same kernels
clear: the rows of dpd_stats_async after each step of a run without a ring."""
import numpy as np
import pytest

import oercel_b200 as ob
from gpu_util import params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,rho,mode", [
    (24.0, 4.0, 2), (190.0, 3.0, 2), (445.0, 3.0, 2), (24.0, 11.0, 2), (24.0, 4.0, 0), (24.0, 4.0, 1)])
def test_rows_of_each_sort(cuda_ok, L, rho, mode):
    import torch
    kv = dict(dt=0.01, noise="philox", stir_A=0.3, f_lip=0.3)
    ps = [params(L=L, rho=rho, seed=6, **kv), params(L=11.0, rho=rho, seed=7, **kv)]
    a, b = ob.Engine(ps), ob.Engine(ps)
    for e in (a, b):
        e.set_tuning(sort_mode=mode)
        for r in range(2):
            e.load_soup(r)
        e.prime()
    ring = torch.zeros((8, 16), dtype=torch.int64, pin_memory=True).numpy().view(np.uint64)
    a.stats_ring(0, ring)
    a.set_graph_steps(2)
    b.set_graph_steps(1)
    for k in (1, 4, 3):
        a.step(k)
        rows = {int(r[6]): r.copy() for r in ring}
        for _ in range(k):
            b.step(1)
            raw = np.zeros(16, np.uint64)
            b.stats_async(0, raw)
            b.sync()
            got = rows[b.step_no]
            got[6] = 0
            assert np.array_equal(got, raw), b.step_no
    for r in range(2):
        u, v = a.state(r), b.state(r)
        for k in ("x", "y", "vhx", "fx", "fy", "gid"):
            assert np.array_equal(u[k], v[k]), k
