"""The storage of differentiated windows stays within what its rule allows: the
larger of what the intervals of the handle's windows asked for and the limit
set, and the scratch, however the windows' shapes change."""
import numpy as np
import pytest

import oercel_b200 as ob
from gpu_util import params

pytestmark = pytest.mark.gpu

L, SLACK = 128.0, 6 << 20  # (the allocator's granularity)


def asked(n, c, nsteps, ckpt):
    """a checkpoint every ckpt steps, ckpt configurations: 44 and 32 bytes a bead, 4 a cell, each array's padding"""
    k = -(-nsteps // ckpt)
    return n * (44 * k + 32 * ckpt) + (4 * c + 7 * 320) * (k + ckpt)


@pytest.mark.parametrize("limit", [0, 100 << 20])
@pytest.mark.parametrize("windows", [
    [(100, 10, 2), (24, 24, 2), (60, 1, 2)], [(60, 1, 2), (24, 24, 2)], [(40, 40, 40), (400, 20, 100)]])
def test_storage_within_the_limit(cuda_ok, limit, windows):
    import torch
    e = ob.Engine(params(L=L, seed=3))
    e.load_soup(0)
    e.prime()
    n, c = e.n_beads[0], len(e.cells(0)) - 1

    def run(nsteps, ckpt, last):
        spec = e.rdf_spec(ta=2, tb=2, nbin=40, rmax=2.0, sigma=0.05, last_steps=last)
        e.window_adjoint(nsteps, ckpt, spec, np.zeros(40))

    for w in windows:  # what the kernels' first launches take
        run(*w)
    e.set_window_memory(limit)
    free = torch.cuda.mem_get_info()[0]
    most = limit
    for w in windows:
        run(*w)
        most = max(most, asked(n, c, *w[:2]))
        assert free - torch.cuda.mem_get_info()[0] <= most + 104 * n + SLACK, w
    e.set_window_memory(limit)
    assert abs(free - torch.cuda.mem_get_info()[0]) <= SLACK
