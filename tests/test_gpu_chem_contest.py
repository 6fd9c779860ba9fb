"""Growth and bonding requests for the same free H beads in one check (growth is
decided first, and a T whose nearest H went to a growing chain takes its next
one), in boxes of single H, T and P beads where every draw succeeds: types,
links and events against the oracle's serial statement."""
import numpy as np
import pytest

import oracle as O
import oercel_b200 as ob
from gpu_util import engine_with, oracle_params, oracle_state, params

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,shares,rates", [
    (6.0, (0.1, 0.3, 0.3, 0.3), (1.0, 1.0)),     # few H, wanted by many
    (14.0, (0.2, 0.3, 0.3, 0.2), (1.0, 1.0)),
    (40.0, (0.3, 0.1, 0.5, 0.1), (1.0, 1.0)),    # over a CTA's threads of bonding requests
    (40.0, (0.9, 0.04, 0.03, 0.03), (1.0, 1.0)),
    (14.0, (0.3, 0.3, 0.4, 0.0), (1.0, 1.0)),    # no growth
    (14.0, (0.2, 0.3, 0.2, 0.3), (1.0, 0.0)),    # no bonding
    (14.0, (0.2, 0.3, 0.3, 0.2), (0.2, 1.0)),
])
def test_contested_ends(cuda_ok, L, shares, rates):
    n = int(4 * L * L)
    p = params(L=L, seed=7, noise="philox", chem=1, n_chem=1, p_grow=rates[0], p_bond=rates[1], p_break=0.3, r_grow=1.0,
               r_bond=0.8, n_t_min=1, max_chain=4)
    rng = np.random.default_rng(int(100 * L) + int(100 * shares[1]))
    x, y = (rng.uniform(0, L, n).astype(np.float32) for _ in range(2))
    top = np.nextafter(np.float32(L), np.float32(0))
    v = np.zeros(n, np.float32)
    none = np.full(n, -1, np.int32)
    e = engine_with(p, np.minimum(x, top), np.minimum(y, top), v, v, rng.choice(4, n, p=shares).astype(np.uint8), none,
                    none.copy())
    e.build_cells()
    op = oracle_params(p)
    oc = O.chem(p_break=p.p_break, p_grow=p.p_grow, p_bond=p.p_bond, r_grow=p.r_grow, r_bond=p.r_bond,
                n_t_min=p.n_t_min, max_chain=p.max_chain)
    for step in range(1, 5):
        st = oracle_state(e.state())
        _, ev = O.chemistry(op, oc, st, e.cells(), step)
        e.chemistry(step)
        t = e.state()
        for k in ("type", "prev", "next"):
            assert np.array_equal(t[k], st[k]), (step, k)
        assert sorted((k, g, q) for (_, k, g, q, *_) in e.events()) == sorted((k, g, q) for (_, k, g, q, *_) in ev)
