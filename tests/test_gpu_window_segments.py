"""The segments of a differentiated window: its forward pass, loss and gradients
whether all differentiated steps are kept, or some stepped again from
checkpoints, in segments as short as the caller's interval or longer, with a
shorter first one, with and without a horizon."""
import numpy as np
import pytest

import oercel_b200 as ob

pytestmark = pytest.mark.gpu

PHYS = dict(rho=4, dt=0.02, chem=0, warmup=0, f_Ka=0, k_angle=0, c_N=0.01)


def run(memory, nsteps, ckpt, last, horizon, replicas, stir):
    e = ob.Engine([ob.Params(L=9.0 + 2 * r, f_lip=0.3, seed=5 + r, stir_A=stir, **PHYS) for r in range(replicas)])
    for r in range(replicas):
        e.load_soup(r)
    e.prime()
    e.step(20)
    e.set_window_memory(memory)
    spec = e.rdf_spec(ta=2, tb=2, nbin=40, rmax=2.0, sigma=0.05, last_steps=last, horizon=horizon)
    target = np.tile(np.linspace(0.0, 1.0, 40), (replicas, 1))
    call = e.window_adjoint if horizon else e.window_adjoint_state
    out = [call(nsteps, ckpt, spec, target) for _ in range(2)]  # the second from the first's end, in its storage
    return out, [e.state(r) for r in range(replicas)]


@pytest.mark.parametrize("replicas,stir", [(1, 0.0), (2, 0.3)])
@pytest.mark.parametrize("nsteps,ckpt,last,horizon", [
    (1, 1, 1, 0),     # one step
    (12, 5, 3, 0),    # a shorter first segment
    (12, 1, 4, 3),    # a checkpoint a step, loss steps in more than one segment
    (17, 4, 2, 6),    # the horizon inside an interval
    (17, 17, 9, 20),  # a horizon past the start
    (40, 7, 36, 2),   # more loss steps than one launch of their kernels takes
])
def test_segments_agree(cuda_ok, replicas, stir, nsteps, ckpt, last, horizon):
    bead = 4 * 9.0 ** 2 * 33
    want, state = run(None, nsteps, ckpt, last, horizon, replicas, stir)  # small boxes: every step kept
    for memory in (0, int(8 * bead), int(20 * bead)):
        got, st = run(memory, nsteps, ckpt, last, horizon, replicas, stir)
        for a, b in zip(want, got):
            np.testing.assert_allclose(b[0], a[0], rtol=1e-12)
            # FP64 sums in another order; the state's cotangents go through FP32 weights of such sums
            np.testing.assert_allclose(b[1], a[1], rtol=1e-6, atol=1e-6 * np.abs(a[1]).max())
            for u, v in zip(a[3:], b[3:]):
                np.testing.assert_allclose(v, u, rtol=1e-6, atol=1e-6 * np.abs(u).max())
        for a, b in zip(state, st):
            for k in ("x", "y", "vhx", "vhy", "fx", "fy"):
                if k in a:
                    assert np.array_equal(a[k], b[k]), k
