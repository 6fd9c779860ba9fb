"""The force VJP on the boxes that its launch rule gives two lanes a bead (2 and 4
CTAs an SM) and their neighbours on either side of its lines, with and without
the fused update: each replica of a batch against the same box alone, whose
few chunks take eight lanes.  A bead's terms are added in one order (each lane has
at most 32 candidates here), so the products are the same bits; the parameters'
gradients are FP64 sums in another order."""
import numpy as np
import pytest

import oercel_b200 as ob
from gpu_util import params

pytestmark = pytest.mark.gpu
ROUND = 1e-10  # FP64 sums of 1e4 terms (1e-12 of their sizes), at most a hundred times the largest sum

BOX = dict(rho=3, dt=0.02, f_lip=0.3, noise="philox")


def boxes(n):
    return [params(L=L, seed=11 + k, **BOX) for k, L in enumerate((24.0, 20.3, 16.5, 31.0)[:n])]


def primed(ps):
    e = ob.Engine(ps)
    for r in range(len(ps)):
        e.load_soup(r)
    e.prime()
    e.step(3)
    return e


def chunks(e):
    return sum(-(-n // 256) for n in e.n_beads)


@pytest.mark.parametrize("copies,want", [
    (18, (112, 148)), (36, (223, 296)), (50, (297, 444)), (72, (445, 592)), (90, (593, 666)), (110, (667, 1000))])
def test_batch_equals_single_boxes(cuda_ok, copies, want):
    ps = boxes(1) * copies
    e, one = primed(ps), primed(boxes(1))
    assert want[0] <= chunks(e) <= want[1] and chunks(one) * 8 <= 2 * 148
    n, nc = one.n_beads[0], 24
    c = np.diff(one.cells(0)).reshape(nc, nc)
    near = sum(np.roll(c, (i, j), (0, 1)) for i in (-1, 0, 1) for j in (-1, 0, 1))
    assert near.max() <= 2 * 32
    rng = np.random.default_rng(5)
    g = rng.normal(size=(2, n)).astype(np.float32)
    w = one.force_vjp(0, 3, g[0], g[1])
    for r in (0, copies // 2, copies - 1):
        v = e.force_vjp(r, 3, g[0], g[1])
        for k in range(4):
            assert np.array_equal(v[k], w[k]), (r, k)
        np.testing.assert_allclose(v[4], w[4], rtol=0, atol=ROUND * np.abs(w[4]).max())


@pytest.mark.parametrize("copies", [11, 13, 40])
def test_windows_of_a_batch(cuda_ok, copies):
    """the update of the adjoint state in the same kernel: window gradients of uneven boxes"""
    ps = [q for _ in range(copies) for q in boxes(4)[:2]]
    e = primed(ps)
    spec = e.rdf_spec(ta=2, tb=2, nbin=40, rmax=2.0, sigma=0.05, last_steps=3)
    got = e.window_adjoint_state(6, 6, spec, np.linspace(0.0, 1.0, 40))
    at = np.concatenate([[0], np.cumsum(e.n_beads)])
    for q in range(2):
        one = primed([boxes(4)[q]])
        want = one.window_adjoint_state(6, 6, spec, np.linspace(0.0, 1.0, 40))
        for r in (q, 2 * (copies // 2) + q, 2 * (copies - 1) + q):
            np.testing.assert_allclose(got[0][r], want[0][0], rtol=1e-12)
            # FP64 sums in another order; the cotangents go through FP32 weights of such sums
            np.testing.assert_allclose(got[1][r], want[1][0], rtol=1e-6, atol=1e-6 * np.abs(want[1]).max())
            for u, v in zip(got[3:], want[3:]):
                np.testing.assert_allclose(u[at[r]:at[r + 1]], v, rtol=1e-6, atol=1e-6 * np.abs(v).max())
