"""The smoothed pair distribution at the edges of its kernel's split: the blocks
of 256 bins, and pairs that reach one bin more than the sixteen lanes of a half
warp (or twice those), of configurations taken one and several at a time.  The
loss's g(r) and its gradient against every pair on the CPU in FP64."""
import numpy as np
import pytest

import oercel_b200 as ob
from test_gpu_rdf import PHYS, smoothed

pytestmark = pytest.mark.gpu
DR = 2.0 / 64


@pytest.mark.parametrize("nbin,rmax,sigma", [
    (255, 1.5, 0.02), (256, 1.5, 0.02), (257, 1.5, 0.02), (512, 1.5, 0.02), (513, 1.5, 0.02),
    (64, 2.0, 14.5 * DR / 8), (64, 2.0, 15.5 * DR / 8), (64, 2.0, 16.5 * DR / 8), (64, 2.0, 31.5 * DR / 8)])
def test_bins_and_reaches(cuda_ok, nbin, rmax, sigma):
    e = ob.Engine(ob.Params(L=12.0, f_lip=0.3, seed=3, **PHYS))
    e.load_soup(0)
    e.prime()
    e.step(40)
    spec = e.rdf_spec(ta=2, tb=2, nbin=nbin, rmax=rmax, sigma=sigma, last_steps=1)
    target = np.linspace(0.0, 1.0, nbin)
    loss, grad, rdf, xbar, vhbar, _ = e.window_adjoint_state(1, 1, spec, target)
    s = e.state(0)
    x, y = s["x"].astype(np.float64), s["y"].astype(np.float64)
    g, norm, dk, i, j, d, r = smoothed(x, y, s["type"], 12.0, 2, 2, nbin, rmax, sigma)
    # a pair at the edge of its 4 sigma cut may fall on either side in FP32: e^-8 of its peak
    peak = norm * (rmax / nbin) * 0.3989422804 / sigma
    np.testing.assert_allclose(rdf[0], g, rtol=2e-5, atol=np.exp(-8) * peak.max() * 2)
    # F_bar = 0 at the window's end, so the loss's own gradient is vhbar / dt
    dl = (2.0 * (g - target) / nbin * norm * dk).sum(1)
    want = np.zeros((len(x), 2))
    for c in range(2):
        np.add.at(want[:, c], i, dl * d[c] / r)
        np.add.at(want[:, c], j, -dl * d[c] / r)
    got = vhbar[s["gid"].astype(np.int64)] / np.float32(0.02)
    assert np.abs(got - want).max() < 2e-3 * np.abs(want).max()


@pytest.mark.parametrize("last", [2, 31, 32, 33, 40])
def test_configurations_together(cuda_ok, last):
    """up to 32 stored configurations a launch: the mean of the steps' own distributions"""
    mk = lambda: ob.Engine(ob.Params(L=12.0, f_lip=0.3, seed=3, **PHYS))
    a, b = mk(), mk()
    for e in (a, b):
        e.load_soup(0)
        e.prime()
    target = np.linspace(0.0, 1.0, 64)
    spec = a.rdf_spec(ta=2, tb=2, nbin=64, rmax=2.0, sigma=0.05, last_steps=last)
    _, _, rdf, *_ = a.window_adjoint_state(44, 44, spec, target)
    one = b.rdf_spec(ta=2, tb=2, nbin=64, rmax=2.0, sigma=0.05, last_steps=1)
    b.step(44 - last)
    mean = np.mean([b.window_loss(1, one, target)[1][0] for _ in range(last)], 0)
    np.testing.assert_allclose(rdf[0], mean, rtol=1e-11)  # FP64 sums in another order
