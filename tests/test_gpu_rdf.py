"""The smoothed pair distribution of a window and its position gradient over
the shapes the kernel splits by: bins within one lane round, past it, past a
block of 128; clusters with more than 32 neighbours of the types; windows of
cells as wide as the box; two different types.  The loss's g(r) against every
pair on the CPU in FP64, the gradient against its FP64 derivative."""
import numpy as np
import pytest

import oercel_b200 as ob

pytestmark = pytest.mark.gpu

PHYS = dict(rho=4, dt=0.02, chem=0, warmup=0, f_Ka=0, k_angle=0, c_N=0.01)


def smoothed(x, y, t, L, ta, tb, nbin, rmax, sigma):
    """g(r) of the bins and dg_b / dr of every pair, FP64, as the documented
    definition: a Gaussian of width sigma per pair, cut at 4 sigma around r"""
    dr = rmax / nbin
    i, j = np.triu_indices(len(x), 1)
    m = ((t[i] == ta) & (t[j] == tb)) | ((t[i] == tb) & (t[j] == ta))
    i, j = i[m], j[m]
    npairs = len(i)
    d = np.stack([x[i] - x[j], y[i] - y[j]])
    d -= L * np.rint(d / L)
    r = np.hypot(*d)
    m = (r < rmax + 4 * sigma) & (r > 0)
    i, j, d, r = i[m], j[m], d[:, m], r[m]
    b = np.arange(nbin)
    rb = (b + 0.5) * dr
    e = r[:, None] - rb[None, :]
    lo = np.maximum(0, np.floor((r - 4 * sigma) / dr))[:, None]
    hi = np.minimum(nbin - 1, np.floor((r + 4 * sigma) / dr))[:, None]
    k = np.where((b >= lo) & (b <= hi), dr * 0.3989422804 / sigma * np.exp(-e * e / (2 * sigma * sigma)), 0.0)
    norm = L * L / (npairs * 2 * np.pi * rb * dr)
    return (k.sum(0) * norm, norm, -e / sigma ** 2 * k, i, j, d, r)


@pytest.mark.parametrize("L,f_lip,ta,tb,nbin,rmax,sigma", [
    (6.0, 0.9, 2, 2, 7, 1.0, 0.1),        # one lane round; a window as wide as the box
    (12.0, 0.3, 2, 2, 64, 2.0, 0.05),     # the fits' shape
    (9.3, 0.95, 2, 2, 64, 2.0, 0.05),     # over 32 neighbours a bead
    (12.0, 0.3, 1, 2, 65, 2.0, 0.05),     # two types, one bin past the two lane rounds
    (12.0, 0.3, 2, 0, 300, 1.5, 0.02),    # past one block of bins
])
def test_window_rdf_and_gradient(cuda_ok, L, f_lip, ta, tb, nbin, rmax, sigma):
    e = ob.Engine(ob.Params(L=L, f_lip=f_lip, seed=3, **PHYS))
    e.load_soup(0)
    e.prime()
    e.step(40)
    spec = e.rdf_spec(ta=ta, tb=tb, nbin=nbin, rmax=rmax, sigma=sigma, last_steps=1)
    target = np.linspace(0.0, 1.0, nbin)
    loss, grad, rdf, xbar, vhbar, _ = e.window_adjoint_state(1, 1, spec, target)
    s = e.state(0)
    Lf = float(np.float32(L))
    x, y = s["x"].astype(np.float64), s["y"].astype(np.float64)
    g, norm, dk, i, j, d, r = smoothed(x, y, s["type"], Lf, ta, tb, nbin, rmax, sigma)
    # a pair at the edge of its 4 sigma cut may fall on either side in FP32: e^-8 of its peak
    peak = norm * (rmax / nbin) * 0.3989422804 / sigma
    np.testing.assert_allclose(rdf[0], g, rtol=2e-5, atol=np.exp(-8) * peak.max() * 2)
    assert abs(loss[0] - np.mean((g - target) ** 2)) < 1e-3 * max(loss[0], 1e-3)
    # one step of length 1 with the loss at its end: v_bar at the start = dt x_bar at the end (plus the force
    # VJP's share, which F_bar = 0 leaves out), so the loss's own gradient is vhbar / dt
    dl = (2.0 * (g - target) / nbin * norm * dk).sum(1)
    want = np.zeros((len(x), 2))
    for c in range(2):
        np.add.at(want[:, c], i, dl * d[c] / r)
        np.add.at(want[:, c], j, -dl * d[c] / r)
    gid = s["gid"].astype(np.int64)
    got = vhbar[gid] / np.float32(0.02)
    assert np.abs(got - want).max() < 2e-3 * np.abs(want).max()
