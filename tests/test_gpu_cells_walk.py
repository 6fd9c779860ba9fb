"""Cell detection on sheets whose walk has frontiers of hundreds of beads (a
lane per frontier bead) and on thin rings (sixteen lanes): a scene of positions
on a power-of-two grid moved by whole pixels across the periodic edges must
give the same lumens, lipids and membranes, though every walk starts elsewhere
and crosses the box edges."""
import numpy as np
import pytest

from oercel_b200 import cells

pytestmark = pytest.mark.gpu


def sheet(L, size, holes, step):
    """a square sheet of H-T-T-T lipids (one lipid per `step`) with round holes
    of water, water around it, all coordinates multiples of 1/64"""
    g = np.arange(0, size, step)
    X, Y = (v.ravel() + (L - size) / 2 for v in np.meshgrid(g, g, indexing="ij"))
    keep = np.ones(len(X), bool)
    for x, y, r in holes:
        keep &= np.hypot(X - x, Y - y) >= r
    X, Y = X[keep], Y[keep]
    k = np.arange(4) * 8 / 64
    lx, ly = (X[:, None] + k).ravel(), (Y[:, None] + 0 * k).ravel()
    nl = len(X)
    w = np.arange(0, L, 0.5) + 0.25
    wx, wy = (v.ravel() for v in np.meshgrid(w, w, indexing="ij"))
    inside = (np.abs(wx - L / 2) < size / 2 + 1) & (np.abs(wy - L / 2) < size / 2 + 1)
    for x, y, r in holes:
        inside &= ~(np.hypot(wx - x, wy - y) < r - 1)
    wx, wy = wx[~inside], wy[~inside]
    t = np.concatenate([np.tile(np.array([1, 2, 2, 2], np.uint8), nl), np.zeros(len(wx), np.uint8)])
    i = np.arange(4 * nl).reshape(-1, 4)
    b = np.stack([i[:, :3].ravel(), i[:, 1:].ravel()], 1).astype(np.int64)
    return np.concatenate([lx, wx]), np.concatenate([ly, wy]), t, b


CFG = dict(min_exposure=0.0, min_aqueous_frac=0.0, inner_frac_range=(0.0, 1.0), leaflet_max=30.0, wall_extra=20.0)


@pytest.mark.parametrize("L,size,holes,step", [
    (64.0, 48.0, [(20.0, 20.0, 4.0), (40.0, 30.0, 6.0), (30.0, 48.0, 3.0)], 0.5),
    (64.0, 40.0, [(32.0, 32.0, 18.5)], 0.5),
    (32.0, 20.0, [(16.0, 16.0, 5.0)], 0.75)])
def test_shifted_scene_has_the_same_cells(cuda_ok, L, size, holes, step):
    x, y, t, b = sheet(L, size, holes, step)
    order = np.random.default_rng(3).permutation(len(t))  # bead numbers in no spatial order
    inv = np.argsort(order)
    x, y, t, b = x[order], y[order], t[order], inv[b]
    got = []
    for sx, sy in ((0, 0), (7, 0), (L / 2, L / 2), (L - 9.25, 13.75)):
        d = cells.detect(cells.Snapshot(0, 0.0, L, (x + sx) % L, (y + sy) % L, t, b), CFG)
        got.append((d["summary"], sorted((c["area"], c["n_lipids"], c["n_W"], c["inner_heads"]) for c in d["cells"]),
                    sorted(np.unique(d["label"], return_counts=True)[1].tolist())))
    assert len(got[0][1]) == len(holes)
    for g in got[1:]:
        assert g == got[0]
