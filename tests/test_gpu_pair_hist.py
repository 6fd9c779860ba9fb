"""The pair-distance histogram against every pair binned in FP64 on the CPU:
boxes of three cells and up (windows as wide as the box, odd sides), few and
many bins (the lane-private and the shared counters), one type, two types and
all, and distances that fall on the bins' edges."""
import numpy as np
import pytest

import oercel_b200 as ob

pytestmark = pytest.mark.gpu


def brute(x, y, t, L, ta, tb, rmax, nbin, window):
    """np.histogram's bins of every pair's FP64 nearest-image distance; pairs of
    cells more than `window` columns or rows apart are out of the search"""
    nc = int(np.floor(L))
    cx, cy = (np.minimum((v * (nc / L)).astype(int), nc - 1) for v in (x, y))
    i, j = np.triu_indices(len(x), 1)
    if ta >= 0:
        m = ((t[i] == ta) & (t[j] == tb)) | ((t[i] == tb) & (t[j] == ta))
        i, j = i[m], j[m]
    for c in (cx, cy):
        d = np.abs(c[i] - c[j])
        m = np.minimum(d, nc - d) <= window
        i, j = i[m], j[m]
    dx, dy = x[i] - x[j], y[i] - y[j]
    dx -= L * np.rint(dx / L)
    dy -= L * np.rint(dy / L)
    r = np.hypot(dx, dy)
    r = r[r <= rmax]
    step = rmax / nbin
    b = np.minimum((r * (nbin / rmax)).astype(int), nbin - 1)
    low = r < b * step
    up = ~low & (b + 1 < nbin) & (r >= (b + 1) * step)
    return np.bincount(b - low + up, minlength=nbin)


@pytest.mark.parametrize("L,rho,grid", [(3.0, 12, 0), (5.7, 6, 0), (6.0, 9, 0.25), (7.99, 4, 0), (9.0, 5, 0.5),
                                        (16.0, 4, 0.1), (31.3, 3, 0), (40.0, 3, 0.125)])
@pytest.mark.parametrize("ta,tb", [(-1, -1), (2, 2), (0, 2)])
@pytest.mark.parametrize("rmax,nbin", [(3.0, 30), (0.4, 1), (2.0, 256), (2.5, 257), (3.0, 4096)])
def test_counts_equal_fp64_binning(cuda_ok, L, rho, grid, ta, tb, rmax, nbin):
    rng = np.random.default_rng(int(100 * L) + nbin)
    Lf = float(np.float32(L))
    n = max(int(rho * L * L), 2)
    x, y = rng.uniform(0, Lf, (2, n)).astype(np.float32)
    if grid:  # distances on the bins' edges
        x, y = ((np.round(v / grid) * grid) % L for v in (x, y))
    x, y = (np.where(v >= np.float32(Lf), 0, v).astype(np.float32) for v in (x, y))
    t = rng.choice([0, 2], n, p=[0.7, 0.3]).astype(np.uint8)
    e = ob.Engine(ob.Params(L=L, chem=0), n_beads=n)
    z = np.zeros(n, np.float32)
    e.set_state(0, x, y, z, z, t)
    e.build_cells()
    nc = int(np.floor(L))
    window = min(int(np.ceil(rmax * (nc / Lf))), (nc - 1) // 2)
    want = brute(x.astype(np.float64), y.astype(np.float64), t, Lf, ta, tb, rmax, nbin, window)
    assert np.array_equal(e.pair_hist(0, ta, tb, rmax, nbin).astype(np.int64), want)
