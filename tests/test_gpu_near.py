"""The contact searches of the analysis (eight lanes a listed bead, FP32 with
FP64 at the thresholds) against every pair in FP64 on the CPU: boxes of three
cells and up, odd sides, distances on the thresholds, few and many beads of the
type, and clusters across the edges."""
import numpy as np
import pytest
from scipy.sparse import coo_matrix
from scipy.sparse.csgraph import connected_components

import oercel_b200 as ob

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("L,rho,frac,grid", [(3.0, 8, 0.5, 0), (4.9, 5, 1.0, 0), (8.0, 4, 0.3, 0.25), (17.3, 3, 0.05, 0),
                                             (25.0, 4, 0.2, 0.5), (40.0, 3, 0.19, 0.1)])
@pytest.mark.parametrize("rcut", [1.0, 0.8, 0.5])
def test_clusters_and_aggregates_equal_fp64(cuda_ok, L, rho, frac, grid, rcut):
    rng = np.random.default_rng(int(10 * L))
    Lf = float(np.float32(L))
    n = int(rho * L * L)
    x, y = rng.uniform(0, Lf, (2, n))
    if grid:
        x, y = (np.round(v / grid) * grid for v in (x, y))
    x, y = (np.where(v.astype(np.float32) >= np.float32(Lf), 0, v).astype(np.float32) for v in (x, y))
    t = np.where(rng.random(n) < frac, 2, 0).astype(np.uint8)
    e = ob.Engine(ob.Params(L=L, chem=0), n_beads=n)
    z = np.zeros(n, np.float32)
    e.set_state(0, x, y, z, z, t)
    e.build_cells()
    X, Y = x.astype(np.float64), y.astype(np.float64)
    at = np.nonzero(t == 2)[0]
    dx, dy = X[at][:, None] - X[None], Y[at][:, None] - Y[None]
    dx, dy = dx - Lf * np.rint(dx / Lf), dy - Lf * np.rint(dy / Lf)
    r2 = dx * dx + dy * dy
    near = r2 <= 1.0
    near[np.arange(len(at)), at] = False
    link = r2[:, at] <= rcut * rcut
    nc, lab = connected_components(coo_matrix(link), directed=False)
    size = np.bincount(lab, minlength=max(nc, 1))
    got = e.type_clusters(0, 2, rcut)
    want = dict(n=len(at), clusters=nc, largest=int(size.max(initial=0)), sum_sq=int((size.astype(np.int64) ** 2).sum()),
                nb_all=int(near.sum()), nb_same=int(near[:, at].sum()))
    assert {k: got[k] for k in want} == want
    agg = e.aggregates(0, r_tail=rcut, min_lipids=3, labels=True)  # every T is a molecule of its own
    assert agg["n_molecules"] == len(at) and agg["n_aggregates"] == nc
    assert agg["n_membranes"] == int((size >= 3).sum()) and agg["largest_aggregate"] == int(size.max(initial=0))
    first = np.full(max(nc, 1), n)
    np.minimum.at(first, lab, at)
    labels = np.full(n, -1)
    labels[at] = first[lab]
    assert np.array_equal(agg["labels"], labels)
