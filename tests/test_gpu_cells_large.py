"""Cell detection on one connected aggregate of 640,000 beads, walked by a cluster
of CTAs: the holes, lipids and membranes of the scene, the same wherever the
walk starts, and in no more time than level by level over the whole GPU (53 ms)."""
import time

import numpy as np
import pytest

from oercel_b200 import cells
from test_gpu_cells_walk import CFG, sheet

pytestmark = pytest.mark.gpu


def test_one_large_aggregate(cuda_ok):
    L = 256.0
    holes = [(60.0, 60.0, 6.0), (128.0, 100.0, 9.0), (180.0, 190.0, 4.0)]
    x, y, t, b = sheet(L, 200.0, holes, 0.5)
    order = np.random.default_rng(3).permutation(len(t))
    inv = np.argsort(order)
    x, y, t, b = x[order], y[order], t[order], inv[b]
    got = []
    for sx, sy in ((0, 0), (L / 2, L - 9.25)):
        s = cells.Snapshot(0, 0.0, L, (x + sx) % L, (y + sy) % L, t, b)
        d = cells.detect(s, CFG)
        got.append((d["summary"], sorted((c["area"], c["n_lipids"], c["n_W"], c["inner_heads"]) for c in d["cells"])))
    assert len(got[0][1]) == len(holes) and got[0] == got[1]
    assert got[0][0]["n_aggregates"] == 1 and got[0][0]["largest_aggregate"] == got[0][0]["n_molecules"]
    took = []
    for _ in range(5):
        t0 = time.perf_counter()
        cells.detect(s, CFG)
        took.append(time.perf_counter() - t0)
    assert min(took) < 0.05, took
