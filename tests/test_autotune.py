"""The autotuner's choices on an engine whose kernel times are given."""
import pytest

from oercel_b200.autotune import autotune


class Timed:
    """kernel times of a step: the sort's four, permute, forces"""
    n_beads = [4096]

    def __init__(self, sort, forces):
        self.sort, self.forces = sort, forces
        self.t = dict(force_kernel=0, tile_w=8, tile_h=8, tile_threads=256, sort_mode=2)

    def set_tuning(self, **kv):
        self.t.update(kv)

    def tuning(self):
        return dict(self.t)

    def profile_step(self):
        m = self.t["sort_mode"]
        return [*self.sort[m], 5.0, self.forces[m] * (1.0 if self.t["tile_w"] == 4 else 2.0)]


@pytest.mark.parametrize("forces,want", [([20.0, 20.0, 24.0], 1), ([20.0, 20.0, 20.5], 2), ([20.0, 25.0, 25.0], 0)])
def test_sort_is_judged_with_the_forces_it_bins_in(forces, want):
    """mode 2 moves a part of the sort into the force kernel: its own kernels alone are always the fewest here"""
    sort = [[3.0, 2.0, 2.0, 2.0], [3.0, 0.0, 2.0, 2.0], [0.0, 0.0, 0.0, 4.5]]
    e = Timed(sort, forces)
    out = autotune(e, candidates=[dict(tile_w=2), dict(tile_w=4)], use_cache=False)
    assert (out["tuning"]["sort_mode"], out["tuning"]["tile_w"]) == (want, 4)
    assert out["sort_ms"] == sum(sort[want])


class Shaped(Timed):
    """the force kernel's time by tile shape"""

    def __init__(self, best):
        super().__init__([[1.0] * 4] * 3, None)
        self.best = best
        self.t = dict(force_kernel=0, tile_w=7, tile_h=12, tile_threads=256, sort_mode=2)

    def profile_step(self):
        return [1.0, 1.0, 1.0, 1.0, 5.0, 20.0 if (self.t["tile_w"], self.t["tile_h"]) == self.best else 25.0]


@pytest.mark.parametrize("best", [(7, 12), (10, 18)])
def test_the_engines_own_shape_is_a_candidate(best):
    out = autotune(Shaped(best), use_cache=False)
    assert (out["tuning"]["tile_w"], out["tuning"]["tile_h"]) == best
