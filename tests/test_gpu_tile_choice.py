"""The default tile shape of a handle: within the limits dpd_set_tuning takes,
for any size, density and mix of boxes."""
import pytest

import oercel_b200 as ob


@pytest.mark.gpu
@pytest.mark.parametrize("boxes", [[(3.0, 36)], [(8.0, 256)], [(32.0, 4096)], [(64.0, 12288), (9.5, 300)],
                                   [(128.0, 65536)], [(20.0, 8000)], [(300.2, 270000)],
                                   [(12.0 + r, int(4 * (12 + r) ** 2)) for r in range(40)]])
def test_default_tile_is_a_shape_the_kernel_takes(cuda_ok, boxes):
    e = ob.Engine([ob.Params(L=L, chem=0) for L, _ in boxes], [n for _, n in boxes])
    t = e.tuning()
    assert t["force_kernel"] == 0 and t["tile_threads"] == 256
    assert t["tile_w"] >= 1 and t["tile_h"] >= 1 and (t["tile_w"] + 2) * (t["tile_h"] + 2) <= 256
    densest = max(n / int(L) ** 2 for L, n in boxes)
    if densest <= 9:  # staged in shared memory: 1,408 beads with the halo
        assert (t["tile_w"] + 2) * (t["tile_h"] + 2) * densest <= 1408
    e.set_tuning(**t)
