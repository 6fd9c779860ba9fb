"""State and VJP calls on device pointers: an array shorter than the replica is
refused whichever array it is, and leaves the state as it was; arrays inside a
larger allocation, at any 4-byte offset, are read and written in place."""
import numpy as np
import pytest

import oercel_b200 as ob
from oercel_b200 import _capi
from gpu_util import params

pytestmark = pytest.mark.gpu
KEYS = ("x", "y", "vhx", "vhy", "vtx", "vty", "fx", "fy", "type", "gid", "prev", "next")


class Owned:
    """device memory in allocations of its own"""

    def __init__(self):
        import ctypes as C
        self.rt, self.C, self.p = C.CDLL("libcudart.so.12"), C, []

    def __call__(self, nbytes):
        p = self.C.c_void_p()
        assert self.rt.cudaMalloc(self.C.byref(p), self.C.c_size_t(nbytes)) == 0
        self.p.append(p)
        return p.value

    def free(self):
        for p in self.p:
            assert self.rt.cudaFree(p) == 0


@pytest.fixture
def engine(cuda_ok):
    e = ob.Engine(params(L=512.0, seed=3))  # 4 MB an array
    e.load_soup(0)
    e.prime()
    return e


def test_short_arrays_are_refused(engine):
    e, n = engine, engine.n_beads[0]
    own = Owned()
    try:
        full, short = own(4 * n), own(4096)
        before = e.state(0)
        for k in [k for k in range(12) if KEYS[k] != "type"]:
            args = [None] * 12
            args[k] = short
            assert e.lib.dpd_get_state(e.h, 0, *args) != 0
            if k != 0:
                args[0] = full
                assert e.lib.dpd_get_state(e.h, 0, *args) != 0
        for k in range(4):
            args = [full] * 4
            args[k] = short
            assert e.lib.dpd_set_state(e.h, 0, *args, full, None, None, None) != 0
        for g in ((short, full), (full, short)):
            assert e.lib.dpd_force_vjp(e.h, 0, 1, *g, None, None, None, None, None) != 0
        after = e.state(0)
        for k in KEYS:
            assert np.array_equal(before[k], after[k]), k
    finally:
        own.free()


@pytest.mark.parametrize("offset", [0, 4, 12])
def test_arrays_inside_an_allocation(engine, offset):
    import torch
    e, n = engine, engine.n_beads[0]
    want = e.state(0)
    pool = torch.zeros(12 * (4 * n + 64) + 64, dtype=torch.uint8, device="cuda")
    at = [pool.data_ptr() + offset + k * (4 * n + 64) for k in range(12)]
    torch.cuda.synchronize()
    _capi.check(e.lib.dpd_get_state(e.h, 0, *at))
    for k, name in enumerate(KEYS):
        w = want[name]
        o = offset + k * (4 * n + 64)
        assert np.array_equal(pool[o:o + w.nbytes].cpu().numpy().view(w.dtype), w), name
    by = dict(zip(KEYS, at))
    _capi.check(e.lib.dpd_set_state(e.h, 0, *[by[k] for k in ("x", "y", "vhx", "vhy", "type", "gid", "prev", "next")]))
    s = e.state(0)
    for k in ("x", "y", "type", "gid", "prev", "next"):
        assert np.array_equal(s[k], want[k]), k
