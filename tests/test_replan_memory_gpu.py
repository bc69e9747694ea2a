"""A change of tile shape that the device has no memory for reports it and
leaves the handle as it was: with the memory back, its steps give the bits of a
handle that was never asked, at whichever of the plan's arrays the memory ran
out."""
import ctypes as C

import numpy as np
import pytest

from dgswem_b200 import Deck, HydroStep, decks
from dgswem_b200._abi import DgswemError

pytestmark = pytest.mark.gpu

MB = 1 << 20


class DeviceFill:
    """Holds all of the device's free memory but `leave` bytes."""

    def __init__(self, leave):
        self.cu = C.CDLL("libcuda.so.1")
        self.cu.cuMemAlloc_v2.argtypes = [C.POINTER(C.c_uint64), C.c_size_t]
        self.cu.cuMemFree_v2.argtypes = [C.c_uint64]
        self.held = []
        kept = self._alloc(leave) if leave else None
        size = 16 << 30
        while size >= 2 * MB:
            p = self._alloc(size)
            if p is None:
                size //= 2
            else:
                self.held.append(p)
        if kept is not None:
            self.cu.cuMemFree_v2(kept)

    def _alloc(self, size):
        p = C.c_uint64()
        return p.value if self.cu.cuMemAlloc_v2(C.byref(p), size) == 0 else None

    def release(self):
        for p in self.held:
            assert self.cu.cuMemFree_v2(p) == 0
        self.held = []


@pytest.mark.parametrize("variant", ["strict", "mixed"])
def test_shape_change_without_memory(built, tmp_path, variant):
    path = decks.sloping_beach(tmp_path / "sb", nx=400, ny=100, nsteps=8, dramp=0.01)
    deck = Deck(path)
    kw = dict(mixed=variant == "mixed")
    with HydroStep(deck, **kw) as hs:
        hs.run(1, 6)
        want = hs.state()
    with HydroStep(deck, **kw) as hs:
        st = hs.state()
        for shape in (1, 0):  # both shapes' kernels loaded before the memory goes
            hs.set_shapes(tile=shape)
            hs.run(1, 1)
            hs.synchronize()
        failed = 0
        for leave in range(0, 24, 4):
            hs.set_state(*st)
            hs.run(1, 2)
            hs.synchronize()
            fill = DeviceFill(leave * MB)
            try:
                hs.set_shapes(tile=1)
            except DgswemError as e:
                assert "memory" in str(e)
                failed += 1
                assert hs.get_shapes()[0] == 0
            finally:
                fill.release()
            hs.run(3, 4)
            got = hs.state()
            for a, b in zip(got, want):
                np.testing.assert_array_equal(a, b)
            hs.set_shapes(tile=0)
        assert failed > 0
