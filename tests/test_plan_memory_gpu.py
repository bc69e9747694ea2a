"""Device memory of a mixed handle against a strict one of the same mesh: the
FP32 copy of the geometry table (18 rows, 72 bytes an element) more, and the
plan's normals and front fluxes (eight numbers a task, at least 1.5 tasks an
element) in four bytes instead of eight, 48 bytes an element less."""
import ctypes as C

import pytest

from dgswem_b200 import Deck, HydroStep, decks

pytestmark = pytest.mark.gpu


def _free():
    cu = C.CDLL("libcuda.so.1")
    free, total = C.c_size_t(), C.c_size_t()
    assert cu.cuMemGetInfo_v2(C.byref(free), C.byref(total)) == 0
    return free.value


def test_mixed_plan_in_its_own_type(built, tmp_path):
    deck = Deck(decks.sloping_beach(tmp_path / "sb", nx=1000, ny=200, nsteps=2))
    HydroStep(deck).close()  # the context and the kernels' module
    used = {}
    for mixed in (False, True):
        before = _free()
        with HydroStep(deck, mixed=mixed):
            used[mixed] = before - _free()
    slack = 8 << 20  # allocations are rounded up to 2 MB; a few arrays differ
    assert used[True] - used[False] <= (72 - 48) * deck.s.ne + slack
