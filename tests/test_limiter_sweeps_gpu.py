"""Limiter sweeps on rough states: steep slopes, steps between neighbours and
columns with no gradient at all, so that clamped, shared and idle sweeps meet in
one warp, on meshes that end just before, at and after a block of 64 elements.
The strict build equals the oracle bit for bit, whichever block size runs."""
import numpy as np
import pytest

from dgswem_b200 import Deck, HydroStep, decks
from oracle_lib import Oracle

pytestmark = pytest.mark.gpu


def _rough(deck, seed):
    ne = deck.s.ne
    rng = np.random.default_rng(seed)
    ze, qx, qy = (deck.real_array(n, 3 * ne).reshape(ne, 3).copy() for n in ("ze", "qx", "qy"))
    wd = deck.int_array("wdflg", ne)
    wet = wd == 1
    for q, scale in ((ze, 0.02), (qx, 0.05), (qy, 0.05)):
        q[wet] += scale * rng.normal(size=(ne, 3))[wet]
        flat = wet & (rng.random(ne) < 0.2)
        q[flat, 1:] = 0.0
        steep = wet & (rng.random(ne) < 0.2)
        q[steep, 1:] *= 5.0
    return ze, qx, qy, wd


@pytest.mark.parametrize("nx,ny", [(1, 1), (31, 1), (8, 4), (3, 11), (5, 19), (24, 8)])
@pytest.mark.parametrize("shape", [0, 1, 2])
def test_rough_states(built, tmp_path, nx, ny, shape):
    path = decks.sloping_beach(tmp_path / "sb", nx=nx, ny=ny, lx=100.0 * nx, ly=100.0 * ny, nsteps=3, dt=0.1)
    deck = Deck(path)
    assert deck.s.ne == 2 * nx * ny
    orc = Oracle(path, threads=1)
    st = _rough(deck, 100 * nx + ny)
    with HydroStep(deck) as hs:
        hs.set_shapes(limiter=shape)
        hs.set_state(*st)
        hs.run(1, 3)
        got = hs.state()
    orc.set_state(*st)
    orc.run(1, 3)
    for a, b in zip(got, orc.state()):
        np.testing.assert_array_equal(a, b)
