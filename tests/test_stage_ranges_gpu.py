"""Stage kernel values outside the range of its straight-line reciprocals and
roots (cr_math.cuh): states whose depths, speeds or momenta are tiny, subnormal
or zero, or whose columns are far too deep, in some elements of every tile and
of the last, partly filled one.  The strict build equals the oracle bit for
bit, as on ordinary states."""
import numpy as np
import pytest

from dgswem_b200 import Deck, HydroStep, decks
from oracle_lib import Oracle

pytestmark = pytest.mark.gpu


def _state(deck, kind):
    ne = deck.s.ne
    rng = np.random.default_rng(11)
    ze, qx, qy = (deck.real_array(n, 3 * ne).reshape(ne, 3).copy() for n in ("ze", "qx", "qy"))
    wd = deck.int_array("wdflg", ne)
    wet = wd == 1
    for q in (qx, qy):
        q[wet] = rng.normal(0.0, 0.1, (ne, 3))[wet]
    some = wet & (rng.random(ne) < 0.2)
    if kind == "still":
        qx[some], qy[some] = 0.0, 0.0
    elif kind == "tiny momentum":  # squares underflow, products are subnormal
        qx[some] *= 1e-170
        qy[some] *= 1e-305
    elif kind == "subnormal":
        qx[some] = rng.integers(-40, 40, (ne, 3))[some] * 5e-324
        qy[some] = rng.integers(-40, 40, (ne, 3))[some] * 5e-324
    elif kind == "deep":  # depth beyond 2^30 m
        ze[some, 0] = 3e9
    return ze, qx, qy, wd


@pytest.mark.parametrize("kind", ["still", "tiny momentum", "subnormal", "deep"])
def test_values_out_of_range(built, tmp_path, kind):
    path = decks.sloping_beach(tmp_path / "sb", nx=35, ny=11, lx=3500.0, ly=1100.0, nsteps=4, dt=0.2)
    deck = Deck(path)
    assert deck.s.ne % 128 != 0
    orc = Oracle(path, threads=1)
    with HydroStep(deck) as hs:
        st = _state(deck, kind)
        hs.set_state(*st)
        orc.set_state(*st)
        n = 1 if kind == "deep" else 4
        hs.run(1, n)
        got = hs.state()
    orc.run(1, n)
    want = orc.state()
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
