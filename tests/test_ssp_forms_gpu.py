"""Every Runge-Kutta scheme the decks accept, whose stages combine one, two or
up to seven earlier states and right-hand sides, with terms left out between
them: p=1 and p=2, strict build against the oracle bit for bit."""
import numpy as np
import pytest

from dgswem_b200 import Deck, HydroStep, decks
from oracle_lib import Oracle

pytestmark = pytest.mark.gpu

SCHEMES = [(1, 1), (2, 2), (3, 2), (4, 2), (5, 2), (6, 2), (8, 2), (3, 3)]


@pytest.mark.parametrize("rk", SCHEMES)
@pytest.mark.parametrize("order", [1, 2])
def test_scheme_bitwise(built, tmp_path, rk, order):
    kw = dict(extra=dict(pl=2, ph=2, px=2)) if order == 2 else dict(slopeflag=5, nolibf=1, cf=0.0025)
    path = decks.quarter_annulus(tmp_path / "qa", nr=7, nth=13, nsteps=4, dt=2.0, rk_stage=rk[0], rk_order=rk[1], **kw)
    deck = Deck(path)
    dof = deck.s.dofh
    rng = np.random.default_rng(rk[0])
    st = [s * rng.normal(size=(deck.s.ne, dof)) for s in (0.02, 0.05, 0.05)]
    orc = Oracle(path, threads=1)
    with HydroStep(deck) as hs:
        hs.set_state(*st)
        hs.run(1, 4)
        got = hs.state()
    orc.set_state(*st, np.ones(deck.s.ne, np.int32))
    orc.run(1, 4)
    for a, b in zip(got[:3], orc.state()[:3]):
        np.testing.assert_array_equal(a, b)
