"""An edge point whose one side has depth zero and no flow: that side's normal
velocity is 0 / 0.  The mass flux takes the other side's speed, whichever side
of the edge that is, so one forward-Euler stage leaves every water level finite
(the discharges next to the column are not, and the run reports it).  Where the
oracle, whose maximum skips a NaN on one side of the edge only, has finite
levels too, the strict build has the same bits."""
import numpy as np
import pytest

from dgswem_b200 import Deck, HydroStep, decks
from dgswem_b200._abi import DgswemError
from oracle_lib import Oracle

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("variant", ["strict", "fast", "mixed"])
def test_mass_flux_beside_an_empty_column(built, tmp_path, variant):
    path = decks.quarter_annulus(tmp_path / "qa", nr=9, nth=17, nsteps=2, dt=1.0, rk_stage=1, rk_order=1)
    deck = Deck(path)
    ne = deck.s.ne
    rng = np.random.default_rng(4)
    ze, qx, qy = (0.05 * rng.normal(size=(ne, 3)) for _ in range(3))
    empty = rng.choice(ne, 7, replace=False)
    ze[empty] = -deck.real_array("hb", 3 * ne).reshape(ne, 3)[empty]
    qx[empty] = qy[empty] = 0.0
    with HydroStep(deck, fast=variant == "fast", mixed=variant == "mixed") as hs:
        hs.set_state(ze, qx, qy)
        hs.timestep(1)
        with pytest.raises(DgswemError, match="NaN"):
            hs.synchronize()
        got = hs.state()[0]
    assert np.isfinite(got).all()
    if variant != "strict":
        return
    orc = Oracle(path, threads=1)
    orc.set_state(ze, qx, qy, deck.int_array("wdflg", ne))
    orc.run(1, 1)
    want = orc.state()[0]
    same = np.isfinite(want)
    assert same.any() and (~same).any()
    np.testing.assert_array_equal(got[same], want[same])
