"""Node bounds over stars of every length: a fan of n triangles round one node
gives a star of n elements (the rim nodes' have one or two), so that the star's
batches end full, one short and two short.  The strict build equals the oracle
bit for bit on random states with some zeros of either sign."""
import numpy as np
import pytest

from dgswem_b200 import Deck, HydroStep, decks
from oracle_lib import Oracle

pytestmark = pytest.mark.gpu


def _fan(path, n):
    """Fan of n triangles: n = 1 or 2 and open, else closed round node 1."""
    ctl = decks.Controls(title="fan", nolibf=1, nolifa=2, cf=0.0025, dt=0.1, nsteps=2, rk_stage=2, rk_order=2,
                         slopeflag=5, h0=0.01, nramp=1, dramp=1.0)
    m = n if n > 2 else n + 1
    ang = 2.0 * np.pi * np.arange(m) / max(m, 3)
    x = np.concatenate([[0.0], 1000.0 * np.cos(ang)])
    y = np.concatenate([[0.0], 1000.0 * np.sin(ang)])
    tri = np.array([[1, 2 + i, 2 + (i + 1) % m] for i in range(n)])
    rim = [2 + i for i in range(m)]
    land = rim + [rim[0]] if n > 2 else [1] + rim + [1]
    return decks.write_deck(path, x, y, np.full(m + 1, 10.0), tri, [], [(land, 0)], ctl)


@pytest.mark.parametrize("n", [1, 2, 3, 4, 5, 6, 7, 8])
def test_star_lengths(built, tmp_path, n):
    path = _fan(tmp_path / "fan", n)
    deck = Deck(path)
    assert deck.s.ne == n
    rng = np.random.default_rng(n)
    st = [0.1 * rng.normal(size=(n, 3)) for _ in range(3)]
    for q in st[1:]:
        q[rng.random((n, 3)) < 0.3] = 0.0
        q[rng.random((n, 3)) < 0.1] = -0.0
    st.append(np.ones(n, np.int32))
    orc = Oracle(path, threads=1)
    with HydroStep(deck) as hs:
        hs.set_state(*st)
        hs.run(1, 2)
        got = hs.state()
    orc.set_state(*st)
    orc.run(1, 2)
    for a, b in zip(got, orc.state()):
        np.testing.assert_array_equal(a, b)
