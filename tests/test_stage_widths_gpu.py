"""The stage kernel runs in blocks twice as wide on meshes of at most 148 tiles
(18,944 elements).  The bits do not depend on the width: copies of a small deck
side by side, each with a state of its own, in one handle above that line give
what each gives alone below it, and a mesh above it what its partitions below
it give -- in every build, over the boundary kinds, friction laws, forcings,
coordinates and Runge-Kutta forms."""
import numpy as np
import pytest

from conftest import golden_dir
from dgswem_b200 import Deck, HydroStep, decks
from dgswem_b200.hydro import PartitionedRun

pytestmark = pytest.mark.gpu

WIDE = 148 * 128  # elements up to which blocks are wide
QUAD = dict(nolibf=1, cf=0.0025)


def _annulus(**kw):
    return lambda p: decks.quarter_annulus(p, nr=23, nth=41, nsteps=10, dt=2.0, **kw)


DECKS = {
    "linear_friction": _annulus(),
    "wind_quadratic": _annulus(nws=1, **QUAD),
    "flow_radiation_limiter": _annulus(flow_amp=0.05, radiation=True, slopeflag=5, **QUAD),
    "hybrid_friction": _annulus(nolibf=2, cf=0.0025),
    "linear_equations": _annulus(nolifa=0, nolica=0, nolicat=0),
    "ssp52": _annulus(rk_stage=5, **QUAD),
    "rain": _annulus(rainfall=1),
    "beach": lambda p: decks.sloping_beach(p, nx=61, ny=17, lx=6100.0, ly=1700.0, nsteps=10, dt=0.2),
    "barriers": lambda p: golden_dir("wetdry"),
    "spherical": lambda p: golden_dir("mass_conservation"),
}
VARIANTS = {"strict": {}, "fast": dict(fast=True), "mixed": dict(mixed=True)}


def _state(deck, rng):
    ne = deck.s.ne
    st = [deck.real_array(n, 3 * ne).reshape(ne, 3).copy() for n in ("ze", "qx", "qy")]
    wd = deck.int_array("wdflg", ne)
    for q, scale in zip(st, (0.02, 0.05, 0.05)):
        q[wd == 1] += scale * rng.normal(size=(ne, 3))[wd == 1]
    return [*st, wd]


@pytest.fixture(scope="module")
def deck_dir(tmp_path_factory):
    return tmp_path_factory.mktemp("widths")


@pytest.mark.parametrize("variant", sorted(VARIANTS))
@pytest.mark.parametrize("name", sorted(DECKS))
def test_copies_side_by_side(built, deck_dir, name, variant):
    path = deck_dir / name
    deck = Deck(DECKS[name](path) if not path.exists() else path)
    ne, npn, steps = deck.s.ne, deck.s.np, 4
    assert ne <= WIDE
    n = WIDE // ne + 1
    rng = np.random.default_rng(21)
    states = [_state(deck, rng) for _ in range(n)]
    met = [1e-4 * rng.normal(size=npn), 1e-4 * rng.normal(size=npn), 0.1 * rng.normal(size=npn)]
    wind = deck.s.nws != 0
    with HydroStep(Deck.merge([deck] * n), **VARIANTS[variant]) as hs:
        assert hs.ne > WIDE
        if wind:
            hs.set_met(*(np.tile(m, n) for m in met))
        hs.set_state(*(np.concatenate([s[k] for s in states]) for k in range(4)))
        hs.run(1, steps)
        got = hs.state()
    for i in sorted({0, n // 2, n - 1}):
        with HydroStep(deck, **VARIANTS[variant]) as hs:
            if wind:
                hs.set_met(*met)
            hs.set_state(*states[i])
            hs.run(1, steps)
            want = hs.state()
        for a, b in zip(got, want):
            np.testing.assert_array_equal(a[i * ne:(i + 1) * ne], b)


@pytest.mark.parametrize("variant", sorted(VARIANTS))
def test_partitions_of_a_larger_mesh(built, deck_dir, variant):
    path = deck_dir / "larger"
    deck = Deck(path if path.exists() else
                decks.sloping_beach(path, nx=173, ny=57, lx=17300.0, ly=5700.0, nsteps=10, dt=0.2))
    assert WIDE < deck.s.ne < 2 * WIDE
    kw = dict(strict=False) if variant == "fast" else VARIANTS[variant]
    st = _state(deck, np.random.default_rng(22))
    with HydroStep(deck, **kw) as hs:
        hs.set_state(*st)
        hs.run(1, 4)
        want = hs.state()
    with PartitionedRun(deck, 2, **kw) as pr:
        for p in pr.parts:
            p.set_state(*st)
        pr.run(1, 4)
        pr.synchronize()
        got = pr.state()
    for a, b in zip(got, want):
        np.testing.assert_array_equal(a, b)
