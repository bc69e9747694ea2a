"""Handles stepped from several threads at once, on meshes whose stage tiles need
different amounts of shared memory: each gives the bits it gives alone, launched
step by step and captured in graphs."""
import threading

import numpy as np
import pytest

from dgswem_b200 import Deck, HydroStep, decks

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("order", [1, 2])
def test_handles_in_threads(built, tmp_path, order):
    kw = dict(nsteps=2000, dt=1.0, **(dict(rk_stage=3, rk_order=3, extra=dict(pl=2, ph=2, px=2)) if order == 2 else {}))
    small = Deck(decks.quarter_annulus(tmp_path / "small", nr=2, nth=2, **kw))  # one tile, no halo
    large = Deck(decks.quarter_annulus(tmp_path / "large", nr=9, nth=40, nws=1, **kw))
    steps, rounds = 240, 6

    def run(deck, graph):
        with HydroStep(deck) as hs:
            if graph:
                hs.set_graph(graph)
            hs.run(1, steps)
            return hs.state()

    want = {id(d): run(d, 0) for d in (small, large)}
    failures = []

    def work(deck, graph):
        try:
            for _ in range(rounds):
                for a, b in zip(run(deck, graph), want[id(deck)]):
                    np.testing.assert_array_equal(a, b)
        except Exception as e:  # reported by the main thread
            failures.append(repr(e))

    threads = [threading.Thread(target=work, args=(d, g)) for d in (small, large) for g in (0, 0, 4)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not failures
