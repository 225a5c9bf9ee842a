"""Lanes tuned on one engine and pinned on another do not take a small world off the
one-launch substep; lanes given at creation do."""
import numpy as np
import pytest

from sunaengine_gb300 import scenes
from sunaengine_gb300.engine import Batch, Engine

pytestmark = pytest.mark.gpu


def _block(n, seed=5):
    return scenes.jittered_block(n, 1.1, np.random.Generator(np.random.PCG64(seed)))


def test_tuned_lanes_keep_the_route():
    sc = _block(3000)
    a, b, c = Engine(max_particles=sc.n), Engine(max_particles=sc.n), Engine(max_particles=sc.n, lanes=4)
    for e in (a, b, c):
        e.load_scene(sc)
    ran = a.autotune(1)
    b.set_lanes(a.lanes())
    for e, k in ((a, 6), (b, ran + 6), (c, ran + 6)):
        e.step(k)
    assert a.last_timing()[1] == 6 and b.last_timing()[1] == ran + 6
    assert c.last_timing()[1] > 20 * (ran + 6)
    assert a.chain_hex() == b.chain_hex() == c.chain_hex()
    assert b.lanes() == a.lanes()


def test_batch():
    out = []
    for pin in (False, True):
        b = Batch(max_particles=9000, max_scenes=2)
        ids = [b.add_scene(_block(n, seed=n)) for n in (2500, 1200)]
        if pin:
            b.set_lanes({'solveA': 1, 'colours': 8, 'post1': 2, 'post2': 4, 'nbr': 1})
        b.step(4)
        assert b.last_timing()[1] == 4
        out.append([b.chain_hex(i) for i in ids])
    assert out[0] == out[1]
