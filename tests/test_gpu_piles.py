"""Cells that hold hundreds to tens of thousands of particles, in the fused substeps.

A cell above a few hundred particles is put in order by a whole CTA; the words have
to be the per-phase kernels', and the substep must not grow with the square of
the pile.
"""
import numpy as np
import pytest

from sunaengine_gb300 import scenes, tables3d
from sunaengine_gb300.engine import Batch, Engine
from sunaengine_gb300.engine3d import Engine3D

pytestmark = pytest.mark.gpu

ONE, H3 = scenes.ONE, 1 << 17


def _piles(n, piles, seed=5):
    """A block, its first particles moved into free cells above it and held there."""
    sc = scenes.jittered_block(n, 1.1, np.random.Generator(np.random.PCG64(seed)))
    rng = np.random.Generator(np.random.PCG64(seed + 1))
    sc.flags = np.zeros(sc.n, np.uint32)
    at = 0
    order = rng.permutation(sc.nFluid)
    for k, p in enumerate(piles):
        who = order[at:at + p]
        sc.pos[who] = np.array([(10 + 8 * k) * ONE, 6 * ONE]) + rng.integers(-ONE, ONE, (p, 2))
        sc.flags[who] = 4
        at += p
    return sc


def _same(a, b, steps):
    for k in steps:
        a.step(k)
        b.step(k)
        assert a.digest().hex == b.digest().hex
    assert np.array_equal(a.read_state(), b.read_state())
    assert np.array_equal(a.read_cell_start(), b.read_cell_start())
    for x, y in zip(a.read_fields(), b.read_fields()):
        assert np.array_equal(x, y)
    a.check_errors()


@pytest.mark.parametrize('n,piles,room', [(3000, [512], 0), (3000, [513], 0), (9000, [511, 700, 514, 2000], 0),
                                          (40000, [30000, 1000], 0), (1500, [900], 150000), (700, [640], 120000)])
def test_2d(n, piles, room):
    sc = _piles(n, piles)
    a, b = (Engine(max_particles=max(room, sc.n), lanes=k).load_scene(sc) for k in (0, 4))
    _same(a, b, [1, 3])
    assert a.last_timing()[1] == 3  # one launch a substep


def test_2d_batch():
    out = []
    for lanes in (0, 4):
        b = Batch(max_particles=40000, max_scenes=3, lanes=lanes)
        ids = [b.add_scene(_piles(n, p, seed=n)) for n, p in ((4000, [900, 600]), (500, []), (5000, [3000]))]
        b.step(3)
        out.append([(b.digest(i).hex, b.chain_hex(i), b.read_state(i).tobytes()) for i in ids])
    assert out[0] == out[1]


def _pile3(n, piles):
    sc = tables3d.initial_state(n, 'pool', 30, 30, 30)
    rng = np.random.Generator(np.random.PCG64(n))
    order = rng.permutation(sc.n)
    at = 0
    for k, p in enumerate(piles):
        who = order[at:at + p]
        sc.pos[who] = np.array([3 + 5 * k, 27, 3 + 9 * (k % 3)]) * H3 + H3 // 2 + rng.integers(-H3 // 3, H3 // 3, (p, 3))
        at += p
    return sc


@pytest.mark.parametrize('n,piles,room', [(4000, [512], 0), (4000, [513], 0), (9000, [511, 700, 514, 2000], 0),
                                          (30000, [20000, 1000], 0), (1200, [900], 150000)])
def test_3d(n, piles, room):
    sc = _pile3(n, piles)
    a, b = (Engine3D(max_particles=max(room, sc.n), lanes=k).load_scene(sc) for k in (0, 1))
    for k in (1, 2):
        a.step(k)
        b.step(k)
        assert a.chain_hex() == b.chain_hex()
    assert np.array_equal(a.read_state(), b.read_state())
    assert a.last_timing()[1] == 2 and b.last_timing()[1] > 20


def test_time_does_not_grow_with_the_square():
    """30,000 of 40,000 particles held in one cell: the fused substep stays the
    faster route (it took three times the per-phase one's time)."""
    sc = _piles(40000, [30000])
    us = []
    for lanes in (0, 2):
        e = Engine(max_particles=sc.n, lanes=lanes).load_scene(sc)
        e.step(4)
        t = []
        for _ in range(7):
            e.step(4)
            t.append(e.last_timing()[0])
        us.append(sorted(t)[3])
    assert us[0] < us[1]
