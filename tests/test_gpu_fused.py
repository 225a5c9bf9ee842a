"""The fused substep of small worlds against the per-phase kernels.

A pinned lane split keeps a world on the per-phase path, so the two engines
below advance the same scene on the two routes; every word has to be equal.
Sizes sit at the edges of what the fused kernel chooses by: one particle, the
lane splits' limits, the largest world it takes and one above it.
"""
import numpy as np
import pytest

from sunaengine_gb300 import scenes
from sunaengine_gb300.data import mat_id
from sunaengine_gb300.engine import Batch, Engine

pytestmark = pytest.mark.gpu


def _block(n, seed=5):
    return scenes.jittered_block(n, 1.1, np.random.Generator(np.random.PCG64(seed)))


def _pair(sc, extra=0, **kw):
    return (Engine(max_particles=sc.n + extra, **kw).load_scene(sc),
            Engine(max_particles=sc.n + extra, lanes=4, **kw).load_scene(sc))


def _same(a, b, steps):
    for k in steps:
        a.step(k)
        b.step(k)
        assert a.digest().hex == b.digest().hex
        assert np.array_equal(a.read_state(), b.read_state())
    assert a.chain_hex() == b.chain_hex()
    assert np.array_equal(a.read_scratch(), b.read_scratch())
    assert np.array_equal(a.read_bonds(), b.read_bonds())
    assert np.array_equal(a.read_cell_start(), b.read_cell_start())
    for x, y in zip(a.read_fields(), b.read_fields()):
        assert np.array_equal(x, y)
    a.check_errors()
    b.check_errors()


@pytest.mark.parametrize('n', [4, 37, 1000, 18500, 19300, 37500, 38300, 74000, 76500, 90000, 110000])
def test_sizes(n):
    a, b = _pair(_block(n))
    _same(a, b, [1, 7])
    if n <= 90000:
        assert a.last_timing()[1] == 7  # one launch a substep
    assert b.last_timing()[1] > 7 * 20


@pytest.mark.parametrize('iters', [1, 3, 4])
def test_iterations(iters):
    a, b = _pair(_block(3000), iters=iters)
    _same(a, b, [5])


@pytest.mark.parametrize('name', ['overdense_v1', 'gel', 'sand', 'sealed_box', 'no_chain'])
def test_rows(name):
    if name == 'gel' or name == 'sand':
        sc = scenes.make_scene('pool_v1', mat=mat_id(name.upper()), w=60, h=20)
    elif name == 'sealed_box':
        sc = scenes.sealed_box()
    else:
        sc = scenes.make_scene('overdense_v1')
    a, b = _pair(sc, chain=name != 'no_chain')
    _same(a, b, [1, 12])


def test_crowded_cells():
    """A column stacked into one edge cell: box culling and long rank loops."""
    sc = _block(4000)
    sc.pos[:900, 0] = scenes.ONE // 4
    sc.pos[:900, 1] = scenes.ONE // 2 + np.arange(900) % 64
    a, b = _pair(sc)
    _same(a, b, [1, 6])


def test_spawn_past_the_captured_size():
    sc = _block(3000)
    a, b = _pair(sc, extra=2600)
    _same(a, b, [2])
    drops = [{'x': (20 + i % 50) * scenes.ONE, 'y': (6 + i // 50 // 2) * scenes.ONE + i} for i in range(2500)]
    for e in (a, b):
        e.spawn_fluid(drops)
    _same(a, b, [2, 4])


def test_batch_with_a_gap():
    """Scenes of uneven sizes, one removed (its slots stay as a gap) and one
    added into part of the gap."""
    out = []
    for lanes in (0, 4):
        b = Batch(max_particles=40000, max_scenes=5, lanes=lanes)
        ids = [b.add_scene(_block(n, seed=n)) for n in (5000, 900, 7000)]
        b.schedule_impulse(ids[2], 3, 20 * scenes.ONE, 20 * scenes.ONE, 4 * scenes.ONE, 9000, -4000)
        b.step(4)
        b.remove_scene(ids[1])
        b.step(3)
        ids[1] = b.add_scene(_block(600, seed=9))
        b.step(5)
        out.append([(b.digest(i).hex, b.chain_hex(i), b.read_state(i).tobytes()) for i in ids])
        b.check_errors()
    assert out[0] == out[1]
