"""The fused substep of small worlds with rigid bodies against the per-phase
kernels: every word of the state, the body records and the chain has to be
equal. Sizes sit on both sides of the lane splits' limits, with fewer and with
more bodies than the GPU has SMs.
"""
import numpy as np
import pytest

from sunaengine_gb300 import scenes
from sunaengine_gb300.data import mat_id
from sunaengine_gb300.engine import Batch, Engine

pytestmark = pytest.mark.gpu

ONE = scenes.ONE


def _bodies(e, sc):
    for slots in sc.meta['planks']:
        e.make_rigid_body(slots)
    for slots, (cx, cy) in zip(sc.meta['wheels'], sc.meta['wheel_pivots']):
        e.make_axis_body(slots, cx, cy)


def _pair(sc):
    out = Engine(max_particles=sc.n).load_scene(sc), Engine(max_particles=sc.n, lanes=4).load_scene(sc)
    for e in out:
        _bodies(e, sc)
    return out


def _same(a, b, steps):
    for k in steps:
        a.step(k)
        b.step(k)
        assert a.digest().hex == b.digest().hex
        assert np.array_equal(a.read_state(), b.read_state())
    assert a.chain_hex() == b.chain_hex()
    assert np.array_equal(a.read_bodies(), b.read_bodies())
    a.check_errors()
    b.check_errors()


@pytest.mark.parametrize('tiles', [1, 2, 3, 6, 7, 12, 13, 24, 25, 28])
def test_sites(tiles):
    a, b = _pair(scenes.construction_site(tiles=tiles, seed=tiles))
    _same(a, b, [1, 7, 32])
    assert a.last_timing()[1] == 32  # one launch a substep
    assert b.last_timing()[1] > 32 * 20


def _blocks(n, side=3):
    """n metal squares over a shallow pool, in rows of twenty."""
    pos, mat, planks = [], [], []
    w, h = 20 * (side + 2) + 8, (n + 19) // 20 * (side + 2) + 24
    for k in range(n):
        ox, oy = 4 + k % 20 * (side + 2), 4 + k // 20 * (side + 2)
        planks.append(list(range(len(pos), len(pos) + side * side)))
        pos += [((ox + c) * ONE + ONE // 2, (oy + r) * ONE + ONE // 2) for r in range(side) for c in range(side)]
        mat += [mat_id('METAL')] * side * side
    for r in range(10):
        for c in range(w - 8):
            pos.append(((c + 4) * ONE + ONE // 2, (h - 14 + r) * ONE + ONE // 2))
            mat.append(mat_id('WATER'))
    sc = scenes._assemble(pos, np.array(mat, np.uint32), scenes.boundary_ring(w, h, h - 4), w, h, f'blocks_{n}')
    sc.meta = {'planks': planks, 'wheels': [], 'wheel_pivots': []}
    return sc


@pytest.mark.parametrize('n', [1, 151, 153, 200])
def test_body_counts(n):
    a, b = _pair(_blocks(n))
    _same(a, b, [1, 9, 60])


def test_bodies_come_and_go():
    """Worlds that gain and lose their bodies change route and back."""
    sc = scenes.construction_site(tiles=2, seed=9)
    a, b = Engine(max_particles=sc.n).load_scene(sc), Engine(max_particles=sc.n, lanes=4).load_scene(sc)
    _same(a, b, [3])
    _bodies(a, sc)
    _bodies(b, sc)
    _same(a, b, [5])
    assert a.dissolve_all_bodies() == b.dissolve_all_bodies()
    _same(a, b, [5])


def test_batch_with_and_without_bodies():
    site, pool = scenes.construction_site(tiles=2, seed=3), scenes.make_scene('dambreak_v1')
    out = []
    for kw in ({}, {'lanes': 4}):
        bt = Batch(max_particles=site.n + pool.n, max_scenes=2, **kw)
        i, j = bt.add_scene(site), bt.add_scene(pool)
        for slots in site.meta['planks']:
            bt.make_rigid_body(i, slots)
        bt.step(20)
        out.append([bt.read_state(k) for k in (i, j)] + [bt.chain_hex(k) for k in (i, j)])
    for x, y in zip(*out):
        assert np.array_equal(x, y)
