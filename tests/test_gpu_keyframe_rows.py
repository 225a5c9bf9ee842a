"""Keyframes of scenes whose bond rows are empty, and chains read after every way
a chain changes."""
import numpy as np
import pytest

from sunaengine_gb300 import scenes, tables3d
from sunaengine_gb300.checkpoints import CheckpointPool
from sunaengine_gb300.data import mat_id
from sunaengine_gb300.engine import Batch, Engine
from sunaengine_gb300.engine3d import Engine3D

pytestmark = pytest.mark.gpu


def _water(n=1500, seed=3):
    return scenes.jittered_block(n, 1.0, np.random.Generator(np.random.PCG64(seed)))


@pytest.mark.parametrize('lanes', [0, 4])
def test_empty_rows_come_back_empty(lanes):
    sc = _water()
    e = Engine(max_particles=sc.n, lanes=lanes).load_scene(sc)
    pool = CheckpointPool(2 * e.ckpt_bytes() + 4096)
    e.step(5)
    want = e.read_state().copy()
    key = e.ckpt_save(pool)
    rows = np.zeros((sc.nFluid, 48), np.uint32)
    rows[0, 0] = (1000 << 17) | 1
    rows[1, 0] = 1000 << 17
    e.write_bonds(rows.reshape(-1))
    e.step(3)
    e.ckpt_load(pool, key)
    assert not e.read_bonds().any()
    assert np.array_equal(e.read_state(), want)
    e.step(4)
    f = Engine(max_particles=sc.n).load_scene(sc)
    f.step(9)
    assert e.digest().hex == f.digest().hex and e.chain_hex() == f.chain_hex()


def test_live_rows_come_back():
    sc = scenes.make_scene('pool_v1', mat=mat_id('RUBBER'), w=20, h=10)
    e = Engine(max_particles=sc.n).load_scene(sc)
    pool = CheckpointPool(2 * e.ckpt_bytes() + 4096)
    e.step(5)
    rows = e.read_bonds().copy()
    assert rows.any()
    key = e.ckpt_save(pool)
    e.step(7)
    late = e.digest().hex
    f = Engine(max_particles=sc.n).load_scene(sc)  # no row of this world is live yet
    f.ckpt_load(pool, key)
    assert np.array_equal(f.read_bonds(), rows)
    f.step(7)
    assert f.digest().hex == late and f.chain_hex() == e.chain_hex()


def test_chains_after_loads_resets_and_scrubs():
    sc = _water()
    e = Engine(max_particles=sc.n).load_scene(sc)
    c0 = e.chain_hex()
    pool = CheckpointPool(2 * e.ckpt_bytes() + 4096)
    e.step(2)
    c2, key = e.chain_hex(), e.ckpt_save(pool)
    e.step(1)
    c3 = e.chain_hex()
    assert len({c0, c2, c3}) == 3
    e.ckpt_load(pool, key)
    assert e.chain_hex() == c2
    e.step(1)
    assert e.chain_hex() == c3
    e.reset_chain()
    assert e.chain_hex() == c0
    e.load_scene(sc)
    assert e.chain_hex() == c0
    b = Batch(max_particles=6000, max_scenes=2)
    i = b.add_scene(sc)
    b.step(2)
    j = b.add_scene(_water(900, 5))
    assert b.chain_hex(i) == c2 and b.chain_hex(j) == c0
    b.step(1)
    assert b.chain_hex(i) == c3 and b.chain_hex(j) != c0


def test_chains_3d():
    sc = tables3d.initial_state(2000)
    e = Engine3D(max_particles=sc.n).load_scene(sc)
    c0 = e.chain_hex()
    pool = CheckpointPool(e.ckpt_bytes() + 4096)
    e.step(2)
    c2, key = e.chain_hex(), e.ckpt_save(0, pool)
    e.step(1)
    c3, d3 = e.chain_hex(), e.digest().hex
    e.ckpt_load(0, pool, key)
    assert e.chain_hex() == c2 and e.digest().hex != d3
    e.step(1)
    assert e.chain_hex() == c3 and e.digest().hex == d3
    e.load_scene(sc)
    assert e.chain_hex() == c0
