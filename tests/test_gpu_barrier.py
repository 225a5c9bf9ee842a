"""A grid barrier that runs out: no word of the half-run substep is given out.

The wait is cut to nothing, so the first CTAs at a barrier give up, the kernel
ends by itself and the engine has to refuse every read until the scene is loaded
again or takes a checkpoint.
"""
import numpy as np
import pytest

from sunaengine_gb300 import scenes, tables3d
from sunaengine_gb300.checkpoints import CheckpointPool
from sunaengine_gb300.engine import Batch, Engine, EngineError
from sunaengine_gb300.engine3d import Engine3D

pytestmark = pytest.mark.gpu

WAIT = 1 << 31
TEXT = 'grid barrier'


def _block(n, seed=5):
    return scenes.jittered_block(n, 1.1, np.random.Generator(np.random.PCG64(seed)))


def _refused(*calls):
    for call in calls:
        with pytest.raises(EngineError, match=TEXT):
            call()


def _give_up(e):
    e.set_barrier_wait(0)
    e.step(2)  # queued: the second launch finds the first one's error
    _refused(e.sync)
    e.set_barrier_wait(WAIT)
    _refused(lambda: e.step(1))


@pytest.mark.parametrize('persistent', [False, True])
def test_engine_refuses_until_loaded(persistent):
    sc = _block(3000)
    want = Engine(max_particles=sc.n).load_scene(sc)
    want.step(6)
    e = Engine(max_particles=sc.n).set_persistent(persistent).load_scene(sc)
    with CheckpointPoolOf(e.ckpt_bytes()) as pool:
        e.step(3)
        key = e.ckpt_save(pool)
        digest = e.digest().hex
        for restore in (lambda: e.load_scene(sc), lambda: e.ckpt_load(pool, key)):
            _give_up(e)
            _refused(e.digest, e.chain_hex, e.read_state, e.read_scratch, e.read_bonds, e.read_fields,
                     e.check_errors, lambda: e.ckpt_save(pool))
            restore()
            e.check_errors()
            e.step(6 - e.substep_count)
            assert e.digest().hex == want.digest().hex and e.chain_hex() == want.chain_hex()
            assert np.array_equal(e.read_state(), want.read_state())
        e.ckpt_load(pool, key)
        assert e.digest().hex == digest


def test_batch_keeps_the_other_scenes_refused():
    b = Batch(max_particles=12000, max_scenes=3)
    scs = [_block(n, seed=n) for n in (2000, 1500)]
    ids = [b.add_scene(sc) for sc in scs]
    with CheckpointPoolOf(b.ckpt_bytes(ids[0]) * 2) as pool:
        b.step(2)
        key = b.ckpt_save(ids[0], pool)
        b.step(1)
        want = b.digest(ids[0]).hex, b.chain_hex(ids[0])
        _give_up(b)
        third = b.add_scene(_block(900))  # the world runs again, the others are void
        b.step(1)
        alone = Engine(max_particles=4000).load_scene(_block(900))
        alone.step(1)
        assert b.digest(third).hex == alone.digest().hex and b.chain_hex(third) == alone.chain_hex()
        for s in ids:
            _refused(lambda: b.digest(s), lambda: b.chain_hex(s), lambda: b.read_state(s))
        _refused(b.check_errors)
        b.ckpt_load(ids[0], pool, key)
        b.step(1)
        assert (b.digest(ids[0]).hex, b.chain_hex(ids[0])) == want
        _refused(lambda: b.digest(ids[1]))
        b.remove_scene(ids[1])
        b.check_errors()


def test_3d_refuses_until_restored():
    sc = tables3d.initial_state(6000, 'pool', 20, 20, 20)
    want = Engine3D(max_particles=2 * sc.n).load_scene(sc)
    want.step(5)
    e = Engine3D(max_particles=2 * sc.n, max_scenes=2)
    s = e.add_scene(sc)
    other = e.add_scene(sc)
    with CheckpointPoolOf(e.ckpt_bytes(s) * 2) as pool:
        e.step(2)
        key = e.ckpt_save(s, pool)
        words, chain = e.read_state(s), e.chain_words(s)
        for restore in (lambda: e.ckpt_load(s, pool, key), lambda: e.write_state(words, 2, chain, s)):
            _give_up(e)
            _refused(lambda: e.digest(s), lambda: e.chain_hex(s), lambda: e.chain(s), lambda: e.read_state(s),
                     lambda: e.ckpt_save(s, pool))
            restore()
            e.step(3)
            assert e.digest(s).hex == want.digest().hex and e.chain_hex(s) == want.chain_hex()
            assert np.array_equal(e.read_state(s), want.read_state())
            _refused(lambda: e.digest(other))


class CheckpointPoolOf:
    """A pool for a few checkpoints of `nbytes`, closed at the end."""

    def __init__(self, nbytes):
        self.pool = CheckpointPool(4 * (nbytes + 256))

    def __enter__(self):
        return self.pool

    def __exit__(self, *exc):
        self.pool.close()
