"""The grid's sort at the edges of its tile rule: the slots of a world (its
capacity) are the keys, so one scene at several capacities has to advance the
same way. Below, at and above the capacities where a tile takes more items.
"""
import functools

import numpy as np
import pytest

from sunaengine_gb300 import scenes
from sunaengine_gb300.engine import Engine

pytestmark = pytest.mark.gpu

SC = scenes.jittered_block(9000, 1.3, np.random.Generator(np.random.PCG64(11)))


def _run(cap):
    e = Engine(max_particles=cap, lanes=4).load_scene(SC)
    e.step(4)
    out = e.chain_hex(), e.read_state()[:SC.n * 8]
    e.check_errors()
    e.destroy()
    return out


@functools.lru_cache(None)
def _tight():
    return _run(SC.n)


@pytest.mark.parametrize('cap', [k * 131072 + d for k in (1, 2, 4, 8, 16) for d in (-1, 0, 1)])
def test_capacities(cap):
    chain, state = _run(cap)
    assert chain == _tight()[0]
    assert np.array_equal(state, _tight()[1])
