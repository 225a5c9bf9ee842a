"""Several engines in flight at once: the words are those of each alone, and from the
third on small worlds leave the SMs to the others (the per-phase launches)."""
import threading
import time

import numpy as np
import pytest

from sunaengine_gb300 import scenes, tables3d
from sunaengine_gb300.engine import Engine
from sunaengine_gb300.engine3d import Engine3D

pytestmark = pytest.mark.gpu

LONG = 1500  # substeps: tens of milliseconds of work, queued in a few


def _block(n, seed):
    return scenes.jittered_block(n, 1.1, np.random.Generator(np.random.PCG64(seed)))


def _make(kind, i):
    if kind == '3d':
        sc = tables3d.initial_state(2000 + 500 * i, 'pool', 16, 16, 16)
        return Engine3D(max_particles=sc.n).load_scene(sc)
    sc = _block(2000 + 500 * i, i)
    return Engine(max_particles=sc.n).load_scene(sc)


@pytest.mark.parametrize('kind', ['2d', '3d'])
def test_the_third_shares(kind):
    time.sleep(0.1)
    es = [_make(kind, i) for i in range(4)]
    for e in es:
        e.step(2)
        e.sync()
    launches = []
    for e, k in zip(es, (LONG, LONG, 5, 5)):
        e.step(k)
    for e, k in zip(es, (LONG, LONG, 5, 5)):
        launches.append(e.last_timing()[1] / k)
        e.sync()
    assert launches[0] == launches[1] == 1 and launches[2] > 10 and launches[3] > 10
    time.sleep(0.3)  # a crowd is remembered for a moment
    for i, (e, k) in enumerate(zip(es, (LONG, LONG, 5, 5))):
        e.step(3)
        assert e.last_timing()[1] == 3
        one = _make(kind, i)
        one.step(k + 5)
        assert e.chain_hex() == one.chain_hex() and e.digest().hex == one.digest().hex


def test_an_engine_nobody_waited_for_is_not_counted():
    time.sleep(0.1)
    es = [_make('2d', i) for i in range(3)]
    for e in es[:2]:
        e.step(2)
    es[2].step(20)
    es[2].sync()  # the others finished long ago, though no call waited for them
    time.sleep(0.3)
    for _ in range(3):
        es[2].step(4)
        es[2].sync()
    assert es[2].last_timing()[1] == 4


def test_threads():
    es = [_make(k, i) for i, k in enumerate(('2d', '2d', '3d', '2d', '3d', '2d'))]
    out = [None] * len(es)

    def frames(i):
        for _ in range(30):
            es[i].step(2)
            es[i].digest()
        out[i] = es[i].chain_hex()

    ts = [threading.Thread(target=frames, args=(i,)) for i in range(len(es))]
    for t in ts:
        t.start()
    for t in ts:
        t.join()
    for i, k in enumerate(('2d', '2d', '3d', '2d', '3d', '2d')):
        one = _make(k, i)
        one.step(60)
        assert out[i] == one.chain_hex()
