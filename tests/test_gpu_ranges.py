"""The release build's shortened arithmetic at the ends of its ranges.

Release and debug engines have to agree word by word where the densities pass
the closed form's last shifts (a mean above 4 and 8 rest densities), and where
a material row lies outside what the release kernels take (those worlds run the
debug kernels).
"""
import numpy as np
import pytest

from sunaengine_gb300 import data, scenes
from sunaengine_gb300.engine import Engine

pytestmark = pytest.mark.gpu


def _same(sc, steps, **kw):
    es = [Engine(max_particles=sc.n, **k, **kw).load_scene(sc) for k in ({}, {'lanes': 1}, {'debug': True})]
    for _ in range(steps):
        for e in es:
            e.step(1)
        d = [e.digest().hex for e in es]
        assert d[0] == d[1] == d[2]
    for e in es:
        e.check_errors()
    return es


@pytest.mark.parametrize('spread', [64, 20000, 60000])
def test_piled_particles(spread):
    """Hundreds of particles inside a fraction of the kernel radius."""
    sc = scenes.jittered_block(600, 1.0, np.random.Generator(np.random.PCG64(3)))
    rng = np.random.Generator(np.random.PCG64(spread))
    sc.pos[:400] = np.array([10 * scenes.ONE, 12 * scenes.ONE]) + rng.integers(-spread, spread + 1, (400, 2))
    _same(sc, 4)


def test_held_pile():
    """Anchored particles keep their pile: full lists at 10 rest densities."""
    sc = scenes.jittered_block(600, 1.0, np.random.Generator(np.random.PCG64(3)))
    rng = np.random.Generator(np.random.PCG64(8))
    sc.pos[:300] = np.array([10 * scenes.ONE, 12 * scenes.ONE]) + rng.integers(-9000, 9001, (300, 2))
    sc.flags = np.zeros(sc.n, np.uint32)
    sc.flags[:200] = 4
    rho, _ = _same(sc, 4)[0].read_fields()
    assert rho.max() > 8 << 20


@pytest.mark.parametrize('word,value', [(4, 1 << 19), (4, (1 << 19) + 1), (4, -(1 << 29)), (5, 2047), (5, 2048),
                                        (5, 1 << 22)])
def test_rows_at_the_range(word, value):
    mats = np.asarray(data.mats()).reshape(-1, 48).copy()
    mats[0, word] = value
    sc = scenes.jittered_block(900, 1.0, np.random.Generator(np.random.PCG64(4)))
    _same(sc, 3, mats=mats)
