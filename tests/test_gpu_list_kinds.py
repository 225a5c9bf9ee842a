"""Neighbour lists of worlds with live SEAL or CONGEAL particles: the filtered
build has to raise the same list flags as the debug build's scan of every
candidate, also for hits past a full list. Cells are filled to the edges of a
filter word and far past what a list holds, the seal particles last in slot
order (past the cut), first, or spread.
"""
import numpy as np
import pytest

from sunaengine_gb300 import scenes
from sunaengine_gb300.data import mat_id
from sunaengine_gb300.engine import Engine

pytestmark = pytest.mark.gpu
CELL = 1 << 18


def _scene(per_cell, where, seal):
    rng = np.random.Generator(np.random.PCG64([per_cell, len(where)]))
    n = per_cell * 9
    pos = np.zeros((n, 2), np.int64)
    cell = np.arange(n) % 9
    pos[:, 0] = (1 + cell % 3) * CELL + rng.integers(0, CELL, n)
    pos[:, 1] = (2 + cell // 3) * CELL + rng.integers(0, CELL, n)
    mat = np.zeros(n, np.uint32)
    k = max(1, n // 40)
    at = {'last': slice(n - k, n), 'first': slice(0, k), 'spread': slice(0, n, 40)}[where]
    mat[at] = mat_id(seal)
    sc = scenes._assemble(pos, mat, scenes.boundary_ring(24, 24, 20), 24, 24, 'kinds')
    fl = np.zeros(sc.n, np.uint32)
    fl[:n][at] = 4  # held
    sc.flags = fl
    return sc


@pytest.mark.parametrize('lanes', [0, 1, 2, 4, 8])
@pytest.mark.parametrize('where', ['last', 'first', 'spread'])
@pytest.mark.parametrize('per_cell', [3, 31, 33, 61, 66, 130])
def test_kinds(per_cell, where, lanes):
    for seal in ('RUBBER', 'STONE'):
        sc = _scene(per_cell, where, seal)
        a = Engine(max_particles=sc.n, lanes=lanes).load_scene(sc)
        b = Engine(max_particles=sc.n, debug=True).load_scene(sc)
        for _ in range(3):
            a.step(1)
            b.step(1)
            assert a.digest().hex == b.digest().hex
            for x, y in zip(a.read_fields(), b.read_fields()):
                assert np.array_equal(x, y)
        a.check_errors()
        b.check_errors()
