"""Bond gather and formation with several lanes to a row, against one lane.

Rows near their 48 entries (a pile of gel at a third of its spacing), sparse
rows written by the host (a zero word ends a row, whatever follows it), rows
with tombstones, and formation on and off the clock.
"""
import numpy as np
import pytest

from sunaengine_gb300 import scenes
from sunaengine_gb300.data import mat_id
from sunaengine_gb300.engine import Engine

pytestmark = pytest.mark.gpu


def _pile(mat, spacing):
    side, one = 26, scenes.ONE
    pos = [(12 * one + int(x * spacing * one), 20 * one + int(y * spacing * one))
           for y in range(side) for x in range(side)]
    return scenes._assemble(pos, np.full(len(pos), mat_id(mat), np.uint32), scenes.boundary_ring(48, 48, 40), 48, 48,
                            'pile')


@pytest.mark.parametrize('lanes', [0, 1, 2, 4, 8])
@pytest.mark.parametrize('mat,spacing', [('GEL', 0.35), ('GEL', 1.0), ('RUBBER', 0.9), ('ICE', 0.5)])
def test_formation(mat, spacing, lanes):
    sc = _pile(mat, spacing)
    a = Engine(max_particles=sc.n, lanes=lanes).load_scene(sc)
    b = Engine(max_particles=sc.n, debug=True, lanes=1).load_scene(sc)
    _same(a, b, 9)


@pytest.mark.parametrize('lanes', [0, 2, 8])
def test_host_rows(lanes):
    sc = _pile('GEL', 1.0)
    a = Engine(max_particles=sc.n, lanes=lanes).load_scene(sc)
    b = Engine(max_particles=sc.n, debug=True, lanes=1).load_scene(sc)
    a.step(5)  # the pool bonds at its second formation
    b.step(5)
    rows = b.read_bonds().reshape(-1, 48).copy()
    assert (rows[:, 0] != 0).any()
    rng = np.random.Generator(np.random.PCG64(6))
    for r in range(0, len(rows), 3):
        n = int((rows[r] != 0).sum())
        if n > 3:
            rows[r, rng.integers(0, n)] = 0            # a gap: the rest of the row is not read
            rows[r, rng.integers(0, n)] |= 0x40000000  # a tombstone (or a lone one in the gap)
    for e in (a, b):
        e.write_bonds(rows.reshape(-1))
    _same(a, b, 7)


def _same(a, b, steps):
    for _ in range(steps):
        a.step(1)
        b.step(1)
        assert a.digest().hex == b.digest().hex
        assert np.array_equal(a.read_bonds(), b.read_bonds())
    assert np.array_equal(a.read_state(), b.read_state())
    a.check_errors()
    b.check_errors()
