"""The fused 3D substep against the per-phase kernels (a pinned lane split keeps a
world on those): sizes at the lane splits' limits, the largest it takes and one
above, rows of candidates past two filter words, bonds, ball, stir, several
scenes, spawns."""
import numpy as np
import pytest

from sunaengine_gb300 import tables3d
from sunaengine_gb300.engine3d import Engine3D

pytestmark = pytest.mark.gpu


def _column(side, g=None):
    g = g or min(52, max(8, side))
    return tables3d.column_fast(side, side, side, g, g, g)


def _pair(sc, extra=0, load=None, **kw):
    out = []
    for lanes in (0, 1):
        e = Engine3D(max_particles=sc.n + extra, lanes=lanes, **kw)
        e.load_scene(sc, **(load or {}))
        out.append(e)
    return out


def _same(a, b, steps):
    for k in steps:
        a.step(k)
        b.step(k)
        assert a.digest().hex == b.digest().hex
        assert a.chain() == b.chain()
    assert a.chain_hex() == b.chain_hex()
    assert np.array_equal(a.read_state(), b.read_state())
    assert np.array_equal(a.read_bonds(), b.read_bonds())
    a.sync()
    b.sync()


@pytest.mark.parametrize('side', [1, 2, 7, 21, 22, 26, 27, 33, 34, 47, 50, 52])
def test_sizes(side):
    sc = _column(side)
    a, b = _pair(sc, max_cells=1 << 18)
    _same(a, b, [1, 5])
    assert (a.last_timing()[1] == 5) == (side <= 50)  # one launch a substep
    assert b.last_timing()[1] > 5 * 10


@pytest.mark.parametrize('iters', [1, 3, 4])
def test_iterations_ball_and_stir(iters):
    sc = tables3d.initial_state(6000)
    es = _pair(sc, iters=iters, load={'stir_amp': 900})
    for e in es:
        e.set_ball(True, 14.0, 9.0, 12.0, 3.0)
    _same(*es, [1, 6])


def test_overdense_rows():
    """0.4 wu spacing: rows of well over 64 candidates, every list truncated."""
    sc = tables3d.initial_state(9000, 'overdense')
    _same(*_pair(sc), [1, 4])


def test_bonds():
    sc = _column(16, 20)
    rows = tables3d.bond_rows(sc, tables3d.lattice_bonds(16, 16, 16, 900, 4))
    es = _pair(sc)
    for e in es:
        e.write_bonds(rows, tables3d.DAM3D_BOND_K, 70000)
    _same(*es, [1, 30])


def test_spawn_and_scenes():
    sc = tables3d.initial_state(3000)
    es = []
    for lanes in (0, 1):
        e = Engine3D(max_particles=9000, max_scenes=3, lanes=lanes)
        e.add_scene(sc, cap=4000)
        e.step(2)
        e.spawn(0, 20.0, 30.0, 20.0, 700)
        sid = e.add_scene(_column(11), cap=1500)
        e.step(3)
        e.remove_scene(sid)
        e.step(2)
        e.add_scene(_column(9), cap=800)
        es.append(e)
    _same(*es, [3])
