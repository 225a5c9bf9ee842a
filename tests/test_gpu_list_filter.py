"""The list build's candidate filter against the general scan.

Debug engines scan every candidate exactly; release engines filter them by
their place in 64ths of a cell first. Lists decide every later word, so equal
states, counts and densities mean equal lists. Cells are filled to the edges of
what a filter word (32) and the dealt cells (64) hold; positions sit on cell
borders and outside the domain; larger cells make the filter coarser.
"""
import numpy as np
import pytest

from sunaengine_gb300 import scenes
from sunaengine_gb300.data import mat_id
from sunaengine_gb300.engine import Engine

pytestmark = pytest.mark.gpu
CELL = 1 << 18


def _scene(per_cell, seed, cell_shift=18, dead=False):
    rng = np.random.Generator(np.random.PCG64([per_cell, seed]))
    dom = 24
    n = per_cell * 9 + 60
    pos = np.zeros((n, 2), np.int64)
    k = 0
    for cy in range(2, 5):  # nine full cells
        for cx in range(1, 4):
            pos[k:k + per_cell, 0] = cx * CELL + rng.integers(0, CELL, per_cell)
            pos[k:k + per_cell, 1] = cy * CELL + rng.integers(0, CELL, per_cell)
            pos[k:k + 4] = [(cx * CELL, cy * CELL), (cx * CELL, (cy + 1) * CELL - 1),
                            ((cx + 1) * CELL - 1, cy * CELL), (cx * CELL + 4096, cy * CELL + 4095)]
            k += per_cell
    # pairs around the kernel radius, on the axes and the diagonal
    r = 163840
    for j in range(20):
        pos[k:k + 3] = [(2 * CELL + 7 * j, CELL // 2), (2 * CELL + 7 * j + r + j - 10, CELL // 2),
                        (2 * CELL + 7 * j + 115852 + j - 10, CELL // 2 + 115852 + j - 10)]
        k += 3
    mat = np.zeros(n, np.uint32)
    if dead:
        mat[::5] = mat_id('VOID')
    sc = scenes._assemble(pos, mat, scenes.boundary_ring(dom, dom, dom - 4), dom, dom, 'filter')
    sc.cellShift = cell_shift
    return sc


@pytest.mark.parametrize('lanes', [0, 1, 2, 4, 8])
@pytest.mark.parametrize('per_cell', [4, 29, 32, 33, 61, 65, 130])
def test_cell_occupancies(per_cell, lanes):
    _compare(_scene(per_cell, 1), lanes)


@pytest.mark.parametrize('cell_shift', [19, 20, 24])
def test_larger_cells(cell_shift):
    for lanes in (0, 1, 4):
        _compare(_scene(20, 2, cell_shift), lanes)


def test_dead_particles():
    for lanes in (0, 1, 4):
        _compare(_scene(31, 3, dead=True), lanes)


def _compare(sc, lanes):
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
