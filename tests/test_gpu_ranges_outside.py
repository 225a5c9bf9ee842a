"""Rows and tables on both sides of what the release arithmetic is built for.

Every route has to give the debug engine's words, and the oracle's: rows outside
run the wide form of the two post sweeps, tables outside the debug kernels.
"""
import numpy as np
import pytest

import oracle
from sunaengine_gb300 import data, scenes, tables3d
from sunaengine_gb300.engine import Engine
from sunaengine_gb300.engine3d import Engine3D

pytestmark = pytest.mark.gpu

XSPH, COH, CUR, ADHESION, COND, CORRODE, CORR_PT, CORR_TO = 2, 4, 5, 6, 8, 28, 29, 30
BOUNDS = {XSPH: 1 << 22, COH: 1 << 19, CUR: 2047, ADHESION: 1 << 22, COND: 1 << 17, CORRODE: 1 << 24}


def _scene():
    """Water and oil mixed against the walls, every pair's temperatures further
    apart than the conducted difference is clamped to, velocities at random."""
    sc = scenes.make_scene('pool_v1', w=40, h=16)
    rng = np.random.Generator(np.random.PCG64(11))
    k = rng.integers(0, 2, sc.nFluid)
    sc.matId[:sc.nFluid] = np.where(k, data.mat_id('WATER'), data.mat_id('OIL'))
    sc.temp = np.zeros(sc.n, np.int32)
    sc.temp[:sc.nFluid] = np.where(k, 1 << 25, -(1 << 24))
    sc.vel[:sc.nFluid] = rng.integers(-65536, 65537, (sc.nFluid, 2))
    return sc


def _agree(sc, steps, **kw):
    es = [Engine(max_particles=sc.n, **k, **kw).load_scene(sc)
          for k in ({}, {'lanes': 1}, {'lanes': 8}, {'debug': True})]
    o = oracle.OracleEngine(sc.n, **{'luts' if k == 'tables' else k: v for k, v in kw.items()}).load_scene(sc)
    for _ in range(steps):
        o.step(1)
        for e in es:
            e.step(1)
        assert [e.digest().hex for e in es] == [o.digest()] * len(es)
    return es


@pytest.mark.parametrize('word', sorted(BOUNDS))
@pytest.mark.parametrize('over', ['at', 'past', 'far', 'negative'])
def test_rows(word, over):
    b = BOUNDS[word]
    mats = np.asarray(data.mats()).reshape(-1, 48).copy()
    rows = [data.mat_id('WATER'), data.mat_id('OIL')]
    mats[rows, word] = {'at': b, 'past': b + 1, 'far': 1 << 29, 'negative': -4 * b}[over]
    if word == CORRODE:  # rows that do corrode: a threshold that a few full terms reach
        mats[rows, CORR_PT] = 1 << 18
        mats[rows, CORR_TO] = rows[::-1]
    _agree(_scene(), 3, mats=mats)


def test_a_row_minted_outside_and_cleared():
    """set_material moves a running world to the wide sweeps and back."""
    sc = scenes.jittered_block(900, 1.0, np.random.Generator(np.random.PCG64(4)))
    a, b = Engine(max_particles=sc.n).load_scene(sc), Engine(max_particles=sc.n, debug=True).load_scene(sc)
    row = np.asarray(data.mats()).reshape(-1, 48)[data.mat_id('WATER')].copy()
    row[COND] = 1 << 20
    launches = []
    for change in (None, lambda e: e.set_material(len(data.mats()), row), lambda e: e.clear_materials()):
        for e in (a, b):
            if change:
                change(e)
            e.step(2)
        launches.append(a.last_timing()[1])
        assert a.digest().hex == b.digest().hex
    assert launches[0] == launches[2] == 2 and launches[1] > 40


@pytest.mark.parametrize('table', ['W', 'G', 'C', 'A'])
def test_2d_tables(monkeypatch, table):
    luts = np.asarray(data.luts()).astype(np.int64).reshape(5, -1)
    i = 'WGCA'.index(table)
    luts[i] *= {'W': 2, 'G': 2, 'C': 4, 'A': 4}[table]
    luts = luts.reshape(-1).astype(np.int32)
    monkeypatch.setattr(data, 'TABLE_HASH', data.table_hash(luts))
    es = _agree(_scene(), 2, tables=luts)
    assert es[0].last_timing()[1] > 20


def test_3d_tables(monkeypatch):
    luts = np.asarray(tables3d.luts3d()).astype(np.int64)
    luts[2049:2 * 2049] *= 2
    luts = luts.astype(np.int32)
    monkeypatch.setattr(tables3d, 'luts3d', lambda: luts)
    sc = tables3d.initial_state(3000, 'pool', 16, 16, 16)
    es = [Engine3D(max_particles=sc.n, **k).load_scene(sc) for k in ({}, {'lanes': 1}, {'debug': True})]
    for _ in range(4):
        for e in es:
            e.step(1)
        assert len({e.chain_hex() for e in es}) == 1
    assert es[0].last_timing()[1] > 4
