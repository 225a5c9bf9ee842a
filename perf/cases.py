"""The work that users of this framework have it do, as cases to time.

Each case is one pass through the public entry points (`Engine`, `Batch`,
`Engine3D`, `CheckpointPool`): an interactive page's frame, a replay from a
device keyframe, a scene load, a serving quantum over many scenes. A pass ends
as its caller's does, with the state digest, the chain and the state words read
back. All outputs are 32-bit words that have to be equal, not near.

Kinds:

* ``frame``  -- ``Engine.frame()`` (2 substeps) on a scene that keeps running;
* ``replay`` -- ``ckpt_load`` of a keyframe, then ``step(steps)`` (scrubbing, a
  replay job): every pass starts from the same keyframe;
* ``load``   -- ``load_scene`` from host arrays, then ``step(steps)``;
* ``batch``  -- ``Batch.step(steps)`` over scenes of uneven sizes with queued
  stir impulses (lockstep peers, a serving quantum);
* ``site``   -- ``frame`` of a scene with rigid bodies and seal rails;
* ``frame3d``, ``replay3d`` -- the 3D engine's frame and replay.
"""
from __future__ import annotations

import math

import numpy as np

from sunaengine_gb300 import data, scenes, serving, tables3d
from sunaengine_gb300.checkpoints import CheckpointPool
from sunaengine_gb300.engine import Batch, Engine
from sunaengine_gb300.engine3d import Engine3D

ONE = scenes.ONE


def listed():
    return [
        # the 4096-particle dam break, one page frame: the smallest call
        {'name': 'frame_4k', 'kind': 'frame', 'scene': 'block', 'n': 4096, 'steps': 2, 'settle': 60},
        # the page at the particle count its own performance notes quote
        {'name': 'frame_40k', 'kind': 'frame', 'scene': 'block', 'n': 40000, 'steps': 2, 'settle': 100},
        # a pool of gel: friction rows, live bonds and bond formation
        {'name': 'gel_6k', 'kind': 'frame', 'scene': 'gel', 'n': 6100, 'steps': 4, 'settle': 40},
        # 48 rigid bodies and held seal rails in a 74k-particle tank
        {'name': 'site_74k', 'kind': 'site', 'n': 74384, 'bays': 24, 'steps': 4, 'settle': 20},
        # a scrub inside one checkpoint interval of a small serving job
        {'name': 'replay_15k', 'kind': 'replay', 'scene': 'block', 'n': 15427, 'steps': 50, 'settle': 100},
        # the two-fluid thermal scene at a quarter of its size, settled
        {'name': 'replay_262k', 'kind': 'replay', 'scene': 'two_fluid', 'n': 262144, 'steps': 20, 'settle': 200},
        # the two-fluid thermal scene at its stated size
        {'name': 'replay_1m', 'kind': 'replay', 'scene': 'two_fluid', 'n': 1048576, 'steps': 10, 'settle': 60},
        # opening a scene: upload, checks, packing, the first frame
        {'name': 'load_131k', 'kind': 'load', 'scene': 'two_fluid', 'n': 131044, 'steps': 2, 'settle': 0},
        # a serving quantum over uneven scenes, 1k to 64k particles each
        {'name': 'batch_48', 'kind': 'batch', 'scenes': 48, 'n_lo': 1024, 'n_hi': 65536, 'n': 756000, 'steps': 25},
        # lockstep peers: twins of one small size
        {'name': 'batch_16x4k', 'kind': 'batch', 'scenes': 16, 'n_lo': 4096, 'n_hi': 4097, 'n': 65536, 'steps': 25},
        # the 3D page's starting pool, one frame
        {'name': 'frame3d_16k', 'kind': 'frame3d', 'n': 16000, 'steps': 2, 'settle': 60},
        # the 3D dam break with its lattice bonds
        {'name': 'replay3d_262k', 'kind': 'replay3d', 'n': 262144, 'bonds': 4096, 'steps': 20, 'settle': 60},
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def draw(rng):
    kind = rng.choice(['frame', 'frame', 'gel', 'site', 'replay', 'replay', 'two_fluid', 'two_fluid', 'load',
                       'batch', 'batch', 'frame3d', 'replay3d', 'replay3d'])
    if kind == 'frame':
        return {'kind': 'frame', 'scene': 'block', 'n': _log(rng, 1024, 80000), 'steps': 2,
                'settle': rng.randint(10, 120)}
    if kind == 'gel':
        return {'kind': 'frame', 'scene': 'gel', 'n': _log(rng, 600, 6100), 'steps': rng.randint(2, 4),
                'settle': rng.randint(10, 60)}
    if kind == 'site':
        bays = _log(rng, 2, 24)
        return {'kind': 'site', 'n': 3100 * bays, 'bays': bays, 'steps': rng.randint(2, 4),
                'settle': rng.randint(5, 30)}
    if kind == 'replay':
        return {'kind': 'replay', 'scene': 'block', 'n': _log(rng, 2000, 262144), 'steps': rng.randint(10, 50),
                'settle': rng.randint(20, 120)}
    if kind == 'two_fluid':
        n = _log(rng, 16384, 1048576)
        return {'kind': 'replay', 'scene': 'two_fluid', 'n': n, 'steps': rng.randint(5, 10),
                'settle': rng.randint(20, 60)}
    if kind == 'load':
        return {'kind': 'load', 'scene': rng.choice(['block', 'two_fluid']), 'n': _log(rng, 4096, 524288),
                'steps': 2, 'settle': 0}
    if kind == 'batch':
        count, lo = rng.randint(4, 48), _log(rng, 1024, 8192)
        hi = max(lo + 1, _log(rng, 8192, 65536))
        mean = (hi - lo) / math.log(hi / lo)
        return {'kind': 'batch', 'scenes': count, 'n_lo': lo, 'n_hi': hi, 'n': int(count * mean),
                'steps': rng.randint(10, 25)}
    if kind == 'frame3d':
        return {'kind': 'frame3d', 'n': _log(rng, 2000, 60000), 'steps': 2, 'settle': rng.randint(10, 80)}
    n = _log(rng, 4096, 262144)
    return {'kind': 'replay3d', 'n': n, 'bonds': n // 64, 'steps': rng.randint(5, 20),
            'settle': rng.randint(20, 80)}


def _scene2d(case, seed):
    """The case's scene, its positions jittered from the seed."""
    n = case['n']
    if case['scene'] == 'two_fluid':
        return scenes.large_two_fluid(side=max(8, round(math.sqrt(n))), seed=seed)
    if case['scene'] == 'gel':
        h = max(6, min(61, round(math.sqrt(0.61 * n))))
        sc = scenes.make_scene('pool_v1', mat=data.mat_id('GEL'), w=max(10, min(100, round(n / h))), h=h)
        rng = np.random.Generator(np.random.PCG64(seed))
        sc.pos[:sc.nFluid] += rng.integers(-ONE // 16, ONE // 16 + 1, size=(sc.nFluid, 2)).astype(np.int32)
        return sc
    # the block's shape goes by its size, from tall to wide
    return scenes.jittered_block(n, 0.7 + n % 10 / 10, np.random.Generator(np.random.PCG64(seed)))


def _engine2d(case, seed):
    sc = scenes.construction_site(tiles=case['bays'], seed=seed % 0x7fffffff + 1) if case['kind'] == 'site' \
        else _scene2d(case, seed)
    e = Engine(max_particles=sc.n).load_scene(sc)
    if case['kind'] == 'site':
        for slots in sc.meta['planks']:
            e.make_rigid_body(slots)
        for slots, (cx, cy) in zip(sc.meta['wheels'], sc.meta['wheel_pivots']):
            e.make_axis_body(slots, cx, cy)
    return sc, e


def _batch(case, seed):
    """Scenes of log-uniform sizes and aspect ratios in [0.5, 2] (drawn from the
    case), their jitter and their stir schedules (drawn from the seed)."""
    size = np.random.Generator(np.random.PCG64([case['scenes'], case['n_lo'], case['n_hi']]))
    out = []
    for k in range(case['scenes']):
        n = round(math.exp(size.uniform(math.log(case['n_lo']), math.log(case['n_hi']))))
        aspect = float(size.uniform(0.5, 2.0))
        rng = np.random.Generator(np.random.PCG64([seed, k]))
        sc = scenes.jittered_block(n, aspect, rng)
        out.append((sc, scenes.stir_schedule(sc, 6000, rng)))
    return out


def _scene3d(case):
    """A water column in the corner of a box, as the serving jobs lay it out."""
    side = max(4, round(case['n'] ** (1 / 3)))
    g = min(52, max(8, math.ceil((side + 3) * 1.5 / 2)))
    return side, tables3d.column_fast(side, side, side, g, min(52, max(8, math.ceil((side + 3) / 2) + 6)), g)


def prepare(case, seed):
    st = {'kind': case['kind'], 'steps': case['steps']}
    kind = case['kind']
    if kind == 'batch':
        scs, sched = zip(*_batch(case, seed))
        b = Batch(max_particles=sum(s.n for s in scs), max_scenes=len(scs),
                  max_cells=sum(serving.scenes_cells_2d(s) for s in scs))
        ids = []
        for sc, ev in zip(scs, sched):
            sid = b.add_scene(sc)
            for e in ev:
                b.schedule_impulse(sid, *e)
            ids.append(sid)
        b.step(1)
        st.update(batch=b, ids=ids, at=np.cumsum([0] + [s.n * 8 for s in scs]))
        st['words'] = np.zeros(int(st['at'][-1]), np.int32)
    elif kind in ('frame3d', 'replay3d'):
        rng = np.random.Generator(np.random.PCG64(seed))
        stir = int(rng.integers(200, 1500))
        if kind == 'frame3d':
            sc = tables3d.initial_state(case['n'])
            e = Engine3D(max_particles=sc.n).load_scene(sc, stir_amp=stir)
            e.set_ball(True, *(float(v) for v in rng.uniform(8.0, 24.0, 3)), 3.0)
        else:
            side, sc = _scene3d(case)
            e = Engine3D(max_particles=sc.n, max_cells=sc.gx * sc.gy * sc.gz, iters=4).load_scene(sc, stir_amp=stir)
            e.write_bonds(tables3d.bond_rows(sc, tables3d.lattice_bonds(side, side, side, case['bonds'], seed)),
                          tables3d.DAM3D_BOND_K, tables3d.DAM3D_BOND_BRK)
        e.step(case['settle'])
        st.update(engine=e, words=np.zeros(sc.n * 8, np.int32))
        if kind == 'replay3d':
            st['pool'] = CheckpointPool(e.ckpt_bytes() + (1 << 20))
            st['key'] = e.ckpt_save(0, st['pool'])
    else:
        if kind == 'load':
            sc = _scene2d(case, seed)
            st.update(engine=Engine(max_particles=sc.n), scene=sc)
        else:
            sc, e = _engine2d(case, seed)
            e.step(case['settle'])
            st['engine'] = e
            if kind == 'replay':
                st['pool'] = CheckpointPool(e.ckpt_bytes() + (1 << 20))
                st['key'] = e.ckpt_save(st['pool'])
        st['words'] = np.zeros(sc.n * 8, np.int32)
    return st


def run(st):
    kind = st['kind']
    if kind == 'batch':
        b, at, words = st['batch'], st['at'], st['words']
        b.step(st['steps'])
        digests = np.concatenate([b.digest(i).acc for i in st['ids']])
        for k, i in enumerate(st['ids']):
            b.read_state(i, out=words[at[k]:at[k + 1]])
        return {'digests': digests, 'state': words}
    e = st['engine']
    if kind in ('frame3d', 'replay3d'):
        if kind == 'replay3d':
            e.ckpt_load(0, st['pool'], st['key'])
        e.run_substeps(st['steps'])
        return {'digest': e.digest().acc, 'chain': e.chain_words(), 'state': e.read_state(out=st['words'])}
    if kind == 'load':
        e.load_scene(st['scene'])
    elif kind == 'replay':
        e.ckpt_load(st['pool'], st['key'])
    e.step(st['steps'])
    return {'digest': e.digest().acc, 'chain': e.chain_words(), 'state': e.read_state(out=st['words'])}


def work(case):
    """The phase-minimal bytes of a particle-substep (each dependent phase of
    the substep reads each particle's fields once and writes its outputs once:
    792 B in 2D at 4 iterations, 432 and 520 B in 3D at 3 and 4), and its
    integer operations: about 20 (3D: 30) neighbours in each sweep of the
    list (2D 14, 3D 7 and 9) at about 30 operations a pair."""
    ps = case['n'] * case['steps']
    if case['kind'] == 'frame3d':
        return {'bytes': 432 * ps, 'flops': 30 * 7 * 30 * ps}
    if case['kind'] == 'replay3d':
        return {'bytes': 520 * ps, 'flops': 30 * 9 * 30 * ps}
    return {'bytes': 792 * ps, 'flops': 20 * 14 * 30 * ps}


def exact(case, seed):
    """None: every output is a word of the deterministic integer state, its
    digest or its chain. None of them is a rounded number, so they are equal
    or they are wrong."""
    return None
