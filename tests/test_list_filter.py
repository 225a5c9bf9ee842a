"""The list build's candidate filter restated in numpy, against the exact rule.

No neighbour may be dropped, nothing outside the kernel may be taken as near,
a dead particle's code is always dropped: over every cell size, pairs about the
kernel radius, places on cell borders and outside the cells (which are clamped).
"""
import numpy as np
import pytest

HS, H2S = 10240, 104857600


def _in_kernel(d):
    a = (np.abs(d) + 8) >> 4
    return (a.max(1) <= HS) & ((a * a).sum(1) < H2S)


def _dot(word):
    b = [(word >> (8 * k)) & 0xff for k in range(4)]
    return sum(np.where(v > 127, v - 256, v) ** 2 for v in b)


@pytest.mark.parametrize('cell_shift', [18, 19, 20, 24, 27])
@pytest.mark.parametrize('margin', [0, 200000])
def test_filter_bounds(cell_shift, margin):
    rng = np.random.default_rng([cell_shift, margin])
    sh = cell_shift - 6
    far = -((((4 * (HS + 1) * 16) >> sh) + 1 + 9) ** 2 // 16 + 4)
    near = -(max(((4 * (HS * 16 - 12)) >> sh) - 9, 0) ** 2 // 16)
    for cells in (1, 2, 3, 7):
        n, span = 200000, cells << cell_shift
        pi = rng.integers(-margin, span + margin, (n, 2))
        ang = rng.uniform(0, 2 * np.pi, n)
        rad = np.where(rng.random(n) < 0.5, 163840 + rng.integers(-12000, 12000, n), rng.uniform(0, 200000, n))
        pj = pi + np.stack([rad * np.cos(ang), rad * np.sin(ang)], 1).astype(np.int64)
        qi, qj = (np.clip(p >> sh, 0, cells * 64 - 1) for p in (pi, pj))
        ci, cj = qi >> 6, qj >> 6
        ok = (np.abs(cj - ci) <= 1).all(1) & (pj >= -margin).all(1) & (pj < span + margin).all(1)
        pi, pj, qi, qj, ci, cj = (x[ok] for x in (pi, pj, qi, qj, ci, cj))
        own = (qi[:, 0] & 63) | (qi[:, 1] & 63) << 16
        bias = (cj - ci)[:, 0] * 64 + (cj - ci)[:, 1] * (64 << 16) - own
        dot = _dot(((qj[:, 0] & 63 | (qj[:, 1] & 63) << 16) + bias) & 0xffffffff)
        want = _in_kernel(pj - pi)
        assert (dot + far < 0)[want].all()
        exact_only = (pi >> cell_shift != ci).any(1) | ((cj == 0) | (cj == cells - 1)).any(1)
        assert want[(dot + near < 0) & ~exact_only].all()
        assert (_dot((0x4000 + bias) & 0xffffffff) + far >= 0).all()


@pytest.mark.parametrize('cells', [1, 2, 7, 52])
def test_filter_bounds_3d(cells):
    """The 3D filter: places modulo 256, three bytes, r2q's floored axes."""
    rng = np.random.default_rng(cells)
    n, span, margin = 400000, cells << 17, 32768
    pi = rng.integers(margin, span - margin + 1, (n, 3))
    v = rng.normal(size=(n, 3))
    rad = np.where(rng.random(n) < 0.7, 131072 + rng.integers(-9000, 9000, n), rng.uniform(0, 200000, n))
    pj = pi + (v / np.linalg.norm(v, axis=1)[:, None] * rad[:, None]).astype(np.int64)
    ok = ((pj >> 17) - (pi >> 17) >= -1).all(1) & ((pj >> 17) - (pi >> 17) <= 1).all(1)
    ok &= (pj >= margin).all(1) & (pj <= span - margin).all(1)
    pi, pj = pi[ok], pj[ok]
    code = lambda p: ((p >> 11) & 255) @ np.array([1, 256, 65536])
    dot = _dot((code(pj) - code(pi)) & 0xffffffff)
    q = (pj - pi) >> 8
    want = (q * q).sum(1) < 262144
    assert (dot <= 4520)[want].all()
    assert want[dot < 3694].all()
    assert want.any()
