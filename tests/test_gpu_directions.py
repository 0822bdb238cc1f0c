"""Types and steepest-path labels at the edges of tiles (32 x 8 x 4) and of
grids, with ties, infinities and signed zeros: against an exhaustive evaluation
in numpy over (value, id)."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIRS = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (-1, 1, 0), (1, -1, 0),
        (0, 1, 1), (0, -1, -1), (-1, 0, 1), (1, 0, -1), (-1, 1, 1), (1, -1, -1)]


def roots(f, ascent):
    """Steepest-path roots: the largest (smallest) of (value, id) over the closed
    star, followed to its fixed point."""
    d, h, w = f.shape
    ids = np.arange(f.size).reshape(f.shape)
    best_v, best_i = f.copy(), ids.copy()
    for dx, dy, dz in DIRS:
        src = [slice(max(0, o), n + min(0, o)) for o, n in ((dz, d), (dy, h), (dx, w))]
        dst = [slice(max(0, -o), n + min(0, -o)) for o, n in ((dz, d), (dy, h), (dx, w))]
        v, i = f[tuple(src)], ids[tuple(src)]
        bv, bi = best_v[tuple(dst)], best_i[tuple(dst)]
        take = (v > bv) | ((v == bv) & (i > bi)) if ascent else (v < bv) | ((v == bv) & (i < bi))
        best_v[tuple(dst)] = np.where(take, v, bv)
        best_i[tuple(dst)] = np.where(take, i, bi)
    p = best_i.ravel()
    while True:
        q = p[p]
        if np.array_equal(p, q):
            return p
        p = q


SHAPES = [(32, 8, 4), (33, 9, 5), (31, 7, 3), (64, 16, 8), (65, 17, 9), (40, 24, 13), (34, 1, 6),
          (1, 9, 5), (96, 24, 1), (2, 2, 2), (36, 10, 12)]


@pytest.mark.parametrize("w,h,d", SHAPES)
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("kind", ["noise", "ties", "zeros", "inf"])
def test_labels_and_types(w, h, d, dtype, kind):
    import torch
    from extrem_z_b200 import api
    from oracle import ffi
    rng = np.random.default_rng(w * 10007 + h * 101 + d)
    f = rng.standard_normal((d, h, w))
    if kind == "ties":
        f = np.round(f * 2)
    elif kind == "zeros":
        f = np.where(rng.random(f.shape) < 0.5, 0.0, -0.0) + np.where(rng.random(f.shape) < 0.3, f, 0.0)
        f[rng.random(f.shape) < 0.3] *= -0.0
    elif kind == "inf":
        f[rng.random(f.shape) < 0.02] = np.inf
        f[rng.random(f.shape) < 0.02] = -np.inf
    f = np.ascontiguousarray(f.astype(dtype))
    t, up, down = api.context(0).classify(torch.from_numpy(f).cuda())
    assert np.array_equal(up.cpu().numpy().ravel(), roots(f, True))
    assert np.array_equal(down.cpu().numpy().ravel(), roots(f, False))
    assert np.array_equal(t.cpu().numpy().ravel(), np.asarray(ffi.classify(f)[0]).ravel())
