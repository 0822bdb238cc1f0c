"""Property test (CPU) of the tile search of light manifold rounds: starting
from the tiles whose pointers are recomputed, a tile whose halo holds a touched
label (an old label of a vertex in a recomputed tile) leads to the halo vertex's
tile.  Every vertex whose label changes, and every vertex that carries a touched
label at all, lies in a tile found that way."""

import numpy as np
import pytest

DIRS = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (-1, 1, 0), (1, -1, 0),
        (0, 1, 1), (0, -1, -1), (-1, 0, 1), (1, 0, -1), (-1, 1, 1), (1, -1, -1)]
TX, TY, TZ = 8, 4, 2  # smaller than the kernels' tiles, so that labels cross several


def labels(f, ascent):
    d, h, w = f.shape
    ids = np.arange(f.size).reshape(f.shape)
    bv, bi = f.copy(), ids.copy()
    for dx, dy, dz in DIRS:
        src = tuple(slice(max(0, o), n + min(0, o)) for o, n in ((dz, d), (dy, h), (dx, w)))
        dst = tuple(slice(max(0, -o), n + min(0, -o)) for o, n in ((dz, d), (dy, h), (dx, w)))
        v, i = f[src], ids[src]
        take = ((v > bv[dst]) | ((v == bv[dst]) & (i > bi[dst])) if ascent else
                (v < bv[dst]) | ((v == bv[dst]) & (i < bi[dst])))
        bv[dst] = np.where(take, v, bv[dst])
        bi[dst] = np.where(take, i, bi[dst])
    p = bi.ravel()
    while not np.array_equal(p, p[p]):
        p = p[p]
    return p.reshape(f.shape)


@pytest.mark.parametrize("seed", range(6))
def test_found_tiles_cover_the_touched_labels(seed):
    rng = np.random.default_rng(seed)
    shape = (9 + seed, 13, 21 + 3 * seed)
    f = rng.standard_normal(shape)
    for axis in range(3):  # smooth, so that labels span tiles
        f = f + np.roll(f, 1, axis) + np.roll(f, -1, axis)
    old = [labels(f, True), labels(f, False)]
    g = f.copy()
    changed = rng.random(shape) < 0.002
    changed.flat[rng.integers(f.size)] = True
    g[changed] -= rng.random(int(changed.sum())) * 5
    new = [labels(g, True), labels(g, False)]
    z, y, x = np.indices(shape)
    tile = np.stack([z // TZ, y // TY, x // TX], -1)
    grid = [-(-n // t) for n, t in zip(shape, (TZ, TY, TX))]
    # Recomputed: tiles whose halo holds a changed vertex.
    found = set()
    for v in np.argwhere(changed):
        lo, hi = np.maximum(v - 1, 0), np.minimum(v + 1, np.array(shape) - 1)
        for c in range(lo[0] // TZ, hi[0] // TZ + 1):
            for b in range(lo[1] // TY, hi[1] // TY + 1):
                for a in range(lo[2] // TX, hi[2] // TX + 1):
                    found.add((c, b, a))
    recomputed = np.zeros(grid, bool)
    for t in found:
        recomputed[t] = True
    inside = recomputed[tuple(tile[..., k] for k in range(3))]
    touched = [np.isin(o, np.unique(o[inside])) for o in old]
    hot = touched[0] | touched[1]
    queue = list(found)
    while queue:
        c, b, a = queue.pop()
        lo = [max(0, c * TZ - 1), max(0, b * TY - 1), max(0, a * TX - 1)]
        hi = [min(shape[0], (c + 1) * TZ + 1), min(shape[1], (b + 1) * TY + 1),
              min(shape[2], (a + 1) * TX + 1)]
        box = tuple(slice(l, h) for l, h in zip(lo, hi))
        for t in {tuple(t) for t in tile[box][hot[box]]}:
            if t not in found:
                found.add(t)
                queue.append(t)
    covered = np.zeros(grid, bool)
    for t in found:
        covered[t] = True
    covered = covered[tuple(tile[..., k] for k in range(3))]
    assert covered[hot].all()
    for o, n in zip(old, new):
        assert covered[o != n].all()
        assert hot[o != n].all()
