"""Saddle rows of fields with a few NaN voxels: a NaN neighbour is on neither side
of a saddle, in the original field's rows as in the decompressed field's.  The NaNs
lie where they change no other vertex's type and end no path, and the decompressed
field differs elsewhere only, so the mismatch census and the correction equal the
oracle's."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu

DIRS = [(1, 0, 0), (-1, 0, 0), (0, 1, 0), (0, -1, 0), (0, 0, 1), (0, 0, -1), (-1, 1, 0), (1, -1, 0),
        (0, 1, 1), (0, -1, -1), (-1, 0, 1), (1, 0, -1), (-1, 1, 1), (1, -1, -1)]


def neighbours(shape, v):
    d, h, w = shape
    x, y, z = v % w, v // w % h, v // (w * h)
    return [(z + c) * h * w + (y + b) * w + x + a for a, b, c in DIRS
            if 0 <= x + a < w and 0 <= y + b < h and 0 <= z + c < d]


def plant(f, count, rng):
    """Sets `count` voxels of f to NaN: each an upper neighbour of a 2-saddle, none where
    it changes a neighbour's type (with the NaN taken as above everything, or as
    nothing) or leaves a neighbour without a higher one."""
    from oracle import ffi
    flat = f.ravel()
    base = ffi.classify(f)[0].ravel()
    spots = []
    for v in rng.permutation(f.size):
        near = neighbours(f.shape, v)
        if len(near) < 14 or any(r in spots for u in near for r in [u] + neighbours(f.shape, u)):
            continue
        if not any(base[s] in (2, 3) and flat[v] > flat[s] for s in near):
            continue
        if any(not any(flat[r] > flat[u] for r in neighbours(f.shape, u) if r != v) for u in near):
            continue
        keep = flat[v]
        types = []
        for value in (np.inf, np.nan):
            flat[v] = value
            t = ffi.classify(f)[0].ravel()
            types.append(np.delete(t, spots + [v]))
        if np.array_equal(types[0], np.delete(base, spots + [v])) and np.array_equal(*types):
            spots.append(int(v))
        else:
            flat[v] = keep
        if len(spots) == count:
            break
    return spots


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("w,h,d,seed", [(33, 21, 13, 1), (40, 24, 12, 2)])
def test_rows_next_to_a_nan(w, h, d, seed, dtype):
    import torch
    from extrem_z_b200 import api
    from oracle import ffi
    rng = np.random.default_rng(seed)
    f = rng.standard_normal((d, h, w))
    f[:, :, : w // 2] += np.sin(np.arange(w // 2))
    f = np.ascontiguousarray(f.astype(dtype))
    spots = plant(f, 5, rng)
    assert len(spots) >= 4
    far = np.ones(f.shape, bool)
    for v in spots:
        z, y, x = v // (w * h), v // w % h, v % w
        far[max(0, z - 4):z + 5, max(0, y - 4):y + 5, max(0, x - 4):x + 5] = False
    assert far.sum() > 100
    g = f.copy()
    g[far] -= dtype(0.05) * rng.random(int(far.sum())).astype(dtype)
    ctx = api.context(0)
    tf = torch.from_numpy(f).cuda()
    ref = ffi.census(f, g)
    got = ctx.mismatch_census(tf, torch.from_numpy(g).cuda())
    assert got["counters"] == ref
    out, rep, _ = ffi.correct(f, g, 0.05, q=4, edit_type=1, max_outer=30)
    tg = torch.from_numpy(g.copy()).cuda()
    r, _ = ctx.correct_device(tf, tg, 0.05, max_outer=30)
    assert np.array_equal(tg.cpu().numpy().view(np.uint8), out.view(np.uint8))
    assert r.status == rep["status"] and r.counters == rep["counters"]
