"""The tile search of light manifold rounds by itself (k_touched_tiles), several
fields in a launch of more blocks than the device holds at once: it finds exactly the
tiles of numpy's search, or asks for the pass over every vertex when more than a 64th
of the tiles are listed or more than a quarter found."""

import ctypes
import os
import subprocess

import numpy as np
import pytest

from test_touched_tiles import labels

pytestmark = pytest.mark.gpu

HERE = os.path.dirname(os.path.abspath(__file__))
TX, TY, TZ = 32, 8, 4


@pytest.fixture(scope="module")
def search(tmp_path_factory):
    from extrem_z_b200 import build
    lib = str(tmp_path_factory.mktemp("search") / "touched_tiles.so")
    subprocess.run([build.nvcc(), *build.NVCC_FLAGS, "-I", build.CSRC,
                    os.path.join(HERE, "native", "touched_tiles.cu"), "-o", lib], check=True)
    return ctypes.CDLL(lib).touched_tiles


def closure(shape, hot, listed):
    """Tiles found outwards from the listed ones through halos with a touched label."""
    grid = [-(-n // t) for n, t in zip(shape, (TZ, TY, TX))]
    found, queue = set(listed), list(listed)
    while queue:
        t = queue.pop()
        c, b, a = t // (grid[1] * grid[2]), t // grid[2] % grid[1], t % grid[2]
        lo = [max(0, c * TZ - 1), max(0, b * TY - 1), max(0, a * TX - 1)]
        hi = [min(n, (k + 1) * s + 1) for n, k, s in zip(shape, (c, b, a), (TZ, TY, TX))]
        z, y, x = np.nonzero(hot[tuple(slice(l, h) for l, h in zip(lo, hi))])
        near = ((z + lo[0]) // TZ * grid[1] + (y + lo[1]) // TY) * grid[2] + (x + lo[2]) // TX
        for u in set(near.tolist()) - found:
            found.add(u)
            queue.append(u)
    return found


@pytest.mark.parametrize("smooth", [0, 2, 5, 9])
@pytest.mark.parametrize("nlist", [1, 4, 5])
def test_finds_the_tiles(search, smooth, nlist):
    rng = np.random.default_rng(10 * smooth + nlist)
    shape = (37, 45, 131)
    n, jobs, nt = int(np.prod(shape)), 5, 10 * 6 * 5
    z, y, x = np.indices(shape)
    tile = (z // TZ * 6 + y // TY) * 5 + x // TX
    lab, touch, listed, hot = [[], []], [[], []], [], []
    for _ in range(jobs):
        f = rng.standard_normal(shape)
        for _ in range(smooth):  # labels of a few vertices to ones across many tiles
            for axis in range(3):
                f = f + np.roll(f, 1, axis) + np.roll(f, -1, axis)
        mine = rng.choice(nt, nlist, replace=False)
        inside = np.isin(tile, mine)
        h = np.zeros(shape, bool)
        for side in (0, 1):
            lb = labels(f, side == 0)
            t = np.zeros(-(-n // 32) * 32, bool)
            t[lb[inside]] = True
            h |= t[lb]
            lab[side].append(lb.astype(np.int32).ravel())
            touch[side].append(np.packbits(t, bitorder="little").view(np.uint32))
        listed.append(mine.astype(np.int32))
        hot.append(h)
    arg = [np.ascontiguousarray(np.concatenate(a)) for a in (*lab, *touch, listed)]
    want = [closure(shape, h, m.tolist()) for h, m in zip(hot, listed)]
    for rep in range(20):
        dense, count = np.zeros(jobs, np.int32), np.zeros(jobs, np.int32)
        queue = np.zeros((jobs, nt), np.int32)
        rc = search(jobs, shape[2], shape[1], shape[0], *[a.ctypes.data_as(ctypes.c_void_p) for a in arg],
                    nlist, 3 + rep, 1500, *[a.ctypes.data_as(ctypes.c_void_p)
                                            for a in (dense, count, queue)])
        assert rc == 0
        for j in range(jobs):
            if nlist > nt // 64:
                assert dense[j] and count[j] == nlist
            elif len(want[j]) > nt // 4:
                assert dense[j] and count[j] > nt // 4
            else:
                assert not dense[j] and count[j] == len(want[j])
                assert sorted(queue[j][:count[j]].tolist()) == sorted(want[j])
