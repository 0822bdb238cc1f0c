"""Merge vertices of the persistence pairing at the edges of its compaction
blocks (1024 ids per block, 32 per word): the pairs against the union-find
oracle, exactly."""

import numpy as np
import pytest

from extrem_z_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,d", [(31, 33, 1), (32, 32, 1), (41, 25, 1), (16, 16, 4), (5, 5, 41),
                                   (17, 19, 7), (3, 2, 2), (64, 32, 4)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_pairs_at_block_edges(w, h, d, dtype):
    import torch
    from extrem_z_b200 import api
    from oracle import ffi
    fld = synth.make_field(w, h, d, n_gauss=6, seed=w * h + d, rel=1e-2, dtype=dtype)
    for field in (fld.f, fld.decp):
        mx, mn = api.context(0).persistence_pairs(torch.from_numpy(field).cuda())
        rmx, rmn = ffi.persistence_pairs(field)
        assert np.array_equal(mx, rmx)
        assert np.array_equal(mn, rmn)
