"""The final join pass of jobs that keep the 1-saddles' rows (preserve_join)
and of jobs that look at them once, alone and in one batch: byte-equal to the
oracle at sizes around warps and tiles."""

import numpy as np
import pytest

from extrem_z_b200 import synth

pytestmark = pytest.mark.gpu

SHAPES = [(33, 9, 5), (32, 8, 4), (40, 31, 27), (3, 17, 64), (65, 64, 1)]


def _field(k, dtype):
    w, h, d = SHAPES[k]
    return synth.make_field(w, h, d, n_gauss=10, seed=40 + k, rel=3e-3, dtype=dtype)


@pytest.mark.parametrize("dtype", [np.float32, np.float64])
@pytest.mark.parametrize("k", range(len(SHAPES)))
def test_alone(k, dtype):
    import torch
    from extrem_z_b200 import api
    from oracle import ffi
    fld = _field(k, dtype)
    for final_join in (True, False):
        for preserve_join in (False, True):
            kw = dict(final_join=final_join, preserve_join=preserve_join, max_outer=60)
            ref, rrep, _ = ffi.correct(fld.f, fld.decp, fld.eb, q=4, edit_type=1, **kw)
            g = torch.from_numpy(fld.decp.copy()).cuda()
            rep, _ = api.context(0).correct_device(torch.from_numpy(fld.f).cuda(), g, fld.eb, **kw)
            assert np.array_equal(g.cpu().numpy().view(np.uint8), ref.view(np.uint8)), kw
            assert rep.status == rrep["status"] and rep.counters == rrep["counters"], kw


def test_both_kinds_in_one_batch():
    import torch
    from extrem_z_b200 import api
    from oracle import ffi
    items, refs = [], []
    for k in range(len(SHAPES)):
        for preserve_join in (False, True):
            fld = _field(k, np.float64)
            kw = dict(preserve_join=preserve_join, max_outer=60)
            refs.append(ffi.correct(fld.f, fld.decp, fld.eb, q=4, edit_type=1, final_join=True,
                                    **kw)[0])
            items.append((torch.from_numpy(fld.f).cuda(), torch.from_numpy(fld.decp.copy()).cuda(),
                          fld.eb, kw))
    api.context(0).correct_batch(items)
    for it, ref in zip(items, refs):
        assert np.array_equal(it[1].cpu().numpy().view(np.uint8), ref.view(np.uint8))
