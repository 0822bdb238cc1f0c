"""Corrections that compute more than 256 manifold rounds, so that the round's
stamp outgrows a byte: byte-equal to the oracle, with equal traces.  A
persistence filter of half the bound at a loose bound keeps the wrong-extremum
checks busy until the cap on outer iterations."""

import numpy as np
import pytest

from extrem_z_b200 import synth

pytestmark = pytest.mark.gpu


# An odd vertex count and two that are multiples of four; with and without the
# join tree's checks.
@pytest.mark.parametrize("w,h,d,seed,preserve_join", [(49, 47, 45, 2, False), (48, 40, 32, 1, True),
                                                      (64, 64, 16, 2, True)])
def test_rounds_past_a_byte(w, h, d, seed, preserve_join):
    import torch
    from extrem_z_b200 import api
    from oracle import ffi
    fld = synth.make_field(w, h, d, n_gauss=12, seed=seed, rel=0.3, alpha=2.0)
    kw = dict(thr=0.5 * fld.eb, q=4, edit_type=1, preserve_join=preserve_join, max_outer=250,
              trace_cap=200000)
    ref, rrep, rtrace = ffi.correct(fld.f, fld.decp, fld.eb, final_join=True, **kw)
    g = torch.from_numpy(fld.decp.copy()).cuda()
    rep, trace = api.context(0).correct_device(torch.from_numpy(fld.f).cuda(), g, fld.eb, **kw)
    assert rep.manifold_rounds - rep.manifold_reused > 256
    assert np.array_equal(trace, rtrace)
    assert np.array_equal(g.cpu().numpy().view(np.uint8), ref.view(np.uint8))
    assert rep.counters == rrep["counters"] and rep.status == rrep["status"]
