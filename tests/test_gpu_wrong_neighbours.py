"""The wrong-neighbour steps of later rounds at list lengths around one block's
share, a cluster's share and beyond (loose bounds make long lists): byte-equal to
the oracle, in both resolution orders."""

import numpy as np
import pytest

from extrem_z_b200 import synth

pytestmark = pytest.mark.gpu

SHAPES = [(24, 20, 16, 2e-2), (48, 40, 32, 2e-2), (80, 72, 64, 1e-2), (96, 96, 80, 3e-2),
          (33, 31, 29, 5e-2)]


@pytest.mark.parametrize("w,h,d,rel", SHAPES)
@pytest.mark.parametrize("order", ["lockstep", "ascending"])
def test_later_rounds(w, h, d, rel, order):
    import torch
    from extrem_z_b200 import api
    from oracle import ffi
    fld = synth.make_field(w, h, d, n_gauss=12, seed=w + d, rel=rel, dtype=np.float32)
    kw = dict(q=4, edit_type=1, max_outer=6)
    ref, rrep, _ = ffi.correct(fld.f, fld.decp, fld.eb, final_join=True,
                               wn_order=order, **kw)
    g = torch.from_numpy(fld.decp.copy()).cuda()
    rep, _ = api.context(0).correct_device(torch.from_numpy(fld.f).cuda(), g, fld.eb,
                                           wn_order=order, **kw)
    assert np.array_equal(g.cpu().numpy().view(np.uint8), ref.view(np.uint8))
    assert rep.counters == rrep["counters"] and rep.status == rrep["status"]
