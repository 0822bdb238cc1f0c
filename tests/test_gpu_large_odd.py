"""A field large enough for the light rounds' tile search, of odd edges (no tile
or quad boundary divides it): byte-equal to the oracle."""

import numpy as np
import pytest

from extrem_z_b200 import synth

pytestmark = pytest.mark.gpu


def test_large_odd_field():
    import torch
    from extrem_z_b200 import api
    from oracle import ffi
    w, h, d = 325, 321, 323
    assert w * h * d >= 1 << 25
    fld = synth.make_field(w, h, d, n_gauss=256, seed=77, rel=5e-5, dtype=np.float32)
    ref, rrep, _ = ffi.correct(fld.f, fld.decp, fld.eb, q=4, edit_type=1)
    g = torch.from_numpy(fld.decp.copy()).cuda()
    rep, _ = api.context(0).correct_device(torch.from_numpy(fld.f).cuda(), g, fld.eb)
    assert np.array_equal(g.cpu().numpy().view(np.uint8), ref.view(np.uint8))
    assert rep.counters == rrep["counters"] and rep.status == rrep["status"]
