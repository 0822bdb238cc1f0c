"""extremz_classify into buffers that can be written in place and into ones
that cannot (missing, not 4-byte aligned, overlapping the field): the same
types and labels, equal to the oracle's types."""

import numpy as np
import pytest

from extrem_z_b200 import synth

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,h,d", [(32, 8, 4), (33, 9, 5), (150, 40, 1), (31, 7, 3)])
@pytest.mark.parametrize("dtype", [np.float32, np.float64])
def test_outputs_by_copy_equal_outputs_in_place(w, h, d, dtype):
    import torch
    from extrem_z_b200 import api
    from oracle import ffi
    fld = synth.make_field(w, h, d, n_gauss=6, seed=w + h, rel=1e-2, dtype=dtype)
    n, code = w * h * d, api.F32 if dtype == np.float32 else api.F64
    f = torch.from_numpy(fld.decp).cuda()
    ctx = api.context(0)
    want = [x.cpu().numpy().ravel() for x in ctx.classify(f)]
    assert np.array_equal(want[0], ffi.classify(fld.decp)[0].ravel())

    def call(field, t, ds, as_):
        st = api.load().extremz_classify(ctx._h, field, code, w, h, d, t, ds, as_,
                                         torch.cuda.current_stream().cuda_stream)
        assert st == api.OK

    t = torch.zeros(n, dtype=torch.int8, device="cuda")
    raw = torch.zeros(8 * n + 16, dtype=torch.uint8, device="cuda")
    # Labels one byte off alignment.
    call(f.data_ptr(), t.data_ptr(), raw.data_ptr() + 1, raw.data_ptr() + 1 + 4 * n)
    host = raw.cpu().numpy()
    assert np.array_equal(t.cpu().numpy(), want[0])
    assert np.array_equal(host[1:1 + 4 * n].copy().view(np.int32), want[1])
    assert np.array_equal(host[1 + 4 * n:1 + 8 * n].copy().view(np.int32), want[2])
    # One output only.
    t.zero_()
    call(f.data_ptr(), t.data_ptr(), None, None)
    assert np.array_equal(t.cpu().numpy(), want[0])
    # A label buffer that lies over the field.
    g = f.clone()
    ds = torch.zeros(n, dtype=torch.int32, device="cuda")
    call(g.data_ptr(), t.data_ptr(), ds.data_ptr(), g.data_ptr())
    assert np.array_equal(ds.cpu().numpy(), want[1])
    assert np.array_equal(g.flatten().view(torch.int32)[:n].cpu().numpy(), want[2])


@pytest.mark.parametrize("off", [4, 8, 12])
@pytest.mark.parametrize("w,h,d", [(33, 9, 5), (32, 8, 4)])
def test_labels_in_place_at_any_word(off, w, h, d):
    """Label buffers at a word that is no 16-byte boundary are written in place,
    vertex by vertex, and nothing beside them is."""
    import torch
    from extrem_z_b200 import api
    fld = synth.make_field(w, h, d, n_gauss=6, seed=off, rel=1e-2, dtype=np.float32)
    n = w * h * d
    f = torch.from_numpy(fld.decp).cuda()
    ctx = api.context(0)
    want = [x.cpu().numpy().ravel() for x in ctx.classify(f)]
    t = torch.zeros(n, dtype=torch.int8, device="cuda")
    a, b = (torch.full((n + 8,), -7, dtype=torch.int32, device="cuda") for _ in range(2))
    st = api.load().extremz_classify(ctx._h, f.data_ptr(), api.F32, w, h, d, t.data_ptr(),
                                     a.data_ptr() + off, b.data_ptr() + off,
                                     torch.cuda.current_stream().cuda_stream)
    assert st == api.OK
    for x, y in ((a, want[1]), (b, want[2])):
        x = x.cpu().numpy()
        k = off // 4
        assert np.array_equal(x[k:k + n], y)
        assert (x[:k] == -7).all() and (x[k + n:] == -7).all()
    assert np.array_equal(t.cpu().numpy(), want[0])
