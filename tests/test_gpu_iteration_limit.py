"""The smallest device iteration limits that a correction needs: a path whose exit
from a tile is its root takes no hop beyond the exit."""

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("w,peak,limit", [(36, 32, 2), (36, 33, 3), (37, 32, 2), (68, 64, 3)])
def test_limit_of_a_path(w, peak, limit):
    """Ramps up to `peak` and down again: tiles are 32 wide, so the paths to the peak
    leave their tile at vertex 32 (and 64).  The last look of a chain, which finds
    its root, counts one, and so does the end of the setup's chase."""
    import torch
    from extrem_z_b200 import api
    x = np.arange(w, dtype=np.float64)
    f = np.where(x <= peak, x, peak - 40.0 * (x - peak)).reshape(1, 1, w)
    tf = torch.from_numpy(np.ascontiguousarray(f)).cuda()
    ctx = api.context(0)
    rep, _ = ctx.correct_device(tf, tf.clone(), 0.5, device_iter_cap=limit)
    assert rep.status == api.OK
    with pytest.raises(api.ExtremzError) as e:
        ctx.correct_device(tf, tf.clone(), 0.5, device_iter_cap=limit - 1)
    assert e.value.status == api.DEVICE_TIMEOUT
