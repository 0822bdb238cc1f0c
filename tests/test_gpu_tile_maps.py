"""Tile maps of successive jobs in one slot."""

import pytest

pytestmark = pytest.mark.gpu


def test_alternating_fields_of_one_shape():
    """Fields of one shape at different addresses take the same job slot in
    turn, so its tile map is rewritten between launches (and the launches
    become a replayed graph): each call must see its own field.  A label is a
    local extremum's id: no vertex lies above its ascent root or below its
    descent root."""
    import torch
    from extrem_z_b200 import api
    ctx = api.context(0)
    fields, want = [], []
    for seed in range(3):
        g = torch.Generator(device="cuda").manual_seed(seed)
        fields.append(torch.rand((128, 128, 256), generator=g, dtype=torch.float64, device="cuda"))
    for rep in range(12):
        for k, f in enumerate(fields):
            t, up, down = ctx.classify(f)
            flat = f.flatten()
            assert bool((flat[up.flatten().long()] >= flat).all())
            assert bool((flat[down.flatten().long()] <= flat).all())
            if rep == 0:
                want.append((t, up, down))
            assert all(torch.equal(a, b) for a, b in zip((t, up, down), want[k]))
