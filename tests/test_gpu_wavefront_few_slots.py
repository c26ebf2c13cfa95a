"""Renders whose sample groups fill the slots more than eight times over keep groups as items; with more
slots the same frame takes single samples.  The images are the same, bit for bit."""
from __future__ import annotations

import pytest

from cudapathtracing_gb300 import abi, api, procedural as P

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("batch", [False, True])
@pytest.mark.parametrize("width,spp", [(400, 2), (362, 9)])
def test_groups_over_few_slots_equal_single_samples(cptlib, width, spp, batch):
    import torch
    ctx = api.Context(0)
    s = api.Scene(ctx, P.cornell_box(width=width)).init()
    cfg = dict(max_depth=6, rr_depth=3, rr_prob=0.8, spp=spp, seed=3)
    got = []
    for slots in (4096, 1 << 21):   # 160,000 and 262,088 groups (131,044 pixels), all above 8 x 4,096
        ctx.set_wavefront(slots)
        o = dict(rgb=torch.zeros(s.height, s.width, 3, device="cuda"), gbuffer=torch.zeros(s.height, s.width, 8, device="cuda"))
        if batch:
            rays = api.render_batch(ctx, [dict(scene=s, **cfg, **o)])["rays"]
        else:
            rays = s.render(estimator=abi.ESTIMATOR_CONFIG, integrator=abi.INTEGRATOR_WAVEFRONT, **cfg, **o)["rays"]
        got.append((o["rgb"], o["gbuffer"], rays))
    s.close()
    ctx.close()
    assert torch.equal(got[0][0], got[1][0]) and torch.equal(got[0][1], got[1][1]) and got[0][2] == got[1][2]
    assert bool((got[0][0] > 0).any())
