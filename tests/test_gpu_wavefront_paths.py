"""How a wavefront render is run must not show in its image: a frame whose items are sample groups,
traced by the queue kernels and handed over for its last paths, equals the same frame in bands of
rows that are small enough for single-sample items and for the one-launch path kernel alone —
radiance, display bytes, G-buffer and ray counts, bit for bit (every pixel draws its own streams)."""
from __future__ import annotations

import numpy as np
import pytest

from cudapathtracing_gb300 import abi, api, procedural as P

pytestmark = pytest.mark.gpu

CFG = dict(estimator=abi.ESTIMATOR_CONFIG, integrator=abi.INTEGRATOR_WAVEFRONT, max_depth=12, rr_depth=3, rr_prob=0.8)


def frame(torch, s, spp, rows, flags=0):
    out = dict(rgb=torch.zeros((s.height, s.width, 3), device="cuda"),
               rgba8=torch.zeros((s.height, s.width, 4), dtype=torch.uint8, device="cuda"),
               gbuffer=torch.zeros((s.height, s.width, 8), device="cuda"))
    rays = 0
    for r in rows:
        rays += s.render(spp=spp, seed=9, rows=r, flags=flags, **CFG, **out)["rays"]
    return {k: v.cpu().numpy() for k, v in out.items()}, rays


@pytest.mark.parametrize("layout", ["bvh2", "bvh2q", "bvh8"])
@pytest.mark.parametrize("scene,width,spp,bands", [
    ("random", 1104, 9, (0, 1, 20, 21, 60, 400, 1104)),   # 2.4M groups whole; bands of 10K to 6.9M samples
    ("random", 512, 2, (0, 3, 100, 512)),                 # 262,144 groups whole: single samples, queue kernels
    ("cornell", 96, 17, (0, 95, 96)),                     # three groups, the last of one sample
    ("cornell", 33, 1, (0, 32, 33)),
])
def test_bands_equal_the_whole_frame(ctx, layout, scene, width, spp, bands):
    import torch
    ctx.set_bvh_width(8 if layout == "bvh8" else 2)
    ctx.set_bvh_compression(layout == "bvh2q")
    try:
        d = P.random_scene(900003, width=width, max_level=5) if scene == "random" else P.cornell_box(width=width)
        s = api.Scene(ctx, d).init()
        whole, rays = frame(torch, s, spp, [(0, 0)])
        parts, prays = frame(torch, s, spp, list(zip(bands[:-1], bands[1:])))
        s.close()
    finally:
        ctx.set_bvh_width(2)
        ctx.set_bvh_compression(False)
    assert rays == prays
    for k in whole:
        assert np.array_equal(whole[k], parts[k]), k
    assert (whole["gbuffer"][..., 3] < 999999.0).any()


def test_few_slots_and_loop_limits(ctx):
    """1,024 slots (items wait for slots, also in the path kernel) give the same image; a render that
    needs more iterations than the limit allows still times out and leaves the context usable."""
    import torch
    s = api.Scene(ctx, P.random_scene(900001, width=120, max_level=4)).init()
    ref, rays = frame(torch, s, 3, [(0, 0)])
    try:
        ctx.set_wavefront(1024)
        few, frays = frame(torch, s, 3, [(0, 0)])
        ctx.set_loop_limits(max_replays=1)
        with pytest.raises(Exception, match="TIMEOUT"):
            frame(torch, s, 3, [(0, 0)])
    finally:
        ctx.set_loop_limits()
        ctx.set_wavefront(1 << 21)
    again, _ = frame(torch, s, 3, [(0, 0)])
    s.close()
    assert rays == frays
    for k in ref:
        assert np.array_equal(ref[k], few[k]) and np.array_equal(ref[k], again[k]), k
