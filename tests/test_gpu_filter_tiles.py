"""The bilateral filter's row and column kernels at the edges of their tiles (four pixels a thread, 128
a warp, windows of any remainder by four) and where the short windows' kernels take over, against the FP64 oracle.

Tolerance: 33 to 513 taps, each weight within 2 ulp of exp of an argument whose own rounding error
is below 8 eps (|argument| <= 8 here): under 2e-5 of a weighted mean of values in [0, 1], and a
second pass doubles it.  1e-4 bounds both."""
from __future__ import annotations

import numpy as np
import pytest

from cudapathtracing_gb300 import abi, api

filters = pytest.importorskip("filters")
pytestmark = pytest.mark.gpu


def _images(W, H, seed):
    rng = np.random.default_rng(seed)
    rgb = rng.uniform(size=(H, W, 3)).astype(np.float32)
    gb = np.zeros((H, W, 8), np.float32)
    gb[..., :3] = rng.uniform(-0.2, 0.2, size=(H, W, 3))
    gb[..., 3] = rng.uniform(1.0, 1.5, size=(H, W))
    return rgb, gb


def _run(ctx, rgb, gb, prm):
    import torch
    out = api.filter_bilateral(ctx, torch.from_numpy(rgb).cuda(), torch.from_numpy(gb).cuda(), params=prm)
    torch.cuda.synchronize()
    return out.cpu().numpy()


@pytest.mark.parametrize("W,H", [(1, 1), (3, 130), (131, 35)])
@pytest.mark.parametrize("radius", [0, 6, 7, 8, 9, 16, 41, 256])
def test_tile_edges(ctx, W, H, radius):
    prm = abi.filter_params(max(radius, 1) / 2.0, 5.0, 0.5, 0.5, radius)
    rgb, gb = _images(W, H, 7 * W + radius)
    want = filters.bilateral(rgb, gb[..., :4].astype(np.float64), prm.sigma_g, prm.sigma_r, prm.sigma_n, prm.sigma_d,
                             prm.radius)
    np.testing.assert_allclose(_run(ctx, rgb, gb, prm), want, rtol=0, atol=1e-4)


@pytest.mark.parametrize("radius", [5, 9])
def test_values_outside_the_window_are_not_read_into_it(ctx, radius):
    """An infinite colour reaches the pixels whose window holds it, and no other."""
    prm = abi.filter_params(4.0, 5.0, 0.5, 0.5, radius)
    rgb, gb = _images(70, 41, 3)
    plain = _run(ctx, rgb, gb, prm)
    rgb[20, 33, 1] = np.inf
    got = _run(ctx, rgb, gb, prm)
    inside = np.zeros((41, 70), bool)
    inside[20 - radius:21 + radius, 33 - radius:34 + radius] = True
    assert np.isnan(got[inside][:, 1]).all()
    np.testing.assert_array_equal(got[~inside], plain[~inside])
