"""The bilateral filter's two forms, a pixel a thread and four, give the same bits: the library's filter
against a build of it that takes the first at every radius."""
from __future__ import annotations

import ctypes as C

import pytest

from cudapathtracing_gb300 import abi, api
from variant_lib import variant

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def plain(tmp_path_factory):
    lib = variant(tmp_path_factory.mktemp("plain"), {"filter.cu": ["-DCPT_FILTER_SMALL_RADIUS=256"]})
    lib.cpt_filter_bilateral.argtypes = [C.c_void_p] * 4 + [C.c_int32] * 2 + [C.POINTER(abi.cpt_filter_params), C.c_void_p]
    ctx = C.c_void_p()
    assert lib.cpt_context_create(0, C.byref(ctx)) == 0
    yield lib, ctx
    lib.cpt_context_destroy(ctx)


@pytest.mark.parametrize("W,H", [(1, 1), (131, 37), (640, 360)])
@pytest.mark.parametrize("radius", [7, 16, 45, 256])
def test_both_forms_give_the_same_bits(ctx, plain, W, H, radius):
    import torch
    lib, h = plain
    g = torch.Generator(device="cuda").manual_seed(W + radius)
    rgb = torch.rand(H, W, 3, device="cuda", generator=g)
    gb = torch.rand(H, W, 8, device="cuda", generator=g)
    gb[..., 3] = torch.where(gb[..., 4] < 0.2, torch.full_like(gb[..., 3], 999999.0), gb[..., 3])   # sky
    prm = abi.filter_params(max(2.0, radius / 2), 0.5, 0.3, 0.4, radius)
    want = torch.empty_like(rgb)
    assert lib.cpt_filter_bilateral(h, rgb.data_ptr(), gb.data_ptr(), want.data_ptr(), W, H, C.byref(prm), None) == 0
    got = api.filter_bilateral(ctx, rgb, gb, params=prm)
    torch.cuda.synchronize()
    assert torch.equal(want.view(torch.int32), got.view(torch.int32))
