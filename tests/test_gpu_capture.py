"""Calls that only queue work (device buffers, no statistics) can be captured in a CUDA graph, also as
their context's first call; a replay gives the bits of a plain call."""
from __future__ import annotations

import ctypes as C

import pytest

from cudapathtracing_gb300 import abi, api, procedural as P
from cudapathtracing_gb300._lib import check, lib

pytestmark = pytest.mark.gpu


def _ptr(t):
    return C.c_void_p(t.data_ptr())


def _case(kind, ctx):
    """(call(stream), outputs) of one kind on the context's scene."""
    import torch
    gen = torch.Generator(device="cuda").manual_seed(5)
    if kind == "filter":
        rgb = torch.rand(37, 150, 3, device="cuda", generator=gen)
        gb = torch.rand(37, 150, 8, device="cuda", generator=gen)
        out = torch.zeros_like(rgb)

        def call(st, keep=(rgb, gb)):
            check(lib().cpt_filter_bilateral(ctx.h, _ptr(keep[0]), _ptr(keep[1]), _ptr(out), 150, 37, None, st), kind)
        return call, [out]
    s = api.Scene(ctx, P.cornell_box(width=48))
    check(lib().cpt_lbvh_build(s.h, None, None), "build")
    if kind == "trace":
        rays = torch.rand(1000, 8, device="cuda", generator=gen) * 2 - 1
        rays[:, 3], rays[:, 7] = 0.001, 999999.0
        out = torch.zeros(1000, 4, device="cuda")

        def call(st, keep=(s, rays)):
            check(lib().cpt_trace_closest(s.h, _ptr(keep[1]), 1000, _ptr(out), 1, st), kind)
        return call, [out]
    if kind == "build":
        def call(st):
            check(lib().cpt_lbvh_build(s.h, st, None), kind)
        return call, []
    est = abi.ESTIMATOR_CONFIG if kind == "render_config" else abi.ESTIMATOR_REFERENCE
    out = torch.zeros(s.height, s.width, 3, device="cuda")
    prm = abi.render_params(2, est, abi.INTEGRATOR_MEGAKERNEL, 8, 3, 0.8, 7, 0, 0, 0)
    dst = abi.cpt_render_output(out.data_ptr(), None, None, 1, 0)

    def call(st, keep=s):
        check(lib().cpt_render(keep.h, C.byref(prm), C.byref(dst), st, None), kind)
    return call, [out]


@pytest.mark.parametrize("first", [True, False])
@pytest.mark.parametrize("kind", ["filter", "trace", "build", "render_config", "render_reference"])
def test_captured_call_equals_plain_call(cptlib, kind, first):
    import torch
    plain = api.Context(0)                 # loads the kernels
    call, want = _case(kind, plain)
    call(None)
    torch.cuda.synchronize()
    ctx = api.Context(0)
    call2, got = _case(kind, ctx)
    if not first:
        call2(None)
        for g in got:
            g.zero_()
    torch.cuda.synchronize()
    graph, stream = torch.cuda.CUDAGraph(), torch.cuda.Stream()
    with torch.cuda.graph(graph, stream=stream):
        call2(C.c_void_p(stream.cuda_stream))
    for _ in range(2):
        for g in got:
            g.zero_()
        graph.replay()
        torch.cuda.synchronize()
        for a, b in zip(got, want):
            a, b = a.view(torch.int32), b.view(torch.int32)   # a miss is primitive -1, not a float
            assert torch.equal(a, b) and bool((b != 0).any())
