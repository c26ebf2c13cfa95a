"""Idle workspace memory: shared by a device's contexts, bounded, given back on request and before an
allocation fails (csrc/workspace.cu), also to the serving loop's other allocations."""
from __future__ import annotations

import numpy as np
import pytest

from cudapathtracing_gb300 import abi, api, serve as S
from cudapathtracing_gb300._lib import CptError

MB = 1 << 20


class _Ctx:
    trims = 0

    def trim(self):
        self.trims += 1


def _executor():
    ex = S.GpuExecutor.__new__(S.GpuExecutor)
    ex.ctx = [_Ctx(), _Ctx()]
    return ex


@pytest.mark.parametrize("kind", ["torch", "library"])
def test_serving_gives_idle_memory_back_before_a_job_fails(kind):
    import torch
    ex, calls = _executor(), []

    def oom():
        if kind == "torch":
            raise torch.cuda.OutOfMemoryError("CUDA out of memory")
        raise CptError(abi.CPT_ERR_OUT_OF_MEMORY, "cpt_render", "workspace allocation: out of memory")

    def run(job, lane):
        calls.append((job, lane, ex.ctx[0].trims))
        if len(calls) == 1:
            oom()
        return 7

    ex._run = ex._run_batch = run
    assert ex.run("job", 1) == 7
    assert calls == [("job", 1, 0), ("job", 1, 1)]
    calls.clear()
    assert ex.run_batch(["job"], 0) == 7
    assert calls == [(["job"], 0, 1), (["job"], 0, 2)]


def test_other_failures_are_not_repeated():
    ex, calls = _executor(), []

    def run(job, lane):
        calls.append(job)
        raise CptError(abi.CPT_ERR_INVALID_ARGUMENT, "cpt_render", "spp must be positive")

    ex._run = run
    with pytest.raises(CptError):
        ex.run("job", 0)
    assert calls == ["job"] and ex.ctx[0].trims == 0


def _free():
    import torch
    torch.cuda.synchronize()
    return torch.cuda.mem_get_info()[0]


def _filter(ctx, images):
    import torch
    api.filter_bilateral(ctx, *images, params=abi.filter_params(2.0, 5.0, 0.1, 0.2, 2))
    torch.cuda.synchronize()


@pytest.fixture
def images():
    """An image whose filter takes 384 MB of workspace."""
    import torch
    rgb, gb = torch.rand(4096, 8192, 3, device="cuda"), torch.rand(4096, 8192, 8, device="cuda")
    return rgb, gb, torch.empty_like(rgb)


@pytest.mark.gpu
def test_contexts_share_the_idle_workspace_and_give_it_back(cptlib, images):
    ctxs = [api.Context(0) for _ in range(3)]
    for c in ctxs:
        c.trim()
    _filter(ctxs[0], images)
    ctxs[0].trim()
    free = _free()
    for c in ctxs:
        _filter(c, images)
    held = free - _free()
    assert 300 * MB < held < 600 * MB, held      # one filter's, not three
    ctxs[1].trim()
    assert free - _free() < 64 * MB
    _filter(ctxs[2], images)
    for c in ctxs[:2]:
        c.close()
    _filter(ctxs[2], images)                     # the pool lives with its last context
    ctxs[2].close()


@pytest.mark.gpu
def test_an_allocation_that_does_not_fit_takes_the_idle_workspace_first(cptlib, images):
    """A wavefront of 2^29 slots and 30 lights needs 1.1 TB, more than any device has: it is refused
    before anything is launched, after the idle memory was given back; the context stays usable."""
    import torch
    ctx = api.Context(0)
    d = abi.SceneDesc()
    d.add_material((0.5, 0.5, 0.5), 0.5, 0.5, abi.M_LAMBERTIAN)
    d.tri_vertices = np.array([[-1, 0, -1, 1, 0, -1, 0, 0, 1], [-1, 1, -1, 1, 1, -1, 0, 1, 1]], np.float32)
    d.tri_material = np.zeros(2, np.uint32)
    d.bounds_min, d.bounds_max = (-1.0, 0.0, -1.0), (1.0, 1.0, 1.0)
    d.lights = [dict(center=(0.1 * k, 3.0, 0.0), normal=(0.0, -1.0, 0.0), width=0.1, height=0.1,
                     color=(1.0, 1.0, 1.0), visible=1) for k in range(30)]
    d.camera = abi.Camera(8192, 1.0, (0, 0.5, 5), (0, 0.5, 0), 40.0)
    s = api.Scene(ctx, d).init()
    rgb = torch.zeros(8192, 8192, 3, device="cuda")
    cfg = dict(estimator=abi.ESTIMATOR_CONFIG, integrator=abi.INTEGRATOR_WAVEFRONT, max_depth=2, rr_depth=3,
               rr_prob=0.8, rgb=rgb)
    ctx.trim()
    free = _free()
    _filter(ctx, images)
    assert free - _free() > 300 * MB
    ctx.set_wavefront(1 << 29)
    with pytest.raises(CptError) as e:
        s.render(spp=64, **cfg)
    assert e.value.status == abi.CPT_ERR_OUT_OF_MEMORY
    assert free - _free() < 64 * MB
    ctx.set_wavefront(1 << 18)
    s.render(spp=1, rows=(0, 64), **cfg)
    s.close()
    ctx.close()
