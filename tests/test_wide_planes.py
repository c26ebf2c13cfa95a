"""The 8-wide walk's box test (WideWalk::axis and the comparison in step, csrc/cpt_trace.cuh) restated in
FP32: a ray that meets a stored box passes, also when it only grazes an edge of it and comes from 10^6
grid steps away, in either form that the compiler's contraction may choose."""
from __future__ import annotations

import numpy as np
import pytest

f, d = np.float32, np.float64
FAR_SLACK = f(1 + 2.0 ** -20)


def _fma(a, b, c):
    """a * b + c rounded once: the FP64 product of FP32 numbers is exact; the sum's own rounding (2^-53)
    is far below what is tested."""
    return (a.astype(d) * b.astype(d) + c.astype(d)).astype(f)


def _planes(p, o, scale, idir, q, fused):
    """Near and far distances (m, 3) of planes q[0] <= q[1]."""
    A = (scale * idir) * f(32768.0)
    b = p - o
    c = _fma(b, idir, -A) if fused else b * idir - A
    k = np.full_like(A, f(2.0 ** -22))
    lo, hi = (_fma(-np.abs(A), k, c), _fma(np.abs(A), k, c)) if fused else (c - np.abs(A) * k, c + np.abs(A) * k)
    up = idir > 0
    first, last = np.where(up, q[0], q[1]), np.where(up, q[1], q[0])
    return [_fma((1.0 + x * 2.0 ** -15).astype(f), A, y) for x, y in ((first, lo), (last, hi))]


@pytest.mark.parametrize("fused", [False, True])
@pytest.mark.parametrize("extent", [0.05, 50.0, 3000.0])
def test_rays_that_meet_a_stored_box_pass(extent, fused):
    rng = np.random.default_rng(int(extent) + 1)
    m = 400_000
    p, o = rng.uniform(-1, 1, (m, 3)).astype(f), (rng.uniform(-1, 1, (m, 3)) * extent).astype(f)
    scale = np.ldexp(f(1), rng.integers(-16, -5, (m, 3))).astype(f)
    q = np.sort(rng.integers(0, 256, (2, m, 3)), 0)
    corner = [p.astype(d) + x * scale.astype(d) for x in q]
    # a point on an edge of the box: two coordinates on its planes, the third between them
    x = np.where(rng.random((m, 3)) < 0.5, corner[0], corner[1])
    free = np.arange(3)[None] == rng.integers(0, 3, (m, 1))
    x = np.where(free, corner[0] + rng.random((m, 3)) * (corner[1] - corner[0]), x)
    dirs = (x - o).astype(f)
    dirs = np.where(np.abs(dirs) < 1e-6, f(1e-6), dirs)
    idir = (f(1) / dirs)
    # the exact intersection, for the inverse direction that the walk has
    t = [(c - o.astype(d)) * idir.astype(d) for c in corner]
    enter, leave = np.minimum(*t).max(1), np.maximum(*t).min(1)
    meets = (enter <= leave) & (leave >= 0.001)
    near, far = _planes(p, o, scale, idir, q, fused)
    tn, tf = np.maximum(near.max(1), f(0.001)), far.min(1)
    passes = ~np.signbit(_fma(tf, np.full_like(tf, FAR_SLACK), -tn))
    assert meets.sum() > m // 20
    assert (passes | ~meets).all()
    # and little more: what passes comes within a grid step and the slack of the box
    step = np.abs(scale * idir).max(1)
    assert (enter - leave <= step + 2.0 ** -19 * np.abs(leave))[passes & (leave >= 0.001)].all()
