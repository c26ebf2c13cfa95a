"""The 8-wide layout against the binary one: the same closest hits, bit for bit, on triangle soups
(no shared edges, so no exact ties) of every small size, at several scales, for rays of all octants
and along the axes."""
from __future__ import annotations

import numpy as np
import pytest

from cudapathtracing_gb300 import abi, api


def soup(n: int, scale: float, seed: int) -> abi.SceneDesc:
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1, 1, (n, 1, 3))
    tri = ((c + rng.normal(0, 0.25, (n, 3, 3))) * scale).astype(np.float32).reshape(n, 9)
    d = abi.SceneDesc()
    d.add_material((0.5, 0.5, 0.5))
    d.tri_vertices, d.tri_material = tri, np.zeros(n, np.uint32)
    pts = tri.reshape(-1, 3).astype(np.float64)
    d.bounds_min, d.bounds_max = tuple(pts.min(0)), tuple(pts.max(0))
    d.camera = abi.Camera(8, 1.0, (0, 0, 5), (0, 0, 0), 40.0)
    return d


def soup_rays(m: int, scale: float, seed: int) -> np.ndarray:
    rng = np.random.default_rng(seed)
    rays = np.zeros(m + 96, abi.RAY_DTYPE)
    rays["origin"] = rng.uniform(-2, 2, (m + 96, 3)) * scale
    rays["direction"][:m] = rng.normal(size=(m, 3))
    axes = np.concatenate([np.eye(3), -np.eye(3)])
    rays["direction"][m:] = np.repeat(axes, 16, 0)
    rays["tmin"], rays["tmax"] = 0.001, 999999.0
    return rays


@pytest.mark.gpu
@pytest.mark.parametrize("scale", [0.05, 3.0, 40.0])
@pytest.mark.parametrize("n", [1, 2, 3, 7, 8, 9, 10, 64, 65, 1000, 20011])
def test_wide_hits_equal_binary_hits(ctx, n, scale):
    d, rays = soup(n, scale, n), soup_rays(2000, scale, n + 1)
    hits = {}
    try:
        for width in (2, 8):
            ctx.set_bvh_width(width)
            s = api.Scene(ctx, d).init()
            hits[width] = s.trace(rays)
            s.close()
    finally:
        ctx.set_bvh_width(2)
    for k in ("prim", "t", "u", "v"):
        assert np.array_equal(hits[2][k], hits[8][k]), k
    assert (hits[8]["prim"] >= 0).any() or n < 3


def test_plane_offsets_contain_the_stored_box():
    """The walk's plane distances, restated in FP32: byte q as 1 + q 2^-15 times A plus an offset that
    is moved outwards.  The near distance may not lie beyond the exact plane and the far distance not
    before it, but for the rounding of the offset (p - o) * idir itself (three roundings of 2^-24)."""
    f = np.float32
    rng = np.random.default_rng(0)
    m = 400_000
    p, o = rng.uniform(-50, 50, m).astype(f), rng.uniform(-50, 50, m).astype(f)
    scale = np.ldexp(f(1), rng.integers(-18, 1, m)).astype(f)
    idir = (1 / rng.uniform(1e-3, 1, m) * np.where(rng.random(m) < 0.5, -1, 1)).astype(f)
    q = rng.integers(0, 256, m)
    A = (scale * idir) * f(32768.0)
    c = (p - o) * idir - A
    e = np.abs(A) * f(2.0 ** -22)
    byte = 1.0 + q * 2.0 ** -15                       # exact in FP32 and FP64
    near = (byte * A.astype(np.float64) + (c - e).astype(np.float64)).astype(f)   # one rounding: an FMA
    far = (byte * A.astype(np.float64) + (c + e).astype(np.float64)).astype(f)
    exact = (p.astype(np.float64) - o + q * scale.astype(np.float64)) * idir
    slack = 3 * 2.0 ** -24 * (np.abs((p.astype(np.float64) - o) * idir) + np.abs(exact))
    assert (near <= exact + slack).all()
    assert (far >= exact - slack).all()
    assert (np.abs(near - exact) <= slack + 2.0 ** -6 * np.abs(scale * idir)).all()
