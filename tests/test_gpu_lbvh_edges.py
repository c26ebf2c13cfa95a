"""LBVH builds at the sizes where a kernel's split of the work changes: the hierarchy's blocks of 512
keys, the sort's tiles (1,024 / 4,096 / 8,192 keys, up to 32,768 / 524,288 / more primitives) — keys,
order, topology and boxes bit for bit against the FP64 oracle.  Distributions: spread triangles; all
in one Morton cell (equal codes, ordered by primitive); two far clusters of very different size (a
hierarchy whose nodes reach across many blocks)."""
from __future__ import annotations

import numpy as np
import pytest

from conftest import outward_f32
from cudapathtracing_gb300 import abi, api

pytestmark = pytest.mark.gpu


def scene(n: int, kind: str) -> abi.SceneDesc:
    rng = np.random.default_rng(n)
    if kind == "spread":
        c = rng.uniform(-3, 3, (n, 3))
    elif kind == "one_cell":
        c = np.full((n, 3), 0.25) + rng.uniform(0, 1e-5, (n, 3))
    else:
        far = rng.random(n) < 0.001
        c = np.where(far[:, None], rng.uniform(2.0, 2.1, (n, 3)), rng.uniform(-3.0, -2.98, (n, 3)))
    e = rng.uniform(0, 0.02, (n, 6))
    tri = np.concatenate([c, c + e[:, :3], c + e[:, 3:]], 1).astype(np.float32)
    d = abi.SceneDesc()
    d.add_material((0.5, 0.5, 0.5))
    d.tri_vertices, d.tri_material = tri, np.zeros(n, np.uint32)
    d.bounds_min, d.bounds_max = (-3.0,) * 3, (3.0,) * 3
    d.camera = abi.Camera(8, 1.0, (0, 0, 5), (0, 0, 0), 40.0)
    return d


@pytest.mark.parametrize("kind", ["spread", "one_cell", "clusters"])
@pytest.mark.parametrize("n", [2, 3, 511, 512, 513, 1023, 1025, 32768, 32769, 36865, 524288, 524297])
def test_build_equals_oracle(ctx, oracle_mod, n, kind):
    d = scene(n, kind)
    s = api.Scene(ctx, d).init()
    L, G = s.export_lbvh(), oracle_mod.OracleScene(d).lbvh()
    s.close()
    for k in ("keys", "order", "child_a", "child_b"):
        assert np.array_equal(L[k], G[k]), k
    for k in ("node_boxes", "leaf_boxes"):
        lo, hi = outward_f32(G[k][:, :3], G[k][:, 3:])
        assert np.array_equal(L[k], np.concatenate([lo, hi], 1)), k
