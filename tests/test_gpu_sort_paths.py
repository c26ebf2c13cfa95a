"""The sort's two paths that ordinary builds do not take: counts of earlier tiles that are not there when
they are looked for are counted from the keys (taken by a tile that waits too long; here every tile, with
no looks at all), and chains of 64-bit words (2^30 primitives and more; here from 524,289 on).  Both give
the library's own trees, bit for bit."""
from __future__ import annotations

import ctypes as C

import numpy as np
import pytest

from cudapathtracing_gb300 import _lib
from variant_lib import variant

pytestmark = pytest.mark.gpu


def _bind(lib):
    lib.cpt_lbvh_scratch_bytes.restype, lib.cpt_lbvh_scratch_bytes.argtypes = C.c_size_t, [C.c_uint32]
    D = C.POINTER(C.c_double)
    lib.cpt_lbvh_build_device.argtypes = [C.c_uint32, C.c_void_p, C.c_void_p, C.c_uint32, C.c_void_p, D, D] + \
        [C.c_void_p] * 7 + [C.c_size_t, C.c_void_p]
    return lib


@pytest.fixture(scope="module")
def counted(tmp_path_factory):
    return _bind(variant(tmp_path_factory.mktemp("counted"), {"lbvh.cu": ["-DCPT_CHAIN_POLLS=0"]}))


@pytest.fixture(scope="module")
def wide_words(tmp_path_factory):
    return _bind(variant(tmp_path_factory.mktemp("wide"), {"lbvh.cu": ["-DCPT_CHAIN_WIDE_FROM=524289"]}))


def _build(lib, tri, n):
    import torch
    out = [torch.zeros(n, dtype=torch.int64, device="cuda"), torch.zeros(n, dtype=torch.int32, device="cuda"),
           torch.zeros(n - 1, 2, dtype=torch.int32, device="cuda"), torch.zeros(n - 1, 2, dtype=torch.int32, device="cuda"),
           torch.zeros(n - 1, 8, device="cuda"), torch.zeros(n, 8, device="cuda")]
    scratch = torch.zeros(lib.cpt_lbvh_scratch_bytes(n), dtype=torch.uint8, device="cuda")
    lo, hi = (C.c_double * 3)(-3, -3, -3), (C.c_double * 3)(3, 3, 3)
    assert lib.cpt_lbvh_build_device(0, None, None, n, tri.data_ptr(), lo, hi, *[o.data_ptr() for o in out],
                                     scratch.data_ptr(), scratch.numel(), None) == 0
    torch.cuda.synchronize()
    return out


def _same(variant_lib, n, kind):
    import torch
    g = torch.Generator(device="cuda").manual_seed(n)
    c = torch.rand(n, 3, device="cuda", generator=g) * (6.0 if kind == "spread" else 1e-5) - 3.0
    e = torch.rand(n, 6, device="cuda", generator=g) * 0.02
    tri = torch.cat([c, c + e[:, :3], c + e[:, 3:]], 1).contiguous()
    want, got = _build(_lib.lib(), tri, n), _build(variant_lib, tri, n)
    assert all(torch.equal(a, b) for a, b in zip(want, got))
    assert np.array_equal(np.sort(got[1].cpu().numpy()), np.arange(n))


@pytest.mark.parametrize("kind", ["spread", "one_cell"])
@pytest.mark.parametrize("n", [1025, 32768, 36865, 262147, 524297])
def test_counts_taken_from_the_keys(cptlib, counted, n, kind):
    _same(counted, n, kind)


@pytest.mark.parametrize("kind", ["spread", "one_cell"])
@pytest.mark.parametrize("n", [524289, 1310720, 2000003])
def test_chains_of_wide_words(cptlib, wide_words, n, kind):
    _same(wide_words, n, kind)
