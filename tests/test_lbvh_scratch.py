"""cpt_lbvh_scratch_bytes on the host: scratch for n primitives also holds every smaller build."""
from __future__ import annotations

import pytest


@pytest.mark.parametrize("edge", [1 << 15, 1 << 16, 1 << 19, 1 << 20, 1 << 30])
def test_scratch_for_a_capacity_holds_every_smaller_build(cptlib, edge):
    """Around the sizes where the sort takes another tile or another chain word."""
    sizes = [edge + d for d in range(-9000, 9001, 7)] + [edge - 1, edge, edge + 1]
    need = [cptlib.cpt_lbvh_scratch_bytes(n) for n in sorted(set(sizes))]
    assert all(a <= b for a, b in zip(need, need[1:]))


def test_scratch_of_the_largest_static_build_fits_its_array(cptlib):
    assert cptlib.cpt_lbvh_scratch_bytes(65536) <= 3 << 20
