"""The adjoint line's rays are those that were traced: a call that keeps the
vertices reports the rays of two passes and traces one."""
from __future__ import annotations

import pytest

import bench


@pytest.mark.parametrize("depth", [1, 3, 8])
def test_rays_of_kept_and_of_replayed_vertices(depth):
    st = {"extension_rays": 2000, "shadow_rays": 1400}
    assert bench.adjoint_rays_traced({**st, "frames": depth + 2}, max_depth=depth) == (1000, 700)
    assert bench.adjoint_rays_traced({**st, "frames": 2 * depth + 3}, max_depth=depth) == (2000, 1400)
