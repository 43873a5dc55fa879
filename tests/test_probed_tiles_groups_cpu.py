"""The launch bound of probed voxel grids for every CTA size that calls it: 128 voxels with one lane per voxel,
64, 32, 16 and 8 with the frame groups."""

from __future__ import annotations

import random

import pytest

from tests.test_probed_tiles_cpu import lib  # noqa: F401  (the compiled bound)


@pytest.mark.parametrize("voxels", [8, 16, 32, 64, 128])
@pytest.mark.parametrize("wf", [1, 2, 4, 8, 16])
def test_bound_covers_every_extent(lib, voxels, wf):  # noqa: F811
    if wf > voxels:
        pytest.skip("the planner clamps the warp tile to the CTA")
    rng = random.Random(100 * voxels + wf)
    shapes = [(16, 128), (17, 128), (16, 129), (31, 129), (65535, 128), (16, 100000), (16, 128 * 128 + 1)]
    shapes += [(rng.randint(16, 700), rng.randint(128, 700)) for _ in range(400)]
    for fast, outer in shapes:
        n = fast * outer
        bound = lib.tiles(n, voxels, wf)
        assert -(-n // voxels) <= bound  # no grid found
        assert -(-outer * wf // voxels) * -(-fast // wf) <= bound
