"""The nodes above the tiles of a light BVH build around the sizes where their kernels change (24,576 leaves: one CTA for
walks, rows and header; 65,536: the walks by one CTA or by a grid, as many as there are), with lights spread in a
box and along a line (far fewer walks), bit for bit the oracle's."""
import numpy as np
import pytest

import oracle_lib
from caelix_b200 import workloads
from test_lt_build_gpu import assert_same_build, gpu_build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("line", [False, True])
@pytest.mark.parametrize("n,launches", [(24575, 11), (24576, 11), (24577, 14), (30011, 14), (40009, 14), (65536, 14), (65537, 13)])
def test_sizes_around_the_changes(cuda_device, oracle, n, launches, line):
    rec, _, _ = workloads.brick_light_records(n, grid_bricks=32, seed=9, stream=n)
    if line:
        for k in ("box_lo", "box_hi"):
            rec[k] &= np.uint32(0x3FF)  # all on the x axis, boxes flat
    g = gpu_build(cuda_device, rec)
    assert g["stats"].status == 0
    assert g["stats"].kernel_launches == launches
    assert_same_build(g, oracle_lib.lt_build(oracle, rec, leaf_capacity=n), n)
