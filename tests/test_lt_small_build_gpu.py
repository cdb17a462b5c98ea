"""The light BVH builds on both sides of the sizes where their kernels change (4,096 leaves: ranks in the
place of radix passes; 16,384: one CTA for the nodes above the tiles), bit for bit the oracle's, with
distinct and with many equal Morton codes, and a sequence of builds in one object."""
import numpy as np
import pytest

import oracle_lib
from caelix_b200 import workloads
from test_lt_build_gpu import assert_same_build, gpu_build

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [2, 4, 31, 33, 63, 65, 127, 129, 255, 257, 513, 4093, 4095, 4096, 4097, 16383, 16384, 16385])
@pytest.mark.parametrize("grid", [32, 2])
def test_sizes_around_the_changes(cuda_device, oracle, n, grid):
    rec, _, _ = workloads.brick_light_records(n, grid_bricks=grid, seed=5, stream=n)
    g = gpu_build(cuda_device, rec)
    assert g["stats"].status == 0
    assert_same_build(g, oracle_lib.lt_build(oracle, rec, leaf_capacity=n), n)


def test_powerless_records_and_one_place(cuda_device, oracle):
    """Every box in one place (one Morton code, extent 0) and half of the powers zero."""
    rec, _, _ = workloads.brick_light_records(3001, grid_bricks=32, seed=6)
    for k in ("box_lo", "box_hi", "pos"):
        rec[k] = rec[k][0]
    rec["face"][::2] = 0.0
    g = gpu_build(cuda_device, rec)
    assert_same_build(g, oracle_lib.lt_build(oracle, rec, leaf_capacity=3001), 3001)
