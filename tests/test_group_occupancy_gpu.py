"""The groups that hold bricks, found a warp's run of bricks at a time: rows of bricks that end inside a warp, at its end
and after it; the group that loses its bricks takes the next life, every other one keeps its generation."""
import numpy as np
import pytest

from test_staging_gpu import generation_state, groups_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [7, 31, 32, 33, 63, 65, 255, 256, 257, 1025])
def test_rows_of_bricks(cuda_device, n):
    import caelix_b200

    keys = np.zeros((n, 3), np.int32)
    keys[:, 0] = np.arange(n)
    scene = caelix_b200.Scene(cuda_device, group_shift=1)  # groups of two bricks along the row
    scene.upload_bricks(keys, np.full((n, 512), 0x8001, np.uint16))
    scene.set_brick_power(keys, np.zeros(n, np.float32))
    scene.flush()
    gen, _, lit, grid = generation_state(scene)
    assert not lit and not gen.any()
    # The first group, one in the middle and the last but one, each in a flush of its own; the row's ends stay.
    for at in (2, n // 4 * 2, (n - 3) // 2 * 2):
        members = keys[at:at + 2]
        scene.remove_bricks(members)
        scene.flush()
        now, _, _, grid_now = generation_state(scene)
        assert grid_now == grid
        want = gen.copy()
        for g in groups_of(members, grid):
            want[g] = ((int(gen[g]) >> 16) + 1) << 16
        assert np.array_equal(now, want)
        scene.upload_bricks(members, np.full((2, 512), 0x8001, np.uint16))
        scene.set_brick_power(members, np.zeros(2, np.float32))
        scene.flush()
        gen, _, _, _ = generation_state(scene)
        assert np.array_equal(gen, want)
    scene.close()
