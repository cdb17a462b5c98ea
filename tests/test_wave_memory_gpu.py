"""The device memory of a render's path state: 280 bytes a slot, without the adjoint's arrays (40 more)."""
import gc

import pytest

from caelix_b200 import workloads

pytestmark = pytest.mark.gpu


def test_render_keeps_no_adjoint_arrays(cuda_device):
    import torch

    import caelix_b200

    vs = workloads.noise_world(grid_bricks=(8, 6, 8), brick_occupancy=0.4, emissive_fraction=0.06, seed=13)
    scene = caelix_b200.Scene.from_voxel_scene(cuda_device, vs)
    first = caelix_b200.Renderer(cuda_device, scene)  # (loads the kernels)
    w, h, spp = 1024, 1024, 4
    out, d = torch.zeros(h, w, 3, device="cuda"), torch.ones(h, w, 3, device="cuda")
    grads = torch.zeros(65536, 3, device="cuda"), torch.zeros(vs.brick_count, device="cuda")
    first.render(out, 32, 32, vs.camera, bounces=1, seed=1, spp=2)
    first.backward(d, 32, 32, vs.camera, *grads, bounces=1, seed=1, spp=2)

    def taken(call):
        gc.collect()
        torch.cuda.synchronize()
        before = torch.cuda.mem_get_info()[0]
        call()
        torch.cuda.synchronize()
        return before - torch.cuda.mem_get_info()[0]

    slots, slack = w * h * spp, 64 << 20  # the buffers' rounding and the allocator's
    r = caelix_b200.Renderer(cuda_device, scene)
    render = taken(lambda: r.render(out, w, h, vs.camera, bounces=1, seed=1, spp=spp))
    assert 280 * slots <= render <= 280 * slots + slack
    more = taken(lambda: r.backward(d, w, h, vs.camera, *grads, bounces=1, seed=1, spp=spp))
    assert (40 + 12) * slots <= more <= (40 + 12) * slots + slack  # and each sample's radiance
    r.close()
    first.close()
    scene.close()
