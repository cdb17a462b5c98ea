"""The walks of the wavefront's light kernel, one lane or four lanes per item (four for waves of at
most 65,536 paths): the same frames bit for bit, the per-pixel kernel's, on light trees of one leaf, of
nodes with two to four children and of many levels, with lights in both trees."""
import numpy as np
import pytest

from caelix_b200 import workloads

pytestmark = pytest.mark.gpu

W, H = 288, 240  # 69,120 paths in one wave: one lane per item; split into two waves: four lanes


def frames(cuda_device, scene, camera):
    import torch

    import caelix_b200

    r = caelix_b200.Renderer(cuda_device, scene)
    out = []
    for mode, capacity in ((r.TRACE_MEGAKERNEL, 0), (r.TRACE_WAVEFRONT, 0), (r.TRACE_WAVEFRONT, 1 << 16),
                           (r.TRACE_WAVEFRONT, 4096)):
        r.set_trace_mode(mode, capacity)
        image = torch.full((H, W, 3), -1.0, device="cuda")
        r.render(image, W, H, camera, bounces=3, seed=3)
        st = r.stats()
        out.append((image.cpu().numpy().tobytes(), st.primary_rays, st.bounce_rays, st.shadow_rays))
    r.close()
    return out


@pytest.mark.parametrize("paths", [(1 << 17) - 32, (1 << 17) + 32, 3 << 17])
@pytest.mark.parametrize("origin", [(0, 0, 0), (-37, 1000, -2000)])
def test_refilled_rays_equal(cuda_device, paths, origin):
    """Waves on both sides of the 2^17 paths from which finished lanes take new rays: the per-pixel
    kernel's frame, on a sparse grid far from the origin and on one at it; two views of a batch, whose
    rays share the warps, equal their plain renders."""
    import torch

    import caelix_b200

    vs = workloads.noise_world(grid_bricks=(20, 9, 14), brick_occupancy=0.15, emissive_fraction=0.05, seed=21)
    camera = dict(vs.camera)
    camera["position"] = camera["position"] + 8.0 * np.asarray(origin, np.float32)
    vs = vs.like(keys=vs.keys + np.asarray(origin, np.int32))
    scene = caelix_b200.Scene.from_voxel_scene(cuda_device, vs)
    r = caelix_b200.Renderer(cuda_device, scene)
    w, h = paths // 4 // 64, 64 * 4  # whole 8 x 4 blocks, or a block more than whole rows
    images = []
    for mode in (r.TRACE_MEGAKERNEL, r.TRACE_WAVEFRONT):
        r.set_trace_mode(mode, 0)
        image = torch.full((h, w, 3), -1.0, device="cuda")
        r.render(image, w, h, camera, bounces=3, seed=9)
        st = r.stats()
        images.append((image.cpu().numpy().tobytes(), st.primary_rays, st.bounce_rays, st.shadow_rays))
    assert images[0] == images[1]
    outs = [torch.zeros(h * w * 3, device="cuda"), torch.zeros(96 * 96 * 3, device="cuda")]
    batch = caelix_b200.Batch(cuda_device, [(r, outs[0], w, h, camera, 3, 9, 1), (r, outs[1], 96, 96, camera, 2, 4, 1)])
    batch.run()
    torch.cuda.synchronize()
    assert outs[0].cpu().numpy().tobytes() == images[0][0]
    ref = torch.zeros_like(outs[1])
    r.render(ref, 96, 96, camera, bounces=2, seed=4)
    torch.cuda.synchronize()
    assert torch.equal(ref, outs[1])
    batch.close()
    r.close()
    scene.close()


@pytest.mark.parametrize("lights", [1, 2, 3, 5, 16, 500])
def test_walks_equal(cuda_device, lights):
    import caelix_b200

    vs = workloads.noise_world(grid_bricks=(14, 10, 14), brick_occupancy=0.3, emissive_fraction=0.0, seed=11)
    rng = np.random.default_rng(lights)
    power = np.zeros(vs.brick_count, np.float32)
    power[rng.choice(vs.brick_count, lights, replace=False)] = rng.lognormal(0.0, 2.0, lights)
    scene = caelix_b200.Scene.from_voxel_scene(cuda_device, vs.like(power=power))
    got = frames(cuda_device, scene, vs.camera)
    assert all(g == got[0] for g in got[1:])
    scene.close()


def test_walks_equal_with_entity_lights(cuda_device):
    import caelix_b200

    vs = workloads.noise_world(grid_bricks=(10, 8, 10), brick_occupancy=0.3, emissive_fraction=0.03, seed=12)
    scene = caelix_b200.Scene.from_voxel_scene(cuda_device, vs)
    rng = np.random.default_rng(5)
    for i in range(6):
        ent = workloads.noise_world(grid_bricks=(2, 2, 2), brick_occupancy=1.0, emissive_fraction=0.5, seed=40 + i)
        q = rng.normal(size=4)
        e = scene.add_entity(tuple(rng.uniform(8.0, 72.0, 3)), tuple(q / np.linalg.norm(q)))
        scene.upload_bricks(ent.keys, ent.voxels, entity=e)
        scene.set_brick_power(ent.keys, ent.power, entity=e)
        scene.set_entity_motion(e, i % 2)
    scene.flush()
    got = frames(cuda_device, scene, vs.camera)
    assert all(g == got[0] for g in got[1:])
    scene.close()
