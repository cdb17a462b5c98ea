"""Waves around the size from which the rays after the camera's take the lanes of finished ones (640,000 paths; 180,000 with several views): one view,
several samples of one view, several views; radiance and ray counts are the per-pixel kernel's, bit for bit."""
import pytest

from caelix_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("views", [[(800, 800, 1)], [(808, 800, 1)], [(333, 251, 8)], [(640, 500, 2), (333, 251, 2)], [(200, 450, 2), (96, 100, 2)], [(200, 400, 2), (96, 100, 2)]])
def test_waves_around_the_change(cuda_device, views):
    import torch

    import caelix_b200

    vs = workloads.noise_world(grid_bricks=(8, 6, 8), brick_occupancy=0.4, emissive_fraction=0.06, seed=13)
    scene = caelix_b200.Scene.from_voxel_scene(cuda_device, vs)
    r = caelix_b200.Renderer(cuda_device, scene)
    want, rays = [], []
    for i, (w, h, spp) in enumerate(views):
        out = torch.full((w * h * 3,), -1.0, device="cuda")
        r.set_trace_mode(r.TRACE_MEGAKERNEL, 0)
        r.render(out, w, h, vs.camera, bounces=3, seed=6 + i, spp=spp)
        st = r.stats()
        want.append(out)
        rays.append((st.primary_rays, st.bounce_rays, st.shadow_rays))
        r.set_trace_mode(r.TRACE_WAVEFRONT, 0)
        got = torch.full_like(out, -1.0)
        r.render(got, w, h, vs.camera, bounces=3, seed=6 + i, spp=spp)
        st = r.stats()
        assert torch.equal(got, out)
        assert (st.primary_rays, st.bounce_rays, st.shadow_rays) == rays[-1]
    outs = [torch.full_like(o, -1.0) for o in want]
    batch = caelix_b200.Batch(cuda_device, [(r, o, w, h, vs.camera, 3, 6 + i, spp)
                                            for i, (o, (w, h, spp)) in enumerate(zip(outs, views))], rebuild_light_trees=False)
    batch.run()
    for i, (o, ref) in enumerate(zip(outs, want)):
        assert torch.equal(o, ref)
        st = batch.view_stats(i)
        assert (st.primary_rays, st.bounce_rays, st.shadow_rays) == rays[i]
    batch.close()
    r.close()
    scene.close()
