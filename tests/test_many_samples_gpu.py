"""More samples per pixel than 16 bits count (a wave's entries keep a sample's place in its wave in 16 bits): the
wavefront render at several splits into waves, a batch that was never tuned and the backward call's image equal the
per-pixel kernel's radiance, bit for bit."""
import pytest

from caelix_b200 import workloads

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("spp", [65_536, 65_539])
def test_samples_past_16_bits(cuda_device, spp):
    import torch

    import caelix_b200

    w, h, items = 4, 3, 32  # one 8 x 4 block
    vs = workloads.noise_world(grid_bricks=(8, 6, 8), brick_occupancy=0.4, emissive_fraction=0.3, seed=21)
    scene = caelix_b200.Scene.from_voxel_scene(cuda_device, vs)
    r = caelix_b200.Renderer(cuda_device, scene)
    want = torch.zeros(w * h * 3, device="cuda")
    r.set_trace_mode(r.TRACE_MEGAKERNEL, 0)
    r.render(want, w, h, vs.camera, bounces=2, seed=9, spp=spp)
    rays = r.stats()
    assert float(want.max()) > 0.0  # (7 of the 12 pixels are lit)
    for capacity in (0, 30_000 * items):  # every sample that fits one wave; three waves
        r.set_trace_mode(r.TRACE_WAVEFRONT, capacity)
        out = torch.full_like(want, -1.0)
        r.render(out, w, h, vs.camera, bounces=2, seed=9, spp=spp)
        st = r.stats()
        assert torch.equal(out, want)
        assert (st.primary_rays, st.bounce_rays, st.shadow_rays) == (rays.primary_rays, rays.bounce_rays, rays.shadow_rays)
    image = torch.full((h, w, 3), -1.0, device="cuda")
    r.backward(torch.ones(h, w, 3, device="cuda"), w, h, vs.camera, torch.zeros(65536, 3, device="cuda"),
               torch.zeros(vs.brick_count, device="cuda"), bounces=2, seed=9, spp=spp, image=image)
    assert torch.equal(image.reshape(-1), want)
    out = torch.full_like(want, -1.0)
    batch = caelix_b200.Batch(cuda_device, [(r, out, w, h, vs.camera, 2, 9, spp)], rebuild_light_trees=False)
    batch.run()
    assert batch.stats().primary_rays == rays.primary_rays
    assert torch.equal(out, want)
    batch.close()
    r.close()
    scene.close()
