"""Several samples of a pixel in one wave: the radiance and the ray counts are those of one sample at
a time, bit for bit, at every split of the samples into waves (the sums are in sample order)."""
import numpy as np
import pytest

from caelix_b200 import workloads

pytestmark = pytest.mark.gpu


def world():
    return workloads.noise_world(grid_bricks=(8, 6, 8), brick_occupancy=0.4, emissive_fraction=0.06, seed=13)


def items(w, h):
    return 32 * ((w + 7) // 8) * ((h + 3) // 4)  # pixel blocks of 8 x 4


@pytest.mark.parametrize("w,h,spp,waves", [(1, 1, 2, 1), (9, 5, 5, 2), (33, 17, 3, 3), (64, 8, 4, 0), (31, 30, 7, 3)])
def test_merged_samples_equal_single_samples(cuda_device, w, h, spp, waves):
    """`waves` samples per wave at most (0: every sample in one wave) against the per-pixel kernel."""
    import torch

    import caelix_b200

    vs = world()
    scene = caelix_b200.Scene.from_voxel_scene(cuda_device, vs)
    r = caelix_b200.Renderer(cuda_device, scene)
    outs, rays = [], []
    for mode, capacity in ((r.TRACE_MEGAKERNEL, 0), (r.TRACE_WAVEFRONT, items(w, h)), (r.TRACE_WAVEFRONT, waves * items(w, h))):
        r.set_trace_mode(mode, capacity)
        out = torch.full((w * h * 3,), -1.0, device="cuda")
        r.render(out, w, h, vs.camera, bounces=3, seed=4, spp=spp)
        st = r.stats()
        outs.append(out.cpu().numpy().tobytes())
        rays.append((st.primary_rays, st.bounce_rays, st.shadow_rays))
    assert outs[0] == outs[1] == outs[2]
    assert rays[0] == rays[1] == rays[2]
    r.close()
    scene.close()


@pytest.mark.parametrize("w,h,spp", [(24, 20, 4), (33, 7, 3)])
def test_adjoint_of_merged_samples(cuda_device, w, h, spp):
    """The backward call with every sample in one wave against one sample per wave: the same image;
    gradients are sums of the same fp32 terms in another order, at most n of them per entry (n = the
    samples times the vertices of a path), so they differ by at most n * 2^-24 of the sum of magnitudes."""
    import torch

    import caelix_b200

    vs = world()
    scene = caelix_b200.Scene.from_voxel_scene(cuda_device, vs)
    r = caelix_b200.Renderer(cuda_device, scene)
    d = torch.ones(h, w, 3, device="cuda")  # one sign: the magnitudes' sum is the sum
    got = []
    for capacity in (items(w, h), 0):
        r.set_trace_mode(r.TRACE_WAVEFRONT, capacity)
        image = torch.full((h, w, 3), -1.0, device="cuda")
        d_albedo = torch.zeros(65536, 3, device="cuda")
        d_power = torch.zeros(vs.brick_count, device="cuda")
        r.backward(d, w, h, vs.camera, d_albedo, d_power, bounces=3, seed=2, spp=spp, image=image)
        got.append([t.cpu().numpy() for t in (image, d_albedo, d_power)])
    assert got[0][0].tobytes() == got[1][0].tobytes()
    bound = w * h * spp * 8 * 2.0 ** -24
    for a, b in zip(got[0][1:], got[1][1:]):
        a, b = a.astype(np.float64), b.astype(np.float64)
        assert a.min() >= -1e-6 * abs(a).max()
        assert np.all(np.abs(a - b) <= bound * np.maximum(np.abs(a), np.abs(b)) + 1e-30)
    r.close()
    scene.close()


def test_batch_of_unequal_samples(cuda_device):
    """A wavefront batch whose views have 1, 4 and 2 samples: the samples that all views have join a
    wave; every view equals its plain render."""
    import torch

    import caelix_b200

    vs = world()
    scene = caelix_b200.Scene.from_voxel_scene(cuda_device, vs)
    r = caelix_b200.Renderer(cuda_device, scene)
    shapes = [(40, 24, 1), (17, 9, 4), (32, 32, 2)]
    outs = [torch.zeros(w * h * 3, device="cuda") for w, h, _ in shapes]
    views = [(r, o, w, h, vs.camera, 3, 5 + i, spp) for i, (o, (w, h, spp)) in enumerate(zip(outs, shapes))]
    batch = caelix_b200.Batch(cuda_device, views, rebuild_light_trees=False)
    batch.set_tuning(kernel=1)
    batch.run()
    torch.cuda.synchronize()
    for i, (o, (w, h, spp)) in enumerate(zip(outs, shapes)):
        ref = torch.zeros_like(o)
        r.render(ref, w, h, vs.camera, bounces=3, seed=5 + i, spp=spp)
        torch.cuda.synchronize()
        assert torch.equal(ref, o)
    batch.close()
    r.close()
    scene.close()


def test_untuned_batch_is_traced_by_the_wavefront_kernels(cuda_device):
    """A batch that was never tuned runs the wavefront kernels; setting the reported tuning runs the
    persistent kernel; both give the plain renders' radiance."""
    import torch

    import caelix_b200

    vs = world()
    scene = caelix_b200.Scene.from_voxel_scene(cuda_device, vs)
    r = caelix_b200.Renderer(cuda_device, scene)
    shapes = [(37, 21, 2), (8, 4, 1)]
    outs = [torch.zeros(w * h * 3, device="cuda") for w, h, _ in shapes]
    refs = [torch.zeros_like(o) for o in outs]
    for i, (ref, (w, h, spp)) in enumerate(zip(refs, shapes)):
        r.render(ref, w, h, vs.camera, bounces=3, seed=5 + i, spp=spp)
    views = [(r, o, w, h, vs.camera, 3, 5 + i, spp) for i, (o, (w, h, spp)) in enumerate(zip(outs, shapes))]
    batch = caelix_b200.Batch(cuda_device, views)
    for tuned in (False, True):
        if tuned:
            assert batch.tuning().kernel == 0
            batch.set_tuning()
        for o in outs:
            o.fill_(-1.0)
        batch.run()
        st = batch.stats()
        # The second view has one sample only, so the views' samples do not join one wave.
        paths = items(37, 21) + items(8, 4)
        assert (st.wavefront == paths) == (not tuned)
        for ref, o in zip(refs, outs):
            assert torch.equal(ref, o)
    batch.close()
    r.close()
    scene.close()
