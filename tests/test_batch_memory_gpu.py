"""A batch whose tuning allows more paths in flight than the device has memory for: the merged samples' path state (a
request of about 300 GB, refused at once) gives way to one sample index per wave, as such a tuning always ran."""
import pytest

from caelix_b200 import workloads

pytestmark = pytest.mark.gpu


def test_merged_samples_that_do_not_fit(cuda_device):
    import torch

    import caelix_b200

    w, h, spp = 2048, 2048, 256
    vs = workloads.noise_world(grid_bricks=(8, 6, 8), brick_occupancy=0.4, emissive_fraction=0.3, seed=21)
    scene = caelix_b200.Scene.from_voxel_scene(cuda_device, vs)
    r = caelix_b200.Renderer(cuda_device, scene)
    r.set_trace_mode(r.TRACE_WAVEFRONT, w * h)  # one sample index per wave
    want, out = torch.zeros(w * h * 3, device="cuda"), torch.full((w * h * 3,), -1.0, device="cuda")
    r.render(want, w, h, vs.camera, bounces=0, seed=9, spp=spp)
    assert float(want.max()) > 0.0
    batch = caelix_b200.Batch(cuda_device, [(r, out, w, h, vs.camera, 0, 9, spp)], rebuild_light_trees=False)
    batch.set_tuning(kernel=1, wavefront=(1 << 31) - 1)
    batch.run()
    assert batch.stats().wavefront == w * h
    assert torch.equal(out, want)
    batch.close()
    r.close()
    scene.close()
