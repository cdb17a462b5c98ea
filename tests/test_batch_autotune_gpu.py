"""Autotuning a batch between two runs: the second run is captured anew (the autotuner rewrites the view tables and may
move the path state that the first run's graph reads), also where the tuning that it picks is the one that ran."""
import pytest

from caelix_b200 import workloads

pytestmark = pytest.mark.gpu


def test_run_autotune_run(cuda_device):
    import torch

    import caelix_b200

    vs = workloads.noise_world(grid_bricks=(8, 6, 8), brick_occupancy=0.4, emissive_fraction=0.06, seed=13)
    scene = caelix_b200.Scene.from_voxel_scene(cuda_device, vs)
    r = caelix_b200.Renderer(cuda_device, scene)
    shapes = [(37, 21, 2), (64, 40, 1), (8, 4, 5)]
    outs = [torch.zeros(w * h * 3, device="cuda") for w, h, _ in shapes]
    refs = [torch.zeros_like(o) for o in outs]
    for i, (ref, (w, h, spp)) in enumerate(zip(refs, shapes)):
        r.render(ref, w, h, vs.camera, bounces=2, seed=3 + i, spp=spp)
    views = [(r, o, w, h, vs.camera, 2, 3 + i, spp) for i, (o, (w, h, spp)) in enumerate(zip(outs, shapes))]
    batch = caelix_b200.Batch(cuda_device, views)
    for captures in (1, 2, 3):  # untuned, then the autotuner's pick twice (mostly the same one)
        if captures > 1:
            batch.autotune(repeats=1)
        for _ in range(2):
            for o in outs:
                o.fill_(-1.0)
            batch.run()
            assert batch.stats().graph_captures == captures
            for ref, o in zip(refs, outs):
                assert torch.equal(ref, o)
    batch.close()
    r.close()
    scene.close()
