"""The path kernel (whole paths per lane) against the stage kernels: the same
samples rendered in passes of the sizes on both sides of each rule, and with
the stage kernels alone (a stage traversal that the path kernel does not
take), give the same image up to the order of the float additions into a
pixel, and trace the same numbers of rays."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu

STAGES_ONLY = 2  # CRT_STAGE_SHARED

# width, height, spp, spp per pass: one lane in use, a few per warp, both
# register budgets, hand-over after one and after two bounces, a remainder
SIZES = [(1, 1, 1, 1), (37, 29, 3, 2), (256, 256, 6, 6), (300, 200, 7, 7), (512, 512, 3, 3), (640, 512, 9, 9)]


def scene(ctx, name, w, h, rr_start=0):
    from cudaraytracer_b200 import Scene, scenes

    if name == "box":
        spec = scenes.cornell_box(width=w, height=h, max_bounces=7, seed=5)
    elif name == "textured":
        spec = scenes.cornell_box(width=w, height=h, max_bounces=5, textured=True, lights=2)
    else:  # 16 displaced spheres of the four materials under an environment
        spec = scenes.icosphere_field(n_spheres=16, level=3, width=w, height=h, max_bounces=9, env_size=(64, 32))
    return Scene.from_spec(ctx, spec)


@pytest.mark.parametrize("name", ["box", "textured", "field"])
@pytest.mark.parametrize("w,h,spp,per_pass", SIZES)
def test_path_kernel_matches_stages(crt_ctx, name, w, h, spp, per_pass):
    import torch

    sc = scene(crt_ctx, name, w, h)
    images, rays = [], []
    for mode in (STAGES_ONLY, 0):
        sc.set_render_params(seed=11, spp_per_pass=per_pass, stage_traversal=mode)
        planes = [torch.zeros((h, w, 4), device="cuda") for _ in range(3)]
        before = sc.ray_counts()
        sc.render_device(planes[0], planes[1], spp, first_sample=3, sumsq=planes[2])
        after = sc.ray_counts()
        images.append([p.cpu().numpy() for p in planes])
        rays.append((after[0] - before[0], after[1] - before[1]))
    crt_ctx.check_device_errors()
    sc.close()
    assert rays[0] == rays[1]
    for a, b in zip(*images):
        np.testing.assert_allclose(b, a, rtol=2e-5, atol=1e-6)


@pytest.mark.parametrize("paths_per_pass", [1000, 300_000, 3_000_000])
def test_path_kernel_in_views(crt_ctx, paths_per_pass):
    import torch

    sc = scene(crt_ctx, "box", 200, 120)
    cams = [dict(sc.camera(), phi_deg=float(p)) for p in (-15.0, 0.0, 20.0)]
    images = []
    for mode in (STAGES_ONLY, 0):
        sc.set_render_params(seed=4, paths_per_pass=paths_per_pass, stage_traversal=mode)
        planes = [torch.zeros((3, 120, 200, 4), device="cuda") for _ in range(2)]
        sc.render_views(cams, planes[0], planes[1], 3 if paths_per_pass < 10_000 else 45)
        images.append([p.cpu().numpy() for p in planes])
    crt_ctx.check_device_errors()
    sc.close()
    for a, b in zip(*images):
        np.testing.assert_allclose(b, a, rtol=2e-5, atol=1e-6)
