"""The stage kernels (extend, shade, shadow per bounce) against the path
kernel, where the settings for them ask for the stages and in passes large
enough to run them by default: the same image up to the order of the float
additions into a pixel, and the same numbers of rays."""
import numpy as np
import pytest

from cudaraytracer_b200 import Scene, scenes

pytestmark = pytest.mark.gpu


def kernel_names(fn):
    """Names of the kernels that fn() launches; skips without a profiler."""
    import torch
    from torch.profiler import ProfilerActivity, profile

    with profile(activities=[ProfilerActivity.CUDA]) as p:
        fn()
        torch.cuda.synchronize()
    names = " ".join(e.key for e in p.key_averages())
    if "k_raygen" not in names:
        pytest.skip("no kernel records from the profiler")
    return names


def scene(ctx, name, w, h):
    if name == "box":
        return Scene.from_spec(ctx, scenes.cornell_box(width=w, height=h, max_bounces=7, seed=5))
    level = 5 if name == "large" else 3  # 81,920 triangles: refill by default; 5,120
    return Scene.from_spec(ctx, scenes.icosphere_field(n_spheres=4, level=level, width=w, height=h, max_bounces=9,
                                                       env_size=(64, 32)))


def render(sc, w, h, spp, **params):
    import torch

    sc.set_render_params(seed=11, **params)
    planes = [torch.zeros((h, w, 4), device="cuda") for _ in range(3)]
    before = sc.ray_counts()
    sc.render_device(planes[0], planes[1], spp, first_sample=3, sumsq=planes[2])
    after = sc.ray_counts()
    return [p.cpu().numpy() for p in planes], (after[0] - before[0], after[1] - before[1])


def same(a, b):
    assert a[1] == b[1]
    for x, y in zip(a[0], b[0]):
        np.testing.assert_allclose(y, x, rtol=2e-5, atol=1e-6)


@pytest.mark.parametrize("var,value,kernels", [
    ("CRT_SHADE_MIN_BLOCKS", "4", ["k_extend(", "k_shade_mb<4>", "k_shadow("]),
    ("CRT_SHADE_MIN_BLOCKS", "6", ["k_shade_mb<6>"]),
    ("CRT_SHADE_MIN_BLOCKS", "10", ["k_shade_mb<10>"]),
    ("CRT_PATH_KERNEL", "0", ["k_extend(", "k_shade(", "k_shade_miss(", "k_shadow("]),
])
def test_settings_of_the_stages_reach_them(crt_ctx, monkeypatch, var, value, kernels):
    sc = scene(crt_ctx, "field", 40, 32)
    want = render(sc, 40, 32, 4)
    monkeypatch.setenv(var, value)
    same(want, render(sc, 40, 32, 4))
    names = kernel_names(lambda: render(sc, 40, 32, 4))
    sc.close()
    assert "k_paths" not in names and all(k in names for k in kernels), names


@pytest.mark.parametrize("name", ["box", "field", "large"])
@pytest.mark.parametrize("mode", [1, 6])  # CRT_STAGE_LOCAL, CRT_STAGE_REFILL
@pytest.mark.parametrize("block", [64, 256])
def test_small_passes_in_stages(crt_ctx, monkeypatch, name, mode, block):
    """Passes of 3,500 paths and a remainder, which the path kernel would take."""
    w, h, spp = 50, 35, 5
    sc = scene(crt_ctx, name, w, h)
    want = render(sc, w, h, spp, spp_per_pass=2)
    monkeypatch.setenv("CRT_PATH_KERNEL", "0")
    same(want, render(sc, w, h, spp, spp_per_pass=2, stage_traversal=mode, stage_block=block))
    crt_ctx.check_device_errors()
    sc.close()


@pytest.mark.parametrize("name,mode", [("box", 6), ("large", 0), ("large", 6), ("field", 6)])
@pytest.mark.parametrize("w,h,spp", [(640, 512, 3), (640, 512, 9)])  # handed over after one and two bounces
def test_refill_in_large_passes(crt_ctx, monkeypatch, name, mode, w, h, spp):
    """The refill stages (the default of 65,536 triangles and more) before
    the path kernel takes over, and throughout, against the shared-stack
    stages."""
    sc = scene(crt_ctx, name, w, h)
    want = render(sc, w, h, spp, spp_per_pass=spp, stage_traversal=2)  # CRT_STAGE_SHARED
    same(want, render(sc, w, h, spp, spp_per_pass=spp, stage_traversal=mode))
    monkeypatch.setenv("CRT_PATH_KERNEL", "0")
    same(want, render(sc, w, h, spp, spp_per_pass=spp, stage_traversal=mode))
    crt_ctx.check_device_errors()
    sc.close()


@pytest.mark.parametrize("use_graph", [False, True])
def test_views_and_noalloc_in_stages(crt_ctx, monkeypatch, use_graph):
    import torch

    w, h = 48, 40
    sc = scene(crt_ctx, "field", w, h)
    sc.set_render_params(seed=6, paths_per_pass=5000)
    cams = [dict(sc.camera(), phi_deg=float(p)) for p in (-15.0, 20.0)]
    got = []
    for stages in (False, True):
        if stages:
            monkeypatch.setenv("CRT_PATH_KERNEL", "0")
        v = [torch.zeros((2, h, w, 4), device="cuda") for _ in range(2)]
        sc.render_views(cams, v[0], v[1], 4, use_graph=use_graph)
        f = [torch.zeros((h, w, 4), device="cuda") for _ in range(2)]
        sc.render_device_noalloc(f[0], f[1], 3)
        torch.cuda.synchronize()
        got.append([p.cpu().numpy() for p in v + f])
    crt_ctx.check_device_errors()
    sc.close()
    for a, b in zip(*got):
        np.testing.assert_allclose(b, a, rtol=2e-5, atol=1e-6)
