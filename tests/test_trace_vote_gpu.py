"""The warp-voting traversal (15) against the lane-refill one (2): the same
bits for batch sizes around warps, chunks and blocks, for closest hits and
shadow queries, over trees from one leaf to thousands of nodes and for rays
that start in order."""
import os

import pytest

pytestmark = pytest.mark.gpu

SIZES = [1, 31, 33, 63, 64, 65, 577, 4097, 200_003, 400_009]


@pytest.mark.parametrize("spheres,level", [(1, 0), (2, 2), (16, 4)])
@pytest.mark.parametrize("n", SIZES)
def test_vote_equals_refill(crt_ctx, spheres, level, n):
    import torch

    from cudaraytracer_b200 import Scene, scenes

    tris = scenes.icosphere_field(n_spheres=spheres, level=level, with_env=False).triangles()
    sc = Scene.from_triangles(crt_ctx, tris)
    r = scenes.random_rays(tris, n, seed=n)
    r[::7, 7] = 0.5  # bounded
    r[::5, 3] = 0.1
    r[n // 2:] = r[n // 2:][r[n // 2:, 0].argsort()]  # half of them in order
    rays = torch.from_numpy(r).cuda()
    q = torch.from_numpy(scenes.random_shadow_queries(tris, n, seed=n)).cuda()
    got = {}
    try:
        for v in ("15", "2"):
            os.environ["CRT_TRAVERSAL"] = v
            got[v] = sc.trace_closest(rays).view(torch.int32), sc.trace_shadow(q)
        del os.environ["CRT_TRAVERSAL"]
        got["default"] = sc.trace_closest(rays).view(torch.int32), sc.trace_shadow(q)
    finally:
        os.environ.pop("CRT_TRAVERSAL", None)
    crt_ctx.check_device_errors()
    sc.close()
    for v in ("15", "default"):
        assert torch.equal(got[v][0], got["2"][0]) and torch.equal(got[v][1], got["2"][1])
