"""The traversal of all triangles of a small scene (14) against the tree
traversal (2) where the margins of its conservative test do not hold: the
same bits, and no read outside the scene's records."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def soup(n, seed):
    rng = np.random.default_rng(seed)
    c = rng.uniform(-1, 1, (n, 1, 3))
    return (c + rng.normal(size=(n, 3, 3)) * 0.4).reshape(n, 9).astype(np.float32)


def random_rays(n, seed):
    rng = np.random.default_rng(seed)
    r = np.zeros((n, 8), np.float32)
    r[:, 0:3] = rng.uniform(-1.5, 1.5, (n, 3))
    r[:, 4:7] = rng.normal(size=(n, 3))
    r[:, 7] = 1e8
    return r


def check(crt_ctx, tris, r, q=None):
    """Both traversals and the default on rays r and queries q: equal bits.
    Returns the primitives hit."""
    import torch

    from cudaraytracer_b200 import Scene, scenes

    if q is None:
        q = scenes.random_shadow_queries(np.nan_to_num(tris), 1 << 14, seed=len(tris))
    r, q = torch.from_numpy(r).cuda(), torch.from_numpy(q).cuda()
    sc = Scene.from_triangles(crt_ctx, tris)
    got = {}
    try:
        for v in ("14", "2"):
            os.environ["CRT_TRAVERSAL"] = v
            got[v] = sc.trace_closest(r).view(torch.int32), sc.trace_shadow(q)
        del os.environ["CRT_TRAVERSAL"]
        got["default"] = sc.trace_closest(r).view(torch.int32), sc.trace_shadow(q)
    finally:
        os.environ.pop("CRT_TRAVERSAL", None)
    crt_ctx.check_device_errors()
    sc.close()
    for v in ("14", "default"):
        assert torch.equal(got[v][0], got["2"][0]) and torch.equal(got[v][1], got["2"][1])
    return got["2"][0][:, 1].cpu().numpy()


@pytest.mark.parametrize("n", [1, 2, 3, 21, 32, 53, 63])
def test_huge_origins(crt_ctx, n):
    """Finite origins so far away that every margin leaves the range: the
    missing second triangle of an odd scene's last pair is no candidate."""
    r = random_rays(1 << 14, n)
    far = np.random.default_rng(n).choice([1e28, 1e33, 1e36, 3e37], (1 << 14, 1)).astype(np.float32)
    r[:, 0:3] *= far
    r[::2, 4:7] = -r[::2, 0:3] / far[::2]  # towards the scene
    check(crt_ctx, soup(n, n), r)


@pytest.mark.parametrize("comp", [0, 3, 5, 7, 8])
@pytest.mark.parametrize("n", [16, 21, 32, 63])
def test_nan_vertices(crt_ctx, n, comp):
    """A triangle with one NaN coordinate, of any of its vertices: the tree
    accepts it with t = NaN or not by the order of its nodes."""
    tris = soup(n, 7 * n)
    tris[n // 3, comp] = np.nan
    check(crt_ctx, tris, random_rays(1 << 14, n + comp))
