"""Closest hits and shadow queries over all triangles of a small scene
(traversal 14) against the tree traversal (2): the same bits, for triangle
counts around the record pairs and the limit, rays from everywhere, from
surfaces and along edges, bounded and unnormalised rays, coplanar and
duplicate triangles, and rays the margins do not cover."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def triangles(n, seed, kind):
    from cudaraytracer_b200 import scenes

    rng = np.random.default_rng(seed)
    if kind == "box":
        return scenes.cornell_box(seed=seed).triangles()[:n]
    if kind == "grid":  # axis-aligned quads on shared planes: edges, corners, ties
        t = []
        for _ in range((n + 1) // 2):
            a, p = rng.integers(0, 3), rng.integers(0, 3, 3).astype(np.float32)
            u, v = np.eye(3, dtype=np.float32)[(a + 1) % 3], np.eye(3, dtype=np.float32)[(a + 2) % 3]
            t += [np.concatenate([p, p + u, p + u + v]), np.concatenate([p, p + u + v, p + v])]
        return np.stack(t)[:n].astype(np.float32)
    c = rng.uniform(-1, 1, (n, 1, 3)) + (50.0 if kind == "far" else 0.0)
    return (c + rng.normal(size=(n, 3, 3)) * (1e-3 if kind == "far" else 0.4)).reshape(n, 9).astype(np.float32)


def rays(tris, n, seed):
    rng = np.random.default_rng(seed)
    t = tris.reshape(-1, 3, 3)
    lo, hi = t.min((0, 1)), t.max((0, 1))
    r = np.empty((n, 8), np.float32)
    r[:, 0:3] = lo + (hi - lo) * rng.uniform(-0.2, 1.2, (n, 3))
    r[:, 4:7] = rng.normal(size=(n, 3))
    r[:, 3], r[:, 7] = 0.0, 1e8
    q = n // 8
    k = rng.integers(0, len(t), 4 * q)
    w = rng.dirichlet((1, 1, 1), 4 * q)
    w[::4] = rng.permuted(np.tile([0.5, 0.5, 0.0], (q, 1)), axis=1)  # edge midpoints
    w[1::4] = np.eye(3)[rng.integers(0, 3, q)]  # vertices
    target = np.einsum("nk,nkc->nc", w, t[k].astype(np.float64))
    r[:2 * q, 4:7] = target[:2 * q] - r[:2 * q, 0:3]  # through points of triangles
    r[2 * q:4 * q, 0:3] = target[2 * q:]  # from points of triangles
    r[4 * q:5 * q, 4:7] = np.eye(3)[rng.integers(0, 3, q)] * rng.choice([-1.0, 1.0], (q, 1))  # along the axes
    r[5 * q:6 * q, 7] = rng.uniform(0, 2, q)
    r[5 * q:6 * q, 3] = rng.uniform(0, 1, q)
    r[6 * q:7 * q, 4:7] *= rng.choice([1e-3, 30.0], (q, 1))
    r[-8:, 0] = [1e20, -1e30, np.inf, np.nan, 0, 0, 0, 0]
    r[-4:, 4] = [1e20, np.inf, np.nan, 0]
    r[-1, 4:7] = 0
    return r


@pytest.mark.parametrize("n", [1, 2, 3, 31, 32, 33, 63, 64, 65])
@pytest.mark.parametrize("kind", ["box", "grid", "soup", "far"])
def test_flat_equals_tree(crt_ctx, n, kind):
    import torch

    from cudaraytracer_b200 import Scene, scenes

    if kind == "box":
        n = min(n, 36)
    tris = triangles(n, n, kind)
    if n > 4:
        tris[n // 2] = tris[n // 3]  # a duplicate: equal t everywhere on it
    sc = Scene.from_triangles(crt_ctx, tris)
    r = torch.from_numpy(rays(tris, 1 << 16, n)).cuda()
    q = torch.from_numpy(scenes.random_shadow_queries(tris, 1 << 16, seed=n)).cuda()
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
