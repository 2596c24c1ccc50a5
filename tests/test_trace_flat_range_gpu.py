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


@pytest.mark.parametrize("n", [2, 13, 32, 63])
@pytest.mark.parametrize("exponent", [-46, -43, -40, -34, -20, 20, 34])
def test_scaled_scenes(crt_ctx, n, exponent):
    """A scene and its rays scaled by a power of two: products of three
    lengths leave the range of normal floats."""
    from cudaraytracer_b200 import scenes

    s = np.float32(2.0 ** exponent)
    tris, r = soup(n, 100 + n), random_rays(1 << 16, n)
    q = scenes.random_shadow_queries(tris, 1 << 14, seed=n)
    t = tris.reshape(-1, 3, 3)
    k, w = np.arange(1 << 14) % n, np.random.default_rng(n).dirichlet((1, 1, 1), 1 << 14)
    r[:1 << 14, 0:3] = np.einsum("nk,nkc->nc", w, t[k])  # from points of triangles
    r[:, 0:3] *= s
    q[:, 0:3] *= s
    q[:, 6:9] *= s
    check(crt_ctx, tris * s, r, q)
    r[:, 4:7] *= np.float32(2.0 ** -30)
    check(crt_ctx, tris * s, r, q)


@pytest.mark.parametrize("n", [2, 3, 32])
def test_products_beyond_the_largest_float(crt_ctx, n):
    """Origin times direction overflows where the triangle test's own
    products do not: rays along the diagonals into triangles around them."""
    d, s = 1e16, 5e23
    tris, r = [], np.zeros((64, 8), np.float32)
    for k in range(max(n, 64)):
        sx, sy, e = (-1) ** (k & 1), (-1) ** (k >> 1 & 1), 1e-6 / (1 + k)
        if k < n:  # facing the origin of the rays of this diagonal
            tris.append([[0, 0, -e / 4], [0, 0, e], [e * sy, -e * sx, -e / 4]])
        if k < 64:
            r[k, 0:3] = np.array([sx, sy, 0]) * s * 2.0 ** -(k >> 2)
            r[k, 4:7] = np.array([-sx, -sy, 0]) * d
    r[:, 7] = 1e8
    prims = check(crt_ctx, np.array(tris, np.float32).reshape(n, 9), r)
    assert (prims >= 0).any()


@pytest.mark.parametrize("tilt", [0.0, 1e-6, 1e-3])
@pytest.mark.parametrize("n", [12, 33, 64])
def test_fans_around_the_origin(crt_ctx, n, tilt):
    """Long, nearly coplanar triangles that share a vertex close to grazing
    rays: the determinants cancel, and t's error is det's."""
    rng = np.random.default_rng(n)
    a, da, m, length = rng.uniform(0, 2 * np.pi, n), rng.uniform(0.01, 1.0, n), 1 << 17, 100.0

    def far(a):
        r = length * rng.uniform(0.5, 1, n)
        return np.stack([r * np.cos(a), r * np.sin(a), r * tilt * rng.normal(size=n)], 1)

    t = np.zeros((n, 3, 3))
    t[:, 1], t[:, 2] = far(a), far(a + da)
    t[::2, 1:] = t[::2, :0:-1]  # both facings
    r = np.zeros((m, 8), np.float32)
    b, c = rng.uniform(0, 2 * np.pi, m), 10 ** rng.uniform(-7, -1, m) * rng.choice([-1, 1], m)
    r[:, 0:3] = rng.normal(size=(m, 3)) * 10 ** rng.uniform(-8, -2, (m, 1))
    r[:, 4:7], r[:, 7] = np.stack([np.cos(b), np.sin(b), c], 1), 1e8
    prims = check(crt_ctx, t.reshape(n, 9).astype(np.float32), r)
    assert (prims >= 0).mean() > 0.05
