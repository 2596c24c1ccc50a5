"""The a-trous passes over sub-lattice tiles against the same passes with
every tap from global memory (CRT_SVGF_TILED=0), for images around the tile
sizes and up to eight passes (steps to 128, past the image). The two differ
in the roundings of the weights; the bound is the filter's own parity bar
against the reference, 1e-3 relative and 1e-4 absolute."""
import os

import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def frames(w, h, n, seed):
    """A static view: patches of two materials and three meshes with smooth
    normals and depths, some background, and noise of its own per frame."""
    import torch

    rng = np.random.default_rng(seed)
    y, x = np.mgrid[0:h, 0:w].astype(np.float32)
    mesh = 1 + ((x // 13 + y // 9) % 3).astype(np.int64)
    mesh[rng.random((h, w)) < 0.03] = 0
    nrm = np.stack([0.3 * np.sin(x / 17), 0.3 * np.cos(y / 11), np.ones_like(x)], -1)
    nrm /= np.linalg.norm(nrm, axis=-1, keepdims=True)
    nm = np.zeros((h, w, 4), np.uint16)
    nm[..., :3] = ((nrm * 0.5 + 0.5) * 65535).astype(np.uint16)
    nm[..., 3] = mesh % 2
    bm = np.zeros((h, w, 4), np.uint16)
    bm[..., 3] = mesh
    md = np.zeros((h, w, 4), np.float32)
    md[..., 2] = 3 + 0.01 * x + 0.02 * y
    md[..., 3] = 0.03
    g = {"pos_tri": torch.zeros((h, w, 4), device="cuda"), "normal_mat": torch.from_numpy(nm.view(np.int16)).cuda(),
         "bary_mesh": torch.from_numpy(bm.view(np.int16)).cuda(), "motion_depth": torch.from_numpy(md).cuda()}
    noisy = [[torch.from_numpy(rng.exponential(1.0, (h, w, 4)).astype(np.float32)).cuda() for _ in range(2)]
             for _ in range(n)]
    return g, noisy


@pytest.mark.parametrize("w,h", [(1, 1), (3, 40), (31, 7), (32, 8), (33, 9), (67, 35), (130, 71), (257, 129)])
@pytest.mark.parametrize("iterations", [1, 2, 5, 8])
def test_lattice_equals_global_taps(crt_ctx, w, h, iterations):
    import torch

    from cudaraytracer_b200 import Svgf
    from cudaraytracer_b200.tracer import default_denoise_params

    p = default_denoise_params()
    p.atrous_iterations = iterations
    g, noisy = frames(w, h, 6, w + iterations)
    got = []
    try:
        for tiled in ("1", "0"):
            os.environ["CRT_SVGF_TILED"] = tiled
            sv = Svgf(crt_ctx, w, h)
            outs = []
            for d, i in noisy:
                od, oi = torch.empty_like(d), torch.empty_like(i)
                sv.frame(g, g, d, i, od, oi, params=p)
                outs.append(torch.stack([od, oi]).cpu().numpy())
            sv.close()
            got.append(np.stack(outs))
    finally:
        os.environ.pop("CRT_SVGF_TILED", None)
    assert np.isfinite(got[0]).all()
    np.testing.assert_allclose(got[0], got[1], rtol=1e-3, atol=1e-4)
