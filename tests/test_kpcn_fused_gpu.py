"""The denoiser's output layer with the filter in its epilogue, and the
concatenated inputs written by the layers they come from: the filtered image
against the logits (of the debug tensor) applied in 64 bits, the logits and
concatenations against the training pass's and their sources, for images
around the tile widths. FP32 softmax and 25 sums of positive terms: 1e-5."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,h,w", [(1, 4, 4), (3, 8, 20), (1, 36, 124), (1, 12, 132), (2, 16, 260), (1, 64, 640)])
def test_filter_and_concatenation(crt_ctx, n, h, w):
    import torch

    from cudaraytracer_b200.kpcn import Kpcn

    rng = np.random.default_rng(h * w)
    net = Kpcn(crt_ctx, seed=2)
    p = net.get_params()
    p[-32:-7] = rng.normal(size=25)  # the filter's bias: not uniform
    net.set_params(p)
    feat = torch.from_numpy(rng.normal(size=(n, h, w, 16)).astype(np.float32)).cuda().bfloat16()
    noisy = torch.from_numpy(rng.exponential(1.0, (n, h, w, 4)).astype(np.float32)).cuda()
    out = net.forward(feat, noisy)
    logits = net.debug_tensor(10, (n, h, w, 32), np.float32)
    cat0 = net.debug_tensor(14, (n, h, w, 96), np.int16)
    cat1 = net.debug_tensor(13, (n, h // 2, w // 2, 160), np.int16)
    e0b, d1b = net.debug_tensor(1, (n, h, w, 32), np.int16), net.debug_tensor(7, (n, h // 2, w // 2, 64), np.int16)
    e1b = net.debug_tensor(3, (n, h // 2, w // 2, 64), np.int16)
    e2b = net.debug_tensor(5, (n, h // 4, w // 4, 96), np.int16)
    up = lambda a: a.repeat(2, 1).repeat(2, 2)  # noqa: E731
    assert np.array_equal(cat0, np.concatenate([up(d1b), e0b], -1))
    assert np.array_equal(cat1, np.concatenate([up(e2b), e1b], -1))
    net.train_step(feat, noisy, noisy, 0.0)
    assert np.array_equal(net.debug_tensor(10, (n, h, w, 32), np.float32), logits)
    crt_ctx.check_device_errors()
    net.close()
    wt = torch.softmax(torch.from_numpy(logits[..., :25]).cuda().double(), -1)
    ys, xs = torch.arange(h, device="cuda"), torch.arange(w, device="cuda")
    ref = torch.zeros((n, h, w, 3), dtype=torch.float64, device="cuda")
    for k in range(25):
        v = noisy[:, (ys + k // 5 - 2).clamp(0, h - 1)][:, :, (xs + k % 5 - 2).clamp(0, w - 1)]
        ref += wt[..., k:k + 1] * v[..., :3].double()
    np.testing.assert_allclose(out[..., :3].double().cpu().numpy(), ref.cpu().numpy(), rtol=1e-5)
    assert not out[..., 3].any()
