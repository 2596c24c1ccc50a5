"""The convolution kernel's tilings (whole rows of 128 pixels, tiles that run
across the rows of a strip, one or several channel stages, resident or
streamed weights, groups of output channels) at the sizes where each can go
wrong, and outputs aligned to 16 but not 32 bytes, against the same sums in
64 bits. The GPU accumulates in FP32: the bound is that of the sum of |terms|
(plus half a BF16 ulp for BF16 outputs), as in test_conv_gpu.py."""
import pytest

pytestmark = pytest.mark.gpu

CASES = [  # n, h, w, cin, cout
    (1, 5, 126, 32, 32), (1, 5, 127, 32, 32), (2, 9, 128, 16, 16), (1, 9, 129, 64, 64), (1, 7, 130, 32, 48),
    (1, 3, 253, 16, 32), (1, 4, 254, 64, 80), (1, 4, 255, 32, 32), (2, 3, 257, 96, 32), (1, 40, 1, 32, 32),
    (1, 1, 700, 64, 96), (3, 33, 37, 96, 96), (8, 32, 32, 64, 96), (1, 61, 131, 160, 64), (2, 31, 66, 64, 160),
    (1, 70, 500, 96, 32), (1, 9, 380, 160, 64), (1, 5, 20, 512, 32), (1, 2, 140, 256, 240), (4, 64, 64, 128, 128),
]


def _taps(x):
    import torch

    h, w = x.shape[1:3]
    p = torch.nn.functional.pad(x, (0, 0, 1, 1, 1, 1))
    return [p[:, t // 3:t // 3 + h, t % 3:t % 3 + w] for t in range(9)]


@pytest.mark.parametrize("n,h,w,cin,cout", CASES)
def test_forward_and_data_gradient_tiles(crt_ctx, n, h, w, cin, cout):
    import torch

    from cudaraytracer_b200 import kpcn

    g = torch.Generator(device="cuda").manual_seed(cin * 7 + cout + w)
    rnd = lambda *s: torch.randn(s, generator=g, device="cuda")  # noqa: E731
    x, gy = rnd(n, h, w, cin).bfloat16(), rnd(n, h, w, cout).bfloat16()
    wt, bias = (rnd(9, cout, cin) / (9 * cin) ** 0.5).bfloat16(), rnd(cout)
    wtt = wt.transpose(1, 2).contiguous()

    def off16(channels):  # a contiguous tensor whose address is 16 modulo 32
        flat = torch.empty(n * h * w * channels + 16, dtype=torch.bfloat16, device="cuda")
        return flat[8:8 + n * h * w * channels].view(n, h, w, channels)

    f32 = torch.empty((n, h, w, cout), device="cuda")
    y = kpcn.conv3x3_forward(crt_ctx, x, wt, bias, relu=True, out=torch.empty_like(gy), out_f32=f32)
    y16 = kpcn.conv3x3_forward(crt_ctx, x, wt, bias, relu=True, out=off16(cout))
    crt_ctx.check_device_errors()
    assert torch.equal(y, y16)

    w64, b64 = wt.double(), bias.double()
    ref = torch.relu(sum(s @ w64[t].T for t, s in enumerate(_taps(x.double()))) + b64)
    tol = 2e-5 * (sum(s @ w64[t].T.abs() for t, s in enumerate(_taps(x.double().abs()))) + b64.abs()) + 1e-6
    assert bool(((f32.double() - ref).abs() <= tol).all())
    assert bool(((y.double() - ref).abs() <= tol + ref.abs() * 2.0 ** -8).all())
    if cin > 256:  # the data gradient's output channels end at 256
        return
    dx = kpcn.conv3x3_backward_data(crt_ctx, gy, wtt, mask=x)
    dx16 = kpcn.conv3x3_backward_data(crt_ctx, gy, wtt, mask=x, out=off16(cin))
    crt_ctx.check_device_errors()
    assert torch.equal(dx, dx16)
    wf = w64.flip(0)
    ref = sum(s @ wf[t] for t, s in enumerate(_taps(gy.double()))) * (x > 0)
    tol = 2e-5 * sum(s @ wf[t].abs() for t, s in enumerate(_taps(gy.double().abs()))) + 1e-6
    assert bool(((dx.double() - ref).abs() <= tol + ref.abs() * 2.0 ** -8).all())
