"""Kpcn.set_params after an inference: no convolution runs, and the logits of
the debug tensor stay the last forward's."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


def test_set_params_after_forward(crt_ctx):
    import torch
    from torch.profiler import ProfilerActivity, profile

    from cudaraytracer_b200.kpcn import Kpcn

    n, h, w = 2, 24, 36
    rng = np.random.default_rng(3)
    feat = torch.from_numpy(rng.normal(size=(n, h, w, 16)).astype(np.float32)).cuda().bfloat16()
    noisy = torch.from_numpy(rng.exponential(1.0, (n, h, w, 4)).astype(np.float32)).cuda()
    nets = [Kpcn(crt_ctx, seed=s) for s in (4, 4, 5)]
    for k, net in enumerate(nets):  # biases of the output layer that differ
        p = net.get_params()
        p[-32:-7] = np.random.default_rng(10 + k // 2).normal(size=25)
        net.set_params(p)
    net, twin, other = nets
    want = []
    for k in (twin, other):
        k.forward(feat, noisy)
        want.append(k.debug_tensor(10, (n, h, w, 32), np.float32))
    assert not np.array_equal(*want)

    net.forward(feat, noisy)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        net.set_params(other.get_params())
        torch.cuda.synchronize()
    names = " ".join(e.key for e in prof.key_averages())
    net.set_params(rng.normal(size=net.num_params))  # (twice: the first one's copy stays)
    net.set_params(other.get_params())
    assert np.array_equal(net.debug_tensor(10, (n, h, w, 32), np.float32), want[0])
    net.forward(feat, noisy)
    assert np.array_equal(net.debug_tensor(10, (n, h, w, 32), np.float32), want[1])
    crt_ctx.check_device_errors()
    for k in nets:
        k.close()
    if "k_weights_bf16" not in names:
        pytest.skip("no kernel records from the profiler")
    assert "k_conv3x3" not in names
