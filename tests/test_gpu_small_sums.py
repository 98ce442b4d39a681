"""Sums of few terms in one launch: dyb200_sum_all / dyb200_squared_norm on one CTA, bias gradients (dynet/nodes-affinetransform.cc:112-157) with both
stages in a CTA, at the edges of where they are used.  Values that are multiples of 2^-3 below 2: every sum is exact in fp32, so any order gives it."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n", [1, 3, 4, 1023, 1025, 4095, 4096, 4097, 5000])
@pytest.mark.parametrize("off", [0, 1])
def test_sum_of_all(n, off):
    import torch
    import gpu_util as g
    ctx = g.ctx()
    x = torch.randint(-15, 16, (n + off,), device="cuda", generator=torch.Generator("cuda").manual_seed(n)).float()[off:] / 8
    out = torch.full((2,), 0.5, device="cuda")
    ctx.sum_all(x.data_ptr(), n, out.data_ptr(), 1)
    ctx.squared_norm(x.data_ptr(), n, out[1:].data_ptr(), 0)
    assert out[0].item() == 0.5 + x.double().sum().item() and out[1].item() == (x.double() ** 2).sum().item()


@pytest.mark.parametrize("n,B", [(1, 17), (31, 33), (32, 64), (33, 257), (45, 520), (256, 1024), (257, 1024), (45, 1025), (5003, 52), (5003, 53)])
def test_bias_gradient(n, B):
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    gen = torch.Generator("cuda").manual_seed(n + B)
    up = torch.randint(-15, 16, (B, n), device="cuda", generator=gen).float() / 8
    db = torch.ones(n, device="cuda")
    b, W, x, y = torch.zeros(n, device="cuda"), torch.zeros(2, n, device="cuda"), torch.zeros(B, 2, device="cuda"), torch.zeros(B, n, device="cuda")
    xs = [g.T(b, [n], 1), g.T(W, [n, 2], 1), g.T(x, [2], B)]
    ctx.bwd("affine_transform", xs, g.T(y, [n], B), g.T(up, [n], B), 0, g.T(db, [n], 1), None)
    assert torch.equal(db, (1 + up.double().sum(0)).float())
    assert ctx.device_errors() == 0
