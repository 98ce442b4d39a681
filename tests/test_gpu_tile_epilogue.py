"""Tensor-pipe products of one tile per CTA: what a tile adds to waits in a stage of the operand ring that the last k-blocks leave
idle.  Reductions of every remainder of the three stages and of the eight k-blocks of an accumulation chunk, rows and destinations in
16-byte pieces and not, stored and added to (dynet/nodes-affinetransform.cc:77-157: y = b + A x, dA += dy x^T)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("add", [0, 1])
@pytest.mark.parametrize("M,N,ldc", [(260, 130, 260), (259, 200, 261), (384, 64, 388), (130, 100, 130)])
@pytest.mark.parametrize("K", [70, 96, 129, 160, 200, 256, 288, 300, 352, 520, 1050, 2080])
def test_epilogue_of_a_tile(K, M, N, ldc, add):
    import torch
    import gpu_util as g
    ctx = g.ctx()
    torch.manual_seed(K + M)
    a, b, c = torch.randn(K, M, device="cuda"), torch.randn(N, K, device="cuda"), torch.randn(N, ldc, device="cuda")
    want = c.double().clone()
    want[:, :M] = b.double() @ a.double() + (want[:, :M] if add else 0)
    ctx.gemm(0, 0, M, N, K, a.data_ptr(), M, b.data_ptr(), K, c.data_ptr(), ldc, add)
    assert ctx.device_errors() == 0
    # a product of the split operands is off by less than 2^-20 of the sum of magnitudes (the dropped lo * lo term 2^-22, the rounding
    # of lo 2^-22, and fp32 sums over chunks of at most 8 k-blocks); an addition by half an ulp of its result
    bound = 2.0 ** -20 * (b.double().abs() @ a.double().abs()) + 2.0 ** -23 * want[:, :M].abs()
    assert ((c.double()[:, :M] - want[:, :M]).abs() <= bound).all()
    assert torch.equal(c.double()[:, M:], want[:, M:])   # the rows past M stay


@pytest.mark.parametrize("M", [260, 259, 388, 1000])
@pytest.mark.parametrize("N,K", [(130, 160), (130, 1050), (130, 2080), (2500, 96)])   # a tile per CTA, its K splits in clusters, the persistent kernel
@pytest.mark.parametrize("off", [0, 1])
def test_bias_of_ragged_rows(M, N, K, off):
    """y = b + W x with rows that end inside a tile, b on 16 bytes and off them, K splits in clusters and through memory."""
    import torch
    import gpu_util as g
    ctx = g.ctx()
    torch.manual_seed(K + M)
    w, x = torch.randn(K, M, device="cuda"), torch.randn(N, K, device="cuda")
    b = torch.randn(M + off, device="cuda")[off:]
    want, sums = b.double() + x.double() @ w.double(), x.double().abs() @ w.double().abs()
    for clusters in (True, False):
        y = torch.full((N, M), 7.0, device="cuda")
        try:
            ctx.cluster_splitk(clusters)
            ctx.fwd("affine_transform", [g.T(b, [M], 1), g.T(w, [M, K], 1), g.T(x, [K], N)], g.T(y, [M], N))
        finally:
            ctx.cluster_splitk(True)
        assert ctx.device_errors() == 0
        assert ((y.double() - want).abs() <= 2.0 ** -20 * sums + 2.0 ** -23 * want.abs()).all()   # (the bound above)


@pytest.mark.parametrize("I,H,B", [(300, 300, 100), (160, 300, 70), (90, 290, 40), (330, 100, 64)])
def test_two_products_in_splits_of_unlike_shares(I, H, B):
    """Wx x + Wh h where the shares of the two reductions end before the number of K splits does (10 + 10 k-blocks in seven): no split is empty."""
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    torch.manual_seed(I + H)
    x, h, c = torch.randn(B, I, device="cuda"), torch.randn(B, H, device="cuda") * 0.5, torch.randn(B, H, device="cuda")
    wx, wh, b = torch.randn(I, 4 * H, device="cuda") * 0.1, torch.randn(H, 4 * H, device="cuda") * 0.1, torch.randn(4 * H, device="cuda")
    z = (x.double() @ wx.double() + h.double() @ wh.double() + b.double()).view(B, 4, H)
    z[:, 1] += 1.0
    want = torch.cat([torch.sigmoid(z[:, :3]), torch.tanh(z[:, 3:])], 1).view(B, 4 * H)
    sums = x.double().abs() @ wx.double().abs() + h.double().abs() @ wh.double().abs() + b.double().abs()
    got = []
    for clusters in (True, False):
        gates, c1, h1 = torch.empty(B, 4 * H, device="cuda"), torch.empty(B, H, device="cuda"), torch.empty(B, H, device="cuda")
        try:
            ctx.cluster_splitk(clusters)
            ctx.lstm_fwd_fused(g.T(x, [I], B), g.T(h, [H], B), g.T(c, [H], B), g.T(wx, [4 * H, I], 1), g.T(wh, [4 * H, H], 1), g.T(b, [4 * H], 1), None, None,
                               capi.LstmGatesAttrs(0, 0.0, 1.0), g.T(gates, [4 * H], B), g.T(c1, [H], B), g.T(h1, [H], B))
        finally:
            ctx.cluster_splitk(True)
        assert ctx.device_errors() == 0
        # the bound above through a function of slope at most one, and a few ulp of values below one for the function itself
        assert ((gates.double() - want).abs() <= 2.0 ** -20 * sums + 2.0 ** -21).all()
        got.append((gates, c1, h1))
    assert all(torch.equal(p, q) for p, q in zip(*got))
