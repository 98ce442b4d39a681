"""Products of at most 64 rows with a reduction of more than 64 (k_gemm_slices, csrc/gemm_narrow.cu) with a bias per row, as the per-token layers of a tagger have one,
and into columns longer than the product, whose rows beyond it stay: every number of columns per lane, slices whose sums meet and tiles
that are stored as they are, rows in fours and one by one, the bias on 16 bytes and off them."""
import pytest

from util import TOL_REDUCE, assert_close

pytestmark = pytest.mark.gpu

SHAPES = [(32, 256, 65), (5, 300, 66), (31, 521, 128), (32, 521, 129), (64, 300, 256), (33, 1183, 131), (60, 1185, 192), (32, 2369, 68), (64, 4737, 200),
          (61, 9473, 255), (32, 37889, 72), (29, 40000, 100), (64, 38000, 130)]


@pytest.mark.parametrize("M,N,K", SHAPES)
@pytest.mark.parametrize("off", [0, 1])
def test_bias(M, N, K, off):
    import torch
    import gpu_util as g
    ctx = g.ctx()
    torch.manual_seed(M + N + K)
    w, x, b = torch.randn(K, M, device="cuda"), torch.randn(N, K, device="cuda"), torch.randn(M + off, device="cuda")[off:]
    y = torch.full((N, M), 7.0, device="cuda")
    before = ctx.launches()
    ctx.fwd("affine_transform", [g.T(b, [M], 1), g.T(w, [M, K], 1), g.T(x, [K], N)], g.T(y, [M], N))
    assert ctx.launches() - before == 1
    # (the bar of test_gpu_narrow.py)
    assert_close(y.cpu().numpy(), (x.double() @ w.double() + b.double()).cpu().numpy(), TOL_REDUCE, floor=0.1 * K ** 0.5, what="narrow product with a bias")
    assert ctx.device_errors() == 0


@pytest.mark.parametrize("M,N,K,ldc", [(32, 256, 65, 36), (32, 521, 129, 33), (31, 521, 128, 32), (64, 4737, 200, 68), (61, 9473, 255, 70), (32, 37889, 72, 40), (64, 300, 256, 65)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_rows_beyond_the_product_stay(M, N, K, ldc, accumulate):
    import torch
    import gpu_util as g
    ctx = g.ctx()
    torch.manual_seed(M + N + K)
    a, b, c0 = torch.randn(K, M, device="cuda"), torch.randn(N, K, device="cuda"), torch.randn(N, ldc, device="cuda")
    c = c0.clone()
    ctx.gemm(0, 0, M, N, K, a.data_ptr(), M, b.data_ptr(), K, c.data_ptr(), ldc, int(accumulate))
    want = b.double() @ a.double() + (c0.double()[:, :M] if accumulate else 0.0)
    assert_close(c[:, :M].cpu().numpy(), want.cpu().numpy(), TOL_REDUCE, floor=0.1 * K ** 0.5, what="narrow product")
    assert torch.equal(c[:, M:], c0[:, M:])
    assert ctx.device_errors() == 0
