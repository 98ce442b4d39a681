"""Deferred weight-gradient products on fp16 pairs made of the accumulator's TF32 planes (csrc/gemm_tc.cu, wgrad_on_f16): either side of the
rule, one and two right operands, widths that are no multiple of 64, rows whose values differ by 2^60, the accumulator used again with fewer
columns.  Against float64; bar on fp16 pairs: 4.5e-7 of |row| |column|, that of every such product, and the last rounding; on TF32 pairs: a
chain of 96 accumulations, each cut off at 2^-24 of a partial sum, 5.7e-6."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N0,N1,k", [(4096, 512, 1024, 300), (3001, 1030, 517, 777), (3000, 1100, 0, 256), (3000, 1100, 0, 255), (1700, 1600, 50, 400), (8000, 100, 800, 500)])
def test_wgrad_products(M, N0, N1, k):
    import torch
    import gpu_util as g
    ctx = g.ctx()
    gen = torch.Generator("cuda").manual_seed(M)
    w = ctx.wgrad_create(M, N0, N1, k)
    try:
        for n in (k, k // 2):
            def mat(rows):
                return torch.randn(n, rows, device="cuda", generator=gen) * torch.exp2(torch.randint(-30, 30, (rows,), device="cuda", generator=gen).float())
            a, bs = mat(M), [mat(N) for N in (N0, N1) if N]
            Cs = [torch.randn(b.shape[1], M, device="cuda", generator=gen) for b in bs]
            before = [C.double() for C in Cs]
            ctx.wgrad_push(w, n, a.data_ptr(), M, bs[0].data_ptr(), N0, None, 0, bs[1].data_ptr() if N1 else None, N1, None, 0)
            ctx.wgrad_flush(w, Cs[0].data_ptr(), M, Cs[1].data_ptr() if N1 else None, M if N1 else 0)
            for b, C, C0 in zip(bs, Cs, before):
                want = b.double().t() @ a.double()
                f16 = n >= 256 and M * (N0 + N1) >= 800 * (M + N0 + N1)
                bar = (4.5e-7 if f16 else 5.7e-6) * b.double().norm(dim=0)[:, None] * a.double().norm(dim=0)[None, :] + 6e-8 * (want.abs() + C0.abs())
                assert bool(((C.double() - C0 - want).abs() <= bar).all())
    finally:
        ctx.wgrad_destroy(w)
    assert ctx.device_errors() == 0
