"""Deferred weight-gradient products on fp16 pairs made of the accumulator's TF32 planes (csrc/gemm_tc.cu, wgrad_on_f16): either side of the
rule, one and two right operands, widths that are no multiple of 64, rows whose values differ by 2^60, the accumulator used again with fewer
columns.  Against float64; bar on fp16 pairs: 4.5e-7 of |row| |column|, that of every such product, and the last rounding; on TF32 pairs: a
chain of 96 accumulations, each cut off at 2^-24 of a partial sum, 5.7e-6 (sides of at most 128 columns have no pairs)."""
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
                f16 = n >= 256 and M * (N0 + N1) >= 800 * (M + N0 + N1) and b.shape[1] > 128
                bar = (4.5e-7 if f16 else 5.7e-6) * b.double().norm(dim=0)[:, None] * a.double().norm(dim=0)[None, :] + 6e-8 * (want.abs() + C0.abs())
                assert bool(((C.double() - C0 - want).abs() <= bar).all())
    finally:
        ctx.wgrad_destroy(w)
    assert ctx.device_errors() == 0


@pytest.mark.parametrize("M,N0,N1,decay", [(2048, 1100, 1024, 20), (2048, 1100, 1024, 26), (2048, 1100, 1024, 40), (3001, 100, 1301, 60), (3001, 1301, 100, 60), (1700, 1600, 0, 110)])
def test_gradients_that_decay_over_the_steps(M, N0, N1, decay):
    """Features that are there in the first steps only, gate gradients that reach them 2^decay smaller than they are in the last: every entry of
    their dW to the error of TF32 pairs, which hold 22 bits of a value whatever the size of the others - also with masked columns (zeros) between."""
    import torch
    import gpu_util as g
    ctx = g.ctx()
    gen = torch.Generator("cuda").manual_seed(M + decay)
    T, B = 40, 16
    k, early = T * B, 3 * B
    t = torch.arange(T, device="cuda").repeat_interleave(B).float()
    a = torch.randn(k, M, device="cuda", generator=gen) * torch.exp2(-decay * (T - 1 - t) / (T - 1))[:, None]
    a[5::16] = 0.0
    bs = [torch.randn(k, N, device="cuda", generator=gen) for N in (N0, N1) if N]
    for b in bs:
        b[early:, ::7] = 0.0
    Cs = [torch.zeros(b.shape[1], M, device="cuda") for b in bs]
    w = ctx.wgrad_create(M, N0, N1, k)
    try:
        ctx.wgrad_push(w, k, a.data_ptr(), M, bs[0].data_ptr(), N0, None, 0, bs[1].data_ptr() if N1 else None, N1, None, 0)
        ctx.wgrad_flush(w, Cs[0].data_ptr(), M, Cs[1].data_ptr() if N1 else None, M if N1 else 0)
        for b, C in zip(bs, Cs):
            want = b.double().t() @ a.double()
            bar = 5.7e-6 * b.double().norm(dim=0)[:, None] * a.double().norm(dim=0)[None, :] + 6e-8 * want.abs()
            bar[::7] = 5.7e-6 * b[:early, ::7].double().norm(dim=0)[:, None] * a[:early].double().norm(dim=0)[None, :] + 6e-8 * want[::7].abs()
            err = (C.double() - want).abs()
            assert bool((err <= bar).all()), "worst error / bar %.3g" % float((err / bar).max())
    finally:
        ctx.wgrad_destroy(w)
    assert ctx.device_errors() == 0
