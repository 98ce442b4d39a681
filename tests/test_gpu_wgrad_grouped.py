"""dWx and dWh as one product over the columns of both operands (csrc/gemm_tc.cu, dyb200_tc_gemm_packed2): widths on either side of a tile, one
tile narrower than the other, 64-column tiles, every form - one tile per CTA, clusters, work items with a second stage, rows that TMA
cannot store - and the accumulator used again.  Against float64; bar: a chain of 96 accumulations on TF32 pairs, each cut off at 2^-24 of
a partial sum, 5.7e-6 of |row| |column|, and the last rounding."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N0,N1,k", [
    (1024, 128, 256, 320), (1000, 129, 127, 1601), (1001, 33, 250, 700), (512, 64, 64, 3000), (256, 7, 65, 31), (130, 40, 64, 1000), (1024, 128, 256, 40000),
    (999, 100, 300, 30001), (4096, 512, 1024, 200), (384, 1, 384, 4000),
])
def test_grouped_products(M, N0, N1, k):
    import torch
    import gpu_util as g
    ctx = g.ctx()
    gen = torch.Generator("cuda").manual_seed(M + k)
    w = ctx.wgrad_create(M, N0, N1, k)
    try:
        for n in (k, max(1, k // 3)):
            a, bs = torch.randn(n, M, device="cuda", generator=gen), [torch.randn(n, N, device="cuda", generator=gen) for N in (N0, N1)]
            pad = 3                                                    # leading dimensions beyond M; what lies between stays as it is
            Cs = [torch.randn(b.shape[1], M + pad, device="cuda", generator=gen) for b in bs]
            before = [C.clone() for C in Cs]
            ctx.wgrad_push(w, n, a.data_ptr(), M, bs[0].data_ptr(), N0, None, 0, bs[1].data_ptr(), N1, None, 0)
            ctx.wgrad_flush(w, Cs[0].data_ptr(), M + pad, Cs[1].data_ptr(), M + pad)
            for b, C, C0 in zip(bs, Cs, before):
                want = b.double().t() @ a.double()
                bar = 5.7e-6 * b.double().norm(dim=0)[:, None] * a.double().norm(dim=0)[None, :] + 6e-8 * (want.abs() + C0[:, :M].double().abs())
                assert bool(((C[:, :M].double() - C0[:, :M].double() - want).abs() <= bar).all())
                assert torch.equal(C[:, M:], C0[:, M:])
    finally:
        ctx.wgrad_destroy(w)
    assert ctx.device_errors() == 0


@pytest.mark.parametrize("M,N,k", [(1024, 128, 320), (256, 100, 31), (1024, 128, 40000), (1700, 1600, 400)])
@pytest.mark.parametrize("layout", ["same", "columns", "rows"])
def test_results_in_one_matrix(M, N, k, layout):
    """One weight read at both places: both products are added to the same matrix, or to one that starts some columns into it; and the two results
    as row blocks of one matrix, which do not meet."""
    import torch
    import gpu_util as g
    ctx = g.ctx()
    gen = torch.Generator("cuda").manual_seed(M + N)
    w = ctx.wgrad_create(M, N, N, k)
    try:
        a, b0, b1 = (torch.randn(k, n, device="cuda", generator=gen) for n in (M, N, N))
        ld = 2 * M if layout == "rows" else M
        C = torch.randn(2 * N, ld, device="cuda", generator=gen)
        want, off = C.double(), dict(same=0, columns=7 * M, rows=M)[layout]
        p0, p1 = b0.double().t() @ a.double(), b1.double().t() @ a.double()
        want[:N, :M] += p0
        if layout == "rows":
            want[:N, M:] += p1
        else:
            want[off // M:off // M + N] += p1
        ctx.wgrad_push(w, k, a.data_ptr(), M, b0.data_ptr(), N, None, 0, b1.data_ptr(), N, None, 0)
        ctx.wgrad_flush(w, C.data_ptr(), ld, C.data_ptr() + 4 * off, ld)
        # (two results of 5.7e-6 of |row| |column| each, and their last roundings)
        bar = 2 * 5.7e-6 * float(a.double().norm(dim=0).max()) * float(torch.cat([b0, b1], 1).double().norm(dim=0).max()) + 2.4e-7 * want.abs().max()
        assert float((C.double() - want).abs().max()) <= float(bar)
    finally:
        ctx.wgrad_destroy(w)
    assert ctx.device_errors() == 0
