"""Large products on fp16 pairs (csrc/gemm_tc.cu): every operand layout, sizes that are no multiple of the tiles, rows and columns
of very different magnitude, infinities and zeros, against float64 on sampled columns.  Bar: the error of one element relative to
|row of A| |column of B| - the fp32 sums of the TF32 pairs they replace were within 4.5e-7 of it, so is this bar."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tA,tB,M,N,K,accumulate", [
    (0, 0, 4099, 3000, 1001, False),     # MN-major A, K-major B, edges everywhere
    (1, 0, 2000, 3007, 2050, True),      # both K-major, accumulate
    (0, 1, 3100, 1030, 4100, True),      # both MN-major
    (1, 1, 1500, 4103, 2111, False),     # K-major A, MN-major B
    (0, 0, 20000, 1500, 520, False),     # many tiles, less than one accumulation chain
    (1, 0, 130, 1200, 80000, False),     # a long reduction over few tiles: K splits
    # a side of at most 128: one SM per tile (those above are products of the pair kernel)
    (0, 1, 50000, 128, 4096, True),      # persistent, 128 columns
    (0, 0, 20000, 64, 4000, False),      # persistent, 64 columns
    (0, 0, 19999, 63, 4004, True),       # ... and edges
    (1, 0, 100, 12000, 12000, True),     # one row of tiles
    (0, 1, 128, 1200, 90000, True),      # K splits
    (1, 0, 128, 300, 120000, False),
    (0, 1, 1030, 128, 100000, False),
])
def test_large_product(tA, tB, M, N, K, accumulate):
    import torch
    import gpu_util as g
    assert 2.0 * M * N * K > 8e9
    gen = torch.Generator("cuda").manual_seed(M + N)
    A = torch.randn(*((M, K) if tA else (K, M)), device="cuda", generator=gen)
    B = torch.randn(*((N, K) if tB == 0 else (K, N)), device="cuda", generator=gen)
    sa = torch.exp2(torch.randint(-30, 30, (M,), device="cuda", generator=gen).float())
    sb = torch.exp2(torch.randint(-30, 30, (N,), device="cuda", generator=gen).float())
    sa[3] = 0.0                                                    # a row of zeros
    A *= sa[:, None] if tA else sa[None, :]
    B *= sb[:, None] if tB == 0 else sb[None, :]
    C = torch.randn(N, M, device="cuda", generator=gen) if accumulate else torch.full((N, M), 7.0, device="cuda")
    C0 = C.clone()
    g.ctx().gemm(tA, tB, M, N, K, A.data_ptr(), K if tA else M, B.data_ptr(), K if tB == 0 else N, C.data_ptr(), M, int(accumulate))
    cols = torch.cat([torch.arange(0, N, max(1, N // 40), device="cuda"), torch.tensor([N - 1], device="cuda")])
    Ad, Bd = (A if tA else A.t()).double(), (B if tB == 0 else B.t())[cols].double()
    want = Bd @ Ad.t() + (C0[cols].double() if accumulate else 0.0)
    # (an accumulated element is rounded once more, at its own size)
    bar = 4.5e-7 * Bd.norm(dim=1)[:, None] * Ad.norm(dim=1)[None, :] + (6e-8 * (want.abs() + C0[cols].abs().double()) if accumulate else 0.0)
    err = (C[cols].double() - want).abs()
    assert bool((err <= bar).all()), "worst error / bar %.3g" % float((err / bar.clamp_min(1e-300)).max())
    assert g.ctx().device_errors() == 0


def test_infinities_stay_in_their_rows():
    import torch
    import gpu_util as g
    M, N, K = 3000, 3000, 1500
    A, B = torch.randn(K, M, device="cuda"), torch.randn(N, K, device="cuda")
    A[7, 5] = float("inf")
    C = torch.empty(N, M, device="cuda")
    g.ctx().gemm(0, 0, M, N, K, A.data_ptr(), M, B.data_ptr(), K, C.data_ptr(), M, 0)
    want = B[:50].double() @ torch.nan_to_num(A, posinf=0.0).double()
    assert not bool(torch.isfinite(C[:, 5]).any())
    keep = torch.arange(M, device="cuda") != 5
    assert float((C[:50].double() - want)[:, keep].abs().max()) < 4.5e-7 * K * 2


@pytest.mark.parametrize("tA", [0, 1])
@pytest.mark.parametrize("cache", [False, True])
def test_parameter_rows_keep_their_own_scale(tA, cache):
    """A parameter operand whose rows differ by 2^60: the same bar as any other product.  With the cache on the second product takes
    the planes of the first, and the transposed product of the same matrix must not get them with the wrong scales."""
    import torch
    from dynet_b200 import capi
    M, N, K = 4100, 2999, 1030
    ctx = capi.Context(0, torch.cuda.current_stream().cuda_stream)
    ctx.param_cache(cache)
    gen = torch.Generator("cuda").manual_seed(7)
    A = torch.randn(*((M, K) if tA else (K, M)), device="cuda", generator=gen)
    A *= torch.exp2(torch.randint(-30, 30, (M,), device="cuda", generator=gen).float()).view((M, 1) if tA else (1, M))
    B = torch.randn(N, K, device="cuda", generator=gen)
    C = torch.empty(N, M, device="cuda")
    for _ in range(2):
        C.fill_(7.0)
        ctx.gemm(tA, 0, M, N, K, A.data_ptr(), K if tA else M, B.data_ptr(), K, C.data_ptr(), M, 0, 1)   # 1: A_IS_PARAM
        Ad = (A if tA else A.t()).double()
        err = (C.double() - B.double() @ Ad.t()).abs() / (B.double().norm(dim=1)[:, None] * Ad.norm(dim=1)[None, :])
        assert float(err.max()) <= 4.5e-7
    # the transposed product: K rows, every one of them with elements of all magnitudes
    D, E = torch.randn(N, M, device="cuda", generator=gen), torch.empty(N, K, device="cuda")
    ctx.gemm(1 - tA, 0, K, N, M, A.data_ptr(), K if tA else M, D.data_ptr(), M, E.data_ptr(), K, 0, 1)   # 1: A_IS_PARAM
    At = (A.t() if tA else A).double()
    err = (E.double() - D.double() @ At.t()).abs() / (D.double().norm(dim=1)[:, None] * At.norm(dim=1)[None, :])
    assert float(err.max()) <= 4.5e-7
    assert ctx.device_errors() == 0


@pytest.mark.parametrize("V,H,n,param", [(12000, 256, 4000, False), (12001, 250, 4003, True), (12000, 128, 8100, False), (12001, 64, 5600, True)])
def test_output_gradient_at_every_row_and_columns_own_scale(V, H, n, param):
    """softmax_output_bwd_fused on fp16 pairs: vocabulary rows whose probability is tiny everywhere, columns whose dE/df differs by 2^40.
    Against float64, every element of dR and dh relative to its own |row| |column|.  Bar: exp of arguments down to -65 (log2: 94) from
    fp32 operands: half an ulp of the argument (2^-18), the rounding of log2(e) (94 x 2^-25) and of z (2^-21), times ln 2, and the
    products' 4.5e-7: below 8e-6.  And the same operands as the node-by-node calls: equal bit for bit."""
    import torch
    from dynet_b200 import capi
    ctx = capi.Context(0, torch.cuda.current_stream().cuda_stream)
    gen = torch.Generator("cuda").manual_seed(V)
    T = lambda t, d, bd=1: capi.DyTensor.of(t.data_ptr(), d, bd)   # noqa: E731
    x = torch.randn(n, V, device="cuda", generator=gen)
    x[:, 1::7] -= 28.0
    x[:, 2::7] -= 50.0
    ids = torch.randint(0, (V - 1) // 7, (n,), device="cuda", generator=gen) * 7
    dE = torch.randn(n, device="cuda", generator=gen) * torch.exp2(torch.randint(-20, 20, (n,), device="cuda", generator=gen).float())
    dE[11] = 0.0
    h, R = torch.randn(n, H, device="cuda", generator=gen), torch.randn(H, V, device="cuda", generator=gen)
    loss, aux = torch.empty(n, device="cuda"), torch.zeros(3 * n, device="cuda")
    aux[2 * n:].view(torch.int32).copy_(ids.int())
    tx, th, tR, tdE, at = T(x, [V], n), T(h, [H], n), T(R, [V, H]), T(dE, [1], n), capi.PickAttrs(None, n)
    ctx.fwd("pickneglogsoftmax", [tx], T(loss, [1], n), at, aux.data_ptr())
    dR, db, dh = torch.zeros(H, V, device="cuda"), torch.zeros(V, device="cuda"), torch.zeros(n, H, device="cuda")
    ctx.softmax_output_bwd_fused(tx, th, tR, tdE, aux.data_ptr(), T(dR, [V, H]), T(db, [V]), T(dh, [H], n), flags=1 if param else 0)
    # node by node
    dx, nR, nh, nb = torch.zeros(n, V, device="cuda"), torch.zeros_like(dR), torch.zeros_like(dh), torch.zeros(V, device="cuda")
    ctx.bwd("pickneglogsoftmax", [tx], T(loss, [1], n), tdE, 0, T(dx, [V], n), at, aux.data_ptr())
    xs, aff = [T(db, [V]), tR, th], capi.AffineAttrs(1 if param else 0)
    for i, d in ((1, T(nR, [V, H])), (2, T(nh, [H], n))):
        ctx.bwd("affine_transform", xs, tx, T(dx, [V], n), i, d, aff)
    d = torch.softmax(x.double(), dim=1)
    d[torch.arange(n, device="cuda"), ids] -= 1.0
    d *= dE.double()[:, None]
    for name, got, want, scale in (("dR", dR, h.double().t() @ d, h.double().norm(dim=0)[:, None] * d.norm(dim=0)[None, :]),
                                   ("dh", dh, d @ R.double().t(), d.norm(dim=1)[:, None] * R.double().norm(dim=1)[None, :])):
        err = (got.double() - want).abs()
        assert bool((err <= 1e-5 * scale).all()), "%s: %.3g" % (name, float((err / scale.clamp_min(1e-300)).max()))
    assert torch.equal(dR, nR) and torch.equal(dh, nh)
    assert ctx.device_errors() == 0
