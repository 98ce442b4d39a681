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
])
def test_large_product(tA, tB, M, N, K, accumulate):
    import torch
    import gpu_util as g
    assert 2.0 * M * N * K > 24e9 or K == 80000
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
