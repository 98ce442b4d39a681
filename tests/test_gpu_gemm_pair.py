"""Products on pairs of SMs (csrc/gemm_pair.cu): one to nineteen k-blocks (a chain is cut after sixteen, the last two and a tile's first
three k-blocks issue their MMAs in another order), tiles that reach past either edge, results that TMA can and cannot address, K splits
of both kinds; against float64 on sampled columns.  Bar: that of test_gpu_gemm_f16.py (4.5e-7 of |row of A| |column of B|, and the
rounding of the sum where the result is accumulated)."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tA,tB,M,N,K,accumulate", [
    (0, 0, 14001, 13999, 63, False),      # part of one k-block; leading dimension no multiple of 4
    (0, 0, 14000, 13999, 64, True),
    (0, 0, 12292, 9996, 100, True),       # two
    (1, 0, 8196, 8001, 190, False),       # three
    (1, 0, 7170, 7000, 256, True),        # four
    (0, 1, 4352, 2816, 1032, True),       # seventeen
    (1, 1, 3332, 3300, 1152, False),      # eighteen
    (1, 1, 3332, 3301, 1216, True),       # nineteen
    (0, 1, 257, 260, 200003, True),       # four tiles, K splits, partial products that TMA cannot address
    (1, 0, 132, 2001, 50001, False),      # half a tile of rows, K splits
    (0, 0, 255, 48000, 1000, True),
])
def test_pair_product(tA, tB, M, N, K, accumulate):
    import torch
    import gpu_util as g
    assert 2.0 * M * N * K > 24e9
    gen = torch.Generator("cuda").manual_seed(M + N + K)
    A = torch.randn(*((M, K) if tA else (K, M)), device="cuda", generator=gen)
    B = torch.randn(*((N, K) if tB == 0 else (K, N)), device="cuda", generator=gen)
    C = torch.randn(N, M, device="cuda", generator=gen) if accumulate else torch.full((N, M), 7.0, device="cuda")
    cols = torch.cat([torch.arange(0, N, max(1, N // 60), device="cuda"), torch.arange(max(0, N - 40), N, device="cuda")])
    C0 = C[cols].double()
    g.ctx().gemm(tA, tB, M, N, K, A.data_ptr(), K if tA else M, B.data_ptr(), K if tB == 0 else N, C.data_ptr(), M, int(accumulate))
    Ad, Bd = (A if tA else A.t()).double(), (B if tB == 0 else B.t())[cols].double()
    want = Bd @ Ad.t() + (C0 if accumulate else 0.0)
    bar = 4.5e-7 * Bd.norm(dim=1)[:, None] * Ad.norm(dim=1)[None, :] + (6e-8 * (want.abs() + C0.abs()) if accumulate else 0.0)
    err = (C[cols].double() - want).abs()
    assert bool((err <= bar).all()), "worst error / bar %.3g" % float((err / bar).max())
    again = C.clone()
    if not accumulate:
        g.ctx().gemm(tA, tB, M, N, K, A.data_ptr(), K if tA else M, B.data_ptr(), K if tB == 0 else N, again.data_ptr(), M, 0)
        assert torch.equal(C, again)
    assert g.ctx().device_errors() == 0


def test_subnormal_results_are_kept():
    """An accumulated product leaves as TMA adds: results and summands below 2^-126 stay what plain adds make of them."""
    import torch
    import gpu_util as g
    M, N, K = 8000, 3000, 512
    gen = torch.Generator("cuda").manual_seed(1)
    A, B = torch.randn(K, M, device="cuda", generator=gen) * 1e-20, torch.rand(N, K, device="cuda", generator=gen) * 1e-21
    A[:, ::2] = 0.0
    C = torch.rand(N, M, device="cuda", generator=gen) * 2e-38 - 1e-38
    C[:, ::4] = 1e-40
    before = C.double()
    g.ctx().gemm(0, 0, M, N, K, A.data_ptr(), M, B.data_ptr(), K, C.data_ptr(), M, 1)
    assert torch.equal(C.double()[:, ::2], before[:, ::2])
    # (the bar above, and the roundings of the product and of the sum to multiples of 2^-149)
    want = B.double() @ A.double() + before
    bar = 4.5e-7 * B.double().norm(dim=1)[:, None] * A.double().norm(dim=0)[None, :] + 2.0 ** -149
    assert bool(((C.double() - want).abs() <= bar).all())
    assert g.ctx().device_errors() == 0
