"""The passes that make fp16 pairs of an operand (csrc/gemm_tc.cu): scales per line and per position, lines that are a warp's, a CTA's or several
CTAs', positions in groups of threads and beyond, edges in both directions, misaligned sources.  Seen through products whose other operand
has a single non-zero per column, so that a result is one element of the operand: it must come back to 2^-22 of itself (2 x 11 bits),
over 2^40 between the rows."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("tA,M,N,K,off", [
    (0, 4100, 4100, 260, 0),       # A: 260 lines of 4100 positions; B: 4100 short lines
    (0, 13003, 1200, 300, 0),      # rows that are no multiple of 4
    (1, 4100, 1300, 2049, 0),      # A: lines beyond a warp's
    (1, 300, 1500, 9001, 1),       # A: lines of two pieces, misaligned
    (0, 135, 400, 90001, 0),       # A: positions in groups of threads
])
def test_values_come_back(tA, M, N, K, off):
    import torch
    import gpu_util as g
    assert 2.0 * M * N * K >= 8e9
    gen = torch.Generator("cuda").manual_seed(M)
    rows = torch.exp2(torch.randint(-20, 20, (M,), device="cuda", generator=gen).float())
    A = torch.randn(M, K, device="cuda", generator=gen) * rows[:, None]
    A[M // 2] = 0.0
    ks = torch.cat([torch.tensor([0, K - 1], device="cuda"), torch.randint(0, K, (N - 2,), device="cuda", generator=gen)])
    B = torch.zeros(N, K, device="cuda")
    B[torch.arange(N, device="cuda"), ks] = 1.0
    buf = torch.empty(M * K + off, device="cuda")
    stored = buf[off:].view(M, K).copy_(A) if tA else buf[off:].view(K, M).copy_(A.t())
    C = torch.empty(N, M, device="cuda")
    g.ctx().gemm(tA, 0, M, N, K, stored.data_ptr(), K if tA else M, B.data_ptr(), K, C.data_ptr(), M, 0)
    want = A[:, ks].t()
    assert bool(((C - want).abs() <= 2.0 ** -22 * want.abs()).all())
    assert g.ctx().device_errors() == 0
