"""Pairs of fp16 made in one pass (csrc/gemm_tc.cu: k_f16_strip, k_f16_line) against the two passes for longer operands: through products whose operands lie
on either side of the line - lines of 8192 and 16384 values, strips of 256, 512 and 1024 lines - with positions and values that fill no quad, strip or
warp, unaligned operands, and rows of zeros and of values 2^90 apart.  Bar: 4.5e-7 of |row| |column|, that of every product on fp16 pairs."""
import pytest

pytestmark = pytest.mark.gpu


# op(A) = A^T: A's lines are its columns of K values; op(A) = A: strips of rows over K lines.  The same for B.
@pytest.mark.parametrize("M,N,K,tA,tB,off", [
    (1500, 3001, 1000, 1, 0, 0), (1500, 3001, 1001, 1, 0, 1),       # lines of 1000 (a warp each), not aligned
    (600, 900, 8192, 1, 0, 0), (600, 900, 8193, 1, 0, 0), (400, 700, 16385, 1, 0, 1),
    (4001, 4099, 256, 0, 1, 0), (4001, 4099, 257, 0, 1, 1),         # strips over 256 lines and one more
    (3001, 2999, 512, 0, 1, 0), (3001, 2999, 513, 0, 1, 0), (2001, 2003, 1024, 0, 1, 1), (2001, 2003, 1025, 0, 1, 0),
    (12290, 600, 1024, 0, 1, 0),                                    # more values than a strip pass takes
])
def test_products_of_pairs_made_in_one_pass(M, N, K, tA, tB, off):
    import torch
    import gpu_util as g
    gen = torch.Generator("cuda").manual_seed(M + K)

    def operand(rows, K, k_fast):
        t = torch.randn((rows, K) if k_fast else (K, rows), device="cuda", generator=gen)
        scale = torch.exp2(torch.randint(-45, 45, (rows,), device="cuda", generator=gen).float())
        scale[::17] = 0.0
        t = t * (scale[:, None] if k_fast else scale)
        buf = torch.zeros(t.numel() + 4, device="cuda")
        buf[off:off + t.numel()] = t.reshape(-1)
        return buf, (t if k_fast else t.t()).double(), buf.data_ptr() + 4 * off

    bA, A, pA = operand(M, K, tA)
    bB, B, pB = operand(N, K, not tB)
    Cm = torch.empty(N, M, device="cuda")
    assert 2.0 * M * N * K >= 8e9
    g.ctx().gemm(tA, tB, M, N, K, pA, K if tA else M, pB, N if tB else K, Cm.data_ptr(), M, 0)
    want = B @ A.t()
    bar = 4.5e-7 * B.norm(dim=1)[:, None] * A.norm(dim=1)[None, :] + 1e-44
    assert bool(((Cm.double() - want).abs() <= bar).all())
    assert g.ctx().device_errors() == 0


@pytest.mark.parametrize("M,N,K,tA,tB", [(1500, 3001, 1000, 1, 0), (600, 900, 8193, 1, 0), (4001, 4099, 257, 0, 1), (2001, 2003, 1024, 0, 1)])
def test_infinities_and_nans_stay_in_their_row(M, N, K, tA, tB):
    import torch
    import gpu_util as g
    gen = torch.Generator("cuda").manual_seed(M)
    A, B = [torch.randn(r, K, device="cuda", generator=gen) for r in (M, N)]

    def product(A, B):
        a, b, C = A if tA else A.t().contiguous(), B if not tB else B.t().contiguous(), torch.empty(N, M, device="cuda")
        g.ctx().gemm(tA, tB, M, N, K, a.data_ptr(), K if tA else M, b.data_ptr(), N if tB else K, C.data_ptr(), M, 0)
        torch.cuda.synchronize()
        return C

    clean = product(A, B)
    A2, B2 = A.clone(), B.clone()
    A2[M - 1, 0], A2[130, K - 1], B2[N - 1, 3] = float("inf"), float("nan"), float("-inf")
    got = product(A2, B2)
    rows, cols = [r for r in range(M) if r not in (130, M - 1)], [n for n in range(N - 1)]
    assert torch.equal(got[cols][:, rows], clean[cols][:, rows])
    assert not bool(torch.isfinite(got[:, [130, M - 1]]).any()) and not bool(torch.isfinite(got[N - 1]).any())
    assert g.ctx().device_errors() == 0
