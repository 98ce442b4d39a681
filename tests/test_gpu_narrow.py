"""Products with a narrow side and a long one (csrc/gemm_narrow.cu) against float64 products, at the edges of its tiles: one row, row
counts around 32 and 64, reductions of one and of several pieces and with remainders, more row blocks than one, column counts on
both sides of the change of tile, operands off a 16-byte boundary; and long reductions whose outputs are one block, several, or a
few that many groups of threads share."""
import numpy as np
import pytest

from util import TOL_REDUCE, assert_close, randn, rng

pytestmark = pytest.mark.gpu


@pytest.fixture(scope="module")
def g():
    import gpu_util
    gpu_util.ctx()
    return gpu_util


@pytest.fixture(autouse=True)
def _release(g):
    yield
    g.release()


def check(g, tA, tB, M, N, K, off, accumulate, floor):
    r = rng(50 + M + N + K)
    A, B, C0 = randn(r, *((M, K) if tA else (K, M))), randn(r, *((K, N) if tB else (N, K))), randn(r, N, M)
    A_, B_, C_ = g.dev(A, off), g.dev(B, off), g.dev(C0, off)
    before = g.ctx().launches()
    g.ctx().gemm(tA, tB, M, N, K, A_.data_ptr(), K if tA else M, B_.data_ptr(), N if tB else K, C_.data_ptr(), M, int(accumulate))
    assert g.ctx().launches() - before == (2 if tB else 1)   # (no operand split: the product itself, and the sum over CTAs)
    a, b = A.astype(np.float64), B.astype(np.float64)
    want = (b.T if tB else b) @ (a.T if tA else a) + (C0 if accumulate else 0.0)
    # fp32 sums of K products of O(1) terms: an error of about sqrt(K) 2^-24 around results of size sqrt(K)
    assert_close(g.host(C_), want, TOL_REDUCE, floor=floor * K ** 0.5, what="narrow product")
    assert g.ctx().device_errors() == 0


@pytest.mark.parametrize("M,N,K,off", [(32, 1100, 256, 0), (45, 20000, 32, 0), (32, 19999, 45, 1), (1, 777, 63, 0), (29, 9999, 40, 0), (48, 5001, 99, 0), (64, 18945, 250, 0),
                                       (33, 256, 250, 2), (256, 19001, 32, 0), (250, 1500, 64, 0), (200, 1301, 61, 3), (100, 512, 1, 0)])
@pytest.mark.parametrize("tA", [0, 1])
@pytest.mark.parametrize("accumulate", [False, True])
def test_few_rows_or_short_reduction(g, M, N, K, off, tA, accumulate):
    check(g, tA, 0, M, N, K, off, accumulate, 0.1)


@pytest.mark.parametrize("M,N,K,off", [(32, 256, 9001, 0), (45, 32, 500, 0), (32, 256, 470, 1), (1, 1, 256, 0), (7, 300, 4099, 1), (64, 1024, 4500, 0),
                                       (1000, 33, 6001, 0), (257, 64, 4097, 3)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_long_reduction(g, M, N, K, off, accumulate):
    check(g, 0, 1, M, N, K, off, accumulate, 0.1)
