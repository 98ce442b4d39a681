"""Products with few columns (csrc/gemm_thin.cu): against float64 products at the edges of its tiles - 1 to 32 columns, row counts
that are no multiple of 32 or 4, reductions longer than the piece of B it keeps in shared memory, misaligned operands - through
dyb200_gemm, and the one-step LSTM call with and without masks against the oracle's node chain."""
import numpy as np
import pytest

from util import TOL_REDUCE, assert_close, glorot, randn, rng

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


@pytest.mark.parametrize("M,N,K,off", [(1024, 1, 2500, 0), (999, 2, 301, 0), (130, 3, 64, 1), (4096, 7, 1024, 0), (333, 16, 2049, 0),
                                       (10000, 17, 256, 0), (64, 32, 40, 3), (31, 5, 7, 0)])
@pytest.mark.parametrize("accumulate", [False, True])
def test_thin_product(g, M, N, K, off, accumulate):
    r = rng(40 + M + N)
    A, B, C0 = randn(r, K, M), randn(r, N, K), randn(r, N, M)
    A_, B_, C_ = g.dev(A, off), g.dev(B, off), g.dev(C0, off)
    g.ctx().gemm(0, 0, M, N, K, A_.data_ptr(), M, B_.data_ptr(), K, C_.data_ptr(), M, int(accumulate))
    want = B.astype(np.float64) @ A.astype(np.float64) + (C0 if accumulate else 0.0)
    # fp32 sums of K products of O(1) terms: an error of about sqrt(K) 2^-24 around results of size sqrt(K)
    assert_close(g.host(C_), want, TOL_REDUCE, floor=0.1 * K ** 0.5, what="thin product")
    assert g.ctx().device_errors() == 0


@pytest.mark.parametrize("I,H,B,mask", [(512, 1024, 1, None), (33, 40, 3, "full"), (200, 301, 8, "one"), (1024, 512, 20, "full"), (16, 8, 32, None)])
def test_thin_lstm_step(oracle, g, I, H, B, mask):
    from dynet_b200 import capi
    r = rng(70 + H + B)
    x, h, c_prev = randn(r, B, I), randn(r, B, H, scale=0.5), randn(r, B, H, scale=0.5)
    Wx, Wh, b = glorot(r, 4 * H, I), glorot(r, 4 * H, H), randn(r, 4 * H, scale=0.1)
    mB = B if mask == "full" else 1
    mx = ((r.random((mB, I)) < 0.8) / 0.8).astype(np.float32) if mask else None
    mh = ((r.random((mB, H)) < 0.8) / 0.8).astype(np.float32) if mask else None
    gates = oracle.lstm_gates_fwd([x], h, Wx, Wh, b, mx, mh)
    c_t = oracle.lstm_c_fwd(c_prev, gates)
    h_t = oracle.lstm_h_fwd(c_t, gates)
    og, oc, oh = (g.dev(np.full_like(a, 9.0)) for a in (gates, c_t, h_t))
    g.ctx().lstm_fwd_fused(g.T(g.dev(x)), g.T(g.dev(h)), g.T(g.dev(c_prev)), g.T(g.dev(Wx), [4 * H, I], 1), g.T(g.dev(Wh), [4 * H, H], 1),
                           g.T(g.dev(b), [4 * H], 1), g.T(g.dev(mx)) if mask else None, g.T(g.dev(mh)) if mask else None,
                           capi.LstmGatesAttrs(1 if mask else 0, 0.0, 1.0), g.T(og), g.T(oc), g.T(oh))
    for name, got, ref in (("gates", og, gates), ("c", oc, c_t), ("h", oh, h_t)):
        assert_close(g.host(got), ref, TOL_REDUCE, floor=0.1, what=name)
    assert g.ctx().device_errors() == 0
