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


@pytest.mark.parametrize("H,B,mask", [(1024, 1, False), (40, 3, True), (301, 8, False), (512, 20, True)])
def test_thin_lstm_step_in_place(g, H, B, mask):
    """h_t on h_tm1 and c_t on c_tm1, and h_t on x (a layer over the one below): the values of separate buffers."""
    import torch
    from dynet_b200 import capi
    gen = torch.Generator("cuda").manual_seed(H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen) * 0.3   # noqa: E731
    x, h, c, Wx, Wh, b = rnd(B, H), rnd(B, H), rnd(B, H), rnd(H, 4 * H) * 0.1, rnd(H, 4 * H) * 0.1, rnd(4 * H)
    masks = [(torch.rand(B, H, device="cuda", generator=gen) < 0.8).float() for _ in range(2)]
    mx, mh = (g.T(masks[0]), g.T(masks[1])) if mask else (None, None)
    at, W = capi.LstmGatesAttrs(1 if mask else 0, 0.0, 1.0), (g.T(Wx, [4 * H, H], 1), g.T(Wh, [4 * H, H], 1), g.T(b, [4 * H], 1))

    def steps(n, onto):
        hs, cs, xs, gates = h.clone(), c.clone(), x.clone(), torch.empty(B, 4 * H, device="cuda")
        for _ in range(n):
            ho, co = (hs, cs) if onto == "state" else (xs, torch.empty_like(c)) if onto == "x" else (torch.empty_like(h), torch.empty_like(c))
            g.ctx().lstm_fwd_fused(g.T(xs), g.T(hs), g.T(cs), *W, mx, mh, at, g.T(gates), g.T(co), g.T(ho))
            hs, cs = ho.clone() if onto == "x" else ho, co
            xs = x.clone()
            torch.cuda.synchronize()
        return hs, cs
    want = steps(5, None)
    for onto in ("state", "x"):
        for got, ref in zip(steps(5, onto), want):
            assert torch.equal(got, ref), onto
    assert g.ctx().device_errors() == 0


@pytest.mark.parametrize("H,B", [(512, 3), (1024, 16), (256, 5), (300, 200)])
def test_sequence_from_a_state_on_its_own_outputs(g, H, B):
    """h0 and c0 on the first step's h and c, or on the last step's (a text read piece by piece into the same buffers)."""
    import torch
    from dynet_b200 import capi
    T, I = 9, 24
    gen = torch.Generator("cuda").manual_seed(H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen) * 0.3   # noqa: E731
    x, h0, c0, Wx, Wh, b = rnd(T * B, I), rnd(B, H), rnd(B, H), rnd(I, 4 * H) * 0.1, rnd(H, 4 * H) * 0.1, rnd(4 * H)
    at, W = capi.LstmGatesAttrs(0, 0.0, 1.0), (g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), g.T(b, [4 * H], 1))
    out = []
    for at_step in (None, 0, T - 1):
        gates, cs, hs = (torch.zeros(T * B, n, device="cuda") for n in (4 * H, H, H))
        hi, ci = (h0, c0) if at_step is None else (hs[at_step * B:(at_step + 1) * B].copy_(h0), cs[at_step * B:(at_step + 1) * B].copy_(c0))
        g.ctx().lstm_seq_fwd(g.T(x, [I], T * B), g.T(hi), g.T(ci), *W, None, None, at, g.T(gates, [4 * H], T * B), g.T(cs, [H], T * B),
                             g.T(hs, [H], T * B), None, T)
        torch.cuda.synchronize()
        out.append((gates, cs, hs))
    for o in out[1:]:
        assert all(torch.equal(p, q) for p, q in zip(o, out[0]))
    assert g.ctx().device_errors() == 0


@pytest.mark.parametrize("n,cols", [(512, 17), (64, 2000)])
def test_product_onto_its_own_operand(g, n, cols):
    """C on B (both paths that read B as it lies give such a product back to the one that splits it first)."""
    import torch
    A, B = torch.randn(n, n, device="cuda"), torch.randn(cols, n, device="cuda")
    want = B.double() @ A.double()
    reps = []
    for _ in range(3):
        C = B.clone()
        g.ctx().gemm(0, 0, n, cols, n, A.data_ptr(), n, C.data_ptr(), n, C.data_ptr(), n, 0)
        torch.cuda.synchronize()
        reps.append(C)
    assert all(torch.equal(r, reps[0]) for r in reps)
    assert float((reps[0].double() - want).abs().max()) <= TOL_REDUCE * n ** 0.5


@pytest.mark.parametrize("M,K", [(4, 3), (1184, 257), (1188, 513), (4736, 65), (4740, 301), (18944, 41), (18948, 67), (49996, 33), (100000, 20)])
@pytest.mark.parametrize("N", [1, 3, 4])
def test_thin_row_shares(g, M, K, N):
    """Plain products of up to four columns at the edges of the row shares (2, 4, 8, 9, 32 quads of rows per CTA on 148 SMs, then rounds of
    smaller CTAs), reductions shorter than the k lanes."""
    import torch
    gen = torch.Generator("cuda").manual_seed(M + N)
    A, B, C = torch.randn(K, M, device="cuda", generator=gen), torch.randn(N, K, device="cuda", generator=gen), torch.randn(N, M, device="cuda", generator=gen)
    want = B.double() @ A.double()
    for accumulate in (0, 1):
        C0 = C.double() if accumulate else 0.0
        got = C.clone()
        g.ctx().gemm(0, 0, M, N, K, A.data_ptr(), M, B.data_ptr(), K, got.data_ptr(), M, accumulate)
        # an fp32 sum of K products, each rounded at the size of the partial sum: below K 2^-24 of |row| |column|, and the last rounding
        bar = (K + 2) * 2.0 ** -24 * (B.double().norm(dim=1)[:, None] * A.double().norm(dim=0)[None, :] + (C.double().abs() if accumulate else 0.0))
        assert bool(((got.double() - want - C0).abs() <= bar).all())
    assert g.ctx().device_errors() == 0
