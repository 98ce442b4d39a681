"""dyb200_ctx_cluster_splitk changes the form of a K split and not its bits: the deferred weight gradients of both operands in one launch
(csrc/gemm_tc.cu, dyb200_tc_gemm_packed2 - splits as clusters, as work items, none at all - and on fp16 pairs) and the recurrence of wide
layers (csrc/lstm_seq.cu, F16), as a sequence and step by step."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N0,N1,k", [(1024, 128, 256, 520), (1024, 128, 256, 320), (512, 64, 64, 3000), (1024, 128, 256, 40000), (1000, 129, 127, 1601),
                                       (2816, 704, 704, 35), (2048, 1100, 1024, 640)])
def test_grouped_weight_gradients(M, N0, N1, k):
    import torch
    import gpu_util as g
    ctx = g.ctx()
    w = ctx.wgrad_create(M, N0, N1, k)
    a, b0, b1 = (torch.randn(k, n, device="cuda") for n in (M, N0, N1))
    out = []
    try:
        for on in (1, 0):
            ctx.cluster_splitk(on)
            C0, C1 = torch.ones(N0, M, device="cuda"), torch.ones(N1, M, device="cuda")
            ctx.wgrad_push(w, k, a.data_ptr(), M, b0.data_ptr(), N0, None, 0, b1.data_ptr(), N1, None, 0)
            ctx.wgrad_flush(w, C0.data_ptr(), M, C1.data_ptr(), M)
            out.append((C0, C1))
    finally:
        ctx.cluster_splitk(1)
        ctx.wgrad_destroy(w)
    assert torch.equal(out[0][0], out[1][0]) and torch.equal(out[0][1], out[1][1])
    assert ctx.device_errors() == 0


@pytest.mark.parametrize("I,H,B,T", [(1024, 1024, 64, 3), (1024, 1024, 128, 3), (512, 512, 64, 2), (1536, 512, 64, 2)])
def test_wide_recurrence(I, H, B, T):
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    gen = torch.Generator("cuda").manual_seed(H + B)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    x, h0, c0, b = rnd(T * B, I), rnd(B, H) * 0.3, rnd(B, H), rnd(4 * H) * 0.1
    Wx, Wh = rnd(I, 4 * H) / I ** 0.5, rnd(H, 4 * H) / H ** 0.5
    W, at = (g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), g.T(b, [4 * H], 1)), capi.LstmGatesAttrs(0, 0.0, 1.0)
    out = []
    try:
        for on, single in ((1, 0), (0, 0), (0, 1)):
            ctx.cluster_splitk(on)
            w = ctx.wgrad_create(4 * H, I, H, T * B)
            gates, cs, hs = (torch.empty(T * B, n, device="cuda") for n in (4 * H, H, H))
            if single:
                for t in range(T):
                    sl, pr = slice(t * B, (t + 1) * B), slice((t - 1) * B, t * B)
                    ctx.lstm_fwd_fused_at(g.T(x[sl]), g.T(hs[pr] if t else h0), g.T(cs[pr] if t else c0), *W, None, None, at, g.T(gates[sl]), g.T(cs[sl]), g.T(hs[sl]), w, t * B)
            else:
                ctx.lstm_seq_fwd(g.T(x, [I], T * B), g.T(h0), g.T(c0), *W, None, None, at, g.T(gates, [4 * H], T * B), g.T(cs, [H], T * B), g.T(hs, [H], T * B), w, T)
            torch.cuda.synchronize()
            ctx.wgrad_destroy(w)
            out.append((gates, cs, hs))
    finally:
        ctx.cluster_splitk(1)
    for o in out[1:]:
        assert all(torch.equal(p, q) for p, q in zip(out[0], o))
    assert ctx.device_errors() == 0
