"""The forward recurrence of wide layers on fp16 pairs (csrc/lstm_seq.cu, F16): reductions that are no multiple of a k-block or longer than a
chain, K splits with even, short and empty last shares, 64- and 128-column tiles, masks per column and for all, an initial state far above 1, columns of x that differ
by 2^60 and a column of zeros, the slots of h in turn.  Step by step against float64 from the device's own h_{t-1} and c_{t-1}.  Bar of a
pre-activation: 4.5e-7 of |row of Wx| |x| + |row of Wh| |h .* mask|, that of every product on fp16 pairs; of a gate: that (its slope is at
most 1) and 3e-6 for the approximate exponential and reciprocal.  The single-step calls must give the same bits, also where
saturated gates leave elements of h far below 2^-28."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


# splits: of the rule on 148 SMs, and where the number of clusters that fit differs between GPUs both
@pytest.mark.parametrize("I,H,B,T,mask,tile,splits", [
    (300, 544, 64, 4, "full", 64, (2,)),       # tails in both reductions
    (1100, 1056, 64, 3, None, 64, (4,)),       # chains cut within both products, lines longer than a warp holds
    (4, 512, 192, 3, "one", 64, (2,)),         # the shortest x, three column blocks
    (512, 1024, 256, 2, "full", 64, (1,)),
    (36, 1024, 512, 3, "one", 128, (1,)),
    (1024, 2048, 128, 2, None, 64, (1,)),      # a reduction of 48 k-blocks
    (1536, 512, 64, 3, "full", 64, (8, 4)),
    (576, 576, 64, 3, None, 64, (4,)),         # 9 + 9 k-blocks: the last share is empty
    (576, 576, 128, 3, "one", 64, (2, 4)),     # (thirty-six clusters of four are more than most GPUs hold)
    (640, 576, 64, 2, "full", 64, (4,)),       # ... or has one
])
def test_sequence_of_a_wide_layer(I, H, B, T, mask, tile, splits):
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    bn, S = C.c_uint32(), C.c_uint32()
    assert ctx.L.dyb200i_seq_f16_tiling(ctx.h, I, H, B, C.byref(bn), C.byref(S)) == 1
    assert bn.value == tile and S.value in splits, (bn.value, S.value)
    gen = torch.Generator("cuda").manual_seed(H + B)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    x, h0, c0, b = rnd(T * B, I), rnd(B, H) * 30.0, rnd(B, H), rnd(4 * H) * 0.1
    x *= torch.exp2(torch.randint(-60, 3, (T * B, 1), device="cuda", generator=gen).float())
    x[5] = 0.0
    Wx, Wh = rnd(I, 4 * H) / I ** 0.5, rnd(H, 4 * H) / H ** 0.5
    mB = B if mask == "full" else 1
    mx, mh = [((torch.rand(mB, n, device="cuda", generator=gen) < 0.8) / 0.8).float() if mask else torch.ones(1, n, device="cuda") for n in (I, H)]
    at, tm = capi.LstmGatesAttrs(1 if mask else 0, 0.0, 1.0), (g.T(mx), g.T(mh)) if mask else (None, None)
    W = (g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), g.T(b, [4 * H], 1))
    out = []
    for single in (False, True):
        w = ctx.wgrad_create(4 * H, I, H, T * B)
        gates, cs, hs = (torch.full((T * B, n), 7.0, device="cuda") for n in (4 * H, H, H))
        if single:
            for t in range(T):
                sl, pr = slice(t * B, (t + 1) * B), slice((t - 1) * B, t * B)
                ctx.lstm_fwd_fused_at(g.T(x[sl]), g.T(hs[pr] if t else h0), g.T(cs[pr] if t else c0), *W, *tm, at, g.T(gates[sl]), g.T(cs[sl]), g.T(hs[sl]), w, t * B)
        else:
            ctx.lstm_seq_fwd(g.T(x, [I], T * B), g.T(h0), g.T(c0), *W, *tm, at, g.T(gates, [4 * H], T * B), g.T(cs, [H], T * B), g.T(hs, [H], T * B), w, T)
        torch.cuda.synchronize()
        ctx.wgrad_destroy(w)
        out.append((gates, cs, hs))
    for p, q in zip(*out):
        assert torch.equal(p, q)
    gates, cs, hs = (o.double().view(T, B, -1) for o in out[0])
    for t in range(T):
        xt, hp, cp = x.double().view(T, B, I)[t] * mx.double(), (hs[t - 1] if t else h0.double()) * mh.double(), cs[t - 1] if t else c0.double()
        pre = xt @ Wx.double() + hp @ Wh.double() + b.double()
        bar = 4.5e-7 * (xt.norm(dim=1)[:, None] * Wx.double().norm(dim=0) + hp.norm(dim=1)[:, None] * Wh.double().norm(dim=0)) + 3e-6
        pre[:, H:2 * H] += 1.0
        want = torch.cat([torch.sigmoid(pre[:, :3 * H]), torch.tanh(pre[:, 3 * H:])], dim=1)
        assert bool(((gates[t] - want).abs() <= bar).all()), "step %d: %.3g" % (t, float(((gates[t] - want).abs() / bar).max()))
        i, f, o, gg = gates[t].split(H, dim=1)
        c = i * gg + f * cp
        assert bool(((cs[t] - c).abs() <= 2e-7 * ((i * gg).abs() + (f * cp).abs())).all())
        assert bool(((hs[t] - o * torch.tanh(cs[t])).abs() <= 5e-7).all())
    assert ctx.device_errors() == 0


@pytest.mark.parametrize("e", [20, 45, 112, -112])
@pytest.mark.parametrize("single", [False, True])
def test_weights_and_inputs_of_other_magnitudes(e, single):
    """Wx 2^e times larger and x as much smaller: Wh and h keep their bits beside them, and no factor leaves fp32's range on the way.  Bar as above."""
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    I, H, B = 512, 512, 64
    gen = torch.Generator("cuda").manual_seed(1)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    x, h0, c0, b = rnd(2 * B, I) * 2.0 ** -e, rnd(B, H) * 0.3, rnd(B, H), rnd(4 * H) * 0.1
    Wx, Wh = rnd(I, 4 * H) / I ** 0.5 * 2.0 ** e, rnd(H, 4 * H) / H ** 0.5
    W, at = (g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), g.T(b, [4 * H], 1)), capi.LstmGatesAttrs(0, 0.0, 1.0)
    gates, cs, hs = (torch.empty(2 * B, n, device="cuda") for n in (4 * H, H, H))
    w = ctx.wgrad_create(4 * H, I, H, 2 * B)
    if single:
        ctx.lstm_fwd_fused_at(g.T(x[:B]), g.T(h0), g.T(c0), *W, None, None, at, g.T(gates[:B]), g.T(cs[:B]), g.T(hs[:B]), w, 0)
    else:
        ctx.lstm_seq_fwd(g.T(x, [I], 2 * B), g.T(h0), g.T(c0), *W, None, None, at, g.T(gates, [4 * H], 2 * B), g.T(cs, [H], 2 * B), g.T(hs, [H], 2 * B), w, 2)
    torch.cuda.synchronize()
    ctx.wgrad_destroy(w)
    xd, hd = x[:B].double(), h0.double()
    pre = xd @ Wx.double() + hd @ Wh.double() + b.double()
    bar = 4.5e-7 * (xd.norm(dim=1)[:, None] * Wx.double().norm(dim=0) + hd.norm(dim=1)[:, None] * Wh.double().norm(dim=0)) + 3e-6
    pre[:, H:2 * H] += 1.0
    want = torch.cat([torch.sigmoid(pre[:, :3 * H]), torch.tanh(pre[:, 3 * H:])], dim=1)
    assert bool(((gates[:B].double() - want).abs() <= bar).all())
    assert ctx.device_errors() == 0
