"""The forward recurrence of wide layers (csrc/lstm_seq.cu, F16) where units and columns do not fill its tiles: batches below and beside whole 64 columns on
64- and 128-column tiles, units that are no multiple of 32 (the last tile of 32 units partly there), inputs of any number of rows, K splits, masks, and calls
without an accumulator, whose inputs are split from x itself.  Step by step against float64 from the device's own h_{t-1} and c_{t-1}; bars as in
test_gpu_lstm_seq_f16.py.  Where the single-step call takes this form too (from 33 columns on, with an accumulator) it must give the same bits."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("I,H,B,T,mask,acc", [
    (300, 600, 30, 8, "full", True),        # 19 tiles of units, the last of 24; one block, 30 columns
    (512, 1000, 100, 8, "one", True),       # the last block has 36 columns
    (7, 388, 9, 9, None, True),             # the smallest of its range; a tile of four units
    (130, 516, 500, 3, "full", True),       # 128-column tiles, the last of 116
    (512, 768, 300, 3, None, True),
    (33, 1020, 65, 3, "full", True),        # a block of one column
    (512, 1024, 64, 8, None, False),
    (128, 412, 17, 8, None, False),
    (300, 777, 100, 8, "full", True),       # units not in fours: a value at a time
    (31, 386, 12, 8, "one", True),
    (64, 1023, 500, 3, None, True),         # ... on 128-column tiles
    (128, 433, 40, 8, None, False),
    (1100, 641, 64, 8, "full", True),       # weights in two passes (more lines than a strip holds)
    (300, 777, 33, 8, "full", True),        # steps of the stacked states start on any four bytes
    (31, 385, 37, 5, "one", True),
    (64, 1022, 131, 3, None, True),         # (on eight)
])
def test_sequence_that_does_not_fill_its_tiles(I, H, B, T, mask, acc):
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    bn, S = C.c_uint32(), C.c_uint32()
    assert ctx.L.dyb200i_seq_f16_tiling(ctx.h, I, H, B, C.byref(bn), C.byref(S)) == 1
    gen = torch.Generator("cuda").manual_seed(H + B)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    x, h0, c0, b = rnd(T * B, I), rnd(B, H) * 3.0, rnd(B, H), rnd(4 * H) * 0.1
    x *= torch.exp2(torch.randint(-40, 3, (T * B, 1), device="cuda", generator=gen).float())
    Wx, Wh = rnd(I, 4 * H) / I ** 0.5, rnd(H, 4 * H) / H ** 0.5
    mB = B if mask == "full" else 1
    mx, mh = [((torch.rand(mB, n, device="cuda", generator=gen) < 0.8) / 0.8).float() if mask else torch.ones(1, n, device="cuda") for n in (I, H)]
    at, tm = capi.LstmGatesAttrs(1 if mask else 0, 0.0, 1.0), (g.T(mx), g.T(mh)) if mask else (None, None)
    W = (g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), g.T(b, [4 * H], 1))
    out, launches = [], []
    for single in (False, True) if acc and B > 32 else (False,):
        w = ctx.wgrad_create(4 * H, I, H, T * B) if acc else None
        gates, cs, hs = (torch.full((T * B + 1, n), 7.0, device="cuda") for n in (4 * H, H, H))     # (a column past the end)
        at0 = ctx.launches()
        if single:
            for t in range(T):
                sl, pr = slice(t * B, (t + 1) * B), slice((t - 1) * B, t * B)
                ctx.lstm_fwd_fused_at(g.T(x[sl]), g.T(hs[pr] if t else h0), g.T(cs[pr] if t else c0), *W, *tm, at, g.T(gates[sl]), g.T(cs[sl]), g.T(hs[sl]), w, t * B)
        else:
            ctx.lstm_seq_fwd(g.T(x, [I], T * B), g.T(h0), g.T(c0), *W, *tm, at, g.T(gates[:T * B], [4 * H], T * B), g.T(cs[:T * B], [H], T * B), g.T(hs[:T * B], [H], T * B), w, T)
        launches.append(ctx.launches() - at0)
        torch.cuda.synchronize()
        if acc:
            ctx.wgrad_destroy(w)
        for o in (gates, cs, hs):
            assert bool((o[T * B] == 7.0).all())
        out.append((gates[:T * B], cs[:T * B], hs[:T * B]))
    assert launches[0] <= 6, launches                        # inputs, weights (up to three launches), pairs, the recurrence
    for p, q in zip(out[0], out[-1]):
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
        assert bool(((cs[t] - (i * gg + f * cp)).abs() <= 2e-7 * ((i * gg).abs() + (f * cp).abs())).all())
        assert bool(((hs[t] - o * torch.tanh(cs[t])).abs() <= 5e-7).all())
    assert ctx.device_errors() == 0


@pytest.mark.parametrize("I,H,B,T,mask", [(64, 400, 9, 7, None), (300, 600, 30, 5, "full"), (31, 777, 12, 2, "one"), (512, 1024, 24, 5, None)])
def test_short_sequence_of_few_columns(I, H, B, T, mask):
    """Fewer than eight steps of up to 32 columns: bit for bit the step calls - plain fp32 where those are (up to 64 M multiply-adds), the wide form in the last row."""
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    gen = torch.Generator("cuda").manual_seed(H + B)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    x, h0, c0, b = rnd(T * B, I), rnd(B, H), rnd(B, H), rnd(4 * H) * 0.1
    Wx, Wh = rnd(I, 4 * H) / I ** 0.5, rnd(H, 4 * H) / H ** 0.5
    mB = B if mask == "full" else 1
    mx, mh = [((torch.rand(mB, n, device="cuda", generator=gen) < 0.8) / 0.8).float() for n in (I, H)]
    at, tm = capi.LstmGatesAttrs(1 if mask else 0, 0.0, 1.0), (g.T(mx), g.T(mh)) if mask else (None, None)
    W, out = (g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), g.T(b, [4 * H], 1)), []
    for single in (False, True):
        w = ctx.wgrad_create(4 * H, I, H, T * B)
        gates, cs, hs = (torch.empty(T * B, n, device="cuda") for n in (4 * H, H, H))
        if single:
            ctx.wgrad_pack_inputs(w, g.T(x, [I], T * B), tm[0], B)
            for t in range(T):
                sl, pr = slice(t * B, (t + 1) * B), slice((t - 1) * B, t * B)
                ctx.lstm_fwd_fused_at(g.T(x[sl]), g.T(hs[pr] if t else h0), g.T(cs[pr] if t else c0), *W, *tm, at, g.T(gates[sl]), g.T(cs[sl]), g.T(hs[sl]), w, t * B)
        else:
            ctx.lstm_seq_fwd(g.T(x, [I], T * B), g.T(h0), g.T(c0), *W, *tm, at, g.T(gates, [4 * H], T * B), g.T(cs, [H], T * B), g.T(hs, [H], T * B), w, T)
        torch.cuda.synchronize()
        ctx.wgrad_destroy(w)
        out.append((gates, cs, hs))
    assert all(torch.equal(p, q) for p, q in zip(*out))
    assert ctx.device_errors() == 0


@pytest.mark.parametrize("I,H,B,acc", [(96, 512, 100, True), (1100, 777, 40, True), (128, 512, 64, False)])
def test_infinities_and_nans_stay_in_their_column_and_gate(I, H, B, acc):
    """In a column of x and of h0, and in a gate row of Wx and of Wh (made into pairs in one pass, or in two above 1024 inputs)."""
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx, T = g.ctx(), 8
    gen = torch.Generator("cuda").manual_seed(H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    x, h0, c0, b, Wx, Wh = rnd(T * B, I), rnd(B, H), rnd(B, H), rnd(4 * H) * 0.1, rnd(I, 4 * H) / I ** 0.5, rnd(H, 4 * H) / H ** 0.5

    def run(x, h0, Wx, Wh):
        w = ctx.wgrad_create(4 * H, I, H, T * B) if acc else None
        out = [torch.empty(T * B, n, device="cuda") for n in (4 * H, H, H)]
        ctx.lstm_seq_fwd(g.T(x, [I], T * B), g.T(h0), g.T(c0), g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), g.T(b, [4 * H], 1), None, None, capi.LstmGatesAttrs(0, 0.0, 1.0),
                         g.T(out[0], [4 * H], T * B), g.T(out[1], [H], T * B), g.T(out[2], [H], T * B), w, T)
        torch.cuda.synchronize()
        if acc:
            ctx.wgrad_destroy(w)
        assert ctx.device_errors() == 0
        return [o.view(T, B, -1) for o in out]

    clean = run(x, h0, Wx, Wh)
    x2, h2 = x.clone(), h0.clone()
    x2[2 * B + 3, I - 1], h2[39, 0] = float("inf"), float("nan")
    got = run(x2, h2, Wx, Wh)
    hit = torch.zeros(T, B, dtype=torch.bool, device="cuda")
    hit[2:, 3] = hit[:, 39] = True
    for p, q in zip(got, clean):
        assert torch.equal(p[~hit], q[~hit])
    assert bool(torch.isnan(got[0][hit]).all())
    Wx2, Wh2 = Wx.clone(), Wh.clone()
    Wx2[5, H + 7], Wh2[H - 1, 4 * H - 1] = float("nan"), float("inf")    # a forget gate, the last unit's candidate
    got = run(x, h0, Wx2, Wh2)
    rest = [r for r in range(4 * H) if r not in (H + 7, 4 * H - 1)]
    assert torch.equal(got[0][0][:, rest], clean[0][0][:, rest]) and bool(torch.isnan(got[0][0][:, H + 7]).all()) and not bool(torch.equal(got[0][0][:, -1], clean[0][0][:, -1]))
