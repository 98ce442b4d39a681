"""The backward pass of wide layers on fp16 pairs (csrc/lstm_bwd_wide.cu): units that are no multiple of a k-block or of a tile, batches that are no
multiple of a column tile, one to four column blocks per CTA, K splits with even, short and empty last shares, an input of one row, masks per column and for
all, columns whose gradients differ by 2^60, a column of zeros.  Step by step against float64 from the device's own dE/dh_t and dE/dc_t.  Bar of a
product: 4.5e-7 of |row| |dgates column|, that of every product on fp16 pairs; dgates themselves are a handful of fp32 operations and a tanhf:
1e-6 of their column, which the product passes on as that much of |row| |column|.  The single-step calls must give the same bits."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu


# blocks: column blocks of 64 per CTA; both of the rule on 148 SMs, where 15 clusters of eight fit, 33 of four, 74 of two
@pytest.mark.parametrize("I,H,B,T,mask,blocks,splits", [
    (512, 1024, 64, 4, "full", 1, 8),
    (1024, 1024, 512, 3, "full", 2, 4),
    (96, 1024, 128, 3, None, 1, 4),
    (256, 1024, 256, 3, "one", 1, 4),
    (512, 512, 64, 3, None, 1, 8),
    (1, 392, 9, 4, "one", 1, 8),           # 28 k-blocks: the last share is empty; the last block of units has eight
    (33, 448, 100, 3, "full", 1, 8),       # ... 64
    (300, 744, 33, 3, "full", 1, 8),       # ... 104: its second half is partly filled
    (130, 904, 300, 3, None, 2, 4),        # five column blocks: the last CTAs have one
    (130, 904, 300, 34, None, 2, 4),       # more steps than the sums of the bias gradient take side by side, 20 tiles each
    (200, 576, 500, 2, "full", 1, 2),
    (64, 2048, 500, 2, "one", 2, 2),
    (40, 2048, 1000, 2, None, 2, 1),
    (8, 3072, 1000, 2, None, 4, 1),
    (388, 388, 70, 3, "one", 1, 8),        # units in fours, not in eights: the gates of the weights' pairs moved apart
    (512, 777, 100, 3, "full", 1, 8),      # in neither: a value at a time
    (30, 514, 64, 3, None, 1, 8),
    (64, 1022, 500, 2, "one", 2, 4),
    (9, 2049, 500, 2, None, 2, 2),
    (9, 2047, 1000, 2, "full", 2, 1),
    (512, 777, 33, 4, "full", 1, 8),       # ... and steps of the stacked states start on any four bytes
    (9, 385, 37, 5, "one", 1, 8),
    (64, 1022, 131, 3, None, 1, 4),        # (on eight)
])
def test_backward_of_a_wide_layer(I, H, B, T, mask, blocks, splits):
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    ncb, S = C.c_uint32(), C.c_uint32()
    assert ctx.L.dyb200i_bwd_wide_tiling(ctx.h, H, B, C.byref(ncb), C.byref(S)) == 1
    assert (ncb.value, S.value) == (blocks, splits)
    gen = torch.Generator("cuda").manual_seed(H + B)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    Wx, Wh = rnd(I, 4 * H) / H ** 0.5, rnd(H, 4 * H) / H ** 0.5
    gates = torch.cat([torch.sigmoid(rnd(T * B, 3 * H)), torch.tanh(rnd(T * B, H))], dim=1)
    cs, c0, x, h0 = rnd(T * B, H), rnd(B, H), rnd(T * B, I), rnd(B, H)
    dh_in, dc_in, dx_in, db_in = rnd(T * B, H), rnd(T * B, H), rnd(T * B, I), rnd(4 * H)
    mag = torch.exp2(torch.randint(-60, 3, (B, 1), device="cuda", generator=gen).float()).repeat(T, 1)
    mag[5::B] = 0.0
    dh_in, dc_in, dx_in = dh_in * mag, dc_in * mag, dx_in * mag
    mB = B if mask == "full" else 1
    mx, mh = [((torch.rand(mB, n, device="cuda", generator=gen) < 0.8) / 0.8).float() if mask else torch.ones(1, n, device="cuda") for n in (I, H)]
    at, tm = capi.LstmGatesAttrs(1 if mask else 0, 0.0, 1.0), (g.T(mx), g.T(mh)) if mask else (None, None)
    W = (g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1))
    outs = []
    for single in (False, True):
        w = ctx.wgrad_create(4 * H, I, H, T * B)
        dh, dc, dx, db = dh_in.clone(), dc_in.clone(), dx_in.clone(), db_in.clone()
        ctx.wgrad_pack_inputs(w, g.T(x, [I], T * B), tm[0], B)
        if single:
            for t in range(T - 1, -1, -1):
                sl, pr = slice(t * B, (t + 1) * B), slice((t - 1) * B, t * B)
                ctx.lstm_bwd_fused_at(g.T(x[sl]), g.T(h0), g.T(cs[pr] if t else c0), *W, *tm, g.T(gates[sl]), g.T(cs[sl]), g.T(dh[sl]), g.T(dc[sl]), g.T(dx[sl]),
                                      g.T(dh[pr]) if t else None, g.T(dc[pr]) if t else None, None, None, g.T(db, [4 * H], 1), at, w, t * B)
        else:
            ctx.lstm_seq_bwd(g.T(x, [I], T * B), g.T(h0), g.T(c0), *W, *tm, at, g.T(gates, [4 * H], T * B), g.T(cs, [H], T * B), g.T(cs, [H], T * B),
                             g.T(dh, [H], T * B), g.T(dc, [H], T * B), g.T(dx, [I], T * B), None, None, g.T(db, [4 * H], 1), w, T)
        torch.cuda.synchronize()
        ctx.wgrad_destroy(w)
        outs.append((dh, dc, dx, db))
    assert ctx.device_errors() == 0
    for p, q in zip(*outs):
        assert torch.equal(p, q)
    dh, dc, dx, db = (o.double() for o in outs[0])
    db_want, db_bar = db_in.double(), torch.zeros(4 * H, device="cuda", dtype=torch.float64)
    for t in range(T - 1, -1, -1):
        sl, pr = slice(t * B, (t + 1) * B), slice((t - 1) * B, t * B)
        i, f, o, gg = gates[sl].double().split(H, dim=1)
        c, cp = cs[sl].double(), (cs[pr] if t else c0).double()
        tc = torch.tanh(c)
        d = dh[sl] * o * (1 - tc * tc) + dc[sl]
        dg = torch.cat([d * gg * i * (1 - i), d * cp * f * (1 - f), dh[sl] * tc * o * (1 - o), d * i * (1 - gg * gg)], dim=1)
        db_want += dg.sum(dim=0)
        db_bar += 2e-6 * dg.norm(dim=0) * B ** 0.5 + 1e-6 * db_want.abs()
        col = dg.norm(dim=1)[:, None]
        want = dx_in[sl].double() + mx.double() * (dg @ Wx.double().t())
        bar = 1.45e-6 * 1.25 * col * Wx.double().norm(dim=1)[None, :] + 1.3e-7 * want.abs() + 1e-44
        assert bool(((dx[sl] - want).abs() <= bar).all()), "dx %d: %.3g" % (t, float(((dx[sl] - want).abs() / bar).max()))
        if t:
            want = dh_in[pr].double() + mh.double() * (dg @ Wh.double().t())
            bar = 1.45e-6 * 1.25 * col * Wh.double().norm(dim=1)[None, :] + 1.3e-7 * want.abs() + 1e-44
            assert bool(((dh[pr] - want).abs() <= bar).all()), "dh %d: %.3g" % (t - 1, float(((dh[pr] - want).abs() / bar).max()))
            want = dc_in[pr].double() + d * f
            assert bool(((dc[pr] - want).abs() <= 1e-6 * (dc_in[pr].double().abs() + (d * f).abs() + (dh[sl] * o * f).abs()) + 1e-44).all()), "dc %d" % (t - 1)
    assert bool(((db - db_want).abs() <= db_bar).all()), float(((db - db_want).abs() / db_bar).max())


@pytest.mark.parametrize("H,B", [(512, 256), (513, 255)])
def test_sequence_without_room_for_its_pairs(H, B):
    """Little device memory: the pairs of all steps (134 MB and more) do not fit, those of one (2 MB) do - the single-step calls run, with the same bits."""
    import contextlib
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    from test_gpu_scratch_limits import room_for
    I, T = 64, 64
    rnd = lambda *s: torch.randn(*s, device="cuda")   # noqa: E731
    x, c0, cs, gates = rnd(T * B, I), rnd(B, H), rnd(T * B, H), torch.sigmoid(rnd(T * B, 4 * H))
    Wx, Wh, dh_in = rnd(I, 4 * H) / H ** 0.5, rnd(H, 4 * H) / H ** 0.5, rnd(T * B, H)
    w = g.ctx().wgrad_create(4 * H, I, H, T * B)
    outs = [[dh_in.clone(), torch.zeros(T * B, H, device="cuda"), torch.zeros(T * B, I, device="cuda"), torch.zeros(4 * H, device="cuda")] for _ in range(2)]
    try:
        for c, (dh, dc, dx, db) in zip((g.ctx(), None), outs):
            with contextlib.nullcontext(c) if c else room_for(48) as ctx:
                ctx.lstm_seq_bwd(g.T(x, [I], T * B), g.T(c0), g.T(c0), g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), None, None, capi.LstmGatesAttrs(0, 0.0, 1.0),
                                 g.T(gates, [4 * H], T * B), g.T(cs, [H], T * B), g.T(cs, [H], T * B), g.T(dh, [H], T * B), g.T(dc, [H], T * B), g.T(dx, [I], T * B),
                                 None, None, g.T(db, [4 * H], 1), w, T)
        torch.cuda.synchronize()
        assert all(torch.equal(p, q) for p, q in zip(*outs))
    finally:
        g.ctx().wgrad_destroy(w)


@pytest.mark.parametrize("I,H,B", [(96, 1024, 64), (33, 448, 100), (9, 777, 500)])
def test_single_step_waits_for_no_other_cluster(I, H, B):
    """A single step's cell pass and the product behind it are launches of their own - one more than where the product is not wanted - so that no CTA waits for
    one beside those of its cluster; the switch for the sequence kernels changes neither that nor the bits."""
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    gen = torch.Generator("cuda").manual_seed(H + B)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    x, c0, cs, gates = rnd(B, I), rnd(B, H), rnd(B, H), torch.sigmoid(rnd(B, 4 * H))
    Wx, Wh, dh, dc, db0 = rnd(I, 4 * H) / H ** 0.5, rnd(H, 4 * H) / H ** 0.5, rnd(B, H), rnd(B, H), rnd(4 * H)
    W, at = (g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1)), capi.LstmGatesAttrs(0, 0.0, 1.0)
    outs = []

    def step(prev):
        w = ctx.wgrad_create(4 * H, I, H, B)
        ctx.wgrad_pack_inputs(w, g.T(x), None, B)
        out = [torch.ones(B, n, device="cuda") for n in (I, H, H)] + [db0.clone()]
        at0 = ctx.launches()
        ctx.lstm_bwd_fused_at(g.T(x), g.T(c0), g.T(c0), *W, None, None, g.T(gates), g.T(cs), g.T(dh), g.T(dc), g.T(out[0]), g.T(out[1]) if prev else None, g.T(out[2]),
                              None, None, g.T(out[3], [4 * H], 1), at, w, 0)
        n = ctx.launches() - at0
        torch.cuda.synchronize()
        ctx.wgrad_destroy(w)
        return n, out

    ctx.param_cache(True)
    try:
        step(True)
        for mode in (1, 2, 0):
            ctx.sequence_kernels(mode)
            with_product, out = step(True)
            outs.append(out)
            assert with_product == step(False)[0] + 1
    finally:
        ctx.sequence_kernels(1)
        ctx.param_cache(False)
    for out in outs[1:]:
        assert all(torch.equal(p, q) for p, q in zip(outs[0], out))
    assert ctx.device_errors() == 0


@pytest.mark.parametrize("append", [False, True])
def test_single_step_without_room_for_its_pairs(append):
    """Little device memory: a step's pairs (11 MB: 1000 columns of dgates, the weights) do not fit, the planes of the weights that the generic form needs (7 MB)
    do - it runs, with the same values to the rounding of either form (2 x 11 bits, sums of 1792: 2e-6 each of a result's norm), and the accumulator holds the
    step once."""
    import contextlib
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    from test_gpu_scratch_limits import room_for
    I, H, B = 32, 448, 1000
    gen = torch.Generator("cuda").manual_seed(H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    x, c0, cs, gates = rnd(B, I), rnd(B, H), rnd(B, H), torch.sigmoid(rnd(B, 4 * H))
    Wx, Wh, dh, dc = rnd(I, 4 * H) / H ** 0.5, rnd(H, 4 * H) / H ** 0.5, rnd(B, H), rnd(B, H)
    outs = []
    spare = [torch.zeros(n, device="cuda") for n in (I * B, H * B, H * B, 4 * H * I, 4 * H * H, 4 * H)]   # (the generic form once with all the memory: its kernels are loaded)
    g.ctx().lstm_bwd_fused(g.T(x), g.T(c0), g.T(c0), g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), None, None, g.T(gates), g.T(cs), g.T(dh), g.T(dc),
                           *(g.T(t, [n], B) for t, n in zip(spare, (I, H, H))), g.T(spare[3], [4 * H, I], 1), g.T(spare[4], [4 * H, H], 1), g.T(spare[5], [4 * H], 1),
                           capi.LstmGatesAttrs(0, 0.0, 1.0))
    for c in (g.ctx(), None):
        out = [torch.ones(B, n, device="cuda") for n in (I, H, H)] + [torch.zeros(n, 4 * H, device="cuda") for n in (1, I, H)]
        w = g.ctx().wgrad_create(4 * H, I, H, B)
        if not append:
            g.ctx().wgrad_pack_inputs(w, g.T(x), None, B)
        with contextlib.nullcontext(c) if c else room_for(11) as ctx:
            ctx.lstm_bwd_fused_at(g.T(x), g.T(c0), g.T(c0), g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), None, None, g.T(gates), g.T(cs), g.T(dh), g.T(dc),
                                  g.T(out[0]), g.T(out[1]), g.T(out[2]), None, None, g.T(out[3], [4 * H], 1), capi.LstmGatesAttrs(0, 0.0, 1.0), w,
                                  ctx.WGRAD_APPEND if append else 0)
        torch.cuda.synchronize()
        if append:
            g.ctx().wgrad_flush(w, out[4].data_ptr(), 4 * H, out[5].data_ptr(), 4 * H)
        torch.cuda.synchronize()
        g.ctx().wgrad_destroy(w)
        outs.append(out)
    for p, q in zip(*outs):
        assert bool((p - q).double().norm() <= 4e-6 * p.double().norm())
    assert not append or float(outs[0][5].abs().max()) > 1.0


def _sweep(I, H, B, T, Wx, Wh, gates, cs, c0, dh_in, dc_in):
    """The sequence call on copies of its gradients: dh, dc of all steps, dx, db."""
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    w = ctx.wgrad_create(4 * H, I, H, T * B)
    dh, dc, dx, db = dh_in.clone(), dc_in.clone(), torch.zeros(T * B, I, device="cuda"), torch.zeros(4 * H, device="cuda")
    x = torch.ones(T * B, I, device="cuda")
    ctx.wgrad_pack_inputs(w, g.T(x, [I], T * B), None, B)
    ctx.lstm_seq_bwd(g.T(x, [I], T * B), g.T(c0), g.T(c0), g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), None, None, capi.LstmGatesAttrs(0, 0.0, 1.0),
                     g.T(gates, [4 * H], T * B), g.T(cs, [H], T * B), g.T(cs, [H], T * B), g.T(dh, [H], T * B), g.T(dc, [H], T * B), g.T(dx, [I], T * B),
                     None, None, g.T(db, [4 * H], 1), w, T)
    torch.cuda.synchronize()
    ctx.wgrad_destroy(w)
    assert ctx.device_errors() == 0
    return dh, dc, dx, db


def _dgates(gates, c, cp, dh, dc, H):
    import torch
    i, f, o, gg = gates.double().split(H, dim=1)
    tc = torch.tanh(c.double())
    d = dh.double() * o * (1 - tc * tc) + dc.double()
    return torch.cat([d * gg * i * (1 - i), d * cp.double() * f * (1 - f), dh.double() * tc * o * (1 - o), d * i * (1 - gg * gg)], dim=1)


# A pair's scale belongs to a column and 128 units of all gates (dgates) or to a row (weights).  Every other `run` of units has gradients 2^-e below the rest; every
# third row of the weights is zero at the rest, every third 2^-e smaller there.  Bar of a result: 1.45e-6 * 1.25 (as above) of the sum of its products'
# magnitudes - never more than |row| |column|, and all that a product or a truncated sum can be off by in proportion - and 2^-22 of what the sum would be with the
# largest value of its quad (four units of a gate, four weights of a row side by side) in the place of one of the factors: a value keeps an absolute error of
# 2^-50 of its scale's largest, and a quad that lies 2^28 below that is added in fp32.  (Runs of four: quads of one magnitude, which keep their own bits.)
@pytest.mark.parametrize("I,H,B,run,e", [(*s, run, e) for s in ((96, 512, 64), (130, 1000, 130), (9, 777, 33)) for run in (1, 4) for e in (10, 20, 27, 28, 29, 30, 40, 50, 90)] +
                         [(3, 4104, 16, 4, 40), (3, 4104, 16, 4, 29)])   # (rows of weights that are made into pairs in two passes)
def test_values_that_differ_within_a_scale(I, H, B, run, e):
    import torch
    T = 2
    gen = torch.Generator("cuda").manual_seed(H + e)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    odd = torch.arange(H, device="cuda") // run % 2 == 1
    weight = [torch.ones(H, device="cuda"), odd.float(), torch.where(odd, 1.0, 2.0 ** -e)]
    Wx, Wh = [torch.stack([weight[j % 3] for j in range(n)]).repeat(1, 4) * rnd(n, 4 * H) / H ** 0.5 for n in (I, H)]
    gates = torch.cat([torch.sigmoid(rnd(T * B, 3 * H)), torch.tanh(rnd(T * B, H))], dim=1)
    cs, c0, small = rnd(T * B, H), rnd(B, H), torch.where(odd, 2.0 ** -e, 1.0)
    dh_in, dc_in = rnd(T * B, H) * small, rnd(T * B, H) * small
    dh, dc, dx, _ = _sweep(I, H, B, T, Wx, Wh, gates, cs, c0, dh_in, dc_in)
    sl, pr = slice(B, 2 * B), slice(0, B)
    dg = _dgates(gates[sl], cs[sl], cs[pr], dh[sl], dc[sl], H)

    def quad(v):   # the largest magnitude of the quad of every value that is not zero
        rows, n = v.shape
        m = torch.nn.functional.pad(v.abs(), (0, -n % 4)).view(rows, -1, 4).amax(dim=2).repeat_interleave(4, dim=1)[:, :n]
        return m * (v != 0)

    qg = torch.cat([quad(g) for g in dg.split(H, dim=1)], dim=1)
    for W, got, old in ((Wx, dx[sl], None), (Wh, dh[pr], dh_in[pr])):
        W = W.double()
        want = dg @ W.t() + (0 if old is None else old.double())
        bar = 1.45e-6 * 1.25 * (dg.abs() @ W.abs().t()) + 2.0 ** -22 * (qg @ W.abs().t() + dg.abs() @ quad(W).t()) + 1.3e-7 * want.abs()
        assert bool(((got - want).abs() <= bar).all()), float(((got - want).abs() / bar).max())


@pytest.mark.parametrize("I,H,B", [(96, 512, 64), (100, 777, 33)])
def test_gradients_that_fade_over_the_steps(I, H, B):
    """2^-20 smaller with every step towards the first, 2^-80 in all; the bar is that of a single magnitude."""
    import torch
    T = 5
    gen = torch.Generator("cuda").manual_seed(H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    Wx, Wh = rnd(I, 4 * H) / H ** 0.5, rnd(H, 4 * H) / H ** 0.5 * 2.0 ** -20
    gates = torch.cat([torch.sigmoid(rnd(T * B, 3 * H)), torch.tanh(rnd(T * B, H))], dim=1)
    gates[:, H:2 * H] *= 2.0 ** -20
    cs, c0, dh_in, dc_in = rnd(T * B, H), rnd(B, H), rnd(T * B, H), rnd(T * B, H)
    dh_in[:-B] = 0.0
    dc_in[:-B] = 0.0
    dh, dc, dx, _ = _sweep(I, H, B, T, Wx, Wh, gates, cs, c0, dh_in, dc_in)
    for t in range(T - 1, -1, -1):
        sl, pr = slice(t * B, (t + 1) * B), slice((t - 1) * B, t * B)
        dg = _dgates(gates[sl], cs[sl], cs[pr] if t else c0, dh[sl], dc[sl], H)
        assert float(dh[sl].abs().max()) < 2.0 ** (5 - 18 * (T - 1 - t))
        for W, got in ((Wx, dx[sl]), (Wh, dh[pr]))[:2 if t else 1]:
            W = W.double()
            assert bool(((got - dg @ W.t()).abs() <= 1.45e-6 * 1.25 * dg.norm(dim=1)[:, None] * W.norm(dim=1)[None, :]).all()), t


@pytest.mark.parametrize("I,H,B", [(96, 512, 100), (2000, 777, 33)])
def test_infinities_and_nans_stay_in_their_column_and_row(I, H, B):
    import torch
    T = 3
    gen = torch.Generator("cuda").manual_seed(H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    Wx, Wh = rnd(I, 4 * H) / H ** 0.5, rnd(H, 4 * H) / H ** 0.5
    gates = torch.cat([torch.sigmoid(rnd(T * B, 3 * H)), torch.tanh(rnd(T * B, H))], dim=1)
    cs, c0, dh_in, dc_in = rnd(T * B, H), rnd(B, H), rnd(T * B, H), rnd(T * B, H)
    clean = _sweep(I, H, B, T, Wx, Wh, gates, cs, c0, dh_in, dc_in)
    bad_h, bad_c = dh_in.clone(), dc_in.clone()
    bad_h[2 * B + 5, 130], bad_h[2 * B + 31, 0], bad_c[B + 32, H - 1] = float("inf"), float("nan"), float("-inf")
    dh, dc, dx, _ = _sweep(I, H, B, T, Wx, Wh, gates, cs, c0, bad_h, bad_c)
    hit = torch.zeros(T, B, dtype=torch.bool, device="cuda")
    hit[:, 5] = hit[:, 31] = hit[:2, 32] = True
    for got, ref in zip((dh, dc, dx), clean):
        assert torch.equal(got[~hit.view(-1)], ref[~hit.view(-1)])
    assert not bool(torch.isfinite(dx[hit.view(-1)]).any())
    Wx2, Wh2 = Wx.clone(), Wh.clone()
    Wx2[7, 3 * H], Wx2[I - 1, 4 * H - 1], Wh2[200, 5] = float("inf"), float("nan"), float("-inf")   # rows 7 and I - 1 of dx; unit 200's dh, from step 1 down all of it
    dh, dc, dx, _ = _sweep(I, H, B, T, Wx2, Wh2, gates, cs, c0, dh_in, dc_in)
    rest = [r for r in range(I) if r not in (7, I - 1)]
    assert torch.equal(dx[2 * B:, rest], clean[2][2 * B:, rest]) and not bool(torch.isfinite(dx[2 * B:, [7, I - 1]]).any())
    units = [r for r in range(H) if r != 200]
    assert torch.equal(dh[B:2 * B, units], clean[0][B:2 * B, units]) and not bool(torch.isfinite(dh[B:2 * B, 200]).any())


@pytest.mark.parametrize("I,H,B", [(64, 1024, 512), (9, 777, 100), (64, 2048, 500)])
@pytest.mark.parametrize("where", ["weights", "dgates"])
def test_small_quads_everywhere(I, H, B, where):
    """Every quad of a scale but one lies 2^-40 below it: the slowest such calls can be, well inside the bounds of the waits, and right."""
    import torch
    T = 3
    gen = torch.Generator("cuda").manual_seed(H)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    keep = torch.arange(H, device="cuda") % 128 < 4                  # (units of quad 0 of every block; H % 4: of gate 0's at least)
    low = torch.where(keep, 1.0, 2.0 ** -40)
    Wx, Wh = [rnd(n, 4 * H) / H ** 0.5 * (torch.where(torch.arange(4 * H, device="cuda") < 4, 1.0, 2.0 ** -40) if where == "weights" else 1.0 - keep.float().repeat(4))
              for n in (I, H)]
    gates = torch.cat([torch.sigmoid(rnd(T * B, 3 * H)), torch.tanh(rnd(T * B, H))], dim=1)
    cs, c0, dh_in, dc_in = rnd(T * B, H), rnd(B, H), rnd(T * B, H), rnd(T * B, H)
    if where == "dgates":
        dh_in *= low
        dc_in *= low
    dh, dc, dx, _ = _sweep(I, H, B, T, Wx, Wh, gates, cs, c0, dh_in, dc_in)
    for t in range(T - 1, -1, -1):
        sl, pr = slice(t * B, (t + 1) * B), slice((t - 1) * B, t * B)
        dg = _dgates(gates[sl], cs[sl], cs[pr] if t else c0, dh[sl], dc[sl], H)
        for W, got, old in ((Wx, dx[sl], None), (Wh, dh[pr], dh_in[pr]))[:2 if t else 1]:
            W = W.double()
            want = dg @ W.t() + (0 if old is None else old.double())
            bar = (1.45e-6 * 1.25 + 2.0 ** -21) * (dg.abs() @ W.abs().t()) + 1.3e-7 * want.abs()
            if where == "dgates" and H % 4 == 0:   # (nothing but small quads meets these rows)
                assert bool(((got - want).abs() <= bar).all()), (t, float(((got - want).abs() / bar).max()))
            bar = 1.45e-6 * 1.25 * dg.norm(dim=1)[:, None] * W.norm(dim=1)[None, :] + 1.3e-7 * want.abs()
            assert bool(((got - want).abs() <= bar).all()), (t, float(((got - want).abs() / bar).max()))
