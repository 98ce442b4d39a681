"""The backward recurrence of 257 - 320 units (csrc/lstm_rec.cu: 32 units per CTA from 8 columns on, up to 320 threads) at the edges of its units and columns, step
by step against float64 from the device's own dE/dh_t and dE/dc_t.  Bar of dE/dh_{t-1}: an fp32 sum of 4H products in slices and trees, at most 80
roundings at 2^-24 of |column of Wh| |dgates|, and 1e-6 of that for dgates themselves."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,B,mask", [(257, 7, None), (257, 8, "full"), (288, 45, None), (300, 31, "one"), (320, 8, None), (320, 130, "full"), (321, 16, None)])
def test_backward_steps(H, B, mask):
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    I, T, ctx = 12, 9, g.ctx()
    gen = torch.Generator("cuda").manual_seed(H + B)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    Wx, Wh, x, c0 = rnd(I, 4 * H) / H ** 0.5, rnd(H, 4 * H) / H ** 0.5, rnd(T * B, I), rnd(B, H)
    gates, cs = torch.cat([torch.sigmoid(rnd(T * B, 3 * H)), torch.tanh(rnd(T * B, H))], dim=1), rnd(T * B, H)
    dh_in, dc_in = rnd(T * B, H), rnd(T * B, H)
    dh, dc, dx, db = dh_in.clone(), dc_in.clone(), torch.zeros(T * B, I, device="cuda"), torch.zeros(4 * H, device="cuda")
    mB = B if mask == "full" else 1
    mx, mh = [((torch.rand(mB, n, device="cuda", generator=gen) < 0.8) / 0.8).float() if mask else torch.ones(1, n, device="cuda") for n in (I, H)]
    at, tm = capi.LstmGatesAttrs(1 if mask else 0, 0.0, 1.0), (g.T(mx), g.T(mh)) if mask else (None, None)
    w = ctx.wgrad_create(4 * H, I, H, T * B)
    ctx.wgrad_pack_inputs(w, g.T(x, [I], T * B), tm[0], B)
    ctx.lstm_seq_bwd(g.T(x, [I], T * B), g.T(c0), g.T(c0), g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), *tm, at, g.T(gates, [4 * H], T * B), g.T(cs, [H], T * B),
                     g.T(cs, [H], T * B), g.T(dh, [H], T * B), g.T(dc, [H], T * B), g.T(dx, [I], T * B), None, None, g.T(db, [4 * H], 1), w, T)
    torch.cuda.synchronize()
    ctx.wgrad_destroy(w)
    db_want = torch.zeros(4 * H, device="cuda", dtype=torch.float64)
    for t in range(T - 1, -1, -1):
        sl, pr = slice(t * B, (t + 1) * B), slice((t - 1) * B, t * B)
        i, f, o, gg = gates[sl].double().split(H, dim=1)
        c, cp, dht = cs[sl].double(), (cs[pr] if t else c0).double(), dh[sl].double()
        tc = torch.tanh(c)
        d = dht * o * (1 - tc * tc) + dc[sl].double()
        dg = torch.cat([d * gg * i * (1 - i), d * cp * f * (1 - f), dht * tc * o * (1 - o), d * i * (1 - gg * gg)], dim=1)
        db_want += dg.sum(dim=0)
        if t:
            want = dh_in[pr].double() + mh.double() * (dg @ Wh.double().t())
            bar = (80 * 2.0 ** -24 + 1e-6) * 1.25 * dg.norm(dim=1)[:, None] * Wh.double().norm(dim=1)[None, :] + 1.3e-7 * want.abs()
            assert bool(((dh[pr].double() - want).abs() <= bar).all()), "dh %d: %.3g" % (t - 1, float(((dh[pr].double() - want).abs() / bar).max()))
            want = dc_in[pr].double() + d * f
            assert bool(((dc[pr].double() - want).abs() <= 1e-6 * (dc_in[pr].double().abs() + (d * f).abs() + (dht * o * f).abs())).all()), "dc %d" % (t - 1)
    assert bool(((db.double() - db_want).abs() <= 2e-6 * (T * B) ** 0.5 * db_want.abs().max()).all())
    assert ctx.device_errors() == 0
