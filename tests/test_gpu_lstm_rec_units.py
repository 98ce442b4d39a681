"""The forward recurrence of 257 - 384 units at the edges of its units per CTA (csrc/lstm_rec.cu: 32 up to 320 units from 8 columns on), step by
step against float64 from the device's own h_{t-1} and c_{t-1}.  Bar of a pre-activation: an fp32 sum of H products in 16 slices and a
tree, at most 40 roundings at 2^-24 of |row of Wh| |h|, and the input product's 5.7e-6 of |row of Wx| |x|; of a gate: that and 3e-6 for the
approximate exponential and reciprocal."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("H,B,mask", [(257, 7, None), (257, 8, "full"), (288, 45, None), (300, 31, "one"), (320, 8, None), (320, 130, "full"), (321, 16, None)])
def test_forward_steps(H, B, mask):
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    I, T, ctx = 12, 9, g.ctx()
    gen = torch.Generator("cuda").manual_seed(H + B)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    x, h0, c0, b = rnd(T * B, I), rnd(B, H), rnd(B, H), rnd(4 * H) * 0.1
    Wx, Wh = rnd(I, 4 * H) / I ** 0.5, rnd(H, 4 * H) / H ** 0.5
    mB = B if mask == "full" else 1
    mx, mh = [((torch.rand(mB, n, device="cuda", generator=gen) < 0.8) / 0.8).float() if mask else torch.ones(1, n, device="cuda") for n in (I, H)]
    at, tm = capi.LstmGatesAttrs(1 if mask else 0, 0.0, 1.0), (g.T(mx), g.T(mh)) if mask else (None, None)
    w = ctx.wgrad_create(4 * H, I, H, T * B)
    gates, cs, hs = (torch.full((T * B, n), 7.0, device="cuda") for n in (4 * H, H, H))
    ctx.lstm_seq_fwd(g.T(x, [I], T * B), g.T(h0), g.T(c0), g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), g.T(b, [4 * H], 1), *tm, at, g.T(gates, [4 * H], T * B),
                     g.T(cs, [H], T * B), g.T(hs, [H], T * B), w, T)
    torch.cuda.synchronize()
    ctx.wgrad_destroy(w)
    gates, cs, hs = (o.double().view(T, B, -1) for o in (gates, cs, hs))
    for t in range(T):
        xt, hp, cp = x.double().view(T, B, I)[t] * mx.double(), (hs[t - 1] if t else h0.double()) * mh.double(), cs[t - 1] if t else c0.double()
        pre = xt @ Wx.double() + hp @ Wh.double() + b.double()
        bar = 5.7e-6 * xt.norm(dim=1)[:, None] * Wx.double().norm(dim=0) + 40 * 2.0 ** -24 * hp.norm(dim=1)[:, None] * Wh.double().norm(dim=0) + 3e-6
        pre[:, H:2 * H] += 1.0
        want = torch.cat([torch.sigmoid(pre[:, :3 * H]), torch.tanh(pre[:, 3 * H:])], dim=1)
        assert bool(((gates[t] - want).abs() <= bar).all()), "step %d" % t
        i, f, o, gg = gates[t].split(H, dim=1)
        c = i * gg + f * cp
        assert bool(((cs[t] - c).abs() <= 2e-7 * ((i * gg).abs() + (f * cp).abs())).all())
        assert bool(((hs[t] - o * torch.tanh(cs[t])).abs() <= 5e-7).all())
    assert ctx.device_errors() == 0
