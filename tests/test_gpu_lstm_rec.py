"""The cluster-resident recurrence (csrc/lstm_rec.cu, csrc/lstm_rec_tc.cu) behind the sequence calls, for layers up to 384 units and sequences of at
least 8 steps: gates, states, every gradient and the weight gradients against the oracle's node chain.  Shapes at the edges of
its tiling: widths that are no multiple of 4, 8 or 32, one CTA / a portable cluster / a 16-CTA cluster, one column, as many
columns as its clusters carry, batch-1 masks."""
import numpy as np
import pytest

from util import TOL_REDUCE, assert_close, glorot, randn, rng, row_floor

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


def _oracle(oracle, x, h0, c0, Wx, Wh, b, mx, mh, up):
    """Forward and backward over the steps, node by node: (h, c, gates) per step, (dx, dh, dc) per step, dWx, dWh, db."""
    T, B, H = len(x), x[0].shape[0], Wh.shape[0]
    h, c, gates = [h0], [c0], []
    for t in range(T):
        gates.append(oracle.lstm_gates_fwd([x[t]], h[-1], Wx, Wh, b, mask_x=mx, mask_h=mh))
        c.append(oracle.lstm_c_fwd(c[-1], gates[t]))
        h.append(oracle.lstm_h_fwd(c[-1], gates[t]))
    dWx, dWh, db = np.zeros_like(Wx), np.zeros_like(Wh), np.zeros_like(b)
    dx = [np.zeros_like(v) for v in x]
    dh = [np.zeros((B, H), np.float32)] + [u.copy() for u in up]
    dc = [np.zeros((B, H), np.float32) for _ in range(T + 1)]
    for t in range(T, 0, -1):
        dg = np.zeros((B, 4 * H), np.float32)
        oracle.lstm_h_bwd(c[t], gates[t - 1], dh[t], 0, dc[t])
        oracle.lstm_h_bwd(c[t], gates[t - 1], dh[t], 1, dg)
        oracle.lstm_c_bwd(c[t - 1], gates[t - 1], dc[t], 0, dc[t - 1])
        oracle.lstm_c_bwd(c[t - 1], gates[t - 1], dc[t], 1, dg)
        for i, tgt in enumerate((dx[t - 1], dh[t - 1], dWx, dWh, db)):
            oracle.lstm_gates_bwd([x[t - 1]], h[t - 1], Wx, Wh, gates[t - 1], dg, i, tgt, mask_x=mx, mask_h=mh)
    return np.concatenate(h[1:]), np.concatenate(c[1:]), np.concatenate(gates), np.concatenate(dx), np.concatenate(dh[1:]), dWx, dWh, db


@pytest.mark.parametrize("I,H,B,T,mask", [
    (20, 12, 5, 8, None),            # one CTA, three column blocks of one
    (33, 33, 3, 9, "full"),          # two CTAs, the second with one unit
    (128, 256, 1, 12, None),         # one column
    (128, 256, 32, 10, "full"),      # two columns per cluster
    (100, 100, 47, 8, "one"),        # batch-1 masks, a cluster of four
    (64, 257, 9, 8, None),           # just beyond the portable cluster
    (200, 300, 30, 9, "full"),       # fifteen CTAs
    (48, 384, 130, 8, None),         # the widest layer, several columns per cluster
    (16, 64, 700, 8, "full"),        # many columns per cluster
    (16, 384, 280, 8, "full"),       # the most columns its clusters carry, or nearly
    # on the tensor pipe (csrc/lstm_rec_tc.cu)
    (24, 256, 70, 9, "full"),        # five columns per cluster
    (24, 256, 301, 8, None),         # twenty-one
    (16, 250, 500, 8, "full"),       # three groups of columns forward; backward more blocks than clusters; a last CTA with 26 units
    (16, 225, 1001, 8, "one"),       # more blocks than clusters both ways; a last CTA with one unit
    (16, 130, 600, 8, None),         # five CTAs, two row tiles
    (16, 97, 1500, 9, "full"),       # four CTAs, one row tile, the second block of the reduction nearly empty
    (8, 31, 3000, 8, None),          # one CTA
])
def test_recurrence_matches_oracle(oracle, g, I, H, B, T, mask):
    import torch
    from dynet_b200 import capi
    r = rng(900 + H + B)
    Wx, Wh, b = glorot(r, 4 * H, I), glorot(r, 4 * H, H), randn(r, 4 * H, scale=0.1)
    mB = B if mask == "full" else 1
    mx = ((r.random((mB, I)) < 0.8) / 0.8).astype(np.float32) if mask else None
    mh = ((r.random((mB, H)) < 0.8) / 0.8).astype(np.float32) if mask else None
    x, up = [randn(r, B, I) for _ in range(T)], [randn(r, B, H) for _ in range(T)]
    h0, c0 = randn(r, B, H, scale=0.5), randn(r, B, H, scale=0.5)
    want = _oracle(oracle, x, h0, c0, Wx, Wh, b, mx, mh, up)
    ctx = g.ctx()
    at = capi.LstmGatesAttrs(1 if mask else 0, 0.0, 1.0)
    D = {k: g.dev(v) for k, v in dict(Wx=Wx, Wh=Wh, b=b, x=np.concatenate(x), h0=h0, c0=c0, dh=np.concatenate(up)).items()}
    tmx, tmh = (g.T(g.dev(mx)), g.T(g.dev(mh))) if mask else (None, None)
    tWx, tWh, tb = g.T(D["Wx"], [4 * H, I], 1), g.T(D["Wh"], [4 * H, H], 1), g.T(D["b"], [4 * H], 1)
    gates, cs, hs = (torch.full((T * B, n), 7.0, device="cuda") for n in (4 * H, H, H))
    dc, dx, db = torch.zeros(T * B, H, device="cuda"), torch.zeros(T * B, I, device="cuda"), torch.zeros(4 * H, device="cuda")
    dWx, dWh = torch.zeros(I, 4 * H, device="cuda"), torch.zeros(H, 4 * H, device="cuda")
    w = ctx.wgrad_create(4 * H, I, H, T * B)
    try:
        l0 = ctx.launches()
        ctx.lstm_seq_fwd(g.T(D["x"], [I], T * B), g.T(D["h0"]), g.T(D["c0"]), tWx, tWh, tb, tmx, tmh, at, g.T(gates, [4 * H], T * B),
                         g.T(cs, [H], T * B), g.T(hs, [H], T * B), w, T)
        ctx.lstm_seq_bwd(g.T(D["x"], [I], T * B), g.T(D["h0"]), g.T(D["c0"]), tWx, tWh, tmx, tmh, at, g.T(gates, [4 * H], T * B),
                         g.T(cs, [H], T * B), g.T(hs, [H], T * B), g.T(D["dh"], [H], T * B), g.T(dc, [H], T * B), g.T(dx, [I], T * B),
                         None, None, g.T(db, [4 * H], 1), w, T)
        assert ctx.launches() - l0 < 14, "the per-step calls ran"
        ctx.wgrad_flush(w, dWx.data_ptr(), 4 * H, dWh.data_ptr(), 4 * H)
        torch.cuda.synchronize()
    finally:
        ctx.wgrad_destroy(w)
    assert ctx.device_errors() == 0
    for name, got, ref in zip(("h", "c", "gates"), (hs, cs, gates), want[:3]):
        assert_close(g.host(got), ref, TOL_REDUCE, floor=0.1, what=name)
    for name, got, ref in zip(("dx", "dh"), (dx, D["dh"]), want[3:5]):
        assert_close(g.host(got), ref, TOL_REDUCE, floor=row_floor(ref, 1, rel=1e-2), what=name + " (per-column scale)")
    for name, got, ref in zip(("dWx", "dWh"), (dWx, dWh), want[5:7]):
        assert_close(g.host(got), ref, TOL_REDUCE, floor=row_floor(ref, 0, rel=1e-2), what=name + " (per-row scale)")
    assert_close(g.host(db), want[7], TOL_REDUCE, floor=float(np.abs(want[7]).max()) * 0.02, what="db")


@pytest.mark.parametrize("I,H,B,T", [(45, 262, 372, 19), (45, 230, 777, 19)])
def test_recurrence_is_the_same_every_time(g, I, H, B, T):
    """Widths whose warps and CTAs finish unevenly (a last CTA with two or six units, nine warps per CTA), many columns: twelve passes
    over the same inputs give the same bits."""
    import torch
    from dynet_b200 import capi
    gen = torch.Generator("cuda").manual_seed(5)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)
    x, Wx, Wh, b, up = rnd(T * B, I), rnd(I, 4 * H) * 0.05, rnd(H, 4 * H) * 0.05, rnd(4 * H) * 0.1, rnd(T * B, H)
    z, at, ctx = torch.zeros(B, H, device="cuda"), capi.LstmGatesAttrs(0, 0.0, 1.0), g.ctx()
    w = ctx.wgrad_create(4 * H, I, H, T * B)
    first = None
    try:
        for _ in range(12):
            gates, cs, hs, dh = (torch.empty(T * B, n, device="cuda") for n in (4 * H, H, H, H))
            dc, dx, db = torch.zeros(T * B, H, device="cuda"), torch.zeros(T * B, I, device="cuda"), torch.zeros(4 * H, device="cuda")
            dh.copy_(up)
            W = (g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1))
            S = (g.T(gates, [4 * H], T * B), g.T(cs, [H], T * B), g.T(hs, [H], T * B))
            ctx.lstm_seq_fwd(g.T(x, [I], T * B), g.T(z), g.T(z), *W, g.T(b, [4 * H], 1), None, None, at, *S, w, T)
            ctx.lstm_seq_bwd(g.T(x, [I], T * B), g.T(z), g.T(z), *W, None, None, at, *S, g.T(dh, [H], T * B), g.T(dc, [H], T * B),
                             g.T(dx, [I], T * B), None, None, g.T(db, [4 * H], 1), w, T)
            dWx, dWh = torch.zeros(I, 4 * H, device="cuda"), torch.zeros(H, 4 * H, device="cuda")
            ctx.wgrad_flush(w, dWx.data_ptr(), 4 * H, dWh.data_ptr(), 4 * H)
            torch.cuda.synchronize()
            out = (gates, cs, hs, dh, dx, db, dWx, dWh)
            first = first or out
            assert all(torch.equal(p, q) for p, q in zip(first, out))
    finally:
        ctx.wgrad_destroy(w)
    assert ctx.device_errors() == 0


def test_more_columns_than_a_grid_holds(g):
    """Past 65 535 clusters the recurrence kernels hand the layer back to the per-step calls."""
    import ctypes as C
    import torch
    from dynet_b200 import capi
    ctx, most = g.ctx(), 65535 * 32
    takes = capi.lib().dyb200i_rec_takes
    takes.argtypes, takes.restype = [C.c_void_p, C.c_uint32, C.c_uint32, C.c_uint32, C.c_int], C.c_int
    assert [takes(ctx.h, 4, 8, most, 1), takes(ctx.h, 4, 8, most + 1, 1), takes(ctx.h, 4, 8, 32767 * 32, 2), takes(ctx.h, 4, 8, 32768 * 32, 2)] == [1, 0, 1, 0]
    I, H, T, B, few = 3, 4, 8, most + 1, 50
    gen = torch.Generator("cuda").manual_seed(9)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen) * 0.5
    x, h0, c0, Wx, Wh, b = rnd(T, B, I), rnd(B, H), rnd(B, H), rnd(I, 4 * H), rnd(H, 4 * H), rnd(4 * H)

    def run(x, h0, c0):
        n = h0.shape[0]
        gates, cs, hs = (torch.empty(T * n, k, device="cuda") for k in (4 * H, H, H))
        ctx.lstm_seq_fwd(g.T(x, [I], T * n), g.T(h0), g.T(c0), g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), g.T(b, [4 * H], 1), None, None,
                         capi.LstmGatesAttrs(0, 0.0, 1.0), g.T(gates, [4 * H], T * n), g.T(cs, [H], T * n), g.T(hs, [H], T * n), None, T)
        torch.cuda.synchronize()
        return hs.view(T, n, H)
    every = run(x, h0, c0)
    for cols in (slice(0, few), slice(B - few, B)):
        want = run(x[:, cols].contiguous(), h0[cols].contiguous(), c0[cols].contiguous())
        assert_close(g.host(every[:, cols]), g.host(want), TOL_REDUCE, floor=0.1, what="h of %d columns" % B)
    assert ctx.device_errors() == 0
