"""Gradient buffers that hold nothing yet: what the drivers' internal calls (csrc/lstm_rec_api.h) write into buffers full of NaNs is, up to the sign of zeros, what the public
calls add to zeros.  Every form of a layer's backward call; the input gradients of AffineTransform and of the output layer on every product path."""
import ctypes as C

import pytest

pytestmark = pytest.mark.gpu

FRESH_DX, FRESH_DC = 1, 2


def _seq_bwd(args, T, fresh):
    import gpu_util as g
    from dynet_b200 import capi
    f = capi.lib().dyb200i_lstm_seq_bwd
    f.restype = C.c_int
    ctx = g.ctx()
    rc = f(*[a if a is None or isinstance(a, C.c_void_p) else C.byref(a) for a in args], C.c_uint32(T), C.c_uint(fresh), C.c_void_p(ctx._hv))
    ctx.check(rc)


def _fresh(name, *args):
    import gpu_util as g
    from dynet_b200 import capi
    f = getattr(capi.lib(), name)
    f.restype = C.c_int
    ctx = g.ctx()
    ctx.check(f(*[C.byref(a) if isinstance(a, capi.DyTensor) else a for a in args], C.c_void_p(ctx._hv)))


# A bit that the drivers once spoke to the kernels with: no public call takes it for anything.
@pytest.mark.parametrize("flags", [0x80000000, 0xfffffffe])
def test_public_calls_add(flags):
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    A, x, d = torch.randn(40, 30, device="cuda"), torch.randn(9, 40, device="cuda"), torch.randn(9, 30, device="cuda")
    for name, at in (("affine_transform", 1), ("matmul", 0)):
        xs = [g.T(d[0].clone(), [30], 1)][:at] + [g.T(A, [30, 40], 1), g.T(x, [40], 9)]
        a, b = torch.ones(9, 40, device="cuda"), torch.ones(9, 40, device="cuda")
        ctx.bwd(name, xs, g.T(d, [30], 9), g.T(d, [30], 9), at + 1, g.T(a, [40], 9))
        ctx.bwd(name, xs, g.T(d, [30], 9), g.T(d, [30], 9), at + 1, g.T(b, [40], 9), capi.AffineAttrs(flags))
        assert torch.equal(a, b), name


@pytest.mark.parametrize("I,H,B,T,mask,spread", [
    (96, 512, 64, 9, "full", 0),        # wide
    (301, 520, 33, 8, "one", 0),        # wide, rows of dx that are no multiple of four
    (1024, 512, 12, 9, None, 0),        # wide, dx in eight CTAs per tile
    (96, 512, 64, 9, None, 60),         # wide, small quads of dgates and of weights
    (45, 517, 40, 8, None, 60),         # the same a value at a time
    (40, 256, 16, 9, "full", 0),        # recurrence in clusters, fp32
    (40, 256, 300, 9, None, 0),         # ... on the tensor pipe
    (128, 256, 64, 8, "one", 0),        # TF32 pairs, all steps in one kernel
    (24, 64, 8, 3, "full", 0),          # launch by launch
    (24, 512, 4, 3, None, 0),
])
def test_layer(I, H, B, T, mask, spread):
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    gen = torch.Generator("cuda").manual_seed(H + B)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    small = torch.ones(H, device="cuda")
    if spread:
        small[H // 2:] = 2.0 ** -spread
    Wx, Wh, x, c0 = rnd(I, 4 * H) / H ** 0.5, rnd(H, 4 * H) / H ** 0.5, rnd(T * B, I), rnd(B, H)
    Wx *= small.repeat(4)[None, :]
    gates, cs, hs = torch.cat([torch.sigmoid(rnd(T * B, 3 * H)), torch.tanh(rnd(T * B, H))], dim=1), rnd(T * B, H), rnd(T * B, H)
    dh_in = rnd(T * B, H) * small
    mB = B if mask == "full" else 1
    mx, mh = [((torch.rand(mB, n, device="cuda", generator=gen) < 0.8) / 0.8).float() for n in (I, H)]
    tm = (g.T(mx), g.T(mh)) if mask else (None, None)
    at = capi.LstmGatesAttrs(1 if mask else 0, 0.0, 1.0)
    got = []
    for fresh in (0, FRESH_DX | FRESH_DC):
        fill = float("nan") if fresh else 0.0
        dh, dc, dx, db = dh_in.clone(), torch.full((T * B, H), fill, device="cuda"), torch.full((T * B, I), fill, device="cuda"), torch.zeros(4 * H, device="cuda")
        w = ctx.wgrad_create(4 * H, I, H, T * B)
        ctx.wgrad_pack_inputs(w, g.T(x, [I], T * B), tm[0], B)
        args = (g.T(x, [I], T * B), g.T(c0), g.T(c0), g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), *tm, at, g.T(gates, [4 * H], T * B), g.T(cs, [H], T * B),
                g.T(hs, [H], T * B), g.T(dh, [H], T * B), g.T(dc, [H], T * B), g.T(dx, [I], T * B), None, None, g.T(db, [4 * H], 1), w)
        if fresh:
            _seq_bwd(args, T, fresh)
        else:
            ctx.lstm_seq_bwd(*args, T)
        torch.cuda.synchronize()
        ctx.wgrad_destroy(w)
        got.append((dh, dx, db))
    assert ctx.device_errors() == 0
    for name, a, b in zip(("dh", "dx", "db"), *got):
        assert torch.equal(a, b), name + ": %d of %d values" % (int((a != b).sum()), a.numel())


# (rows of A, columns of A, batch of B): CUDA cores, thin, narrow (either side), TF32 pairs, fp16 pairs with and without K splits
@pytest.mark.parametrize("M,K,n", [(7, 5, 3), (300, 40, 9), (32, 256, 3000), (45, 130, 5000), (500, 300, 700), (4096, 1024, 2048), (3000, 512, 3001)])
def test_affine_inputs(M, K, n):
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    gen = torch.Generator("cuda").manual_seed(M)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    A, x, b, d, y = rnd(K, M), rnd(n, K), rnd(M), rnd(n, M), torch.empty(n, M, device="cuda")
    xs = [g.T(b, [M], 1), g.T(A, [M, K], 1), g.T(x, [K], n)]
    for i, shape, dims, bd in ((0, (M,), [M], 1), (1, (K, M), [M, K], 1), (2, (n, K), [K], n)):
        zero, nan = torch.zeros(*shape, device="cuda"), torch.full(shape, float("nan"), device="cuda")
        ctx.bwd("affine_transform", xs, g.T(y, [M], n), g.T(d, [M], n), i, g.T(zero, dims, bd))
        _fresh("dyb200i_affine_transform_bwd", (capi.DyTensor * 3)(*xs), C.c_int(3), g.T(y, [M], n), g.T(d, [M], n), C.c_uint(i), g.T(nan, dims, bd), None, None, C.c_int(1))
        assert torch.equal(zero, nan), "argument %d" % i


@pytest.mark.parametrize("V,H,n", [(40, 16, 9), (1001, 200, 300), (6000, 512, 2048)])
def test_output_layer(V, H, n):
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    ctx = g.ctx()
    gen = torch.Generator("cuda").manual_seed(V)
    rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen)   # noqa: E731
    x, h, R, dE = rnd(n, V), rnd(n, H), rnd(H, V) / H ** 0.5, rnd(n)
    aux, loss = torch.zeros(3 * n, device="cuda"), torch.empty(n, device="cuda")
    aux[2 * n:].view(torch.int32).copy_(torch.randint(0, V, (n,), device="cuda", generator=gen))
    ctx.fwd("pickneglogsoftmax", [g.T(x, [V], n)], g.T(loss, [1], n), capi.PickAttrs(None, n), aux.data_ptr())
    got = []
    for fresh in (0, 1):
        dR, db, dh, scratch = torch.zeros(H, V, device="cuda"), torch.zeros(V, device="cuda"), torch.full((n, H), float("nan") if fresh else 0.0, device="cuda"), torch.empty(n, V, device="cuda")
        args = (g.T(x, [V], n), g.T(h, [H], n), g.T(R, [V, H], 1), g.T(dE, [1], n), C.c_void_p(aux.data_ptr()), g.T(dR, [V, H], 1), g.T(db, [V], 1), g.T(dh, [H], n),
                g.T(scratch, [V], n))
        if fresh:
            _fresh("dyb200i_softmax_output_bwd_fused", *args, C.c_uint32(0), C.c_int(1))
        else:
            ctx.softmax_output_bwd_fused(*args[:4], aux.data_ptr(), *args[5:])
        got.append((dR, db, dh))
    for name, a, b in zip(("dR", "db", "dh"), *got):
        assert torch.equal(a, b), name
