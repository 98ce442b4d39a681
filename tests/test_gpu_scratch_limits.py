"""Calls that find little device memory left: where fp16 pairs or partial products do not fit, the form that needs none of them runs - the deferred
weight gradients on the accumulator's TF32 planes or unsplit (csrc/gemm_tc.cu), a product on pairs of SMs unsplit (csrc/gemm_pair.cu), the
sequence of a wide layer step by step (csrc/lstm_seq.cu) - and the context serves the next call, whose arena does not fit either.
Bars as in test_gpu_wgrad_grouped.py and test_gpu_gemm_pair.py."""
import contextlib

import pytest

pytestmark = pytest.mark.gpu


@contextlib.contextmanager
def room_for(mib):
    """A fresh context while all but `mib` MiB of the device's free memory are taken (reserved, not touched)."""
    import torch
    from dynet_b200 import capi
    ctx = capi.Context(0, torch.cuda.current_stream().cuda_stream)
    torch.cuda.synchronize()
    torch.cuda.empty_cache()
    taken = torch.empty(torch.cuda.mem_get_info()[0] - (mib << 20), dtype=torch.uint8, device="cuda")
    try:
        yield ctx
        torch.cuda.synchronize()
        assert ctx.device_errors() == 0
    finally:
        del taken
        torch.cuda.empty_cache()
        ctx.close()


@pytest.mark.parametrize("M,N0,N1,k,mib", [
    (4096, 1024, 1024, 8192, 64),        # pairs: 200 MB
    (1024, 128, 256, 40000, 8),          # work items with partial products: 20 MB and more
])
def test_weight_gradients(M, N0, N1, k, mib):
    import torch
    import gpu_util as g
    w = g.ctx().wgrad_create(M, N0, N1, k)
    try:
        a, b0, b1 = (torch.randn(k, n, device="cuda") for n in (M, N0, N1))
        Cs = [torch.zeros(n, M, device="cuda") for n in (N0, N1)]
        for c in (g.ctx(), None):        # (a first time with all the memory: kernels are loaded, values are right)
            with contextlib.nullcontext(c) if c else room_for(mib) as ctx:
                for _ in range(2 if c is None else 1):
                    for C in Cs:
                        C.zero_()
                    ctx.wgrad_push(w, k, a.data_ptr(), M, b0.data_ptr(), N0, None, 0, b1.data_ptr(), N1, None, 0)
                    ctx.wgrad_flush(w, Cs[0].data_ptr(), M, Cs[1].data_ptr(), M)
            for b, C in zip((b0, b1), Cs):
                want = b.double().t() @ a.double()
                bar = 5.7e-6 * b.double().norm(dim=0)[:, None] * a.double().norm(dim=0)[None, :] + 6e-8 * want.abs()
                assert bool(((C.double() - want).abs() <= bar).all())
    finally:
        g.ctx().wgrad_destroy(w)


def test_product_on_pairs_of_sms():
    import torch
    import gpu_util as g
    M, N, K = 2304, 2300, 8192                                    # planes 151 MB; 81 tiles on 74 pairs of SMs: K splits, 21 MB each
    A, B = torch.randn(K, M, device="cuda"), torch.randn(K, N, device="cuda")
    C = torch.zeros(N, M, device="cuda")
    for c in (g.ctx(), None):
        with contextlib.nullcontext(c) if c else room_for(190) as ctx:
            C.fill_(7.0)
            ctx.gemm(0, 1, M, N, K, A.data_ptr(), M, B.data_ptr(), N, C.data_ptr(), M, 0)
        err = (C.double() - B.double().t() @ A.double()).abs() / (B.double().norm(dim=0)[:, None] * A.double().norm(dim=0)[None, :])
        assert float(err.max()) <= 4.5e-7


def test_sequence_of_a_wide_layer():
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    I, H, B, T = 512, 512, 512, 64                                # pairs of x: 67 MB; of the weights: 8 MB
    rnd = lambda *s: torch.randn(*s, device="cuda")   # noqa: E731
    x, h0, c0, b = rnd(T * B, I), rnd(B, H) * 0.3, rnd(B, H), rnd(4 * H) * 0.1
    Wx, Wh = rnd(I, 4 * H) / I ** 0.5, rnd(H, 4 * H) / H ** 0.5
    w = g.ctx().wgrad_create(4 * H, I, H, T * B)
    outs = [[torch.empty(T * B, n, device="cuda") for n in (4 * H, H, H)] for _ in range(2)]
    try:
        for c, o in zip((g.ctx(), None), outs):
            with contextlib.nullcontext(c) if c else room_for(48) as ctx:
                ctx.lstm_seq_fwd(g.T(x, [I], T * B), g.T(h0), g.T(c0), g.T(Wx, [4 * H, I], 1), g.T(Wh, [4 * H, H], 1), g.T(b, [4 * H], 1), None, None,
                                 capi.LstmGatesAttrs(0, 0.0, 1.0), g.T(o[0], [4 * H], T * B), g.T(o[1], [H], T * B), g.T(o[2], [H], T * B), w, T)
        torch.cuda.synchronize()
        assert all(torch.equal(p, q) for p, q in zip(*outs))       # (the single-step calls give the same bits)
    finally:
        g.ctx().wgrad_destroy(w)
