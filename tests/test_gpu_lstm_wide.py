"""The one-launch recurrence of wide layers with few columns (csrc/lstm_wide.cu) behind the sequence calls, against the oracle's node
chain: one and eight columns, widths just above the cluster kernels', at one, two and three pieces of the reduction, with a last CTA of
two units and unaligned rows, the widest that the SMs hold; masks of one column and of all; and the same bits every time."""
import numpy as np
import pytest

from test_gpu_lstm_rec import _oracle
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


@pytest.mark.parametrize("I,H,B,T,mask", [(12, 386, 8, 8, "full"), (64, 512, 3, 9, "one"), (33, 1021, 2, 10, "full"), (16, 1024, 1, 17, None),
                                          (8, 1184, 5, 8, None)])
def test_wide_recurrence_matches_oracle(oracle, g, I, H, B, T, mask):
    import torch
    from dynet_b200 import capi
    r = rng(700 + H + B)
    Wx, Wh, b = glorot(r, 4 * H, I), glorot(r, 4 * H, H), randn(r, 4 * H, scale=0.1)
    mB = B if mask == "full" else 1
    mx = ((r.random((mB, I)) < 0.8) / 0.8).astype(np.float32) if mask else None
    mh = ((r.random((mB, H)) < 0.8) / 0.8).astype(np.float32) if mask else None
    x, up = [randn(r, B, I) for _ in range(T)], [randn(r, B, H) for _ in range(T)]
    h0, c0 = randn(r, B, H, scale=0.5), randn(r, B, H, scale=0.5)
    want = _oracle(oracle, x, h0, c0, Wx, Wh, b, mx, mh, up)
    ctx, at = g.ctx(), capi.LstmGatesAttrs(1 if mask else 0, 0.0, 1.0)
    D = {k: g.dev(v) for k, v in dict(Wx=Wx, Wh=Wh, b=b, x=np.concatenate(x), h0=h0, c0=c0).items()}
    tmx, tmh = (g.T(g.dev(mx)), g.T(g.dev(mh))) if mask else (None, None)
    tW = (g.T(D["Wx"], [4 * H, I], 1), g.T(D["Wh"], [4 * H, H], 1))
    first = None
    for rep in range(4):
        gates, cs, hs = (torch.full((T * B, n), 7.0, device="cuda") for n in (4 * H, H, H))
        dh = g.dev(np.concatenate(up))
        dc, dx, db = torch.zeros(T * B, H, device="cuda"), torch.zeros(T * B, I, device="cuda"), torch.zeros(4 * H, device="cuda")
        dWx, dWh = torch.zeros(I, 4 * H, device="cuda"), torch.zeros(H, 4 * H, device="cuda")
        S = (g.T(gates, [4 * H], T * B), g.T(cs, [H], T * B), g.T(hs, [H], T * B))
        w = ctx.wgrad_create(4 * H, I, H, T * B)
        try:
            l0 = ctx.launches()
            ctx.lstm_seq_fwd(g.T(D["x"], [I], T * B), g.T(D["h0"]), g.T(D["c0"]), *tW, g.T(D["b"], [4 * H], 1), tmx, tmh, at, *S, w, T)
            assert ctx.launches() - l0 < 8, "a launch per step"
            ctx.lstm_seq_bwd(g.T(D["x"], [I], T * B), g.T(D["h0"]), g.T(D["c0"]), *tW, tmx, tmh, at, *S, g.T(dh, [H], T * B),
                             g.T(dc, [H], T * B), g.T(dx, [I], T * B), None, None, g.T(db, [4 * H], 1), w, T)
            ctx.wgrad_flush(w, dWx.data_ptr(), 4 * H, dWh.data_ptr(), 4 * H)
            torch.cuda.synchronize()
        finally:
            ctx.wgrad_destroy(w)
        assert ctx.device_errors() == 0
        out = (hs, cs, gates)
        first = first or out
        assert all(torch.equal(p, q) for p, q in zip(first, out))
    # (fp32 sums of H products forward; the weight gradients read the operand planes that the recurrence left)
    for name, got, ref in zip(("h", "c", "gates"), (hs, cs, gates), want[:3]):
        assert_close(g.host(got), ref, TOL_REDUCE, floor=0.1, what=name)
    for name, got, ref in zip(("dWx", "dWh"), (dWx, dWh), want[5:7]):
        assert_close(g.host(got), ref, TOL_REDUCE, floor=row_floor(ref, 0, rel=1e-2), what=name + " (per-row scale)")


SHIM = r"""
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) {
  static cudaError_t (*real)(const cudaLaunchConfig_t*, const void*, void**);
  if (!real) real = (cudaError_t (*)(const cudaLaunchConfig_t*, const void*, void**))dlsym(RTLD_NEXT, "cudaLaunchKernelExC");
  for (unsigned k = 0; k < c->numAttrs; ++k)
    if (c->attrs[k].id == cudaLaunchAttributeCooperative) return cudaErrorNotSupported;
  return real(c, f, a);
}
"""
SEQUENCE = """
import sys, torch
from dynet_b200 import capi
H, B, T, I = 520, 3, 9, 16
gen = torch.Generator("cuda").manual_seed(1)
rnd = lambda *s: torch.randn(*s, device="cuda", generator=gen) * 0.2
x, h0, c0, Wx, Wh, b = rnd(T * B, I), rnd(B, H), rnd(B, H), rnd(I, 4 * H), rnd(H, 4 * H) * 0.2, rnd(4 * H)
gates, cs, hs = (torch.zeros(T * B, n, device="cuda") for n in (4 * H, H, H))
t = lambda v, d, n=1: capi.DyTensor.of(v.data_ptr(), d, n)
ctx = capi.Context(0, torch.cuda.current_stream().cuda_stream)
w = ctx.wgrad_create(4 * H, I, H, T * B)
n = []
for _ in range(2):
    l0 = ctx.launches()
    ctx.lstm_seq_fwd(t(x, [I], T * B), t(h0, [H], B), t(c0, [H], B), t(Wx, [4 * H, I]), t(Wh, [4 * H, H]), t(b, [4 * H]), None, None,
                     capi.LstmGatesAttrs(0, 0.0, 1.0), t(gates, [4 * H], T * B), t(cs, [H], T * B), t(hs, [H], T * B), w, T)
    n.append(ctx.launches() - l0)
torch.cuda.synchronize()
assert ctx.device_errors() == 0
torch.save((n, gates.cpu(), cs.cpu(), hs.cpu()), sys.argv[1])
"""


def test_a_refused_gang_launch_runs_step_by_step(tmp_path):
    """A driver that does not take the cooperative attribute (a fake of the launch call that returns cudaErrorNotSupported for it): the same
    sequence, launch by launch, to the rounding of its sums."""
    import os
    import subprocess
    import sys
    from pathlib import Path
    import torch
    (tmp_path / "shim.c").write_text(SHIM)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "shim.so"), str(tmp_path / "shim.c"), "-I/usr/local/cuda/include", "-ldl"])
    out = []
    for name, extra in (("taken", {}), ("refused", {"LD_PRELOAD": str(tmp_path / "shim.so")})):
        p = subprocess.run([sys.executable, "-c", SEQUENCE, str(tmp_path / name)], cwd=Path(__file__).resolve().parent.parent, env=dict(os.environ, **extra),
                           capture_output=True, text=True)
        assert p.returncode == 0, p.stderr[-800:]
        out.append(torch.load(str(tmp_path / name)))
    (n0, *a), (n1, *b) = out
    assert max(n0) < 8 and min(n1) > 9
    for p, q in zip(a, b):
        assert_close(q.numpy(), p.numpy(), TOL_REDUCE, floor=0.1, what="refused")
