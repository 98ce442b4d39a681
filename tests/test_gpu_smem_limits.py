"""A kernel's limit on dynamic shared memory belongs to the function, not to a launch: two host threads with a context each may launch it
with different sizes, so every launch has to ask for the same limit.  A fake of cudaFuncSetAttribute refuses a second value for a
function; products and layers of several sizes run over it, and two threads of them side by side give what they give alone."""
import os
import subprocess
import sys
from pathlib import Path

import pytest

pytestmark = pytest.mark.gpu
ROOT = Path(__file__).resolve().parent.parent

SHIM = r"""
#define _GNU_SOURCE
#include <cuda_runtime_api.h>
#include <dlfcn.h>
static const void* func[4096];
static int value[4096], n;
cudaError_t cudaFuncSetAttribute(const void* f, enum cudaFuncAttribute a, int v) {
  static cudaError_t (*real)(const void*, enum cudaFuncAttribute, int);
  if (!real) real = (cudaError_t (*)(const void*, enum cudaFuncAttribute, int))dlsym(RTLD_NEXT, "cudaFuncSetAttribute");
  if (a == cudaFuncAttributeMaxDynamicSharedMemorySize) {
    int k = 0;
    while (k < n && func[k] != f) ++k;
    if (k < n && value[k] != v) return cudaErrorInvalidValue;
    if (k == n && n < 4096) { func[n] = f; value[n++] = v; }
  }
  return real(f, a, v);
}
"""


def work(seed, device="cuda"):
    """Products and sequences whose kernels take more than 48 KB, in sizes that differ: their results."""
    import torch
    from dynet_b200 import capi
    stream = torch.cuda.Stream()
    out = []
    with torch.cuda.stream(stream):
        ctx = capi.Context(0, stream.cuda_stream)
        gen = torch.Generator("cuda").manual_seed(seed)
        rnd = lambda *s: torch.randn(*s, device=device, generator=gen) * 0.1   # noqa: E731
        T = lambda t, d, n=1: capi.DyTensor.of(t.data_ptr(), d, n)   # noqa: E731
        keep = []
        for M, N, K, tB in ((1000, 16, 2560, 0), (1000, 16, 1100, 0), (1000, 3, 6000, 0), (1000, 3, 4000, 0), (64, 30000, 256, 0), (64, 30000, 200, 0),
                            (250, 30000, 64, 0), (200, 30000, 60, 0), (64, 64, 20000, 1), (8, 8, 20000, 1), (32, 300, 20000, 1)):
            A, B, Cm = rnd(K, M), rnd(K, N) if tB else rnd(N, K), torch.empty(N, M, device=device)
            ctx.gemm(0, tB, M, N, K, A.data_ptr(), M, B.data_ptr(), N if tB else K, Cm.data_ptr(), M, 0)
            out.append(Cm)
            keep += [A, B]
        for H, B in ((1500, 7), (1030, 8), (1184, 8), (256, 1), (256, 32), (256, 45), (300, 30), (300, 200), (384, 9), (250, 70), (130, 600)):
            x, h0, Wx, Wh, b = rnd(8 * B, 16), rnd(B, H), rnd(16, 4 * H), rnd(H, 4 * H), rnd(4 * H)
            gates, cs, hs = (torch.empty(8 * B, k, device=device) for k in (4 * H, H, H))
            dh, dc, dx, db = rnd(8 * B, H), torch.zeros(8 * B, H, device=device), torch.zeros(8 * B, 16, device=device), torch.zeros(4 * H, device=device)
            w, at = ctx.wgrad_create(4 * H, 16, H, 8 * B), capi.LstmGatesAttrs(0, 0.0, 1.0)
            S = (T(gates, [4 * H], 8 * B), T(cs, [H], 8 * B), T(hs, [H], 8 * B))
            ctx.lstm_seq_fwd(T(x, [16], 8 * B), T(h0, [H], B), T(h0, [H], B), T(Wx, [4 * H, 16]), T(Wh, [4 * H, H]), T(b, [4 * H]), None, None, at, *S, w, 8)
            ctx.lstm_seq_bwd(T(x, [16], 8 * B), T(h0, [H], B), T(h0, [H], B), T(Wx, [4 * H, 16]), T(Wh, [4 * H, H]), None, None, at, *S, T(dh, [H], 8 * B),
                             T(dc, [H], 8 * B), T(dx, [16], 8 * B), None, None, T(db, [4 * H]), w, 8)
            stream.synchronize()
            ctx.wgrad_destroy(w)
            out += [gates, cs, hs, dh, dx, db]
            keep += [x, h0, Wx, Wh, b, dc]
        stream.synchronize()
        assert ctx.device_errors() == 0
    return [o.cpu() for o in out]


def test_every_launch_of_a_kernel_asks_for_the_same_limit(tmp_path):
    (tmp_path / "shim.c").write_text(SHIM)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-o", str(tmp_path / "shim.so"), str(tmp_path / "shim.c"), "-I/usr/local/cuda/include", "-ldl"])
    code = "import sys; sys.path.insert(0, 'tests'); import test_gpu_smem_limits as t; t.work(1)"
    p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, LD_PRELOAD=str(tmp_path / "shim.so")), capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-800:]


def test_two_threads_with_a_context_each():
    import threading
    import torch
    want = [work(s) for s in (1, 2)]
    got, errors = {}, []

    def run(k):
        try:
            for rep in range(4):
                got[k, rep] = work(k + 1)
        except Exception as e:
            errors.append(e)
    threads = [threading.Thread(target=run, args=(k,)) for k in range(2)]
    for t in threads:
        t.start()
    for t in threads:
        t.join()
    assert not errors, errors
    for (k, _), outs in got.items():
        assert all(torch.equal(p, q) for p, q in zip(outs, want[k]))
