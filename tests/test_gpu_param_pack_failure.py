"""A parameter's split planes are made in the launch that makes the other operand's. A fake of cudaLaunchKernelExC refuses that launch: the call reports it, and the
next one makes the planes again instead of multiplying with those of the parameter before its update."""
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
int refuse;   /* launches to refuse */
static __thread cudaError_t pending;
cudaError_t cudaLaunchKernelExC(const cudaLaunchConfig_t* c, const void* f, void** a) {
  static cudaError_t (*real)(const cudaLaunchConfig_t*, const void*, void**);
  if (!real) real = (cudaError_t (*)(const cudaLaunchConfig_t*, const void*, void**))dlsym(RTLD_NEXT, "cudaLaunchKernelExC");
  if (refuse) { --refuse; return pending = cudaErrorLaunchOutOfResources; }
  return real(c, f, a);
}
cudaError_t cudaGetLastError(void) {
  static cudaError_t (*real)(void);
  if (!real) real = (cudaError_t (*)(void))dlsym(RTLD_NEXT, "cudaGetLastError");
  const cudaError_t e = pending;
  pending = cudaSuccess;
  return e ? e : real();
}
"""


def work(shim):
    import ctypes
    import torch
    from dynet_b200 import capi
    refuse = ctypes.c_int.in_dll(ctypes.CDLL(shim), "refuse")
    ctx = capi.Context(0, torch.cuda.current_stream().cuda_stream)
    ctx.param_cache(True)
    T = lambda t, d, n=1: capi.DyTensor.of(t.data_ptr(), d, n)   # noqa: E731
    M, K, N = 512, 400, 600
    w, x, b, y = torch.randn(K, M, device="cuda"), torch.randn(N, K, device="cuda"), torch.zeros(M, device="cuda"), torch.empty(N, M, device="cuda")
    call = lambda: ctx.fwd("affine_transform", [T(b, [M]), T(w, [M, K]), T(x, [K], N)], T(y, [M], N), capi.AffineAttrs(1))   # noqa: E731
    for rep in range(2):                     # planes that are not there yet, and planes of the values before an update
        if rep:
            call()
            w.copy_(torch.randn(K, M, device="cuda"))
            ctx.params_changed()
        refuse.value = 1
        try:
            call()
        except capi.Dyb200Error:
            pass
        else:
            raise AssertionError("the refused launch was not reported")
        assert refuse.value == 0
        call()
        want = x.double() @ w.double()
        # (a product of split operands: less than 2^-20 of the sum of magnitudes)
        assert ((y.double() - want).abs() <= 2.0 ** -20 * (x.double().abs() @ w.double().abs()) + 2.0 ** -23 * want.abs()).all()
    assert ctx.device_errors() == 0


def test_planes_whose_launch_was_refused_are_made_again(tmp_path):
    shim = str(tmp_path / "shim.so")
    (tmp_path / "shim.c").write_text(SHIM)
    subprocess.check_call(["gcc", "-shared", "-fPIC", "-o", shim, str(tmp_path / "shim.c"), "-I/usr/local/cuda/include", "-ldl"])
    code = "import sys; sys.path.insert(0, 'tests'); import test_gpu_param_pack_failure as t; t.work(%r)" % shim
    p = subprocess.run([sys.executable, "-c", code], cwd=ROOT, env=dict(os.environ, LD_PRELOAD=shim), capture_output=True, text=True)
    assert p.returncode == 0, p.stderr[-800:]
