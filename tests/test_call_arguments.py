"""How a call of capi.Context hands its arguments over: through the extension and through ctypes alike, and what neither takes is refused
before anything is called.  The entry point is a callback that records what it gets; no GPU is needed."""
import ctypes as C
import subprocess
import sys
import types
from pathlib import Path

import pytest

from dynet_b200 import build, capi

build.build_call()
FWD = [C.POINTER(capi.DyTensor), C.c_int, C.POINTER(capi.DyTensor)] + [C.c_void_p] * 3


def tensor(p, dims, bd=1):
    return capi.DyTensor.of(p, dims, bd)


@pytest.fixture(params=["extension", "ctypes"])
def ctx(request, monkeypatch):
    """A context over fake entry points; ctx.got lists what they received."""
    got = []

    def fake(argtypes, read):
        return C.CFUNCTYPE(C.c_int, *argtypes)(lambda *a: got.append(read(*a)) or 0)
    fwd = fake(FWD, lambda xs, n, fx, attrs, aux, h: ([xs[k].v for k in range(n)], bool(xs), fx[0].v, fx[0].bd,
                                                      C.cast(attrs, C.POINTER(capi.DimAttrs))[0].dimension if attrs else None, aux, h))
    lstm = fake([C.POINTER(capi.DyTensor)] * 8 + [C.POINTER(capi.LstmGatesAttrs)] + [C.POINTER(capi.DyTensor)] * 3 + [C.c_void_p],
                lambda *a: ([bool(t) and t[0].v for t in a[:8] + a[9:12]], a[8][0].forget_gate_bias, a[12]))
    flush = fake([C.c_void_p, C.c_void_p, C.c_uint32, C.c_void_p, C.c_uint32, C.c_void_p], lambda *a: a)
    lookup = fake([C.c_uint, C.POINTER(C.c_uint32)] + [C.c_void_p] * 3 + [C.c_uint, C.c_uint, C.c_void_p],
                  lambda n, ids, *a: (n, [ids[k] for k in range(n)] if ids else None) + a)
    fakes = types.SimpleNamespace(dyb200_softmax_fwd=fwd, dyb200_vanilla_lstm_fwd_fused=lstm, dyb200_wgrad_flush=flush,
                                  dyb200_lookup_accumulate_grads=lookup)
    monkeypatch.setattr(capi, "lib", lambda: fakes)
    monkeypatch.setattr(capi, "_ENTRIES", {})
    if request.param == "ctypes":
        monkeypatch.setattr(capi, "_native_call", lambda *a: NotImplemented)
    c = capi.Context.__new__(capi.Context)
    c.h, c._hv, c._fwd, c._bwd, c.got = None, 0x77, {}, {}, got
    return c


def test_node_arguments(ctx):
    x, y = tensor(0x1000, [4], 2), tensor(0x2000, [4], 3)
    ctx.fwd("softmax", [x, y], y, capi.DimAttrs(1), 0x7fff12345678)
    ctx.fwd("softmax", (x,), y)
    ctx.fwd("softmax", [], x, None, C.c_void_p(0x5000))
    ctx.fwd("softmax", None, x)
    assert ctx.got == [([0x1000, 0x2000], True, 0x2000, 3, 1, 0x7fff12345678, 0x77), ([0x1000], True, 0x2000, 3, None, None, 0x77),
                       ([], False, 0x1000, 2, None, 0x5000, 0x77), ([], False, 0x1000, 2, None, None, 0x77)]


def test_arguments_that_only_ctypes_converts(ctx):
    class Mine(capi.DyTensor):
        pass
    m = Mine()
    m.v, m.bd = 0x3000, 9
    many = [tensor(0x100 + k, [1]) for k in range(300)]            # more than the extension's arena holds
    ctx.fwd("softmax", many, m)
    ctx.lookup_accumulate_grads([3, 1, 4], 0x10, 0x20, 0x30, 8, 99)
    ctx.lookup_accumulate_grads([], 0x10, 0x20, 0x30, 8, 99, n=2)
    assert ctx.got == [([t.v for t in many], True, 0x3000, 9, None, None, 0x77), (3, [3, 1, 4], 0x10, 0x20, 0x30, 8, 99, 0x77),
                       (2, None, 0x10, 0x20, 0x30, 8, 99, 0x77)]


def test_layer_arguments(ctx):
    ts = [tensor(0x1000 + k, [2]) for k in range(9)]
    at = capi.LstmGatesAttrs(0, 0.0, 1.5)
    ctx.lstm_fwd_fused(*ts[:6], None, None, at, *ts[6:])
    ctx.wgrad_flush(C.c_void_p(0x9000), 0xa000, 3)
    assert ctx.got == [([0x1000 + k for k in range(6)] + [False, False] + [0x1006, 0x1007, 0x1008], 1.5, 0x77), (0x9000, 0xa000, 3, None, 0, 0x77)]


# a wild pointer must not reach an entry point: each of these is refused (in a child process: it would read that address otherwise)
REFUSED = ["fwd('softmax', [t], 0x10)", "fwd('softmax', [t], None)", "fwd('softmax', [t], at)", "fwd('softmax', [0x10], t)", "fwd('softmax', [None], t)",
           "fwd('softmax', 0x10, t)", "fwd('softmax', [t], t, 0x10)", "fwd('softmax', [t], t, None, 1.5)", "bwd('softmax', [t], t, 0x10, 0, t)",
           "bwd('softmax', [t], t, t, 0, None)", "bwd('softmax', [t], t, t, 0.5, t)", "lstm_fwd_fused(0x10, t, t, t, t, t, None, None, at, t, t, t)",
           "lstm_fwd_fused(t, t, t, t, t, t, None, None, None, t, t, t)", "lstm_fwd_fused(t, t, t, t, t, t, None, None, t, t, t, t)",
           "lstm_fwd_fused(t, t, t, t, t, t, None, None, 0x10, t, t, t)", "_run('dyb200_wgrad_flush', 0x10)", "wgrad_flush(1.5, 0x10, 1)"]


@pytest.mark.parametrize("call", REFUSED)
def test_refused(call):
    code = """
import ctypes as C
from dynet_b200 import capi
c = capi.Context.__new__(capi.Context)
c.L, c.h, c._hv, c._fwd, c._bwd = capi.lib(), None, None, {}, {}
t, at = capi.DyTensor.of(None, [2], 1), capi.LstmGatesAttrs(0, 0.0, 1.0)
try:
    c.%s
except (TypeError, C.ArgumentError):
    print("refused")
""" % call
    p = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True)
    assert p.returncode == 0 and p.stdout.strip() == "refused", (p.returncode, p.stdout, p.stderr[-500:])


def test_importing_the_bindings_maps_nothing():
    """The reference arm of the benchmark imports them for the synthetic batch and the parameter shapes."""
    code = """
import bench
from dynet_b200 import lm, tagger
lm.synthetic_batch(dict(V=20, E=8, H=8, L=1, T=2, B=3), seed=1, dropout=0.0), lm.param_shapes(20, 8, 8, 1), tagger.param_shapes(20, 8, 8, 4, 3)
print([l.split("/")[-1].strip() for l in open("/proc/self/maps") if "dynet_b200" in l])
"""
    p = subprocess.run([sys.executable, "-c", code], cwd=Path(__file__).resolve().parent.parent, capture_output=True, text=True)
    assert p.returncode == 0 and p.stdout.strip() == "[]", (p.stdout, p.stderr[-500:])
