"""Context.fwd and .bwd as host/py/call.c implements them: the arguments that an entry point receives, the status checked, and what the C route does not take left to the
Python functions.  The entry points are callbacks; no GPU is needed."""
import ctypes as C
import gc
import weakref

import pytest

from dynet_b200 import build, capi

build.build_call()
from dynet_b200 import _call  # noqa: E402

P = C.POINTER(capi.DyTensor)
FWD, BWD = [P, C.c_int, P] + [C.c_void_p] * 3, [P, C.c_int, P, P, C.c_uint, P] + [C.c_void_p] * 3


class Native(capi.Context):
    """The class as its first instance leaves it; the Python functions record that they ran."""
    def _slow_fwd(self, *a, **kw):
        self.slow.append("fwd")
        return capi.Context.fwd(self, *a, **kw)

    def _slow_bwd(self, *a, **kw):
        self.slow.append("bwd")
        return capi.Context.bwd(self, *a, **kw)

    def check(self, rc):
        raise ValueError(rc)


@pytest.fixture(params=["read", "buffers"])
def ctx(request, monkeypatch):
    sample, other = capi.DyTensor(), capi.DyTensor()
    at = C.addressof(sample if request.param == "read" else other)     # (another's address: the layout is not the expected one)
    _call.setup(C.Structure, capi.DyTensor, C.c_void_p, C.sizeof(capi.DyTensor), sample, at)
    got, status = [], [0]
    fwd = C.CFUNCTYPE(C.c_int, *FWD)(lambda xs, n, fx, at, aux, h: (got.append(([xs[k].v for k in range(n)], fx[0].v, at and C.cast(at, C.POINTER(capi.DimAttrs))[0].dimension, aux, h)), status[0])[1])
    bwd = C.CFUNCTYPE(C.c_int, *BWD)(lambda xs, n, fx, d, i, dx, at, aux, h: (got.append(([xs[k].v for k in range(n)], fx[0].v, d[0].v, i, dx[0].v, at, aux, h)), status[0])[1])
    monkeypatch.setattr(Native, "fwd", _call.method(Native._slow_fwd, "_fwd", 6, "_hv", "check"), raising=False)
    monkeypatch.setattr(Native, "bwd", _call.method(Native._slow_bwd, "_bwd", 9, "_hv", "check"), raising=False)
    c = Native.__new__(Native)
    c.h, c._hv, c.got, c.slow, c.status, c.keep = None, 0x77, got, [], status, (fwd, bwd)
    c._fwd = {"softmax": (C.cast(fwd, C.c_void_p).value, b"xitavv", (None,) * 6)}
    c._bwd = {"softmax": (C.cast(bwd, C.c_void_p).value, b"xittitavv", (None,) * 9)}
    yield c
    _call.setup(C.Structure, capi.DyTensor, C.c_void_p, C.sizeof(capi.DyTensor), sample, C.addressof(sample))


def tensor(p):
    return capi.DyTensor.of(p, [4], 2)


def test_arguments(ctx):
    x, y, d = tensor(0x1000), tensor(0x2000), tensor(0x3000)
    ctx.fwd("softmax", [x, y], y, capi.DimAttrs(1), 0x7fff12345678)
    ctx.fwd("softmax", (x,), y)
    ctx.fwd("softmax", [], x, None, C.c_void_p(0x5000))
    ctx.fwd("softmax", None, x)
    ctx.bwd("softmax", [x], y, d, 3, x)
    ctx.bwd("softmax", [x, d], y, d, 0, x, None, 0x99)
    assert ctx.slow == [] and ctx.got == [
        ([0x1000, 0x2000], 0x2000, 1, 0x7fff12345678, 0x77), ([0x1000], 0x2000, None, None, 0x77), ([], 0x1000, None, 0x5000, 0x77), ([], 0x1000, None, None, 0x77),
        ([0x1000], 0x2000, 0x3000, 3, 0x1000, None, None, 0x77), ([0x1000, 0x3000], 0x2000, 0x3000, 0, 0x1000, None, 0x99, 0x77)]


def test_status(ctx):
    ctx.status[0] = 5
    with pytest.raises(ValueError, match="5"):
        ctx.fwd("softmax", [tensor(1)], tensor(2))
    assert len(ctx.got) == 1 and ctx.slow == []


def test_what_is_left_to_the_functions(ctx, monkeypatch):
    x, y = tensor(0x1000), tensor(0x2000)

    class Mine(capi.DyTensor):
        pass
    monkeypatch.setattr(capi, "_native_call", lambda *a: NotImplemented)
    monkeypatch.setattr(capi, "_ctypes_call", lambda name, args: 0)
    monkeypatch.setattr(capi, "_entry", lambda name: None)
    ctx.fwd("softmax", [x], y, aux=7)                      # by keyword
    ctx.fwd("softmax", [Mine()], y)                        # a type of the caller's own
    ctx.fwd("tanh", [x], y)                                # not called before
    ctx.bwd("softmax", [x], y, y, 0.5, x)
    ctx.fwd("softmax", [x], 0x10)
    with pytest.raises(TypeError):
        ctx.fwd("softmax", [x])
    assert ctx.got == [] and ctx.slow == ["fwd", "fwd", "fwd", "bwd", "fwd", "fwd"]


def test_bound_methods_keep_their_context(ctx):
    f, r = ctx.fwd, weakref.ref(ctx)
    f("softmax", [tensor(0x10)], tensor(0x20))
    assert ctx.got == [([0x10], 0x20, None, None, 0x77)] and r() is ctx and f.__self__ is ctx
    del f
    gc.collect()
