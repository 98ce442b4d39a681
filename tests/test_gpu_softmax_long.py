"""Few long columns (a cluster of CTAs per column) and the lengths and column counts around it, against the oracle."""
import numpy as np
import pytest

from util import TOL_REDUCE, assert_close, randn, rng

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("rows,bd", [(2049, 1), (4097, 18), (10000, 1), (32767, 2), (32768, 3), (32769, 2), (5001, 40)])
def test_long_columns(oracle, rows, bd):
    import gpu_util as g
    from dynet_b200 import capi
    r = rng(rows + bd)
    x = randn(r, bd, rows, scale=3.0)
    ids = r.integers(0, rows, bd).astype(np.uint32)
    ids[0] = rows - 1
    x_ = g.dev(x)
    y_ = g.dev(np.zeros_like(x))
    g.ctx().fwd("softmax", [g.T(x_, [rows], bd)], g.T(y_, [rows], bd), capi.DimAttrs(0))
    want = oracle.softmax_fwd(x.reshape(bd, 1, rows), 0).reshape(bd, rows)
    assert_close(g.host(y_), want, TOL_REDUCE, floor=1e-7, what="softmax")
    aux = g.dev(np.zeros(2 * bd, np.float32))
    g.ctx().fwd("log_softmax", [g.T(x_, [rows], bd)], g.T(y_, [rows], bd), None, aux.data_ptr())
    assert_close(g.host(y_), oracle.log_softmax_fwd(x.reshape(bd, 1, rows)).reshape(bd, rows), TOL_REDUCE, floor=1.0, what="log_softmax")
    loss_, paux = g.dev(np.zeros(bd, np.float32)), g.dev(np.zeros(3 * bd, np.float32))
    keep, p = g.u32(ids)
    g.ctx().fwd("pickneglogsoftmax", [g.T(x_, [rows], bd)], g.T(loss_, [1], bd), capi.PickAttrs(p, bd), paux.data_ptr())
    assert_close(g.host(loss_), oracle.pnls_fwd(x, ids)[0], TOL_REDUCE, floor=1.0, what="pnls")
    assert g.ctx().device_errors() == 0
    g.release()


def test_long_columns_beside_other_work():
    """The CTAs of a cluster start unevenly on a GPU that is busy with another stream: the same bits as on a quiet one."""
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    rows, bd = 10000, 3
    x_ = g.dev(randn(rng(3), bd, rows, scale=3.0))
    y_ = torch.empty(200, bd, rows, device="cuda")
    aux = torch.empty(2 * bd, device="cuda")
    a, other = torch.randn(4096, 4096, device="cuda"), torch.cuda.Stream()
    other.wait_stream(torch.cuda.current_stream())
    for k in range(200):
        if k % 5 == 1:
            with torch.cuda.stream(other):
                a = a * 1.0001 + 0.5
        g.ctx().fwd("log_softmax", [g.T(x_, [rows], bd)], g.T(y_[k], [rows], bd), None, aux.data_ptr())
    torch.cuda.synchronize()
    assert all(torch.equal(y_[0], y_[k]) for k in range(200))
    assert g.ctx().device_errors() == 0
    g.release()


@pytest.mark.parametrize("rows", [4100, 8192, 8196, 12288, 12292])
def test_columns_in_registers(rows):
    """Many columns at the lengths where a thread's share of a column changes, with entries of -inf, against float64.  Bar: log-probabilities
    down to -30 from fp32 exponents, an ulp of 30 and of the sum; probabilities to 1e-5 of themselves."""
    import torch
    import gpu_util as g
    from dynet_b200 import capi
    bd = 150
    gen = torch.Generator("cuda").manual_seed(rows)
    x = torch.randn(bd, rows, device="cuda", generator=gen) * 3.0
    x[:, 7::11] = -float("inf")
    x[3] -= 80.0
    y, ly, loss = torch.empty_like(x), torch.empty_like(x), torch.empty(bd, device="cuda")
    aux, paux = torch.empty(2 * bd, device="cuda"), torch.zeros(3 * bd, device="cuda")
    ids = torch.randint(0, rows // 11, (bd,), device="cuda", generator=gen) * 11
    paux[2 * bd:].view(torch.int32).copy_(ids.int())
    g.ctx().fwd("softmax", [g.T(x, [rows], bd)], g.T(y, [rows], bd), capi.DimAttrs(0))
    g.ctx().fwd("log_softmax", [g.T(x, [rows], bd)], g.T(ly, [rows], bd), None, aux.data_ptr())
    g.ctx().fwd("pickneglogsoftmax", [g.T(x, [rows], bd)], g.T(loss, [1], bd), capi.PickAttrs(None, bd), paux.data_ptr())
    want = torch.log_softmax(x.double(), dim=1)
    live = torch.isfinite(want)
    assert bool(((y.double() - want.exp()).abs() <= 1e-5 * want.exp()).all())
    assert bool((ly[live] - want[live]).abs().max() <= 1.6e-5) and bool((ly[~live] == -float("inf")).all())
    assert bool((loss.double() + want[torch.arange(bd), ids]).abs().max() <= 1.6e-5)
    assert g.ctx().device_errors() == 0
    g.release()
