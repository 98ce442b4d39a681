"""Weight normalisation above one CTA's size (csrc/norm.cu), where a thread has less than one, one, four and more vectors of the tensor, and off 16 bytes,
against float64.  Bar: |w|^2 and w . dy are trees of at most 40 roundings (a thread's vectors, a warp, a block, the blocks' sums), so they err by
40 2^-24 of the sum of magnitudes; the root halves that, and the quotient, the products and the sum that follow add six."""
import pytest

pytestmark = pytest.mark.gpu
STEP = 4 * 592 * 256   # floats that four CTAs on each of 148 SMs take at a time, a vector per thread


@pytest.mark.parametrize("n", [16385, 16388, STEP - 4, STEP, STEP + 4, 4 * STEP - 1, 4 * STEP, 4 * STEP + 5, 9 * STEP + 3])
@pytest.mark.parametrize("offset", [0, 1])
def test_sizes(n, offset):
    import torch
    import gpu_util as g
    gen = torch.Generator("cuda").manual_seed(n)
    w, dy, d0 = (torch.randn(n + offset, device="cuda", generator=gen)[offset:] for _ in range(3))
    gain, dg0 = (torch.randn(1, device="cuda", generator=gen) for _ in range(2))
    y, d, dg = torch.empty(n + offset, device="cuda")[offset:], torch.empty(n + offset, device="cuda")[offset:], dg0.clone()
    d.copy_(d0)
    xs = [g.T(w, [n], 1), g.T(gain, [1], 1)]
    ctx = g.ctx()
    ctx.fwd("weight_norm", xs, g.T(y, [n], 1))
    ctx.bwd("weight_norm", xs, g.T(y, [n], 1), g.T(dy, [n], 1), 0, g.T(d, [n], 1))
    ctx.bwd("weight_norm", xs, g.T(y, [n], 1), g.T(dy, [n], 1), 1, g.T(dg, [1], 1))
    torch.cuda.synchronize()
    u, wd, dd = 2.0 ** -24, w.double(), dy.double()
    ss, dot, mag = (wd * wd).sum(), (wd * dd).sum(), (wd * dd).abs().sum()
    sc = gain.double() / ss.sqrt()
    assert bool(((y - wd * sc).abs() <= 26 * u * (wd * sc).abs()).all())
    want = d0.double() + dd * sc - wd * sc * dot / ss
    bar = u * (26 * (dd * sc).abs() + 72 * (wd * sc).abs() * mag / ss + 40 * (wd * sc * dot / ss).abs() + 2 * want.abs())
    assert bool(((d - want).abs() <= bar).all())
    want = dg0.double() + dot / ss.sqrt()
    assert bool((dg - want).abs() <= u * (46 * mag / ss.sqrt() + 26 * (dot / ss.sqrt()).abs() + 2 * want.abs()))
