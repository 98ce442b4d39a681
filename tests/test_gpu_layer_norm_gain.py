"""Layer norm's gain gradient at the edges of `k_layer_norm_dg` (csrc/norm.cu: columns of 1024 - 4096 elements; clusters of eight CTAs, three CTAs per
SM) and beside them, against float64.  Bar: a term up (x - mean) / sigma carries the roundings of a tree over n values in mean (at most 14, in
units of |up| as |x| / sigma is about one) and in sigma (at most 20) and five of its own, the sums over a CTA's columns, a cluster, a warp of
partials and the warps at most 24 more: 2^-24 times 14 |up| + 50 |up x_hat|, summed over the columns, and one rounding of what was there."""
import pytest

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("n,cols", [(1020, 5), (1024, 1), (1024, 444), (1028, 9), (2500, 445), (4092, 1300), (4096, 7), (4096, 1024), (4097, 33), (4100, 33)])
def test_gain_gradient(n, cols):
    import torch
    import gpu_util as g
    gen = torch.Generator("cuda").manual_seed(n + cols)
    x, up = (torch.randn(cols, n, device="cuda", generator=gen) for _ in range(2))
    gain, bias, d0 = (torch.randn(n, device="cuda", generator=gen) for _ in range(3))
    y, d = torch.empty_like(x), d0.clone()
    xs = [g.T(x, [n], cols), g.T(gain, [n], 1), g.T(bias, [n], 1)]
    g.ctx().bwd("layer_norm", xs, g.T(y, [n], cols), g.T(up, [n], cols), 1, g.T(d, [n], 1))
    torch.cuda.synchronize()
    xd, ud = x.double(), up.double()
    c = xd - xd.mean(dim=1, keepdim=True)
    hat = c / ((c * c).mean(dim=1, keepdim=True).sqrt() + 1e-8)
    want = d0.double() + (ud * hat).sum(dim=0)
    bar = 2.0 ** -24 * ((14 * ud.abs() + 50 * (ud * hat).abs()).sum(dim=0) + 2 * want.abs())
    assert bool(((d - want).abs() <= bar).all())
