"""A long reduction onto a narrow product (k_gemm_narrow_k, csrc/gemm_narrow.cu) that finds little device memory: its partial products per group of threads, 19 MB, do not
fit, those per CTA do, and the product is made with them.  Without and with little room, against float64."""
import pytest

from test_gpu_scratch_limits import room_for

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,accumulate", [(32, 256, 0), (250, 32, 1)])
def test_partial_products(M, N, accumulate):
    import contextlib
    import torch
    import gpu_util as g
    K = 60001
    A, B, C0 = torch.randn(K, M, device="cuda"), torch.randn(K, N, device="cuda"), torch.randn(N, M, device="cuda")
    want = B.double().t() @ A.double() + (C0 if accumulate else 0)
    # the largest error of an fp32 sum of K products in 280 stretches of 215, four or two groups each, and of the stretches: at most 2 x 215 + 280 roundings of 2^-24
    bar = 710 * 2.0 ** -24 * (B.double().abs().t() @ A.double().abs() + C0.abs())
    C = C0.clone()
    for c in (g.ctx(), None):        # (a first time with all the memory: the kernels are loaded)
        with contextlib.nullcontext(c) if c else room_for(14) as ctx:
            C.copy_(C0)
            ctx.gemm(0, 1, M, N, K, A.data_ptr(), M, B.data_ptr(), N, C.data_ptr(), M, accumulate)
        assert ((C.double() - want).abs() <= bar).all()
