"""An accumulator's first clear is ordered before the work of the context that creates it.  The context is on a non-blocking stream and the
accumulator's left planes are large: a clear that is not on that stream is still busy with them when the first columns are pushed, and takes
the right planes after that."""
import pytest

pytestmark = pytest.mark.gpu


def test_clear_is_ordered_on_the_contexts_stream():
    import torch
    from dynet_b200 import capi
    M, N, K = 4096, 256, 256
    stream = torch.cuda.Stream()
    with torch.cuda.stream(stream):
        ctx = capi.Context(0, stream.cuda_stream)
        a, b, C = torch.randn(K, M, device="cuda"), torch.randn(K, N, device="cuda"), torch.zeros(N, M, device="cuda")
        for _ in range(3):
            w = ctx.wgrad_create(M, N, 0, 60000)
            ctx.wgrad_push(w, K, a.data_ptr(), M, b.data_ptr(), N)
            torch.cuda.synchronize()
            C.zero_()
            ctx.wgrad_flush(w, C.data_ptr(), M)
            stream.synchronize()
            ctx.wgrad_destroy(w)
            want = b.double().t() @ a.double()
            assert float((C.double() - want).abs().max()) < 1e-4 * float(want.abs().max())
    assert ctx.device_errors() == 0
