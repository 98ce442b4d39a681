"""Products of at most 64 rows with a reduction of more than 64 (k_gemm_slices, csrc/gemm_narrow.cu) against float64: slices of a piece that are empty, short or whole, one
piece and several, tiles of every number of columns per lane, a last column of its own, rows stored in fours and one by one."""
import pytest

from test_gpu_narrow import check

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("M,N,K,off", [
    (32, 256, 65, 0), (5, 300, 66, 0), (32, 257, 127, 0), (31, 521, 128, 1), (32, 521, 129, 0), (64, 300, 256, 0), (33, 1183, 131, 0), (60, 1185, 192, 3),
    (32, 2369, 68, 0), (32, 4737, 500, 0), (64, 4737, 200, 0), (61, 9473, 255, 0), (32, 37889, 72, 0), (29, 40000, 100, 2), (64, 38000, 130, 0)])
@pytest.mark.parametrize("tA,accumulate", [(0, False), (1, True), (0, True)])
def test_products(M, N, K, off, tA, accumulate):
    import gpu_util as g
    g.ctx()
    try:
        check(g, tA, 0, M, N, K, off, accumulate, 0.1)
    finally:
        g.release()
