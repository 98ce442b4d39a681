"""The scatter-add's merge of sorted runs (4096 ids each, eight searched side by side) and its sum over the chunks of 32 of a frequent id (above 32 chunks the eight warps of
a CTA take a stretch each), at the edges of both.  Values that are multiples of 2^-10 below 4 in magnitude: every sum is exact in fp32, so the result is that of any order."""
import pytest

pytestmark = pytest.mark.gpu

N = [31, 32, 33, 1055, 1056, 1057, 1089, 4096, 4097, 8192, 8193, 32768, 32769, 36864, 36865, 69000]


@pytest.mark.parametrize("kind", ["one", "two", "few", "many", "distinct", "wide"])
@pytest.mark.parametrize("E", [4, 128, 132, 512])
def test_sums(E, kind):
    import torch
    import gpu_util as g
    ctx = g.ctx()
    for n in N if E < 512 else N[:12:3]:
        gen = torch.Generator("cuda").manual_seed(n)
        V = {"one": 3, "two": 2, "few": 40, "many": 3000, "distinct": n + 5, "wide": (1 << 20) + 7}[kind]     # (from 2^20 rows on the ids are sorted by 64-bit keys)
        if kind == "wide" and E > 4:
            V = 5000
        ids = torch.randint(0, V, (n,), device="cuda", generator=gen)
        if kind == "one":
            ids[:] = 1
        if kind == "distinct":
            ids = torch.randperm(V, device="cuda", generator=gen)[:n]
        grad = torch.randint(-2048, 2049, (n, E), device="cuda", generator=gen).float() / 1024
        table = torch.randint(-2048, 2049, (V, E), device="cuda", generator=gen).float() / 1024
        want = table.double().index_add_(0, ids, grad.double()).float()
        ids32 = ids.to(torch.int32)
        ctx.lookup_accumulate_grads([], ids32.data_ptr(), grad.data_ptr(), table.data_ptr(), E, V, n=n)
        assert torch.equal(table, want), "n = %d: %d of %d values" % (n, int((table != want).sum()), want.numel())
    assert ctx.device_errors() == 0


@pytest.mark.parametrize("chunks_per_sm", [6, 16, 24])
@pytest.mark.parametrize("E,V", [(128, 3000), (200, 400), (128, 0)])   # (V = 0: no repeats)
def test_sums_where_the_form_changes(chunks_per_sm, E, V):
    """Both sides of the lines up to which chunks go by shared memory: whole chunks and one id more, on (chunk, slice) pairs of the whole GPU."""
    import torch
    import gpu_util as g
    ctx = g.ctx()
    slices = (E + 127) // 128
    at = 32 * (chunks_per_sm * torch.cuda.get_device_properties(0).multi_processor_count // slices)
    for n in (at, at + 1):
        gen = torch.Generator("cuda").manual_seed(n)
        rows = V or n
        ids = torch.randint(0, rows, (n,), device="cuda", generator=gen) if V else torch.randperm(n, device="cuda", generator=gen)
        grad = torch.randint(-2048, 2049, (n, E), device="cuda", generator=gen).float() / 1024
        table = torch.randint(-2048, 2049, (rows, E), device="cuda", generator=gen).float() / 1024
        want = table.double().index_add_(0, ids, grad.double()).float()
        ids32 = ids.to(torch.int32)
        ctx.lookup_accumulate_grads([], ids32.data_ptr(), grad.data_ptr(), table.data_ptr(), E, rows, n=n)
        assert torch.equal(table, want)
    assert ctx.device_errors() == 0
