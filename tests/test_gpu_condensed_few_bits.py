"""Long condensed device rows whose columns keep few bits, one to a warp: they come back, with words off
the pattern and without, and take less time than rows whose columns keep many."""
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

pytestmark = pytest.mark.gpu


def rows_of(g, n, v, wb, kept):
    """Every word keeps its low `kept` bits."""
    bits = 8 * wb
    keep = (1 << kept) - 1
    top = 1 << (bits - 1)
    base = torch.randint(-top, top - 1, (v,), generator=g, device="cuda") & ~keep
    x = base | torch.randint(0, keep + 1, (n, v), generator=g, device="cuda")
    mask = torch.full((v,), ~keep, device="cuda")
    dtype = torch.int64 if wb == 8 else torch.int32
    return x.to(dtype), mask.to(dtype), base.to(dtype)


@pytest.mark.parametrize("stray", [False, True])
@pytest.mark.parametrize("kept", [0, 1, 4, 5])
@pytest.mark.parametrize("wb,v,n", [(4, 129, 40), (4, 1000, 30), (4, 5000, 9), (8, 65, 50),
                                    (8, 257, 20), (8, 2000, 12), (8, 12000, 3)])
def test_rows_come_back(wb, v, n, kept, stray):
    import invariantbitpacking_b200 as ibp
    g = torch.Generator(device="cuda")
    g.manual_seed(10 * v + kept)
    x, m, b = rows_of(g, n, v, wb, kept)
    if stray:
        x = torch.where(torch.rand((n, v), generator=g, device="cuda") < 0.1, ~x, x)
    words, offs = ibp.compress_condensed(x, m, b)
    idx = torch.randint(0, n, (3 * n,), generator=g, device="cuda")
    for k in (None, idx, idx[:1]):
        out = ibp.decompress_fetch_condensed(words, offs, m, b, v, "cuda", k, check=True)
        assert torch.equal(out, x if k is None else x[k])


def test_few_kept_bits_take_less_time():
    import invariantbitpacking_b200 as ibp
    g = torch.Generator(device="cuda")
    g.manual_seed(1)

    def fetch_us(kept):
        x, m, b = rows_of(g, 500, 12000, 8, kept)
        words, offs = ibp.compress_condensed(x, m, b)

        def fetch():
            ibp.decompress_fetch_condensed(words, offs, m, b, 12000, "cuda")

        fetch()
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            for _ in range(5):
                fetch()
            torch.cuda.synchronize()
        took = [e.self_device_time_total for e in prof.key_averages() if "fetch_kernel" in e.key]
        assert took
        return sum(took) / 5

    few, many = fetch_us(2), fetch_us(26)
    assert few < 0.8 * many, (few, many)
