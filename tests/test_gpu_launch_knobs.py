"""nblks and nthreads limit the grid of a fetch of device rows: one block of one warp returns the
same rows in many times the time."""
import pytest
import torch

pytestmark = pytest.mark.gpu


def best_ms(fn):
    fn()
    times = []
    for _ in range(5):
        a, b = torch.cuda.Event(enable_timing=True), torch.cuda.Event(enable_timing=True)
        a.record()
        fn()
        b.record()
        b.synchronize()
        times.append(a.elapsed_time(b))
    return min(times)


@pytest.mark.parametrize("indexed", [False, True])
@pytest.mark.parametrize("v", [33, 100])
def test_a_small_grid_is_honoured(v, indexed):
    import invariantbitpacking_b200 as ibp
    g = torch.Generator(device="cuda")
    g.manual_seed(v)
    n = 100_000
    src = torch.randint(-2**62, 2**62, (n, v), generator=g, device="cuda") & 0xFFFFFFFF
    mask, bitval = ibp.preprocess(src, 0.9)
    comp = src.clone()
    bitmask = ibp.compress_inplace(comp, mask, bitval)
    idx = torch.randint(0, n, (30_000,), generator=g, device="cuda") if indexed else None
    want = src if idx is None else src[idx]
    out = torch.empty_like(want)

    def fetch(nblks, nthreads):
        ibp.decompress_fetch(comp, mask, bitval, bitmask, "cuda", v, idx, nblks, nthreads,
                             output_tensor=out)

    out.zero_()
    whole = best_ms(lambda: fetch(None, None))
    assert torch.equal(out, want)
    for nblks, nthreads, ratio in ((1, 32, 20), (1, None, 8), (2, 64, 8), (10**6, 1000, 0)):
        out.zero_()
        ms = best_ms(lambda: fetch(nblks, nthreads))
        assert torch.equal(out, want)
        assert ms > ratio * whole, (nblks, nthreads, ms, whole)
