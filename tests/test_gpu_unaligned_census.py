"""preprocess of datasets that start anywhere in a 16-byte block: equal masks (against the CPU
oracle), few and many rows, rows narrower than the words before the boundary, host rows; and a census
in about an aligned dataset's time."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from test_gpu_match_chunks import INT, rows_of

pytestmark = pytest.mark.gpu


def put(x, offset, host):
    flat = torch.from_numpy(x.reshape(-1))
    buf = torch.empty(flat.numel() + offset, dtype=flat.dtype, pin_memory=True)
    if not host:
        buf = buf.cuda()
    buf[offset:].copy_(flat)
    return buf[offset:].view(*x.shape)


@pytest.mark.parametrize("host", [False, True])
@pytest.mark.parametrize("wb,v,n", [
    (1, 1, 3), (1, 1, 17), (1, 1, 400), (1, 3, 1), (1, 5, 1000), (1, 16, 50), (1, 65, 333),
    (2, 1, 9), (2, 3, 700), (2, 8, 100), (2, 129, 90), (4, 1, 3), (4, 3, 999), (4, 4, 1),
    (4, 64, 300), (4, 65, 5), (8, 1, 1), (8, 1, 500), (8, 33, 301), (8, 64, 300), (8, 130, 64)])
def test_masks_of_unaligned_data_vs_oracle(oracle, wb, v, n, host):
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(100 * v + 10 * wb + n)
    x = rows_of(rng, n, v, wb)
    for offset in sorted({1, 2, 16 // wb - 1}):
        t = put(x, offset, host)
        for thr in (None, 0.7):
            om, ob, _ = oracle.preprocess(x, thr)
            m, b = ibp.preprocess(t, thr)
            torch.cuda.synchronize()
            assert np.array_equal(m.cpu().numpy(), om.view(INT[wb])), (offset, thr)
            assert np.array_equal(b.cpu().numpy(), ob.view(INT[wb])), (offset, thr)


@pytest.mark.parametrize("wb,v", [(1, 64), (2, 33), (4, 2), (4, 33), (8, 1), (8, 64)])
def test_unaligned_data_is_about_as_fast(wb, v):
    import invariantbitpacking_b200 as ibp
    n = (192 << 20) // (v * wb)
    buf = torch.randint(-128, 128, (n * v * wb + 16,), dtype=torch.int8, device="cuda")
    buf = buf.view(torch.from_numpy(np.zeros(1, INT[wb])).dtype)


    def census_us(t):
        """GPU time of the census kernels alone: the pass after it reads such rows in smaller pieces."""
        ibp.preprocess(t, 0.9)
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            for _ in range(5):
                ibp.preprocess(t, 0.9)
            torch.cuda.synchronize()
        took = [e.self_device_time_total for e in prof.key_averages() if "census" in e.key]
        assert took
        return sum(took) / 5

    aligned = census_us(buf[:n * v].view(n, v))
    off = census_us(buf[1:n * v + 1].view(n, v))
    assert off < 1.5 * aligned, (off, aligned)
