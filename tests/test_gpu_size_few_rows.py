"""get_compress_size of few long rows, which go a row to a warp or to a block, against the CPU oracle
at the edges of both rules (148 SMs: 1184, 4736, 7104 and 18944 rows), with an index and bad positions
and with the running total; and in about the time the same bytes take as many shorter rows."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

from test_gpu_match_chunks import INT, put, rows_of

pytestmark = pytest.mark.gpu


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("wb,v,n", [
    (1, 129, 1184), (1, 600, 1185), (1, 2048, 40), (2, 257, 1300), (2, 1030, 30), (4, 129, 1185),
    (4, 132, 7104), (4, 132, 7105), (4, 131, 18945), (4, 520, 1184), (4, 8300, 35), (4, 60001, 3),
    (8, 65, 1185), (8, 66, 1184), (8, 260, 1300), (8, 4096, 12), (8, 5000, 1)])
def test_sizes_vs_oracle(oracle, wb, v, n, offset):
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(100 * v + 10 * wb + n)
    # few distinct rows where there are many, so that the values are made quickly
    x = rows_of(rng, min(n, 300), v, wb)
    x = np.ascontiguousarray(x[rng.integers(0, len(x), n)])
    om, ob, _ = oracle.preprocess(x[:300], 0.75)
    dm, db = torch.from_numpy(om.view(INT[wb])).cuda(), torch.from_numpy(ob.view(INT[wb])).cuda()
    t = put(x, offset)
    want = oracle.compress_size(x, om, ob)
    total = torch.full((1,), 5, dtype=torch.int64, device="cuda")
    sizes = ibp.get_compress_size(t, dm, db, None, total)
    torch.cuda.synchronize()
    assert np.array_equal(sizes.cpu().numpy(), want)
    assert int(total) == 5 + int(want.sum())
    idx = rng.integers(0, n, 1500 if n > 300 else 45)
    bad = rng.random(len(idx)) < 0.1
    total.zero_()
    sizes = ibp.get_compress_size(t, dm, db, torch.from_numpy(np.where(bad, n, idx)).cuda(), total)
    torch.cuda.synchronize()
    assert np.array_equal(sizes.cpu().numpy(), np.where(bad, 0, want[idx]))
    assert int(total) == int(want[idx][~bad].sum())


@pytest.mark.parametrize("wb,v,rows", [(4, 60000, 600), (8, 8000, 1000)])
def test_few_long_rows_take_about_as_long_as_many(wb, v, rows):
    import invariantbitpacking_b200 as ibp
    x = torch.randint(-128, 128, (rows * v * wb,), dtype=torch.int8, device="cuda")
    x = x.view(torch.from_numpy(np.zeros(1, INT[wb])).dtype)
    m = torch.randint(-128, 128, (v * wb,), dtype=torch.int8, device="cuda").view(x.dtype)

    def size_us(t, k):
        """GPU time of the size kernel."""
        ibp.get_compress_size(t, m[:k], m[:k])
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            for _ in range(6):
                ibp.get_compress_size(t, m[:k], m[:k])
            torch.cuda.synchronize()
        return min(e.device_time for e in prof.events()
                   if "size_kernel" in e.name and e.device_type.name == "CUDA")

    many = size_us(x.view(-1, v // 100), v // 100)
    few = size_us(x.view(rows, v), v)
    assert few < 2 * many, (few, many)
