"""Condensed device rows of one to four chunks of 32 columns, every row with words off the pattern, so
that each takes its offsets and its length from a prefix sum: they come back, rows whose bitmap claims
more than they hold are reported and left alone, and short rows take less time than long ones."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

pytestmark = pytest.mark.gpu

INT = {4: np.int32, 8: np.int64}
UINT = {4: np.uint32, 8: np.uint64}


def rows_of(rng, n, v, wb):
    m = rng.integers(0, 2**64, v, dtype=np.uint64)
    base = rng.integers(0, 2**64, v, dtype=np.uint64) & m
    noise = rng.integers(0, 2**64, (n, v), dtype=np.uint64)
    x = np.where(rng.random((n, v)) < 0.2, noise, (noise & ~m) | base)
    return tuple(torch.from_numpy(a.astype(UINT[wb]).view(INT[wb])).cuda() for a in (x, m, base))


@pytest.mark.parametrize("wb,v", [(4, 3), (4, 31), (4, 32), (4, 33), (4, 64), (4, 65), (4, 127),
                                  (4, 128), (4, 129), (8, 5), (8, 32), (8, 33), (8, 63), (8, 64),
                                  (8, 65)])
def test_rows_come_back_and_bad_ones_are_left_alone(wb, v):
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(10 * v + wb)
    n = 1500
    src, m, b = rows_of(rng, n, v, wb)
    words, offs = ibp.compress_condensed(src, m, b)
    idx = torch.from_numpy(rng.integers(0, n, 4000)).cuda()
    for k in (None, idx, idx[:1]):
        out = ibp.decompress_fetch_condensed(words, offs, m, b, v, "cuda", k, check=True)
        assert torch.equal(out, src if k is None else src[k])
    # rows whose bitmap says that every word is stored whole
    o = offs.cpu().numpy()
    start = np.concatenate([[0], o[:-1]]) // wb
    packed = np.flatnonzero(o // wb - start < v)
    if not len(packed):
        return
    bad = packed[rng.random(len(packed)) < 0.1]
    meta = ((v + 7) // 8 + wb - 1) // wb
    for r in bad:
        words[int(start[r]):int(start[r]) + meta] = 0
    good = torch.ones(n, dtype=torch.bool)
    good[torch.from_numpy(bad)] = False
    good = good.cuda()
    for k in (None, idx):
        want, ok = (src, good) if k is None else (src[k], good[k])
        out = torch.full_like(want, 7)
        try:
            ibp.decompress_fetch_condensed(words, offs, m, b, v, "cuda", k, output_tensor=out,
                                           check=True)
            assert bool(ok.all())
        except RuntimeError as e:
            assert "bitmap" in str(e) and not bool(ok.all())
        assert torch.equal(out[ok], want[ok])
        assert bool((out[~ok] == 7).all())


@pytest.mark.parametrize("wb", [4, 8])
def test_rows_of_16_words_take_less_time_than_rows_of_64(wb):
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(wb)

    def fetch_us(v):
        src, m, b = rows_of(rng, 100_000, v, wb)
        words, offs = ibp.compress_condensed(src.repeat(4, 1), m, b)
        out = torch.empty((400_000, v), dtype=src.dtype, device="cuda")

        def fetch():
            ibp.decompress_fetch_condensed(words, offs, m, b, v, "cuda", output_tensor=out)

        fetch()
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            for _ in range(5):
                fetch()
            torch.cuda.synchronize()
        took = [e.self_device_time_total for e in prof.key_averages() if "fetch_kernel" in e.key]
        assert took
        return sum(took) / 5

    short, long = fetch_us(16), fetch_us(64)
    assert short < 0.8 * long, (short, long)
