"""Fetches of device-resident rows of any length and alignment: rows that start anywhere in a
16-byte block, one group of columns and several, a last group with few columns, rows stored raw
that fit a slot and that do not, rows longer than their first read and than their slot, few rows
and many, every de-duplication mode, and condensed rows.  Output rows equal the source rows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

INT = {4: np.int32, 8: np.int64}
UINT = {4: np.uint32, 8: np.uint64}


def rows_of(rng, n, v, wb, frac):
    W = 8 * wb
    m = np.zeros(v, dtype=np.uint64)
    for b in range(W):
        m |= (rng.random(v) < frac).astype(np.uint64) << np.uint64(b)
    base = rng.integers(0, 2**64, v, dtype=np.uint64) & m
    noise = rng.integers(0, 2**64, (n, v), dtype=np.uint64)
    x = (noise & ~m) | base
    whole = rng.random((n, 1)) < 0.1     # stored raw
    half = rng.random((n, 1)) < 0.1      # much longer than the others
    stray = rng.random((n, v)) < np.where(half, 0.5, 0.02 * (rng.random((n, 1)) < 0.5))
    x = np.where(whole | stray, noise, x)
    return x.astype(UINT[wb]).view(INT[wb]), m.astype(UINT[wb]).view(INT[wb]), \
        base.astype(UINT[wb]).view(INT[wb])


def place(x, offset):
    buf = torch.empty(x.size + offset, dtype=torch.from_numpy(x[:1]).dtype, device="cuda")
    t = buf[offset:].view(*x.shape)
    t.copy_(torch.from_numpy(x))
    return t


@pytest.mark.parametrize("frac", [0.4, 0.95])
@pytest.mark.parametrize("wb,v,n,offset", [
    (4, 1, 50, 0), (4, 7, 900, 1), (4, 33, 300, 0), (4, 64, 500, 1), (4, 99, 2000, 0),
    (4, 128, 1000, 3), (4, 129, 700, 0), (4, 256, 5000, 0), (4, 257, 300, 2), (4, 1100, 60, 0),
    (8, 3, 500, 0), (8, 33, 1000, 0), (8, 63, 700, 1), (8, 64, 300, 1), (8, 65, 2000, 0),
    (8, 128, 3, 0), (8, 200, 400, 1), (8, 512, 3000, 0), (8, 700, 40, 1), (8, 3000, 9, 0)])
def test_device_rows_come_back(wb, v, n, offset, frac):
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(100 * v + wb + n + int(10 * frac))
    x, m, b = rows_of(rng, n, v, wb, frac)
    dm, db = torch.from_numpy(m).cuda(), torch.from_numpy(b).cuda()
    src = torch.from_numpy(x).cuda()
    t = place(x, offset)
    bm = ibp.compress_inplace(t, dm, db)
    for comp_len in (None, 1, max(v // 2, 1), v):
        out = ibp.decompress_fetch(t, dm, db, bm, "cuda", comp_len, check=True)
        assert torch.equal(out, src), comp_len
    idx = torch.from_numpy(rng.integers(0, n, 3 * n // 2 + 5)).cuda()
    try:
        for mode in ("auto", "sort", "hash"):
            ibp.set_fetch_dedup(mode)
            for k in (idx, idx[:1], idx[:0]):
                out = ibp.decompress_fetch(t, dm, db, bm, "cuda", max(v // 2, 1), k, check=True)
                assert torch.equal(out, src[k]), mode
    finally:
        ibp.set_fetch_dedup("auto")
    words, offs = ibp.compress_condensed(src.clone(), dm, db)
    for k in (None, idx, idx[:1]):
        out = ibp.decompress_fetch_condensed(words, offs, dm, db, v, "cuda", k, check=True)
        assert torch.equal(out, src if k is None else src[k])


@pytest.mark.parametrize("wb,v", [(4, 99), (8, 300)])
def test_bad_indices_are_reported_and_the_rest_is_right(wb, v):
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(v)
    x, m, b = rows_of(rng, 400, v, wb, 0.6)
    dm, db = torch.from_numpy(m).cuda(), torch.from_numpy(b).cuda()
    src = torch.from_numpy(x).cuda()
    t = src.clone()
    bm = ibp.compress_inplace(t, dm, db)
    idx = rng.integers(0, 400, 1000)
    bad = rng.random(1000) < 0.1
    k = torch.from_numpy(np.where(bad, rng.choice([-1, 400, 10**12], 1000), idx)).cuda()
    good = torch.from_numpy(~bad).cuda()
    try:
        for mode in ("auto", "sort"):
            ibp.set_fetch_dedup(mode)
            out = torch.full((1000, v), 7, dtype=src.dtype, device="cuda")
            with pytest.raises(RuntimeError, match="out of range"):
                ibp.decompress_fetch(t, dm, db, bm, "cuda", None, k, output_tensor=out, check=True)
            assert torch.equal(out[good], src[k[good]])
            assert bool((out[~good] == 7).all())
    finally:
        ibp.set_fetch_dedup("auto")


@pytest.mark.parametrize("count", [32767, 32768, 32769, 98303, 98304, 98305])
@pytest.mark.parametrize("wb,v", [(8, 33), (8, 64), (4, 128), (4, 129), (4, 300)])
def test_batches_around_the_direct_limit(wb, v, count):
    """Skewed batches on both sides of the size up to which repeats are decoded again, rows of the
    kernel that has no such limit among them; condensed rows too."""
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(count + v)
    x, m, b = rows_of(rng, 3000, v, wb, 0.6)
    dm, db = torch.from_numpy(m).cuda(), torch.from_numpy(b).cuda()
    src = torch.from_numpy(x).cuda()
    t = src.clone()
    bm = ibp.compress_inplace(t, dm, db)
    k = torch.from_numpy(np.minimum(rng.zipf(1.3, count) - 1, 2999)).cuda()
    out = ibp.decompress_fetch(t, dm, db, bm, "cuda", None, k, check=True)
    assert torch.equal(out, src[k])
    words, offs = ibp.compress_condensed(src.clone(), dm, db)
    out = ibp.decompress_fetch_condensed(words, offs, dm, db, v, "cuda", k, check=True)
    assert torch.equal(out, src[k])


@pytest.mark.parametrize("count", [16384, 16385])
def test_long_rows_around_the_direct_limit_in_bytes(count):
    test_batches_around_the_direct_limit(8, 512, count)


@pytest.mark.parametrize("low,high", [(0, 31), (1, 30), (3, 28), (4, 27), (31, 0), (16, 16)])
@pytest.mark.parametrize("wb,v", [(8, 64), (8, 40), (4, 64), (4, 20)])
def test_masks_that_need_few_moves_and_many(wb, v, low, high):
    """Kept bits in one run with `high` dropped bits above and `low` below in every 32-bit half:
    the short-row kernel picks its moves by how many are dropped above."""
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(10 * low + v)
    keep = ((1 << 32) - 1) >> high & ~((1 << low) - 1)
    half = np.uint64(~keep & 0xFFFFFFFF)
    m = np.full(v, half | (half << np.uint64(32)) if wb == 8 else half, dtype=np.uint64)
    noise = rng.integers(0, 2**64, (700, v), dtype=np.uint64)
    base = rng.integers(0, 2**64, v, dtype=np.uint64) & m
    x = (noise & ~m) | base
    x = np.where(rng.random((700, v)) < 0.02 * (rng.random((700, 1)) < 0.3), noise, x)
    x = x.astype(UINT[wb]).view(INT[wb])
    dm = torch.from_numpy(m.astype(UINT[wb]).view(INT[wb])).cuda()
    db = torch.from_numpy(base.astype(UINT[wb]).view(INT[wb])).cuda()
    src = torch.from_numpy(x).cuda()
    t = src.clone()
    bm = ibp.compress_inplace(t, dm, db)
    out = ibp.decompress_fetch(t, dm, db, bm, "cuda", check=True)
    assert torch.equal(out, src)
    k = torch.from_numpy(rng.integers(0, 700, 5000)).cuda()
    out = ibp.decompress_fetch(t, dm, db, bm, "cuda", None, k, check=True)
    assert torch.equal(out, src[k])
