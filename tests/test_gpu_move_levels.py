"""Masks at the edges of the rules that choose how many moves a word's bits need: the short-row fetch
and the packer of rows of one group take one, two or all five moves by how many dropped bits lie above a
kept one in the column that needs most.  For every such number around a power of two: dropped bits in
one run and split between kept ones, in the high half, in the low half and in both; one column in
several and every column; packed bytes equal the CPU oracle's and fetched rows the source."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

INT = {4: np.int32, 8: np.int64}
UINT = {4: np.uint32, 8: np.uint64}


def kept(rng, above, split):
    """Kept bits of a 32-bit half whose lowest one has `above` dropped bits above it."""
    if above == 0:
        n = int(rng.integers(1, 33))           # a run from the top
        return ((1 << n) - 1) << (32 - n)
    if not split:                              # a run right below the dropped ones
        n = int(rng.integers(1, 33 - above))
        return ((1 << n) - 1) << (32 - above - n)
    low = int(rng.integers(0, 32 - above))     # the lowest kept bit; `above` zeros over it
    bits = np.zeros(32 - low - 1, bool)
    bits[:len(bits) - above] = True
    rng.shuffle(bits)
    return (1 << low) | sum(1 << (low + 1 + int(i)) for i in np.flatnonzero(bits))


def places(k):
    """The number the rules look at, by its definition."""
    low = (k & -k).bit_length() - 1
    return sum(not (k >> i) & 1 for i in range(low, 32))


@pytest.mark.parametrize("above", [0, 1, 2, 3, 4, 5, 7, 8, 15, 16, 31])
@pytest.mark.parametrize("split", [False, True])
@pytest.mark.parametrize("wb,v", [(8, 64), (8, 32), (8, 40), (4, 64), (4, 20), (4, 128)])
def test_every_number_of_moves(oracle, wb, v, above, split):
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(100 * above + v + wb + split)
    for halves in (("both",) if wb == 4 else ("high", "low", "both")):
        for everywhere in (False, True):
            most = 0
            m = np.zeros(v, dtype=np.uint64)
            for j in range(v):
                a = above if everywhere or j == v // 3 else int(rng.integers(0, above + 1))
                hi = kept(rng, a if halves != "low" else 0, split)
                lo = kept(rng, a if halves != "high" else 0, split)
                most = max(most, places(lo), places(hi) if wb == 8 else 0)
                keep = (hi << 32 | lo) if wb == 8 else lo
                m[j] = ~keep & (2**64 - 1 if wb == 8 else 2**32 - 1)
            assert most == above
            n = 300
            noise = rng.integers(0, 2**64, (n, v), dtype=np.uint64)
            base = rng.integers(0, 2**64, v, dtype=np.uint64) & m
            x = (noise & ~m) | base
            stray = rng.random((n, v)) < 0.05 * (rng.random((n, 1)) < 0.3)
            x = np.where(stray, noise, x).astype(UINT[wb]).view(INT[wb])
            mw, bw = m.astype(UINT[wb]).view(INT[wb]), base.astype(UINT[wb]).view(INT[wb])
            dm, db = torch.from_numpy(mw).cuda(), torch.from_numpy(bw).cuda()
            src = torch.from_numpy(x).cuda()
            want, want_bits = oracle.compress(x, mw, bw)
            t = src.clone()
            bm = ibp.compress_inplace(t, dm, db)
            torch.cuda.synchronize()
            assert np.array_equal(bm.cpu().numpy(), want_bits)
            assert np.array_equal(t.cpu().numpy(), want.view(INT[wb]))
            idx = torch.from_numpy(rng.integers(0, n, 700)).cuda()
            for k in (None, idx):
                out = ibp.decompress_fetch(t, dm, db, bm, "cuda", None, k, check=True)
                assert torch.equal(out, src if k is None else src[k])
