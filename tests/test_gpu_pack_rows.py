"""Packed rows against the CPU oracle at the edges of the packer: one and several 32-column
chunks, row counts that are no multiple of the rows a warp takes, columns that keep no bit and
columns that keep all, rows stored whole between packed ones, long rows with one and with
several rows per table load, bad indices beside good ones.  Bytes must be equal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

INT = {4: np.int32, 8: np.int64}
UINT = {4: np.uint32, 8: np.uint64}


def rows_of(rng, n, v, wb, frac):
    W = 8 * wb
    m = np.zeros(v, dtype=np.uint64)
    share = np.where(rng.random(v) < 0.2, rng.choice([0.0, 1.0], v), frac)  # some all or nothing
    for b in range(W):
        m |= (rng.random(v) < share).astype(np.uint64) << np.uint64(b)
    base = rng.integers(0, 2**64, v, dtype=np.uint64) & m
    noise = rng.integers(0, 2**64, (n, v), dtype=np.uint64)
    x = (noise & ~m) | base
    whole = rng.random((n, 1)) < 0.1       # rows off the pattern throughout
    stray = (rng.random((n, v)) < 0.05) & (rng.random((n, 1)) < 0.5)
    x = np.where(whole | stray, noise, x)
    return x.astype(UINT[wb]).view(INT[wb]), m.astype(UINT[wb]).view(INT[wb]), \
        base.astype(UINT[wb]).view(INT[wb])


@pytest.mark.parametrize("frac", [0.05, 0.5, 0.97])
@pytest.mark.parametrize("wb,v,n", [(4, 1, 9), (4, 31, 70), (4, 32, 101), (4, 33, 66), (4, 64, 130),
                                    (4, 99, 203), (4, 700, 41), (4, 801, 33), (8, 1, 5),
                                    (8, 16, 67), (8, 32, 33), (8, 63, 101), (8, 64, 1030),
                                    (8, 65, 34), (8, 200, 66), (8, 385, 31), (8, 1025, 18),
                                    (8, 4000, 6)])
def test_packed_bytes_vs_oracle(oracle, wb, v, n, frac):
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(1000 * v + 10 * wb + int(100 * frac))
    x, m, b = rows_of(rng, n, v, wb, frac)
    dm, db = torch.from_numpy(m).cuda(), torch.from_numpy(b).cuda()
    want, want_bits = oracle.compress(x, m, b)
    t = torch.from_numpy(x).cuda()
    bits = ibp.compress_inplace(t, dm, db)
    torch.cuda.synchronize()
    assert np.array_equal(bits.cpu().numpy(), want_bits)
    assert np.array_equal(t.cpu().numpy(), want.view(INT[wb]))
    # an index: every source row read before any is overwritten
    idx = rng.integers(0, n, max(n - 3, 1))
    want, want_bits = oracle.compress(x, m, b, idx)
    t = torch.from_numpy(x).cuda()
    bits = ibp.compress_inplace(t, dm, db, torch.from_numpy(idx).cuda())
    torch.cuda.synchronize()
    assert np.array_equal(bits.cpu().numpy(), want_bits)
    assert np.array_equal(t.cpu().numpy()[:len(idx)], want.view(INT[wb])[:len(idx)])
    # back to back
    words, offs = oracle.compress_condensed(x, m, b)
    cw, co = ibp.compress_condensed(torch.from_numpy(x).cuda(), dm, db)
    torch.cuda.synchronize()
    assert np.array_equal(co.cpu().numpy(), offs)
    assert np.array_equal(cw.cpu().numpy(), words.view(INT[wb]))


def test_bad_indices_leave_the_other_rows_right(oracle):
    """Bad positions beside good ones in one warp's batch: the good rows pack as ever."""
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(3)
    x, m, b = rows_of(rng, 200, 64, 8, 0.5)
    idx = rng.integers(0, 200, 150)
    bad = rng.random(150) < 0.3
    dm, db = torch.from_numpy(m).cuda(), torch.from_numpy(b).cuda()
    words, offs = oracle.compress_condensed(x[idx[~bad]], m, b)
    cw, co = ibp.compress_condensed(torch.from_numpy(x).cuda(), dm, db,
                                    torch.from_numpy(np.where(bad, -1, idx)).cuda())
    torch.cuda.synchronize()
    assert np.array_equal(co.cpu().numpy()[~bad], offs)  # a bad position takes no bytes
    assert np.array_equal(cw.cpu().numpy(), words.view(np.int64))
