"""preprocess and get_compress_size against the CPU oracle at the edges of their row pieces:
every word size, rows of one piece and of many, rows that are no whole number of 16- or 4-byte
chunks, groups of rows that are and the rows left over, row sums past 16 bits, and datasets
that do not start on a 16-byte boundary.  Outputs are integers and must be equal."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu

INT = {1: np.int8, 2: np.int16, 4: np.int32, 8: np.int64}


def rows_of(rng, n, v, wb):
    """Words with invariant bits at several rates (so that thresholds differ) and odd rows."""
    W = 8 * wb
    p = rng.choice([0.02, 0.08, 0.13, 0.22, 0.5, 0.8, 0.93, 0.99, 1.0], size=(v, W))
    x = np.zeros((n, v), dtype=np.uint64)
    for b in range(W):
        x |= (rng.random((n, v)) < p[:, b]).astype(np.uint64) << np.uint64(b)
    keep = rng.random((n, 1)) < 0.8  # most rows: the likely value of every rather likely bit
    m = np.zeros(v, dtype=np.uint64)
    val = np.zeros(v, dtype=np.uint64)
    for b in range(W):
        m |= (np.abs(p[:, b] - 0.5) > 0.25).astype(np.uint64) << np.uint64(b)
        val |= (p[:, b] > 0.75).astype(np.uint64) << np.uint64(b)
    x = np.where(keep, (x & ~m) | val, x)
    return x.astype({1: np.uint8, 2: np.uint16, 4: np.uint32, 8: np.uint64}[wb]).view(INT[wb])


def put(x, offset):
    """x on the GPU, `offset` words past a 16-byte boundary."""
    flat = torch.from_numpy(x.reshape(-1))
    buf = torch.empty(flat.numel() + offset, dtype=flat.dtype, device="cuda")
    buf[offset:].copy_(flat)
    return buf[offset:].view(*x.shape)


SHAPES = [(1, 1, 70), (1, 5, 1000), (1, 16, 333), (1, 33, 517), (1, 130, 200), (1, 600, 90),
          (2, 1, 40), (2, 3, 999), (2, 8, 64), (2, 64, 700), (2, 129, 333), (2, 130, 100),
          (4, 1, 35), (4, 4, 600), (4, 33, 1001), (4, 64, 2000), (4, 140, 65), (4, 2100, 40),
          (8, 1, 100), (8, 2, 500), (8, 16, 300), (8, 17, 301), (8, 64, 5000), (8, 65, 257),
          (8, 1030, 50),
          (4, 32, 900), (4, 36, 331), (4, 128, 700), (4, 132, 300), (8, 62, 401), (8, 66, 150)]


@pytest.mark.parametrize("offset", [0, 1])
@pytest.mark.parametrize("wb,v,n", SHAPES)
def test_masks_and_sizes_vs_oracle(oracle, wb, v, n, offset):
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(100 * v + 10 * wb + n)
    x = rows_of(rng, n, v, wb)
    t = put(x, offset)
    for thr in (None, 0.9, 0.4):
        om, ob, _ = oracle.preprocess(x, thr)
        m, b = ibp.preprocess(t, thr)
        torch.cuda.synchronize()
        assert np.array_equal(m.cpu().numpy(), om.view(INT[wb])), thr
        assert np.array_equal(b.cpu().numpy(), ob.view(INT[wb])), thr
    om, ob, _ = oracle.preprocess(x, 0.75)
    dm, db = torch.from_numpy(om.view(INT[wb])).cuda(), torch.from_numpy(ob.view(INT[wb])).cuda()
    total = torch.full((1,), 5, dtype=torch.int64, device="cuda")
    sizes = ibp.get_compress_size(t, dm, db, None, total)
    want = oracle.compress_size(x, om, ob)
    torch.cuda.synchronize()
    assert np.array_equal(sizes.cpu().numpy(), want)
    assert int(total) == 5 + int(want.sum())
    idx = rng.integers(0, n, 77)
    bad = np.concatenate([idx, [-1, n, 2 * n]]).astype(np.int64)
    sizes = ibp.get_compress_size(t, dm, db, torch.from_numpy(bad).cuda())
    torch.cuda.synchronize()
    assert np.array_equal(sizes.cpu().numpy(), np.concatenate([want[idx], [0, 0, 0]]))


def test_values_outside_the_mask_never_match(oracle):
    """A value bit outside its mask: the word is stored whole, as in the definition."""
    import invariantbitpacking_b200 as ibp
    for wb, v in ((1, 64), (2, 64), (4, 64), (8, 64)):
        x = np.zeros((100, v), dtype=INT[wb])
        m = np.full(v, 0x0F, dtype=INT[wb])
        b = np.zeros(v, dtype=INT[wb])
        b[::3] = 0x10
        sizes = ibp.get_compress_size(torch.from_numpy(x).cuda(), torch.from_numpy(m).cuda(),
                                      torch.from_numpy(b).cuda())
        torch.cuda.synchronize()
        assert np.array_equal(sizes.cpu().numpy(), oracle.compress_size(x, m, b)), wb


def test_host_rows_with_a_remainder(oracle):
    """Rows in pinned memory, staged by the census in pieces and left-over rows."""
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(9)
    for wb, v, n in ((1, 33, 1003), (4, 33, 2050), (8, 64, 3001)):
        x = rows_of(rng, n, v, wb)
        om, ob, _ = oracle.preprocess(x, None)
        m, b = ibp.preprocess(torch.from_numpy(x).pin_memory(), None)
        torch.cuda.synchronize()
        assert np.array_equal(m.cpu().numpy(), om.view(INT[wb]))
        assert np.array_equal(b.cpu().numpy(), ob.view(INT[wb]))
