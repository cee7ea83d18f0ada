"""Bitwise k-means rounds against the CPU oracle at the edges of the tile kernel: rows of odd,
8-byte and 16-byte lengths, cluster counts around the 8- and 16-centroid tiles, rows past one
tile per block, centroids too large for shared memory, clusters of one row and of all rows."""
import numpy as np
import pytest
import torch

pytestmark = pytest.mark.gpu


def mixture(rng, n, v, wb, c, noise):
    W = 8 * wb
    ut = {4: np.uint32, 8: np.uint64}[wb]
    cent = rng.integers(0, 2**63, (c, v), dtype=np.uint64).astype(ut)
    x = cent[rng.integers(0, c, n)]
    for _ in range(noise):
        x ^= (ut(1) << rng.integers(0, W, (n, v)).astype(ut))
    return x.view({4: np.int32, 8: np.int64}[wb])


@pytest.mark.parametrize("wb,v,n,c,noise", [
    (8, 32, 592, 16, 3), (8, 11, 3001, 13, 2), (4, 48, 2000, 15, 4), (4, 33, 1500, 3, 2),
    (4, 1, 100, 2, 1), (4, 6, 40, 8, 1), (8, 64, 5000, 40, 5), (8, 512, 200, 24, 9),
    (4, 3, 700_000, 5, 1), (8, 32, 3000, 1, 0), (4, 64, 20, 17, 3),
])
def test_kmeans_rounds_vs_oracle(oracle, wb, v, n, c, noise):
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(1000 * wb + 10 * v + c)
    x = mixture(rng, n, v, wb, c, noise)
    seeds = rng.choice(n, min(c, n), replace=False).astype(np.int64)
    om, ob, ocl = oracle.preprocess_kmeans(x, c, seeds)
    m, b, cl = ibp.preprocess_kmeans(torch.from_numpy(x).cuda(), c, 0.9, seed_rows=seeds)
    torch.cuda.synchronize()
    assert np.array_equal(cl.numpy(), ocl)
    assert np.array_equal(m.cpu().numpy(), om.view(x.dtype))
    assert np.array_equal(b.cpu().numpy(), ob.view(x.dtype))


def test_kmeans_rounds_of_an_unaligned_view(oracle):
    """Rows of whole 16-byte blocks that start 4 bytes off a 16-byte boundary."""
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(5)
    x = mixture(rng, 1000, 32, 4, 6, 3)
    buf = torch.empty(1000 * 32 + 1, dtype=torch.int32, device="cuda")
    t = buf[1:].view(1000, 32)
    t.copy_(torch.from_numpy(x))
    seeds = rng.choice(1000, 6, replace=False).astype(np.int64)
    om, ob, ocl = oracle.preprocess_kmeans(x, 6, seeds)
    m, b, cl = ibp.preprocess_kmeans(t, 6, 0.9, seed_rows=seeds)
    torch.cuda.synchronize()
    assert np.array_equal(cl.numpy(), ocl)
    assert np.array_equal(m.cpu().numpy(), om.view(np.int32))
