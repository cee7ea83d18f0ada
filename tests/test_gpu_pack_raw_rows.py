"""Rows that stay raw among rows that are packed, against the CPU oracle: all raw, raw up to some
position, rows whose first columns save nothing though the row does, and the other way round; short
rows, rows of several groups of columns, few rows and more than the grid has warps, bad indices.
And packing rows that all stay raw takes less time than packing rows that do not."""
import numpy as np
import pytest
import torch
from torch.profiler import ProfilerActivity, profile

pytestmark = pytest.mark.gpu

INT = {4: np.int32, 8: np.int64}
UINT = {4: np.uint32, 8: np.uint64}


def rows_of(rng, n, v, wb, kind):
    """Half of every word's bits invariant; `kind` says which words are off the pattern."""
    m = rng.integers(0, 2**64, v, dtype=np.uint64)
    base = rng.integers(0, 2**64, v, dtype=np.uint64) & m
    noise = rng.integers(0, 2**64, (n, v), dtype=np.uint64)
    x = (noise & ~m) | base
    first = np.arange(v) < min(v, 512 // wb)     # the first group of columns
    row = np.arange(n)[:, None]
    off = {"all": np.ones((n, v), bool),
           "leading": np.broadcast_to(row < 2 * n // 3, (n, v)),
           "some": np.broadcast_to(rng.random((n, 1)) < 0.3, (n, v)),
           "first": np.broadcast_to(first & (row % 5 != 0), (n, v)),
           "but_first": np.broadcast_to(~first, (n, v))}[kind]
    x = np.where(off, noise, x)
    return tuple(a.astype(UINT[wb]).view(INT[wb]) for a in (x, m, base))


@pytest.mark.parametrize("kind", ["all", "leading", "some", "first", "but_first"])
@pytest.mark.parametrize("wb,v,n", [(4, 1, 50), (4, 64, 300), (4, 127, 333), (4, 128, 90),
                                    (4, 129, 7), (4, 140, 2401), (4, 260, 9700), (4, 1100, 2450),
                                    (8, 2, 70), (8, 33, 101), (8, 64, 130), (8, 65, 2500),
                                    (8, 130, 9600), (8, 700, 5), (8, 4100, 40)])
def test_raw_rows_among_packed_ones(oracle, wb, v, n, kind):
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(100 * v + wb + n)
    x, m, b = rows_of(rng, n, v, wb, kind)
    dm, db = torch.from_numpy(m).cuda(), torch.from_numpy(b).cuda()
    src = torch.from_numpy(x).cuda()
    want, want_bits = oracle.compress(x, m, b)
    t = src.clone()
    bits = ibp.compress_inplace(t, dm, db)
    torch.cuda.synchronize()
    assert np.array_equal(bits.cpu().numpy(), want_bits)
    assert np.array_equal(t.cpu().numpy(), want.view(INT[wb]))
    words, offs = oracle.compress_condensed(x, m, b)
    cw, co = ibp.compress_condensed(src, dm, db)
    torch.cuda.synchronize()
    assert np.array_equal(co.cpu().numpy(), offs)
    assert np.array_equal(cw.cpu().numpy(), words.view(INT[wb]))
    # bad positions among them take no bytes; an index in place reads every row first
    idx = rng.integers(0, n, n)
    bad = rng.random(n) < 0.2
    words, offs = oracle.compress_condensed(x, m, b, idx[~bad])
    cw, co = ibp.compress_condensed(src, dm, db, torch.from_numpy(np.where(bad, n, idx)).cuda())
    torch.cuda.synchronize()
    assert np.array_equal(co.cpu().numpy()[~bad], offs)
    assert np.array_equal(cw.cpu().numpy(), words.view(INT[wb]))
    want, want_bits = oracle.compress(x, m, b, idx)
    t = src.clone()
    bits = ibp.compress_inplace(t, dm, db, torch.from_numpy(idx).cuda())
    torch.cuda.synchronize()
    assert np.array_equal(bits.cpu().numpy(), want_bits)
    assert np.array_equal(t.cpu().numpy(), want.view(INT[wb]))


@pytest.mark.parametrize("wb,v", [(4, 64), (4, 256), (4, 1000), (8, 64), (8, 128), (8, 300)])
def test_raw_rows_take_less_time_than_packed_ones(wb, v):
    import invariantbitpacking_b200 as ibp
    n = (96 << 20) // (v * wb)
    g = torch.Generator(device="cuda")
    g.manual_seed(v)
    dtype = torch.from_numpy(np.zeros(1, INT[wb])).dtype
    noise = torch.randint(-2**63, 2**63 - 1, (n, v), generator=g, device="cuda").to(dtype)
    mask = torch.randint(-2**63, 2**63 - 1, (v,), generator=g, device="cuda").to(dtype)

    def pack_us(x):
        rows = x.clone()
        ibp.compress_inplace(rows, mask, mask)
        torch.cuda.synchronize()
        with profile(activities=[ProfilerActivity.CUDA]) as prof:
            for _ in range(4):
                rows.copy_(x)
                ibp.compress_inplace(rows, mask, mask)
            torch.cuda.synchronize()
        took = [e.self_device_time_total for e in prof.key_averages() if "pack" in e.key]
        assert took
        return sum(took) / 4

    packed = pack_us(noise | mask)
    raw = pack_us(noise)
    assert raw < packed, (raw, packed)


@pytest.mark.parametrize("kind", ["all", "some", "but_first"])
@pytest.mark.parametrize("wb,v,n", [(4, 1, 70), (4, 33, 300), (4, 128, 200), (4, 200, 90),
                                    (8, 2, 90), (8, 3, 40), (8, 64, 130), (8, 65, 300),
                                    (8, 128, 70), (8, 1000, 20), (8, 14000, 3), (8, 14500, 2)])
def test_host_rows(oracle, wb, v, n, kind):
    """Rows in pinned memory: whole 16-byte blocks and not, tiny rows, rows longer than a warp's
    words and image together; in place, back to back, and by an index with bad positions."""
    import invariantbitpacking_b200 as ibp
    rng = np.random.default_rng(100 * v + wb + n)
    x, m, b = rows_of(rng, n, v, wb, kind)
    dm, db = torch.from_numpy(m).cuda(), torch.from_numpy(b).cuda()
    src = torch.from_numpy(x).pin_memory()
    words, offs = oracle.compress_condensed(x, m, b)
    cw, co = ibp.compress_condensed(src, dm, db)
    assert np.array_equal(co.numpy(), offs) and np.array_equal(cw.numpy(), words.view(INT[wb]))
    idx = rng.integers(0, n, n)
    bad = rng.random(n) < 0.2
    words, offs = oracle.compress_condensed(x, m, b, idx[~bad])
    cw, co = ibp.compress_condensed(src, dm, db, torch.from_numpy(np.where(bad, -1, idx)).cuda())
    assert np.array_equal(co.numpy()[~bad], offs) and np.array_equal(cw.numpy(), words.view(INT[wb]))
    want, want_bits = oracle.compress(x, m, b)
    bits = ibp.compress_inplace(src, dm, db)
    assert np.array_equal(bits.cpu().numpy(), want_bits)
    assert np.array_equal(src.numpy(), want.view(INT[wb]))


def test_raw_host_rows_cross_the_link_once():
    """Raw host rows of 8 KiB packed back to back: a kernel that reads them twice over the link takes
    at least two copies' time, as measured here; the copy engine reads no slower than a kernel."""
    import invariantbitpacking_b200 as ibp
    n, v = 8000, 1000
    g = torch.Generator(device="cuda")
    g.manual_seed(1)
    noise = torch.randint(-2**63, 2**63 - 1, (n, v), generator=g, device="cuda")
    mask = torch.randint(-2**63, 2**63 - 1, (v,), generator=g, device="cuda")
    rows = noise.cpu().pin_memory()
    on_device = torch.empty_like(noise)
    on_device.copy_(rows, non_blocking=True)
    ibp.compress_condensed(rows, mask, mask)
    torch.cuda.synchronize()
    with profile(activities=[ProfilerActivity.CUDA]) as prof:
        for _ in range(6):
            on_device.copy_(rows, non_blocking=True)
            torch.cuda.synchronize()
            ibp.compress_condensed(rows, mask, mask)
            torch.cuda.synchronize()

    def best_us(name):
        return min(e.device_time for e in prof.events()
                   if name in e.name and e.device_type.name == "CUDA")

    assert best_us("pack") < 2 * best_us("Memcpy HtoD")


@pytest.mark.parametrize("wb,v", [(4, 64), (4, 99), (4, 300), (8, 2), (8, 64), (8, 300)])
def test_a_set_without_rows_is_never_read(wb, v):
    """An index into a set of no rows: every position is bad, nothing is read or written."""
    import ctypes

    from invariantbitpacking_b200 import _capi
    lib = _capi.lib
    dtype = torch.from_numpy(np.zeros(1, INT[wb])).dtype
    mask = torch.ones(v, dtype=dtype, device="cuda")
    idx = torch.arange(3000, device="cuda")
    offsets = torch.zeros(3000, dtype=torch.int64, device="cuda")
    out = torch.full((8,), 7, dtype=dtype, device="cuda")
    need = lib.ibp_compress_condensed_workspace_size(v, wb)
    ws = torch.empty(need, dtype=torch.uint8, device="cuda")
    status = lib.ibp_compress_condensed(None, 0, v, wb, mask.data_ptr(), mask.data_ptr(),
                                        idx.data_ptr(), 3000, offsets.data_ptr(), out.data_ptr(),
                                        ws.data_ptr(), need, torch.cuda.current_stream().cuda_stream)
    assert status == 0
    word = torch.zeros(1, dtype=torch.int32)
    _capi.check(lib.ibp_read_status(ws.data_ptr(), ctypes.c_void_p(word.data_ptr()),
                                    torch.cuda.current_stream().cuda_stream))
    assert int(word) & 1
    assert bool((out == 7).all())
