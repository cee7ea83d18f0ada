// ibp_kmeans.cu -- bitwise k-means preprocessing (replaces
// include/preproc/ibp_preproc_host.cuh:118-284 and include/preproc/ibp_preproc_kmeans.cuh).
//
// B200 design
//  * a host-resident table is copied to HBM once by the copy engine (when the caller's
//    workspace has room) and all ten rounds read HBM; the reference re-reads pinned host
//    memory over PCIe in every round.
//  * a round is one kernel over row tiles and a small one for the centroids.  The tile kernel
//    takes Hamming distances as an integer matrix product on the tensor cores; ties go to the
//    highest centroid id (a deterministic choice among the reference's racy outcomes, see
//    include/preproc/ibp_preproc_kmeans.cuh:139-146).  It then lists the tile's rows by cluster
//    in shared memory and counts the set bits of each cluster's rows in bit planes
//    (ibp_bitcount.cuh); the reference issues one global atomic per set bit.
//  * centroids too many or too long for shared memory once expanded take their distances in
//    assign_kernel (a warp per row, population counts), and the tile kernel counts only.
//  * the counts of the last round are exactly those of the final assignment, so the
//    final masks need no extra pass over the data.
#include <algorithm>
#include <vector>

#include "ibp_bitcount.cuh"
#include "ibp_common.cuh"
#include "ibp_internal.cuh"

namespace ibp200 {

constexpr int kKmRounds = 10;  // include/preproc/ibp_preproc_host.cuh:191

template <typename U>
__global__ void seed_centroids_kernel(const U *__restrict__ data, int64_t n, int64_t v,
                                      const int64_t *__restrict__ init, int c,
                                      U *__restrict__ cent, int32_t *__restrict__ status) {
    const int64_t seeded = (int64_t)c < n ? (int64_t)c : n;
    const int64_t total = (int64_t)c * v;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < total;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t i = e / v, k = e % v;
        U x = 0;
        if (i < seeded) {
            const int64_t r = i == 0 ? 0 : init[i];
            if (r >= 0 && r < n)
                x = data[r * v + k];
            else if (k == 0)
                atomicOr(status, kStatusBadIndex);
        }
        cent[e] = x;
    }
}

// clusters[i] = argmin_j popcount(row_i ^ centroid_j), highest j on ties.
template <typename U>
__global__ void __launch_bounds__(256)
assign_kernel(const U *__restrict__ data, int64_t n, int64_t v, const U *__restrict__ cent_g,
              int c, bool cent_in_smem, int32_t *__restrict__ clusters) {
    extern __shared__ __align__(16) unsigned char smem[];
    U *cent_s = reinterpret_cast<U *>(smem);
    if (cent_in_smem) {
        for (int64_t e = threadIdx.x; e < (int64_t)c * v; e += blockDim.x) cent_s[e] = cent_g[e];
        __syncthreads();
    }
    const U *cent = cent_in_smem ? cent_s : cent_g;
    const int lane = threadIdx.x & 31;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = warp; i < n; i += nwarps) {
        const U *row = data + i * v;
        int best = 0;
        uint32_t bestd = 0xffffffffu;
        for (int j = 0; j < c; ++j) {
            uint32_t d = 0;
            for (int64_t k = lane; k < v; k += 32) d += popc_w((U)(row[k] ^ cent[(int64_t)j * v + k]));
            d = __reduce_add_sync(0xffffffffu, d);
            if (d <= bestd) {
                bestd = d;
                best = j;
            }
        }
        if (lane == 0) clusters[i] = best;
    }
}

// ------------------------------------------------------------------ one round
// Distances as an integer matrix product.  popc(x ^ c) = popc(x) + popc(c) - 2 popc(x & c),
// and popc(x) is the same for every centroid, so the nearest one minimises
// popc(c) - 2 popc(x & c), and popc(x & c) over all centroids is a product of 0/1 matrices.
// A 32-bit unit of a row becomes eight registers of four bytes, x & (0x01010101 << s): byte
// values 2^s, one AND each.  The centroids are expanded once per block into shared memory
// with byte values 2^(7 - s), so every common bit adds 128 to a 32-bit accumulator of
// mma.m16n8k32 (u8 x u8, exact).  The order of K is free, so a lane takes 16 consecutive
// bytes of a row and no operand is shuffled.  mma.sync rather than tcgen05: A exists only in
// registers and N is the number of centroids: with the rows expanded into tensor memory and
// kind::i8 products of 128 rows x 16 centroids the ten rounds of the table below took 504 us
// a call, with these 451.  Bound: issue (8 ANDs, 4 products and one 16-byte shared read
// per 32 rows x 8 bits of a lane's unit).
__device__ __forceinline__ void mma_u8(int32_t (&d)[4], const uint32_t (&a)[4], uint32_t b0,
                                       uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.u8.s32 {%0,%1,%2,%3}, "
                 "{%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
                 : "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}

constexpr int kRoundThreads = 512;
constexpr int kRoundWarps = kRoundThreads / 32;
constexpr int kTileRows = 4096;   // most rows of a tile (16-bit row numbers in shared memory)
constexpr int kTaskRows = 128;    // rows of a task (a lane's eight bit planes count to 255)
constexpr int kFlushStride = 17;  // words per lane of a warp's flush buffer (16 + 1 of padding)

// Shared memory of kmeans_round_kernel: expanded centroids, their set bits, three words per
// list key (entries, first list entry, first task), the tile's new and old clusters and its
// row list, and a flush buffer per warp.
struct RoundShape {
    int units;    // 32-bit units per row
    int groups;   // 64-byte groups of a row
    int pairs;    // pairs of 8-centroid tiles
    bool assign;  // false: the clusters are already in `assign`
    bool fresh;   // every row is added to zero counts; false: only rows that changed cluster
    __host__ __device__ size_t expanded() const { return assign ? (size_t)pairs * groups * 8192 : 0; }
    size_t bytes(int c) const {
        return expanded() + align_up(sizeof(int32_t) * 16 * (size_t)pairs, 16) +
               align_up(sizeof(uint32_t) * (6 * (size_t)c + 2), 16) + 2 * 4 * (size_t)kTileRows +
               sizeof(uint32_t) * 32 * kFlushStride * kRoundWarps;
    }
};

// Nearest centroids of the 32 rows r0.. (highest centroid on ties), into scl[r - base] and
// `assign` (and `out`, the caller's copy, in the last round); the clusters they had go to
// sold[r - base].  hist counts the list entries: key cl for a row added to cluster cl, key
// c + cl for one taken from it.  V16: rows are 16-byte aligned.
template <bool V16>
__device__ __forceinline__ void assign_rows(const uint32_t *__restrict__ data, int64_t r0,
                                            int64_t rend, int64_t base, const RoundShape &sh,
                                            int c, const uint4 *__restrict__ expanded,
                                            const int32_t *__restrict__ pcs, uint16_t *scl,
                                            uint16_t *sold, uint32_t *hist,
                                            int32_t *__restrict__ assign,
                                            int32_t *__restrict__ out) {
    const int lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
    int bestd[4], bestj[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        bestd[q] = 0x7fffffff;
        bestj[q] = 0;
    }
    const uint32_t *row[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int64_t r = r0 + g + 8 * q;
        row[q] = data + (r < rend ? r : r0) * sh.units;  // rows past the end: a valid row, unused
    }
    for (int p = 0; p < sh.pairs; ++p) {
        const bool two = 16 * p + 8 < c;  // centroids in the pair's second tile
        int32_t acc[2][2][4];
#pragma unroll
        for (int x = 0; x < 16; ++x) acc[x >> 3][(x >> 2) & 1][x & 3] = 0;
        const uint4 *bp = expanded + (size_t)p * sh.groups * 512 + lane;
        for (int k = 0; k < sh.groups; ++k, bp += 512) {
            const int u = 16 * k + 4 * t;
            uint32_t x[4][4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                if constexpr (V16) {
                    uint4 y = make_uint4(0, 0, 0, 0);
                    if (u < sh.units) y = *reinterpret_cast<const uint4 *>(row[q] + u);
                    x[q][0] = y.x, x[q][1] = y.y, x[q][2] = y.z, x[q][3] = y.w;
                } else {
#pragma unroll
                    for (int i = 0; i < 4; ++i) x[q][i] = u + i < sh.units ? row[q][u + i] : 0u;
                }
            }
#pragma unroll
            for (int i = 0; i < 4; ++i) {
#pragma unroll
                for (int s = 0; s < 4; ++s) {
                    const uint4 b = bp[(i * 4 + s) * 32];
                    const uint32_t lo = 0x01010101u << (2 * s), hi = lo << 1;
                    const uint32_t a0[4] = {x[0][i] & lo, x[1][i] & lo, x[0][i] & hi, x[1][i] & hi};
                    const uint32_t a1[4] = {x[2][i] & lo, x[3][i] & lo, x[2][i] & hi, x[3][i] & hi};
                    mma_u8(acc[0][0], a0, b.x, b.y);
                    mma_u8(acc[1][0], a1, b.x, b.y);
                    if (two) {
                        mma_u8(acc[0][1], a0, b.z, b.w);
                        mma_u8(acc[1][1], a1, b.z, b.w);
                    }
                }
            }
        }
        // lane (g, t) holds centroids 2t, 2t+1 of each tile for rows g, g+8 of each 16 rows
#pragma unroll
        for (int x = 0; x < 16; ++x) {
            const int m = x >> 3, nt = (x >> 2) & 1, e = x & 3;
            const int q = 2 * m + (e >> 1), j = 16 * p + 8 * nt + 2 * t + (e & 1);
            const int d = pcs[j] - (acc[m][nt][e] >> 6);  // popc(c) - 2 * (acc / 128)
            if (j < c && d <= bestd[q]) {  // j rises: the highest centroid wins ties
                bestd[q] = d;
                bestj[q] = j;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) {
#pragma unroll
        for (int o = 1; o < 4; o <<= 1) {
            const int d = __shfl_xor_sync(0xffffffffu, bestd[q], o);
            const int j = __shfl_xor_sync(0xffffffffu, bestj[q], o);
            if (d < bestd[q] || (d == bestd[q] && j > bestj[q])) {
                bestd[q] = d;
                bestj[q] = j;
            }
        }
    }
    // lane (g, t) writes row g + 8t
    const int cl = t == 0 ? bestj[0] : (t == 1 ? bestj[1] : (t == 2 ? bestj[2] : bestj[3]));
    const int64_t r = r0 + g + 8 * t;
    if (r < rend) {
        const int old = sh.fresh ? -1 : assign[r];
        scl[r - base] = (uint16_t)cl;
        assign[r] = cl;
        if (out) out[r] = cl;
        if (!sh.fresh) sold[r - base] = (uint16_t)old;
        if (old != cl) {
            atomicAdd(&hist[cl], 1u);
            if (old >= 0) atomicAdd(&hist[c + old], 1u);
        }
    }
}

// bits[u * 32 + b] += (or -=) rows of one task (up to kTaskRows list entries of one key) with
// bit b of unit u set, for the units of one slice of 32 / R lanes x VEC units: every lane
// counts its units' bits over its rows in bit planes (BitPlanes), the planes become byte
// counts, and the warp adds those, 32 consecutive counters at a time, to the global ones.
template <int VEC>
__device__ __forceinline__ void count_task(const uint32_t *__restrict__ data, int64_t base,
                                           const uint16_t *list, int rows, int units, int u0,
                                           int lanes, bool minus, uint32_t *flush,
                                           uint32_t *bits) {
    const int lane = threadIdx.x & 31;
    const int slot = lane / lanes, R = 32 / lanes;
    const int u = u0 + (lane % lanes) * VEC;
    const bool in = u < units;  // VEC divides units
    BitPlanes<VEC> bp;
    bp.clear();
    constexpr int N = 8;
    for (int k = slot; k < rows + slot; k += N * R) {  // same trips in every lane
        uint32_t x[N][VEC];
#pragma unroll
        for (int q = 0; q < N; ++q) {
            const int kk = k + q * R;
            const bool ok = in && kk < rows;
            const uint32_t *p = data + (base + (ok ? list[kk] : 0)) * units + u;
            if constexpr (VEC == 2) {
                const uint2 y = ok ? *reinterpret_cast<const uint2 *>(p) : make_uint2(0, 0);
                x[q][0] = y.x, x[q][1] = y.y;
            } else {
                x[q][0] = ok ? *p : 0u;
            }
        }
        bp.add8(x);
    }
    // byte counts: word s of unit w holds bits s, s + 8, s + 16, s + 24
#pragma unroll
    for (int w = 0; w < VEC; ++w)
#pragma unroll
        for (int s = 0; s < 8; ++s) flush[lane * kFlushStride + w * 8 + s] = bp.bytes(w, s);
    __syncwarp();
    // lane b adds bit b's counter of each unit (the slots of a unit first, where a warp holds
    // several rows at once)
    const int nl = min(lanes, (units - u0) / VEC), sh = 8 * (lane >> 3);
    const uint32_t *f = flush + (lane & 7);
    uint32_t *to = bits + (int64_t)u0 * 32 + lane;
    const uint32_t sign = minus ? ~0u : 1u;
    auto put = [&](uint32_t count, int unit) {
        if (count) atomicAdd(to + unit * 32, count * sign);
    };
    if (R == 1) {
#pragma unroll 4
        for (int l = 0; l < nl; ++l) {
#pragma unroll
            for (int w = 0; w < VEC; ++w)
                put((f[l * kFlushStride + w * 8] >> sh) & 0xffu, l * VEC + w);
        }
    } else {
        for (int l = 0; l < nl; ++l) {
#pragma unroll
            for (int w = 0; w < VEC; ++w) {
                uint32_t count = 0;
                for (int r = 0; r < R; ++r)
                    count += (f[(r * lanes + l) * kFlushStride + w * 8] >> sh) & 0xffu;
                put(count, l * VEC + w);
            }
        }
    }
    __syncwarp();
}

// One round over the rows of a tile at a time: clusters (assign_rows), then the tile's rows
// listed by cluster (a counting sort of row numbers in shared memory), then the set bits of
// each cluster's rows (count_task).  The counts live on from round to round: after the first
// only rows that changed cluster are listed, once to add and once to take away (a fifth of
// the rows in the second round of a 16-cluster mixture, a fiftieth in the last).  The
// reference issues an atomic per set bit, and this kernel's predecessors formed a ballot per
// bit of every word (200k rows of 32 64-bit words, 16 clusters: 777 us a round; this kernel
// 38 us, 12 of them the products at the rate mma.sync reaches, 8 cycles each per scheduler).
// Block: 16 warps, one block per SM, tiles of n / SMs rows, so that a cluster's rows of a
// tile make a task long enough to pay for its flush.
template <bool V16, int VEC>
__global__ void __launch_bounds__(kRoundThreads, 1)
kmeans_round_kernel(const uint32_t *__restrict__ data, int64_t n, const uint32_t *__restrict__ cent,
                    int c, RoundShape sh, int tile, int32_t *__restrict__ assign,
                    int32_t *__restrict__ out, uint32_t *__restrict__ bits,
                    uint32_t *__restrict__ cnt) {
    extern __shared__ __align__(16) unsigned char smem[];
    uint4 *expanded = reinterpret_cast<uint4 *>(smem);
    int32_t *pcs = reinterpret_cast<int32_t *>(smem + sh.expanded());
    uint32_t *hist = reinterpret_cast<uint32_t *>(pcs + 16 * sh.pairs);
    const int keys = sh.fresh ? c : 2 * c;
    uint32_t *first = hist + keys;   // next list entry of each key
    uint32_t *task0 = first + keys;  // first task of each key, then the number of tasks
    uint16_t *scl = reinterpret_cast<uint16_t *>(
        smem + sh.expanded() + align_up(sizeof(int32_t) * 16 * (size_t)sh.pairs, 16) +
        align_up(sizeof(uint32_t) * (6 * (size_t)c + 2), 16));
    uint16_t *sold = scl + kTileRows;
    uint16_t *list = sold + kTileRows;
    uint32_t *flush = reinterpret_cast<uint32_t *>(list + 2 * kTileRows);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int units = sh.units;
    grid_dep_wait();
    grid_dep_release();
    if (sh.assign) {
        const int total = sh.pairs * sh.groups * 512;
        for (int e = threadIdx.x; e < total; e += kRoundThreads) {
            const int ln = e & 31, s = (e >> 5) & 3, i = (e >> 7) & 3;
            const int k = (e >> 9) % sh.groups, p = (e >> 9) / sh.groups;
            const int u = 16 * k + 4 * (ln & 3) + i, j = 16 * p + (ln >> 2);
            uint32_t x0 = 0, x1 = 0;
            if (u < units) {
                if (j < c) x0 = cent[(int64_t)j * units + u];
                if (j + 8 < c) x1 = cent[(int64_t)(j + 8) * units + u];
            }
            auto spread = [](uint32_t x, int b) { return ((x >> b) & 0x01010101u) << (7 - b); };
            expanded[e] = make_uint4(spread(x0, 2 * s), spread(x0, 2 * s + 1), spread(x1, 2 * s),
                                     spread(x1, 2 * s + 1));
        }
        for (int j = warp; j < 16 * sh.pairs; j += kRoundWarps) {
            int pc = 0;
            if (j < c)
                for (int u = lane; u < units; u += 32) pc += __popc(cent[(int64_t)j * units + u]);
            pc = __reduce_add_sync(0xffffffffu, pc);
            if (lane == 0) pcs[j] = pc;
        }
    }
    // lanes of a warp per row in count_task: a power of two that covers the row's units
    int lanes = 32;
    while (lanes > 1 && (lanes / 2) * VEC >= units) lanes >>= 1;
    const int slices = (units + lanes * VEC - 1) / (lanes * VEC);
    for (int64_t base = (int64_t)blockIdx.x * tile; base < n; base += (int64_t)gridDim.x * tile) {
        const int64_t rend = min(base + tile, n);
        const int rows = (int)(rend - base);
        for (int j = threadIdx.x; j < keys; j += kRoundThreads) hist[j] = 0;
        __syncthreads();
        if (sh.assign) {
            for (int r = warp * 32; r < rows; r += kRoundThreads)
                assign_rows<V16>(data, base + r, rend, base, sh, c, expanded, pcs, scl, sold,
                                 hist, assign, out);
        } else {
            for (int r = threadIdx.x; r < rows; r += kRoundThreads) {
                const int cl = assign[base + r];
                scl[r] = (uint16_t)cl;
                if (out) out[base + r] = cl;
                atomicAdd(&hist[cl], 1u);
            }
        }
        __syncthreads();
        if (warp == 0) {  // list entries and tasks before each key
            uint32_t at = 0, tk = 0;
            for (int j0 = 0; j0 < keys; j0 += 32) {
                const int j = j0 + lane;
                const uint32_t h = j < keys ? hist[j] : 0u;
                const uint32_t th = (h + kTaskRows - 1) / kTaskRows;
                uint32_t ih = h, it = th;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const uint32_t y = __shfl_up_sync(0xffffffffu, ih, o);
                    const uint32_t z = __shfl_up_sync(0xffffffffu, it, o);
                    if (lane >= o) {
                        ih += y;
                        it += z;
                    }
                }
                if (j < keys) {
                    first[j] = at + ih - h;
                    task0[j] = tk + it - th;
                }
                at += __shfl_sync(0xffffffffu, ih, 31);
                tk += __shfl_sync(0xffffffffu, it, 31);
            }
            if (lane == 0) task0[keys] = tk;
        }
        __syncthreads();
        for (int r = threadIdx.x; r < rows; r += kRoundThreads) {
            const int cl = scl[r];
            if (sh.fresh || sold[r] != cl) {
                list[atomicAdd(&first[cl], 1u)] = (uint16_t)r;
                if (!sh.fresh) list[atomicAdd(&first[c + sold[r]], 1u)] = (uint16_t)r;
            }
        }
        for (int j = threadIdx.x; j < keys; j += kRoundThreads)
            if (hist[j]) atomicAdd(&cnt[j < c ? j : j - c], j < c ? hist[j] : 0u - hist[j]);
        __syncthreads();  // first[j] is now the end of key j's entries
        const int jobs = (int)task0[keys] * slices;
        for (int job = warp; job < jobs; job += kRoundWarps) {
            const int tk = job / slices, sl = job % slices;
            int lo = 0, hi = keys - 1;  // the last key whose first task is at most tk
            while (lo < hi) {
                const int mid = (lo + hi + 1) >> 1;
                if ((int)task0[mid] <= tk) lo = mid; else hi = mid - 1;
            }
            const int part = tk - (int)task0[lo];
            const int h = (int)hist[lo];
            const bool minus = lo >= c;
            count_task<VEC>(data, base, list + (first[lo] - h) + part * kTaskRows,
                            min(kTaskRows, h - part * kTaskRows), units, sl * lanes * VEC, lanes,
                            minus, flush + warp * 32 * kFlushStride,
                            bits + (int64_t)(minus ? lo - c : lo) * units * 32);
        }
        __syncthreads();
    }
}

// Majority centroids with the reference's per-lane OR accumulation
// (include/preproc/ibp_preproc_kmeans.cuh:219-236): bit set when count > size/2 (int div).
// One block per cluster: a warp per word, a lane per bit (coalesced counts, one ballot per
// 32 bits), then the accumulation over every 32nd word.
template <typename U>
__global__ void __launch_bounds__(256)
majority_kernel(const uint32_t *__restrict__ bits, const uint32_t *__restrict__ cnt, int64_t v,
                U *__restrict__ cent) {
    constexpr int W = 8 * sizeof(U);
    grid_dep_wait();
    grid_dep_release();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const uint32_t *bb = bits + (int64_t)blockIdx.x * v * W;
    U *cc = cent + (int64_t)blockIdx.x * v;
    const int32_t half = (int32_t)cnt[blockIdx.x] / 2;
    for (int64_t id = warp; id < v; id += 8) {
        uint64_t m = 0;
#pragma unroll
        for (int h = 0; h < W; h += 32) {
            const bool on = (int32_t)bb[id * W + h + lane] > half;
            m |= (uint64_t)__ballot_sync(0xffffffffu, on) << h;
        }
        if (lane == 0) cc[id] = (U)m;
    }
    __syncthreads();
    if (threadIdx.x < 32) {
        U acc = 0;
        for (int64_t id = threadIdx.x; id < v; id += 32) {
            acc |= cc[id];
            cc[id] = acc;
        }
    }
}

// Per-cluster masks (include/preproc/ibp_preproc_kmeans.cuh:238-297): counts accumulate in
// float32 there (saturating at 2^24); `>= thr*count` in float32, `<= (1-thr)*count` in
// float64; an empty cluster yields all-ones mask and bitval.  A warp per word, a lane per bit.
template <typename U>
__global__ void __launch_bounds__(256)
cluster_masks_kernel(const uint32_t *__restrict__ bits, const uint32_t *__restrict__ cnt, int64_t v,
                     int c, float thr, U *__restrict__ masks, U *__restrict__ bitvals) {
    constexpr int W = 8 * sizeof(U);
    const int lane = threadIdx.x & 31;
    const int64_t nwarps = (int64_t)gridDim.x * 8;
    for (int64_t e = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); e < (int64_t)c * v;
         e += nwarps) {
        const int32_t count = (int32_t)cnt[e / v];
        const float lim1 = __fmul_rn(thr, (float)count);
        const double lim0 = __dmul_rn(1.0 - (double)thr, (double)count);
        uint64_t m = 0, val = 0;
#pragma unroll
        for (int h = 0; h < W; h += 32) {
            const uint32_t bs = bits[e * W + h + lane];
            const float bsf = bs > 16777216u ? 16777216.0f : (float)bs;
            const bool one = bsf >= lim1;
            const bool inv = one || (double)bsf <= lim0;
            val |= (uint64_t)__ballot_sync(0xffffffffu, one) << h;
            m |= (uint64_t)__ballot_sync(0xffffffffu, inv) << h;
        }
        if (lane == 0) {
            masks[e] = (U)m;
            bitvals[e] = (U)val;
        }
    }
}

size_t kmeans_workspace(int64_t n, int64_t v, int wb, int c) {
    Sizer s;
    s.take<char>(kStatusBytes);
    s.take<int64_t>((size_t)c);                     // seed rows
    s.take<char>((size_t)c * v * wb);               // centroids
    s.take<uint32_t>((size_t)c * v * 8 * wb);       // bit counts
    s.take<uint32_t>((size_t)c);                    // cluster sizes
    s.take<int32_t>((size_t)n);                     // assignments
    return s.total();
}

// The ten rounds: assignment, counts, and (but for the last round) the next centroids.
template <typename U>
static ibp_status kmeans_rounds(const U *rows, int64_t n, int64_t v, int c, U *cent, uint32_t *bits,
                                uint32_t *cnt, int32_t *assign, int32_t *clusters,
                                cudaStream_t st) {
    const int sms = device_sm_count();
    const size_t maxs = (size_t)device_max_smem_optin();
    RoundShape sh;
    sh.units = (int)(v * (int64_t)sizeof(U) / 4);
    sh.groups = (sh.units + 15) / 16;
    sh.pairs = (c + 15) / 16;
    sh.assign = sh.fresh = true;
    if (sh.bytes(c) > maxs) sh.assign = false;
    const size_t smem = sh.bytes(c);
    const uint32_t *data = reinterpret_cast<const uint32_t *>(rows);
    const bool v16 = sh.units % 4 == 0 && (((uintptr_t)rows) & 15) == 0;
    const bool v8 = sh.units % 2 == 0 && (((uintptr_t)rows) & 7) == 0;
    auto rkern = v16 ? kmeans_round_kernel<true, 2>
                     : (v8 ? kmeans_round_kernel<false, 2> : kmeans_round_kernel<false, 1>);
    int per_sm = 0;
    IBP_RET(kernel_blocks_per_sm((const void *)rkern, kRoundThreads, smem, &per_sm));
    int64_t tile = ((n + sms - 1) / sms + 31) / 32 * 32;
    if (tile > kTileRows) tile = kTileRows;
    const int64_t blocks = std::min<int64_t>((n + tile - 1) / tile, sms);
    // fallback assignment
    const size_t cent_bytes = (size_t)c * v * sizeof(U);
    const bool cent_smem = cent_bytes <= 64 * 1024;
    auto akern = assign_kernel<U>;
    if (!sh.assign && cent_smem && cent_bytes > 48 * 1024)
        IBP_CUDA(cudaFuncSetAttribute(akern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                      (int)cent_bytes));
    const int64_t ablocks = std::max<int64_t>(1, std::min<int64_t>((n + 7) / 8, (int64_t)sms * 8));
    for (int it = 0; it < kKmRounds; ++it) {
        const bool last = it + 1 == kKmRounds;
        sh.fresh = it == 0 || !sh.assign;
        if (sh.fresh) {
            IBP_CUDA(cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * c, st));
            IBP_CUDA(cudaMemsetAsync(bits, 0, sizeof(uint32_t) * c * v * 8 * sizeof(U), st));
        }
        if (!sh.assign) {
            akern<<<(unsigned)ablocks, 256, cent_smem ? cent_bytes : 0, st>>>(rows, n, v, cent, c,
                                                                              cent_smem, assign);
            IBP_LAUNCHED("assign_kernel");
        }
        IBP_CUDA(launch_dependent(rkern, (unsigned)blocks, kRoundThreads, smem, st, data, n,
                                  reinterpret_cast<const uint32_t *>(cent), c, sh, (int)tile,
                                  assign, last ? clusters : nullptr, bits, cnt));
        IBP_LAUNCHED("kmeans_round_kernel");
        if (!last) {
            IBP_CUDA(launch_dependent(majority_kernel<U>, (unsigned)c, 256, 0, st, bits, cnt, v,
                                      cent));
            IBP_LAUNCHED("majority_kernel");
        }
    }
    return IBP_OK;
}

template <typename U>
ibp_status kmeans_impl(const U *data, int64_t n, int64_t v, int c, const int64_t *init_rows,
                       U *masks, U *bitvals, int32_t *clusters, void *ws, size_t ws_bytes,
                       cudaStream_t st) {
    constexpr int W = 8 * sizeof(U);
    const int wb = sizeof(U);
    Carver cv{(char *)ws, 0, ws_bytes};
    int32_t *status = cv.take<int32_t>(kStatusBytes / 4);
    int64_t *seed = cv.take<int64_t>((size_t)c);
    U *cent = cv.take<U>((size_t)c * v);
    uint32_t *bits = cv.take<uint32_t>((size_t)c * v * W);
    uint32_t *cnt = cv.take<uint32_t>((size_t)c);
    int32_t *assign = cv.take<int32_t>((size_t)n);
    if (!assign) {
        set_error("preprocess_kmeans: workspace of %zu bytes is below the required %zu",
                  ws_bytes, kmeans_workspace(n, v, wb, c));
        return IBP_ERR_WORKSPACE;
    }
    // optional HBM copy of a host-resident table (room left in the workspace)
    U *stage = cv.take<U>((size_t)(n * v));
    IBP_CUDA(cudaMemsetAsync(status, 0, sizeof(int32_t), st));
    const U *rows = data;
    if (stage && n > 0) {
        cudaPointerAttributes pa{};
        if (cudaPointerGetAttributes(&pa, data) == cudaSuccess && pa.type != cudaMemoryTypeDevice &&
            pa.type != cudaMemoryTypeManaged) {
            IBP_CUDA(cudaMemcpyAsync(stage, data, (size_t)(n * v) * wb, cudaMemcpyDefault, st));
            rows = stage;
        }
        cudaGetLastError();
    }
    const int64_t seeded = (int64_t)c < n ? (int64_t)c : n;
    std::vector<int64_t> h(c > 0 ? c : 1, 0);
    for (int64_t i = 1; i < seeded; ++i) h[i] = init_rows[i];
    IBP_CUDA(cudaMemcpyAsync(seed, h.data(), sizeof(int64_t) * c, cudaMemcpyHostToDevice, st));
    {
        int64_t tot = (int64_t)c * v;
        int blocks = (int)std::min<int64_t>((tot + 255) / 256, 1024);
        seed_centroids_kernel<U><<<blocks, 256, 0, st>>>(rows, n, v, seed, c, cent, status);
        IBP_LAUNCHED("seed_centroids_kernel");
    }
    if (n == 0) {
        IBP_CUDA(cudaMemsetAsync(cnt, 0, sizeof(uint32_t) * c, st));
        IBP_CUDA(cudaMemsetAsync(bits, 0, sizeof(uint32_t) * c * v * W, st));
    }
    // the most clusters a call may ask for (894 of 64-bit words, 1760 of 32-bit words)
    if ((size_t)c * (W + 1) * 4 > (size_t)device_max_smem_optin()) {
        set_error("preprocess_kmeans: %d clusters do not fit shared memory", c);
        return IBP_ERR_CUDA;
    }
    if (n > 0 && v > 0)
        IBP_RET(kmeans_rounds<U>(rows, n, v, c, cent, bits, cnt, assign, clusters, st));
    // the reference's final sweep leaves the masks of its last step, thr = 1.0f
    const ThrList sweep = sweep_thresholds(-1.0f);
    const float last = sweep.v[sweep.count - 1];
    if (c > 0 && v > 0) {
        int blocks = (int)std::min<int64_t>(((int64_t)c * v + 7) / 8, 4096);
        cluster_masks_kernel<U><<<blocks, 256, 0, st>>>(bits, cnt, v, c, last, masks, bitvals);
        IBP_LAUNCHED("cluster_masks_kernel");
    }
    return IBP_OK;
}

template ibp_status kmeans_impl<uint32_t>(const uint32_t *, int64_t, int64_t, int,
                                          const int64_t *, uint32_t *, uint32_t *, int32_t *,
                                          void *, size_t, cudaStream_t);
template ibp_status kmeans_impl<uint64_t>(const uint64_t *, int64_t, int64_t, int,
                                          const int64_t *, uint64_t *, uint64_t *, int32_t *,
                                          void *, size_t, cudaStream_t);

}  // namespace ibp200
