// ibp_compress.cu -- per-row compressed size, in-place bit packing and the condensed layout.
// Replaces include/misc/ibp_misc_{dev,kernels}.cuh (size check), include/compress/*.cuh
// (packer and its launchers) and the size/offset glue of src/compress.cu.
//
// B200 design
//  * sizes: 8, 16 or 32 lanes per row, 16 bytes a lane where rows allow it, 8 rows in flight, the
//    columns' tables in registers (few long rows: a warp or a block each); no shared-memory
//    atomics (the reference uses one 256-thread block per row with smem atomics).
//  * packing: a warp per row and 4 rows in flight; words go from memory to registers once
//    (host rows of whole 16-byte blocks: to shared memory), each lane gathers its words'
//    non-invariant bits with the Hacker's Delight move masks (in registers for rows of up to 512
//    bytes) and ORs them into a shared-memory image of the output row (three 32-bit shared
//    atomics per 64 bits of the row).  The finished row goes back with one coalesced pass; an
//    incompressible row compressed in place is not written at all.
//    No global workspace is cudaMalloc'd or freed per call (the reference does both and
//    thereby blocks the host).
#include <cub/device/device_scan.cuh>

#include <algorithm>

#include "ibp_codec.cuh"
#include "ibp_internal.cuh"
#include "ibp_match.cuh"

namespace ibp200 {

// ------------------------------------------------------------------ sizes
// Bound: reading the rows.  G lanes share a row (8, 16 or 32 by its pieces of A bytes) and
// take 8 rows at a time, all loads before any use, so a warp has up to 4 KiB in
// flight; the columns' mask, values and set bits stay in registers, loaded once when a group
// covers the row and once per 8 rows when it does not (1M rows of 128 16-bit words: 239 us
// with a 2-byte load and two table loads a word, 103 with half the lanes idle, 51 now, 5.2 TB/s;
// 200k rows of 99 32-bit words, in 4-byte pieces: 70 us, 78 with one piece a lane, 28 with four).
constexpr int kSizeRows = 8;

template <typename U, int A, int G, bool INDEX>
__global__ void __launch_bounds__(256, 2)
compress_size_kernel(const U *__restrict__ data, int64_t n, int64_t v,
                     const U *__restrict__ mask, const U *__restrict__ bitval,
                     const int64_t *__restrict__ idx, int64_t nrows,
                     int64_t *__restrict__ sizes, unsigned long long *__restrict__ total,
                     int32_t *__restrict__ status, uint32_t one) {
    using C = Chunk<U, A, G>;
    constexpr int RPW = 32 / G, Q = kSizeRows;
    __shared__ unsigned long long block_sum;
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), gin = lane / G;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t row_bytes = v * (int64_t)sizeof(U);
    const int64_t chunks = row_bytes / A;
    if (threadIdx.x == 0) block_sum = 0;
    __syncthreads();
    unsigned long long acc = 0;
    uint32_t m[C::NR], b[C::NR], pc[C::NW];
    auto tables = [&](int64_t c) {
        C::load_words(mask, c, chunks, m);
        C::load_words(bitval, c, chunks, b);
        C::set_bits(m, pc);
    };
    constexpr int SP = G * C::NS;  // pieces of a step
    const bool once = chunks <= SP;
    if (once && sub < chunks) tables(sub);
    for (int64_t base = warp * RPW * Q; base < nrows; base += nwarps * RPW * Q) {
        // positions i0 + q * RPW; consecutive rows without an index
        const int64_t i0 = base + gin;
        const char *row[INDEX ? Q : 1];
        unsigned okm = 0;
        if constexpr (INDEX) {
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const int64_t r = i0 + q * RPW < nrows ? idx[i0 + q * RPW] : -1;
                const bool ok = r >= 0 && r < n;
                okm |= (unsigned)ok << q;
                row[q] = reinterpret_cast<const char *>(data) + (ok ? r : 0) * row_bytes;
            }
        } else {
            row[0] = reinterpret_cast<const char *>(data) + i0 * row_bytes;
#pragma unroll
            for (int q = 0; q < Q; ++q) okm |= (unsigned)(i0 + q * RPW < nrows) << q;
        }
        uint32_t s[Q];
#pragma unroll
        for (int q = 0; q < Q; ++q) s[q] = 0;
        for (int64_t c = sub; c < chunks; c += SP) {
            uint32_t x[Q][C::NR];
#pragma unroll
            for (int q = 0; q < Q; ++q)
                if ((okm >> q) & 1)
                    C::load(INDEX ? row[INDEX ? q : 0] : row[0] + q * RPW * row_bytes, c, chunks, x[q]);
            if (!once) tables(c);
#pragma unroll
            for (int q = 0; q < Q; ++q)
                if ((okm >> q) & 1)
                    C::matched(s[q], [&](int k) { return (x[q][k] & m[k]) ^ b[k]; }, pc, one);
        }
        group_sums<Q, G>(s, one);
        const int q = group_sums_value<Q, G>(sub);
        const int64_t i = base + q * RPW + gin;
        if ((sub & (group_sums_copies<Q, G>() - 1)) == 0 && i < nrows) {
            if ((okm >> q) & 1) {
                const int64_t sz = compressed_bytes(v, (int)sizeof(U), s[0]);
                sizes[i] = sz;
                acc += (unsigned long long)sz;
            } else {
                sizes[i] = 0;
                if (status) atomicOr(status, kStatusBadIndex);
            }
        }
    }
    if (total) {
        acc = group_sum<32>(acc);
        if (lane == 0 && acc) atomicAdd(&block_sum, acc);
        __syncthreads();
        if (threadIdx.x == 0 && block_sum) atomicAdd(total, block_sum);
    }
}

// Few rows of more than one step: a row to a warp or, with ROWS == 1, to a block of 8 warps, 4 steps
// of a warp in flight.
template <typename U, int A, int ROWS, bool INDEX>
__global__ void __launch_bounds__(256, 4)
few_rows_size_kernel(const U *__restrict__ data, int64_t n, int64_t v,
                     const U *__restrict__ mask, const U *__restrict__ bitval,
                     const int64_t *__restrict__ idx, int64_t nrows,
                     int64_t *__restrict__ sizes, unsigned long long *__restrict__ total,
                     int32_t *__restrict__ status, uint32_t one) {
    using C = Chunk<U, A, 32>;
    constexpr int P = 4, SP = 32 * C::NS, WARPS = 8 / ROWS;  // warps of a row
    __shared__ uint32_t sums[2][8];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int64_t row_bytes = v * (int64_t)sizeof(U);
    const int64_t chunks = row_bytes / A;
    const int part = warp % WARPS;
    unsigned long long acc = 0;
    int now = 0;
    for (int64_t i = (int64_t)blockIdx.x * ROWS + warp / WARPS; i < nrows;
         i += (int64_t)gridDim.x * ROWS) {
        const int64_t r = INDEX ? idx[i] : i;
        if (INDEX && (r < 0 || r >= n)) {
            if (part == 0 && lane == 0) {
                sizes[i] = 0;
                if (status) atomicOr(status, kStatusBadIndex);
            }
            continue;
        }
        const char *row = reinterpret_cast<const char *>(data) + r * row_bytes;
        uint32_t s = 0;
        for (int64_t c = (int64_t)part * P * SP + lane; c < chunks; c += WARPS * P * SP) {
            uint32_t x[P][C::NR];
#pragma unroll
            for (int p = 0; p < P; ++p) C::load(row, c + p * SP, chunks, x[p]);
#pragma unroll
            for (int p = 0; p < P; ++p) {
                uint32_t m[C::NR], b[C::NR], pc[C::NW];
                C::load_words(mask, c + p * SP, chunks, m);
                C::load_words(bitval, c + p * SP, chunks, b);
                C::set_bits(m, pc);
                C::matched(s, [&](int k) { return (x[p][k] & m[k]) ^ b[k]; }, pc, one);
            }
        }
        s = __reduce_add_sync(0xffffffffu, s);
        if constexpr (WARPS > 1) {
            // (two sets of sums: the one read here is next written after the next row's barrier)
            if (lane == 0) sums[now][warp] = s;
            __syncthreads();
            s = __reduce_add_sync(0xffffffffu, lane < WARPS ? sums[now][lane] : 0u);
            now ^= 1;
        }
        if (part == 0 && lane == 0) {
            const int64_t sz = compressed_bytes(v, (int)sizeof(U), s);
            sizes[i] = sz;
            acc += (unsigned long long)sz;
        }
    }
    if (total && acc) atomicAdd(total, acc);
}

template <typename U, int A>
static ibp_status launch_sizes(const U *data, int64_t n, int64_t v, const U *mask,
                               const U *bitval, const int64_t *idx, int64_t nrows,
                               int64_t *sizes, int64_t *total, int32_t *status,
                               cudaStream_t st) {
    const int64_t chunks = v * (int64_t)sizeof(U) / A;
    int per_sm = 0;
    // Rows of several steps, too few for every warp to have 8: a block each up to 8 rows per SM (and
    // of long ones up to 32), a warp each up to 48.  600 rows of 60,000 32-bit words: a warp each
    // and a word a lane 425 us, eight to a warp 545, a block each 50; 3333 of 4096, indexed: 18.7, 31.5,
    // 19.4 (a block each 22); 10,000 of 2000 64-bit words 48, 46 (a block each 50), and off 16-byte
    // boundaries, where eight rows to a warp are slower, 48, 57, 38.
    const int64_t sms = device_sm_count();
    const bool block_each = nrows <= 8 * sms || (nrows <= 32 * sms && v * sizeof(U) >= 32768);
    if (chunks > 32 * Chunk<U, A, 32>::NS && (block_each || nrows <= (A == 16 ? 48 : 128) * sms)) {
        auto few = block_each ? (idx ? few_rows_size_kernel<U, A, 1, true>
                                     : few_rows_size_kernel<U, A, 1, false>)
                              : (idx ? few_rows_size_kernel<U, A, 8, true>
                                     : few_rows_size_kernel<U, A, 8, false>);
        IBP_RET(kernel_blocks_per_sm((const void *)few, 256, 0, &per_sm));
        const int64_t blocks =
            std::min<int64_t>(block_each ? nrows : (nrows + 7) / 8, sms * per_sm);
        few<<<(unsigned)blocks, 256, 0, st>>>(data, n, v, mask, bitval, idx, nrows, sizes,
                                              (unsigned long long *)total, status, 1u);
        IBP_LAUNCHED("few_rows_size_kernel");
        return IBP_OK;
    }
    auto kern = idx ? compress_size_kernel<U, A, 32, true> : compress_size_kernel<U, A, 32, false>;
    int lanes = 32;
    if (chunks <= 8 * Chunk<U, A, 8>::NS) {
        kern = idx ? compress_size_kernel<U, A, 8, true> : compress_size_kernel<U, A, 8, false>;
        lanes = 8;
    } else if (chunks <= 16 * Chunk<U, A, 8>::NS) {
        kern = idx ? compress_size_kernel<U, A, 16, true> : compress_size_kernel<U, A, 16, false>;
        lanes = 16;
    }
    const int64_t per_block = 8 * kSizeRows * (32 / lanes);
    IBP_RET(kernel_blocks_per_sm((const void *)kern, 256, 0, &per_sm));
    const int64_t blocks = std::min<int64_t>((nrows + per_block - 1) / per_block,
                                             (int64_t)device_sm_count() * per_sm);
    kern<<<(unsigned)blocks, 256, 0, st>>>(data, n, v, mask, bitval, idx, nrows, sizes,
                                           (unsigned long long *)total, status, 1u);
    IBP_LAUNCHED("compress_size_kernel");
    return IBP_OK;
}

template <typename U>
ibp_status compress_size_impl(const U *data, int64_t n, int64_t v, const U *mask,
                              const U *bitval, const int64_t *idx, int64_t nrows,
                              int64_t *sizes, int64_t *total, int32_t *status,
                              cudaStream_t st) {
    if (nrows <= 0) return IBP_OK;
    const int a = row_piece_bytes(data, v, sizeof(U));
    if (a == 16)
        return launch_sizes<U, 16>(data, n, v, mask, bitval, idx, nrows, sizes, total, status, st);
    if constexpr (sizeof(U) < 4)
        if (a == 4)
            return launch_sizes<U, 4>(data, n, v, mask, bitval, idx, nrows, sizes, total, status,
                                      st);
    return launch_sizes<U, sizeof(U)>(data, n, v, mask, bitval, idx, nrows, sizes, total, status,
                                      st);
}

// ------------------------------------------------------------------ packing
template <typename U>
struct PackArgs {
    const U *src;
    int64_t n, v;
    ColTables<U> t;
    const int64_t *idx;
    int64_t nrows;
    U *out;             // fixed-stride output rows (nullptr for condensed)
    U *cond;            // condensed output base (word aligned offsets)
    const int64_t *offsets;
    bool in_place;      // out rows alias src rows one to one
    int32_t *bitmask;
    int32_t *status;
    int64_t buf_words;  // shared-memory words per output row
    int64_t stage_words;  // and per input row, for rows in host memory
};

// A lane packs 64 bits of a row at a time, as two halves, high first: one 64-bit word, or two
// neighbouring 32-bit words, each compressible or not on its own.  A chunk is 32 lanes of that
// (32 or 64 columns), a group NC chunks.  The tables of a lane's halves in a group, where each
// lane's bits start and where the group's end when all of it is compressible.
template <typename U, int NC>
struct PackTables {
    static constexpr bool PAIR = sizeof(U) == 4;
    static constexpr int COLS = PAIR ? 64 : 32;      // columns of a chunk
    static constexpr int UNITS = NC * (COLS / 32);   // bitmap units of a group
    uint32_t m[NC][2], bv[NC][2], mv[NC][2][kMoves];
    uint32_t nb[NC], nbh[NC];  // kept bits of both halves, of the first
    uint32_t before[NC], all;
    uint32_t valid;  // lane u < UNITS: the columns of bitmap unit u that exist
    int left;        // columns from this lane's first in the group to the row's end
    int levels;      // moves the group's columns need (gather_left)

    __device__ __forceinline__ static void split(U x, uint32_t (&h)[2]) {
        h[0] = (uint32_t)((uint64_t)x >> 32);
        h[1] = (uint32_t)x;
    }

    __device__ __forceinline__ void load(const ColTables<U> &t, int v, int j0,
                                         bool count_levels = false) {
        const int lane = threadIdx.x & 31;
        uint32_t moves[kMoves] = {};
        const int of_unit = v - j0 - 32 * lane;
        valid = lane >= UNITS || of_unit <= 0 ? 0u : (of_unit >= 32 ? ~0u : (1u << of_unit) - 1u);
        left = v - j0 - (PAIR ? 2 : 1) * lane;
        all = 0;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            // a column past the end: no bits, always compressible
            if constexpr (PAIR) {
                uint32_t k[2];
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int64_t j = j0 + COLS * c + 2 * lane + h;
                    const bool in = j < v;
                    m[c][h] = in ? __ldg(&t.mask[j]) : 0u;
                    bv[c][h] = in ? __ldg(&t.bitval[j]) : 0u;
                    k[h] = in ? (uint32_t)__ldg(&t.nb[j]) : 0u;
#pragma unroll
                    for (int i = 0; i < kMoves; ++i)
                        mv[c][h][i] = in ? __ldg(&t.mv[i * (int64_t)v + j]) : 0u;
                    if (!in) m[c][h] = bv[c][h] = 0;
                }
                nbh[c] = k[0];
                nb[c] = k[0] + k[1];
            } else {
                const int64_t j = j0 + COLS * c + lane;
                const bool in = j < v;
                split(in ? __ldg(&t.mask[j]) : (U)0, m[c]);
                split(in ? __ldg(&t.bitval[j]) : (U)0, bv[c]);
                const uint32_t k = in ? (uint32_t)__ldg(&t.nb[j]) : 0u;
                nb[c] = k & 0xffu;
                nbh[c] = nb[c] - (k >> 8);
#pragma unroll
                for (int i = 0; i < kMoves; ++i) {
                    uint32_t h[2];
                    split(in ? __ldg(&t.mv[i * (int64_t)v + j]) : (U)0, h);
                    mv[c][0][i] = h[0];
                    mv[c][1][i] = h[1];
                }
            }
#pragma unroll
            for (int i = 0; i < kMoves; ++i) moves[i] |= mv[c][0][i] | mv[c][1][i];
            uint32_t incl = nb[c];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += y;
            }
            before[c] = all + incl - nb[c];
            all += __shfl_sync(0xffffffffu, incl, 31);
        }
        levels = kMoves;
        if (count_levels) {
            levels = 0;
#pragma unroll
            for (int i = 0; i < kMoves; ++i)
                if (__any_sync(0xffffffffu, moves[i] != 0)) levels = i + 1;
        }
    }

    // this lane's halves of chunk c of a row (p: the row's word at the lane's first column of the
    // group; wide: pairs of words are 8-byte aligned)
    __device__ __forceinline__ void read(const U *p, int c, int left_, bool wide,
                                         uint32_t (&x)[2]) const {
        x[0] = x[1] = 0;
        if constexpr (PAIR) {
            if (wide) {
                if (COLS * c < left_) {
                    const uint2 y = *reinterpret_cast<const uint2 *>(p + COLS * c);
                    x[0] = y.x;
                    x[1] = y.y;
                }
            } else {
                if (COLS * c < left_) x[0] = p[COLS * c];
                if (COLS * c + 1 < left_) x[1] = p[COLS * c + 1];
            }
        } else {
            if (COLS * c < left_) split(p[COLS * c], x);
        }
    }
};

// Moves `words` words of a row image (units in stream order: a 64-bit word's high half first)
// to global memory and leaves zeros in their place.
template <typename U>
__device__ __forceinline__ void write_image(U *__restrict__ dst, uint32_t *image, int words) {
    const int lane = threadIdx.x & 31;
    int done = 0;
    if ((((uintptr_t)dst) & 15) == 0) {
        uint4 *d4 = reinterpret_cast<uint4 *>(dst), *b4 = reinterpret_cast<uint4 *>(image);
        const int n16 = words * (int)sizeof(U) / 16;
        for (int k = lane; k < n16; k += 32) {
            const uint4 x = b4[k];
            b4[k] = make_uint4(0, 0, 0, 0);
            d4[k] = sizeof(U) == 8 ? make_uint4(x.y, x.x, x.w, x.z) : x;
        }
        done = n16 * (16 / (int)sizeof(U));
    }
    for (int k = done + lane; k < words; k += 32) {
        if constexpr (sizeof(U) == 8) {
            dst[k] = (uint64_t)image[2 * k] << 32 | image[2 * k + 1];
            image[2 * k] = image[2 * k + 1] = 0;
        } else {
            dst[k] = image[k];
            image[k] = 0;
        }
    }
}

// Packs a group of a row (x: this lane's halves): its bitmap units and its words' kept bits are
// ORed into the row's zeroed image (a shared address) from stream bit `at` on, which moves past
// the group.  Offsets come from the tables where the group is all compressible, else from a
// prefix sum.  A row of one group that would end past stream bit `limit` leaves the image alone.
template <typename U, int NC, bool ONE, int LEVELS>
__device__ __forceinline__ void pack_group(const PackTables<U, NC> &t, const uint32_t (&x)[NC][2],
                                           int g, int chunks, uint32_t image, uint32_t &at,
                                           uint32_t limit) {
    using T = PackTables<U, NC>;
    constexpr int H = sizeof(U) / 4;
    const int lane = threadIdx.x & 31;
    uint32_t p0[NC], p1[NC], off[NC];  // the halves' bits, gathered left
    bool c0[NC], c1[NC];               // the halves compress (64-bit words: together)
    bool every = true;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        if (!ONE && c >= chunks) {  // past the row's end
            c0[c] = c1[c] = true;
            p0[c] = p1[c] = 0;
            off[c] = at;
            continue;
        }
        const uint32_t e0 = (x[c][0] & t.m[c][0]) ^ t.bv[c][0];
        const uint32_t e1 = (x[c][1] & t.m[c][1]) ^ t.bv[c][1];
        c0[c] = T::PAIR ? e0 == 0 : (e0 | e1) == 0;
        c1[c] = T::PAIR ? e1 == 0 : c0[c];
        every = every && (e0 | e1) == 0;
        p0[c] = gather_left<LEVELS>(x[c][0], t.m[c][0], t.mv[c][0]);
        p1[c] = gather_left<LEVELS>(x[c][1], t.m[c][1], t.mv[c][1]);
        off[c] = at + t.before[c];
    }
    uint32_t bits = t.valid;  // lane u < UNITS: bitmap unit u of the group
    uint32_t split[NC];       // bits of the first half
#pragma unroll
    for (int c = 0; c < NC; ++c) split[c] = t.nbh[c];
    if (__all_sync(0xffffffffu, every)) {
        at += t.all;
    } else {
        bits = 0;
#pragma unroll
        for (int c = 0; c < NC; ++c) {
            // bitmap units, LSB-first
            if constexpr (T::PAIR) {
                const uint32_t f = (uint32_t)c0[c] | (uint32_t)c1[c] << 1;
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const uint32_t z = __shfl_sync(0xffffffffu, f, 16 * h + (lane >> 1));
                    const uint32_t b = __ballot_sync(0xffffffffu, (z >> (lane & 1)) & 1);
                    if (lane == 2 * c + h) bits = b;
                }
            } else {
                const uint32_t b = __ballot_sync(0xffffffffu, c0[c]);
                if (lane == c) bits = b;
            }
            split[c] = c0[c] ? t.nbh[c] : 32u;
            const uint32_t len = split[c] + (c1[c] ? t.nb[c] - t.nbh[c] : 32u);
            uint32_t incl = len;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t z = __shfl_up_sync(0xffffffffu, incl, o);
                if (lane >= o) incl += z;
            }
            off[c] = at + incl - len;
            at += __shfl_sync(0xffffffffu, incl, 31);
            p0[c] = c0[c] ? p0[c] : x[c][0];
            p1[c] = c1[c] ? p1[c] : x[c][1];
        }
        bits &= t.valid;
    }
    if (ONE && at > limit) return;
    // bitmap units in memory order (units past the row's last are zero and belong to
    // the stream, where an OR of nothing does no harm)
    or_shared(image + (uint32_t)((g * T::UNITS + (lane & (T::UNITS - 1))) ^ (H - 1)) * 4, bits);
#pragma unroll
    for (int c = 0; c < NC; ++c)
        if (ONE || c < chunks)
            put_bits(image, off[c], p0[c] | __funnelshift_rc(p1[c], 0, split[c]),
                     __funnelshift_rc(0, p1[c], split[c]));
}

// Whether the rows at src(0), ..., src(Q - 1) save so few bits that all of them stay raw: the bits
// set in the masks of their matching words are added up, as in the size pass.
template <typename U, int Q, typename Src>
__device__ __forceinline__ bool all_raw(const ColTables<U> &t, int v, Src src) {
    constexpr int N = 8 / Q, P = 16 / sizeof(U);  // blocks of a lane and row in flight, their words
    const int lane = threadIdx.x & 31;
    const U *row[Q];
    uint32_t s[Q];
    bool aligned = v % P == 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        row[q] = src(q);
        s[q] = 0;
        aligned = aligned && (((uintptr_t)row[q]) & 15) == 0;
    }
    if (aligned) {
        const uint4 *mask = reinterpret_cast<const uint4 *>(t.mask);
        const uint4 *value = reinterpret_cast<const uint4 *>(t.bitval);
        for (int i0 = lane; i0 < v / P; i0 += 32 * N) {
            uint4 x[Q][N];
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int k = 0; k < N; ++k)
                    if (i0 + 32 * k < v / P)
                        x[q][k] = reinterpret_cast<const uint4 *>(row[q])[i0 + 32 * k];
#pragma unroll
            for (int k = 0; k < N; ++k) {
                if (i0 + 32 * k >= v / P) break;
                const uint4 m = __ldg(mask + i0 + 32 * k), b = __ldg(value + i0 + 32 * k);
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const uint32_t e[4] = {(x[q][k].x & m.x) ^ b.x, (x[q][k].y & m.y) ^ b.y,
                                           (x[q][k].z & m.z) ^ b.z, (x[q][k].w & m.w) ^ b.w};
                    const uint32_t c[4] = {(uint32_t)__popc(m.x), (uint32_t)__popc(m.y),
                                           (uint32_t)__popc(m.z), (uint32_t)__popc(m.w)};
                    if constexpr (sizeof(U) == 8) {
                        if ((e[0] | e[1]) == 0) s[q] += c[0] + c[1];
                        if ((e[2] | e[3]) == 0) s[q] += c[2] + c[3];
                    } else {
#pragma unroll
                        for (int i = 0; i < 4; ++i)
                            if (e[i] == 0) s[q] += c[i];
                    }
                }
            }
        }
    } else {
        for (int j = lane; j < v; j += 32) {
            const U m = __ldg(t.mask + j), b = __ldg(t.bitval + j);
            const uint32_t saved = popc_w(m);
#pragma unroll
            for (int q = 0; q < Q; ++q)
                if ((U)(row[q][j] & m) == b) s[q] += saved;
        }
    }
    // none saves more than the one that saves most
    uint32_t most = 0;
#pragma unroll
    for (int q = 0; q < Q; ++q) most = max(most, __reduce_add_sync(0xffffffffu, s[q]));
    return compressed_bytes(v, (int)sizeof(U), most) == v * (int64_t)sizeof(U);
}

// Whether the words x of a row's first group save less than a sixteenth of their bits.
template <typename U, int NC>
__device__ __forceinline__ bool saves_little(const ColTables<U> &t, int v, const uint32_t (&x)[NC][2]) {
    using T = PackTables<U, NC>;
    const int lane = threadIdx.x & 31;
    uint32_t s = 0;
#pragma unroll
    for (int c = 0; c < NC; ++c) {
        if constexpr (T::PAIR) {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const int j = T::COLS * c + 2 * lane + h;
                const U m = j < v ? __ldg(t.mask + j) : (U)0;
                if ((x[c][h] & m) == (j < v ? __ldg(t.bitval + j) : (U)0)) s += popc_w(m);
            }
        } else {
            const int j = T::COLS * c + lane;
            const U m = j < v ? __ldg(t.mask + j) : (U)0, y = (U)((uint64_t)x[c][0] << 32 | x[c][1]);
            if ((U)(y & m) == (j < v ? __ldg(t.bitval + j) : (U)0)) s += popc_w(m);
        }
    }
    return __reduce_add_sync(0xffffffffu, s) * 16 <
           (uint32_t)min(v, NC * T::COLS) * 8 * (uint32_t)sizeof(U);
}

// A warp takes Q consecutive positions at a time.  Each row goes through registers once: a
// lane gathers its words' kept bits (left-aligned) and ORs them into the row's zeroed
// shared-memory image at the word's bit offset, and the row's length falls out of the last
// offset; the image is then written and zeroed for the next row.  Rows of up to one group keep
// their tables in registers (ONE), and one that stays raw is known before it reaches its image.
// Longer ones load the tables per group of columns, for Q rows at once.  A warp passes over the
// batches it starts with for as long as all their rows stay raw (long ones are looked through only
// where the first group of the first row saves next to nothing).  96 MiB of rows that all stay raw,
// kernel time, packed and dropped before and now: of 64 32-bit words 129 and 58 us, of 256 100 and
// 31, of 1000 140 and 36; of 64 64-bit words 82 and 37, of 300 93 and 30.
// The words of the next step are loaded while this one is packed.  LEVELS: moves per gather.
template <typename U, int NC, int Q, bool ONE, bool INDEX, int LEVELS>
__device__ __forceinline__ void pack_rows(const PackArgs<U> &a, PackTables<U, NC> &t) {
    using T = PackTables<U, NC>;
    constexpr int W = 8 * sizeof(U), H = sizeof(U) / 4;
    constexpr int GCOLS = T::COLS * NC, STEP = T::PAIR ? 2 : 1;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    uint32_t *images = reinterpret_cast<uint32_t *>(smem) +
                       (int64_t)(threadIdx.x >> 5) * Q * a.buf_words * H;
    const int image_units = (int)a.buf_words * H;
    const uint32_t images_at = (uint32_t)__cvta_generic_to_shared(images);
    const int v = (int)a.v;
    const uint32_t stream0 = (uint32_t)meta_bytes(v, (int)sizeof(U)) * 8;
    const uint32_t limit = (uint32_t)(v - 1) * W;  // last stream bit of a row below the raw one
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t batches = (a.nrows + Q - 1) / Q;
    const int groups = ONE ? 1 : (v + GCOLS - 1) / GCOLS;
    const bool wide = T::PAIR && v % 2 == 0 && (((uintptr_t)a.src) & 7) == 0;
    for (int k = lane; k < Q * image_units; k += 32) images[k] = 0;
    __syncwarp();
    // source row of position batch * Q + q (-1: none)
    auto source = [&](int64_t batch, int q) -> int64_t {
        const int64_t i = batch * Q + q;
        if (i >= a.nrows) return -1;
        if (!INDEX) return i;
        const int64_t r = a.idx[i];
        return r >= 0 && r < a.n ? r : -1;
    };
    auto load = [&](int64_t batch, int g, uint32_t (&x)[Q][NC][2]) {
        const int j = g * GCOLS + STEP * lane;
        if (!INDEX && (batch + 1) * Q <= a.nrows) {  // Q rows one after the other
            const U *p = a.src + batch * Q * v + j;
#pragma unroll
            for (int q = 0; q < Q; ++q, p += v)
#pragma unroll
                for (int c = 0; c < NC; ++c) t.read(p, c, v - j, wide, x[q][c]);
            return;
        }
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int64_t r = source(batch, q);
            const U *p = a.src + (r < 0 ? 0 : r) * v + j;
#pragma unroll
            for (int c = 0; c < NC; ++c) t.read(p, c, r < 0 ? 0 : v - j, wide, x[q][c]);
        }
    };
    // where row i of the output starts
    auto target = [&](int64_t i) -> U * {
        return a.out ? a.out + i * v
                     : reinterpret_cast<U *>(reinterpret_cast<char *>(a.cond) +
                                             (i ? a.offsets[i - 1] : 0));
    };
    // fixed-stride rows of whole 16-byte blocks, at most one per lane
    const int n16 = v * (int)sizeof(U) / 16;
    const bool blocks = ONE && a.out && n16 <= 32 && v * (int)sizeof(U) % 16 == 0 &&
                        (((uintptr_t)a.out) & 15) == 0;
    uint32_t x[Q][NC][2];
    int64_t batch = warp;
    // batches of rows that all stay raw, up to the first other one
    for (; batch < batches; batch += nwarps) {
        if constexpr (!ONE) {
            load(batch, 0, x);
            if (!saves_little<U, NC>(a.t, v, x[0])) break;
        }
        // (a batch with a position that has no row, which must not be read, goes on below)
        bool whole = true;
#pragma unroll
        for (int q = 0; q < Q; ++q) whole = whole && source(batch, q) >= 0;
        if (!whole) break;
        if (!all_raw<U, Q>(a.t, v, [&](int q) { return a.src + source(batch, q) * v; })) break;
#pragma unroll
        for (int q = 0; q < Q; ++q)
            if (!a.in_place)
                warp_copy<U>(target(batch * Q + q), a.src + source(batch, q) * v, v);
    }
    if (ONE && batch < batches) load(batch, 0, x);
    for (; batch < batches; batch += nwarps) {
        uint32_t at[Q];  // stream bits so far
#pragma unroll
        for (int q = 0; q < Q; ++q) at[q] = stream0;
        for (int g = 0; g < groups; ++g) {
            uint32_t y[Q][NC][2];
            const bool more = g + 1 < groups;
            if (more || batch + nwarps < batches)
                load(more ? batch : batch + nwarps, more ? g + 1 : 0, y);
            if (!ONE) t.load(a.t, v, g * GCOLS);
            const int chunks = ONE ? NC : min(NC, (v - g * GCOLS + T::COLS - 1) / T::COLS);
#pragma unroll
            for (int q = 0; q < Q; ++q)
                pack_group<U, NC, ONE, LEVELS>(t, x[q], g, chunks,
                                               images_at + q * image_units * 4, at[q], limit);
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int c = 0; c < NC; ++c)
#pragma unroll
                    for (int h = 0; h < 2; ++h) x[q][c][h] = y[q][c][h];
        }
        __syncwarp();
        unsigned packed = 0;
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int64_t i = batch * Q + q;
            if (i >= a.nrows) break;
            const int64_t r = source(batch, q);
            uint32_t *image = images + q * image_units;
            // bitmap and stream in whole words; stored compressed only when below the raw row
            const int words = (int)((at[q] + W - 1) / W);
            if (r >= 0 && words < v) {
                packed |= 1u << q;
                if (blocks) {
                    if (lane < n16) {
                        uint4 *b4 = reinterpret_cast<uint4 *>(image) + lane;
                        const uint4 x = *b4;
                        *b4 = make_uint4(0, 0, 0, 0);
                        reinterpret_cast<uint4 *>(a.out + i * v)[lane] =
                            H == 2 ? make_uint4(x.y, x.x, x.w, x.z) : x;
                    }
                } else {
                    write_image<U>(target(i), image, a.out ? v : words);
                }
                continue;
            }
            if (r < 0 && lane == 0) atomicOr(a.status, kStatusBadIndex);
            if (r >= 0 && !a.in_place) warp_copy<U>(target(i), a.src + r * v, v);
            if (ONE && words >= v) continue;  // nothing was packed
            for (int k = lane; k < words * H; k += 32) image[k] = 0;
        }
        // Q divides 32 and the batch starts at a multiple of Q: one bitmask word
        if (a.out && packed && lane == 0)
            atomicOr(&a.bitmask[batch * Q >> 5], (int32_t)(packed << (batch * Q & 31)));
        __syncwarp();
    }
}

// Bound: the integer pipe (three operations per move and 32-bit half) and the shared atomics,
// then HBM. 600k rows of 64 64-bit words: 459 us with tables read through L1 and the row staged
// and packed in two passes; 317 with tables in registers; 207 with 32-bit indices and images in
// stream order; 188 with the moves chosen once; 163 without a test per atomic (its branches cost
// more than the atomics of zeros); 137 with the 16-byte epilogue; 120 now, 4.6 TB/s, with raw
// rows out of the loop's way (what else stands in the function decides how the loop is compiled:
// the same loop took 120 to 143 under different ways to pass over raw batches). 32-bit words two
// to a lane rather than one (half the prefix sums, three atomics for two words instead of four):
// 200k rows of 99 words 254 us at first, 110, 92 now; of 400 words 308, 164, 150. Rows whose
// tables stay in registers choose their moves once (LEVELS 2 covers masks that drop at most
// three bits above any kept one, as quantised floats do).
template <typename U, int NC, int Q, bool ONE, bool INDEX>
__global__ void __launch_bounds__(256, 2) pack_rows_kernel(PackArgs<U> a) {
    PackTables<U, NC> t;
    if (ONE) {
        t.load(a.t, (int)a.v, 0, true);
        if (t.levels <= 2) {
            pack_rows<U, NC, Q, ONE, INDEX, 2>(a, t);
            return;
        }
    }
    pack_rows<U, NC, Q, ONE, INDEX, kMoves>(a, t);
}

// Rows in host memory: a warp brings a row over the link once, whole, into shared memory, where
// its size is taken, and writes it from there or packs it.  Bound: the link.  Through
// pack_rows_kernel, whose lanes fetch their own words of four rows and which reads a row that
// stays raw twice: 30k rows of 300 64-bit words in place 2372 us, here 2007; 10k raw ones of 1000
// back to back 6421 and 4605.
template <typename U, int NC, bool ONE, bool INDEX>
__global__ void __launch_bounds__(256, 2) pack_host_rows_kernel(PackArgs<U> a) {
    using T = PackTables<U, NC>;
    constexpr int W = 8 * sizeof(U), H = sizeof(U) / 4, GCOLS = T::COLS * NC;
    extern __shared__ __align__(16) unsigned char smem[];
    const int lane = threadIdx.x & 31;
    U *row = reinterpret_cast<U *>(smem) +
             (int64_t)(threadIdx.x >> 5) * (a.stage_words + a.buf_words);
    uint32_t *image = reinterpret_cast<uint32_t *>(row + a.stage_words);
    const uint32_t image_at = (uint32_t)__cvta_generic_to_shared(image);
    const int v = (int)a.v;
    const uint32_t stream0 = (uint32_t)meta_bytes(v, (int)sizeof(U)) * 8;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int k = lane; k < (int)a.buf_words * H; k += 32) image[k] = 0;
    T t;
    if (ONE) t.load(a.t, v, 0);
    for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; i < a.nrows;
         i += nwarps) {
        const int64_t r = INDEX ? a.idx[i] : i;
        if (INDEX && (r < 0 || r >= a.n)) {
            if (lane == 0) atomicOr(a.status, kStatusBadIndex);
            continue;
        }
        warp_copy<U>(row, a.src + r * v, v);
        __syncwarp();
        uint32_t s = 0;
        for (int j = lane; j < v; j += 32) {
            const U m = __ldg(a.t.mask + j);
            if ((U)(row[j] & m) == __ldg(a.t.bitval + j)) s += popc_w(m);
        }
        s = __reduce_add_sync(0xffffffffu, s);
        U *o = a.out ? a.out + i * v
                     : reinterpret_cast<U *>(reinterpret_cast<char *>(a.cond) +
                                             (i ? a.offsets[i - 1] : 0));
        if (compressed_bytes(v, (int)sizeof(U), s) == v * (int64_t)sizeof(U)) {
            if (!a.in_place) warp_copy<U>(o, row, v);
            __syncwarp();
            continue;
        }
        uint32_t at = stream0;
        for (int j0 = 0, g = 0; j0 < v; j0 += GCOLS, ++g) {
            if (!ONE) t.load(a.t, v, j0);
            const int j = j0 + (T::PAIR ? 2 : 1) * lane;
            uint32_t x[NC][2];
#pragma unroll
            for (int c = 0; c < NC; ++c) t.read(row + j, c, v - j, v % 2 == 0, x[c]);
            pack_group<U, NC, ONE, kMoves>(t, x, g, min(NC, (v - j0 + T::COLS - 1) / T::COLS),
                                           image_at, at, ~0u);
        }
        __syncwarp();
        write_image<U>(o, image, a.out ? v : (int)((at + W - 1) / W));
        if (a.out && lane == 0) atomicOr(&a.bitmask[i >> 5], (int32_t)(1u << (i & 31)));
        __syncwarp();
    }
}

template <typename U, int NC, bool ONE>
static ibp_status launch_pack_host(const PackArgs<U> &a, size_t row, cudaStream_t st) {
    auto kern = a.idx ? pack_host_rows_kernel<U, NC, ONE, true> : pack_host_rows_kernel<U, NC, ONE, false>;
    const int warps = (int)std::max<size_t>(1, std::min<size_t>(8, 96 * 1024 / row));
    int per_sm = 0;
    IBP_RET(kernel_blocks_per_sm((const void *)kern, warps * 32, warps * row, &per_sm));
    const int64_t blocks =
        std::min<int64_t>((a.nrows + warps - 1) / warps, (int64_t)device_sm_count() * per_sm);
    kern<<<(unsigned)blocks, warps * 32, warps * row, st>>>(a);
    IBP_LAUNCHED("pack_host_rows_kernel");
    return IBP_OK;
}

template <typename U, int NC, int Q, bool ONE>
static ibp_status launch_pack_q(const PackArgs<U> &a, int warps, size_t smem, cudaStream_t st) {
    auto kern = a.idx ? pack_rows_kernel<U, NC, Q, ONE, true> : pack_rows_kernel<U, NC, Q, ONE, false>;
    int per_sm = 0;
    IBP_RET(kernel_blocks_per_sm((const void *)kern, warps * 32, smem, &per_sm));
    const int64_t batches = (a.nrows + Q - 1) / Q;
    const int64_t blocks =
        std::min<int64_t>((batches + warps - 1) / warps, (int64_t)device_sm_count() * per_sm);
    kern<<<(unsigned)blocks, warps * 32, smem, st>>>(a);
    IBP_LAUNCHED("pack_rows_kernel");
    return IBP_OK;
}

template <typename U>
static ibp_status launch_pack(PackArgs<U> a, cudaStream_t st) {
    if (a.nrows <= 0) return IBP_OK;
    const int maxs = device_max_smem_optin();
    // the longest rows packed: two raw rows of shared memory (an image can grow past the raw
    // row by its bitmap before it is found incompressible)
    if ((int64_t)(2 * align_up((size_t)a.v + 4, 4) * sizeof(U)) > maxs) {
        set_error("rows of %lld words do not fit the packer's shared-memory staging",
                  (long long)a.v);
        return IBP_ERR_UNSUPPORTED;
    }
    // bitmap and stream, and the units past them that an OR of no bits may touch
    a.buf_words = (int64_t)align_up(
        (size_t)(a.v + meta_bytes(a.v, sizeof(U)) / (int64_t)sizeof(U)) + 16 / sizeof(U),
        16 / sizeof(U));
    const size_t row = (size_t)a.buf_words * sizeof(U);
    constexpr int cols = PackTables<U, 1>::COLS;
    // Host rows of whole 16-byte blocks and at least 512 bytes; and tiny ones packed back to back
    // (500k rows of two 64-bit words 1655 us, here 1242).  Other rows, above all those off 16-byte
    // boundaries, are brought faster four at a time (200k of 99 32-bit words in place 2478 us,
    // here 4567; of 16 words 1192 and 1320; of 64 words 2083 and 2073).
    const int64_t row_bytes = a.v * (int64_t)sizeof(U);
    const bool whole = row_bytes >= 512 && row_bytes % 16 == 0 && (((uintptr_t)a.src) & 15) == 0;
    if ((a.in_place || !a.out) && (whole || (!a.out && row_bytes <= 32))) {
        cudaPointerAttributes pa{};
        if (cudaPointerGetAttributes(&pa, a.src) != cudaSuccess) cudaGetLastError();
        a.stage_words = (int64_t)align_up((size_t)a.v, 16 / sizeof(U));
        const size_t both = row + (size_t)a.stage_words * sizeof(U);
        // (the longest rows' words and image do not both fit)
        if (pa.type == cudaMemoryTypeHost && both <= (size_t)maxs) {
            if (a.v <= cols) return launch_pack_host<U, 1, true>(a, both, st);
            if (a.v <= 2 * cols) return launch_pack_host<U, 2, true>(a, both, st);
            return launch_pack_host<U, 2, false>(a, both, st);
        }
    }
    if (a.v <= cols) return launch_pack_q<U, 1, 4, true>(a, 8, 4 * 8 * row, st);
    if (a.v <= 2 * cols) return launch_pack_q<U, 2, 4, true>(a, 8, 4 * 8 * row, st);
    // longer rows: 4 rows share a load of the tables while two blocks of 8 warps fit an SM,
    // else 1 row and as many warps as fit; and 1 row where every row has a warp of its own
    if (4 * 8 * row <= 100 * 1024 && a.nrows > (int64_t)device_sm_count() * 16)
        return launch_pack_q<U, 2, 4, false>(a, 8, 4 * 8 * row, st);
    const int warps = (int)std::min<size_t>(8, (size_t)maxs / row);
    return launch_pack_q<U, 2, 1, false>(a, warps, (size_t)warps * row, st);
}

template <typename U>
ibp_status compress_rows_impl(const U *src, int64_t n, int64_t v, ColTables<U> t,
                              const int64_t *idx, int64_t nrows, U *out, bool out_is_src,
                              int32_t *bitmask, int32_t *status, cudaStream_t st) {
    if (nrows > 0) IBP_CUDA(cudaMemsetAsync(bitmask, 0, sizeof(int32_t) * ((nrows + 31) / 32), st));
    PackArgs<U> a{};
    a.src = src;
    a.n = n;
    a.v = v;
    a.t = t;
    a.idx = idx;
    a.nrows = nrows;
    a.out = out;
    a.in_place = out_is_src && idx == nullptr;
    a.bitmask = bitmask;
    a.status = status;
    return launch_pack<U>(a, st);
}

template <typename U>
ibp_status compress_condensed_rows(const U *src, int64_t n, int64_t v, ColTables<U> t,
                                   const int64_t *idx, int64_t nrows, const int64_t *offsets,
                                   U *out, int32_t *status, cudaStream_t st) {
    PackArgs<U> a{};
    a.src = src;
    a.n = n;
    a.v = v;
    a.t = t;
    a.idx = idx;
    a.nrows = nrows;
    a.cond = out;
    a.offsets = offsets;
    a.status = status;
    return launch_pack<U>(a, st);
}

// ------------------------------------------------------------------ gather (staging)
template <typename U>
__global__ void gather_rows_kernel(const U *__restrict__ src, int64_t n, int64_t v,
                                   const int64_t *__restrict__ idx, int64_t nrows,
                                   U *__restrict__ out, int32_t *__restrict__ status) {
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = warp; i < nrows; i += nwarps) {
        const int64_t r = idx[i];
        if (r < 0 || r >= n) {
            if ((threadIdx.x & 31) == 0) atomicOr(status, kStatusBadIndex);
            continue;
        }
        warp_copy<U>(out + i * v, src + r * v, v);
    }
}

template <typename U>
ibp_status gather_rows_impl(const U *src, int64_t n, int64_t v, const int64_t *idx,
                            int64_t nrows, U *out, int32_t *status, cudaStream_t st) {
    if (nrows <= 0) return IBP_OK;
    int64_t blocks = (nrows + 7) / 8;
    const int64_t cap = (int64_t)device_sm_count() * 8;
    if (blocks > cap) blocks = cap;
    gather_rows_kernel<U><<<(unsigned)blocks, 256, 0, st>>>(src, n, v, idx, nrows, out, status);
    IBP_LAUNCHED("gather_rows_kernel");
    return IBP_OK;
}

// ------------------------------------------------------------------ offsets
size_t inclusive_offsets_workspace(int64_t nrows) {
    size_t temp = 0;
    cub::DeviceScan::InclusiveSum(nullptr, temp, (int64_t *)nullptr, (int64_t *)nullptr,
                                  (int)(nrows > 0 ? nrows : 1));
    return kStatusBytes + align_up(temp, kAlign);
}

__global__ void copy_last_kernel(const int64_t *offsets, int64_t nrows, int64_t *total) {
    *total = nrows > 0 ? offsets[nrows - 1] : 0;
}

ibp_status inclusive_offsets_impl(int64_t *sizes, int64_t nrows, int64_t *total, void *ws,
                                  size_t ws_bytes, cudaStream_t st) {
    if (nrows > 0x7fffffffLL) {
        set_error("condensed offsets: more than 2^31-1 rows");
        return IBP_ERR_UNSUPPORTED;
    }
    if (nrows > 0) {
        size_t temp = 0;
        IBP_CUDA(cub::DeviceScan::InclusiveSum(nullptr, temp, sizes, sizes, (int)nrows, st));
        if (!ws || ws_bytes < kStatusBytes + temp) {
            set_error("condensed offsets: workspace of %zu bytes is below %zu", ws_bytes,
                      kStatusBytes + temp);
            return IBP_ERR_WORKSPACE;
        }
        IBP_CUDA(cub::DeviceScan::InclusiveSum((char *)ws + kStatusBytes, temp, sizes, sizes,
                                               (int)nrows, st));
    }
    if (total) {
        copy_last_kernel<<<1, 1, 0, st>>>(sizes, nrows, total);
        IBP_LAUNCHED("copy_last_kernel");
    }
    return IBP_OK;
}

#define IBP_INST(U)                                                                          \
    template ibp_status compress_size_impl<U>(const U *, int64_t, int64_t, const U *, const U *, \
                                              const int64_t *, int64_t, int64_t *, int64_t *,  \
                                              int32_t *, cudaStream_t);
IBP_INST(uint8_t)
IBP_INST(uint16_t)
IBP_INST(uint32_t)
IBP_INST(uint64_t)
#undef IBP_INST

#define IBP_INST(U)                                                                            \
    template ibp_status compress_rows_impl<U>(const U *, int64_t, int64_t, ColTables<U>,       \
                                              const int64_t *, int64_t, U *, bool, int32_t *,  \
                                              int32_t *, cudaStream_t);                        \
    template ibp_status compress_condensed_rows<U>(const U *, int64_t, int64_t, ColTables<U>,  \
                                                   const int64_t *, int64_t, const int64_t *,  \
                                                   U *, int32_t *, cudaStream_t);              \
    template ibp_status gather_rows_impl<U>(const U *, int64_t, int64_t, const int64_t *,      \
                                            int64_t, U *, int32_t *, cudaStream_t);
IBP_INST(uint32_t)
IBP_INST(uint64_t)
#undef IBP_INST

}  // namespace ibp200
