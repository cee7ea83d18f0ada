// ibp_preprocess.cu -- invariant-bit census, per-threshold masks, fused saved-bit check and
// on-device threshold selection (replaces include/preproc/ibp_preproc_host.cuh:23-115 and
// include/preproc/ibp_preproc_kernels.cuh:7-77).
//
// B200 design
//  * census: the dataset is taken in 16-byte pieces whatever the word size and wherever it starts
//    (as many bytes as up to 16 rows have are a whole number of pieces, from the first 16-byte
//    boundary on), each thread counting the set bits of one piece's positions in
//    bit planes (ibp_bitcount.cuh), 8 pieces in flight; shared counters per block, one global
//    atomic per (position, block) at the end.  A host-resident dataset is optionally staged
//    into HBM during this pass so the second pass reads HBM instead of PCIe.
//  * all sweep thresholds are checked in ONE pass over the data (the reference makes one
//    PCIe pass and one host round trip per threshold) and the winning mask is selected
//    by a one-block kernel, so preprocess never blocks the host.
#include <algorithm>

#include "ibp_bitcount.cuh"
#include "ibp_common.cuh"
#include "ibp_internal.cuh"
#include "ibp_match.cuh"

namespace ibp200 {

constexpr int kCensusThreads = 256;
constexpr int kCensusCols = 64;   // most 16-byte pieces a block covers side by side

// counts[p] += rows whose bit p (word p / W, bit p % W) is set, over groups of as many bytes as k
// rows have, `pieces` 16-byte pieces each.  `data` is the dataset's first 16-byte boundary, `turn`
// bits from its start: bit p of a group is bit (turn + p) % row_bits of a row.
// Block bx * tiles + tile covers pieces [tile * cpb, tile * cpb + cpb) of every group; the R =
// kCensusThreads / cpb row slots of a tile's blocks take the groups in turn.
// Bound: HBM (600k rows of 512 bytes: 126 -> 54 us, 5.7 TB/s; a thread per word, a
// ripple-carry add into 8 planes and 64 KiB of counters per block before).
__global__ void __launch_bounds__(kCensusThreads, 2)
census_kernel(const uint4 *__restrict__ data, int64_t groups, int64_t pieces, int cpb, int tiles,
              int64_t row_bits, int turn, bool folded, uint32_t *__restrict__ counts,
              uint4 *__restrict__ stage) {
    extern __shared__ uint32_t sc[];  // [128][cpb | 1]
    const int stride = cpb | 1;
    const int R = kCensusThreads / cpb;
    const int c = threadIdx.x % cpb, slot = threadIdx.x / cpb;
    const int64_t col0 = (int64_t)(blockIdx.x % tiles) * cpb, col = col0 + c;
    for (int e = threadIdx.x; e < 128 * stride; e += kCensusThreads) sc[e] = 0;
    __syncthreads();
    BitPlanes<4> bp;
    bp.clear();
    if (slot < R && col < pieces) {
        const int64_t rstride = (int64_t)(gridDim.x / tiles) * R;
        int pending = 0;
        constexpr int N = 8;
        for (int64_t r = (int64_t)(blockIdx.x / tiles) * R + slot; r < groups; r += N * rstride) {
            uint32_t x[N][4];
#pragma unroll
            for (int q = 0; q < N; ++q) {
                const int64_t rr = r + q * rstride;
                uint4 y = make_uint4(0, 0, 0, 0);
                if (rr < groups) y = data[rr * pieces + col];
                x[q][0] = y.x, x[q][1] = y.y, x[q][2] = y.z, x[q][3] = y.w;
            }
            if (stage) {
#pragma unroll
                for (int q = 0; q < N; ++q)
                    if (r + q * rstride < groups)
                        stage[(r + q * rstride) * pieces + col] =
                            make_uint4(x[q][0], x[q][1], x[q][2], x[q][3]);
            }
            bp.add8(x);
            pending += N;
            if (pending > 255 - N || r + N * rstride >= groups) {  // full, or the last rows
#pragma unroll
                for (int w = 0; w < 4; ++w) {
#pragma unroll 1
                    for (int s = 0; s < 8; ++s) {
                        const uint32_t y = bp.bytes(w, s);
#pragma unroll
                        for (int q = 0; q < 4; ++q)
                            atomicAdd(&sc[(w * 32 + s + 8 * q) * stride + c], (y >> (8 * q)) & 0xffu);
                    }
                }
                bp.clear();
                pending = 0;
            }
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < 128 * cpb; e += kCensusThreads) {
        const int cc = e >> 7, b = e & 127;  // consecutive threads: consecutive positions
        const int64_t piece = col0 + cc;
        const uint32_t x = sc[b * stride + cc];
        if (piece < pieces && x) {
            const int64_t p = piece * 128 + b + turn;
            atomicAdd(&counts[folded ? p % row_bits : p], x);
        }
    }
}

// The words the 16-byte pieces leave over, those before `head` and from `tail` to the dataset's
// last: a thread per column, which sees at most 32 of them, an atomic per set bit.
template <typename U>
__global__ void __launch_bounds__(kCensusThreads)
census_rest_kernel(const U *__restrict__ data, int64_t words, int64_t v, int64_t head,
                   int64_t tail, uint32_t *__restrict__ counts, U *__restrict__ stage) {
    constexpr int W = WordBits<U>::value, R = sizeof(U) == 8 ? 2 : 1;
    for (int64_t col = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; col < v;
         col += (int64_t)gridDim.x * blockDim.x) {
        BitPlanes<R> bp;
        bp.clear();
        // words col, col + v, ... of each of the two ranges, eight at a time
        auto count = [&](int64_t from, int64_t to) {
            for (int64_t w = from; w < to; w += 8 * v) {
                uint32_t x[8][R];
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    const bool in = w + q * v < to;
                    const U y = in ? data[w + q * v] : (U)0;
                    if (in && stage) stage[w + q * v] = y;
                    x[q][0] = (uint32_t)y;
                    if constexpr (R == 2) x[q][1] = (uint32_t)((uint64_t)y >> 32);
                }
                bp.add8(x);
            }
        };
        count(col, head);
        count(tail + (col - tail % v + v) % v, words);
#pragma unroll
        for (int b = 0; b < W; ++b) {
            const uint32_t x = (bp.bytes(b / 32, b % 8) >> (8 * (b % 32 / 8))) & 0xffu;
            if (x) atomicAdd(&counts[col * W + b], x);
        }
    }
}

// One mask/bitval pair per threshold: include/preproc/ibp_preproc_kernels.cuh:33-51.
// `count > thr * N` is a float32 product and compare, `count < (1 - thr) * N` float64.
// A lane per bit: 32 consecutive counts make 4 bytes of every mask with two ballots.
template <typename U>
__global__ void __launch_bounds__(256)
masks_from_counts_kernel(const uint32_t *__restrict__ counts, int64_t n, int64_t v, ThrList thr,
                         U *__restrict__ masks, U *__restrict__ bitvals) {
    grid_dep_wait();
    grid_dep_release();
    const int lane = threadIdx.x & 31;
    const int64_t bits = v * WordBits<U>::value, row_bytes = v * (int64_t)sizeof(U);
    const int64_t nwarps = (int64_t)gridDim.x * 8;
    for (int64_t g = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5); g * 32 < bits; g += nwarps) {
        const bool in = g * 32 + lane < bits;
        const int32_t c = in ? (int32_t)counts[g * 32 + lane] : 0;
        for (int t = 0; t < thr.count; ++t) {
            const float lim1 = __fmul_rn(thr.v[t], (float)(unsigned long long)n);
            const double lim0 =
                __dmul_rn(1.0 - (double)thr.v[t], (double)(unsigned long long)n);
            const bool one = (float)c > lim1;
            const unsigned val = __ballot_sync(0xffffffffu, in && one);
            const unsigned m = __ballot_sync(0xffffffffu, in && (one || (double)c < lim0));
            const int64_t at = g * 4 + lane;
            if (lane < 4 && at < row_bytes) {
                reinterpret_cast<uint8_t *>(masks)[t * row_bytes + at] = (uint8_t)(m >> (8 * lane));
                reinterpret_cast<uint8_t *>(bitvals)[t * row_bytes + at] =
                    (uint8_t)(val >> (8 * lane));
            }
        }
    }
}

// saved[t] += sum over rows of max(0, S_t(row) - v), S_t = sum of popc(mask_t[j]) over the
// words with (x & mask_t[j]) == bitval_t[j]: include/preproc/ibp_preproc_kernels.cuh:53-77,
// for every threshold of the sweep in one pass (T == 7), or for one threshold (T == 1).
// In the sweep the masks are nested: thr * N rises and (1 - thr) * N falls with thr, so a bit
// invariant at one threshold is so at every lower one, with the same value (all thresholds are
// above one half); a word matches at threshold t exactly when (x ^ bitval_0) & mask_t is 0.
// Rows as in the size pass (G lanes, pieces of A bytes, Q rows in flight), tables in registers.
// PACK: S_t of a row fits 16 bits, two thresholds to a register in the sums over lanes.
// Bound: the integer pipe, 3 operations per word and threshold there and one on the
// multiply-add pipe (600k rows of 64 64-bit words, 7 thresholds: 550 us with 14 table loads per
// word, 119 with the adds on the integer pipe as well, 100 now; rows of up to 512 bytes take
// check_sweep_kernel).
template <typename U, int A, int G, int T, bool PACK>
__global__ void __launch_bounds__(256, 2)
check_saved_kernel(const U *__restrict__ data, int64_t n, int64_t v, int nthr,
                   const U *__restrict__ masks, const U *__restrict__ bitvals,
                   unsigned long long *__restrict__ saved, uint32_t one) {
    using C = Chunk<U, A, G>;
    constexpr int RPW = 32 / G;
    constexpr int Q = T > 1 ? 4 : 8;
    constexpr int S = T > 1 ? (PACK ? 4 : 8) : 1;  // sums per row
    constexpr int L = Q * S > G ? Q * S / G : 1;   // sums a lane ends with
    __shared__ unsigned long long blk[kMaxThresholds];
    if (threadIdx.x < kMaxThresholds) blk[threadIdx.x] = 0;
    __syncthreads();
    grid_dep_wait();
    grid_dep_release();
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), gin = lane / G;
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t row_bytes = v * (int64_t)sizeof(U);
    const int64_t chunks = row_bytes / A;
    uint32_t b[C::NR], m[T][C::NR], pc[T][C::NW];
    auto tables = [&](int64_t c) {
        C::load_words(bitvals, c, chunks, b);
#pragma unroll
        for (int t = 0; t < T; ++t) {
            if (t < nthr) {
                C::load_words(masks + t * v, c, chunks, m[t]);
            } else {
#pragma unroll
                for (int i = 0; i < C::NR; ++i) m[t][i] = 0;  // saves nothing
            }
            if (PACK && (t & 1))
                C::template set_bits<16>(m[t], pc[t]);
            else
                C::set_bits(m[t], pc[t]);
        }
    };
    constexpr int SP = G * C::NS;  // pieces of a step
    const int64_t steps = (chunks + SP - 1) / SP;  // per row
    if (steps == 1 && sub < chunks) tables(sub);
    unsigned long long acc[L][PACK ? 2 : 1];
#pragma unroll
    for (int l = 0; l < L; ++l) {
        acc[l][0] = 0;
        if (PACK) acc[l][PACK ? 1 : 0] = 0;
    }
    // Batches of RPW * Q rows from the last to the first: the census ended with the last rows,
    // so they are still in L2.  Each step's rows are loaded while the step before is counted.
    const int64_t batches = (n + RPW * Q - 1) / (RPW * Q);
    auto load = [&](int64_t batch, int64_t c, uint32_t (&x)[Q][C::NR]) {
        const int64_t r0 = batch * (RPW * Q) + gin;
        const char *p = reinterpret_cast<const char *>(data) + r0 * row_bytes;
#pragma unroll
        for (int q = 0; q < Q; ++q)
            C::load(p + q * RPW * row_bytes, c, r0 + q * RPW < n ? chunks : 0, x[q]);
    };
    uint32_t x[Q][C::NR];
    int64_t batch = batches - 1 - warp;
    if (batch >= 0) load(batch, sub, x);
    for (; batch >= 0; batch -= nwarps) {
        uint32_t f[Q * S];
#pragma unroll
        for (int i = 0; i < Q * S; ++i) f[i] = 0;
        const int64_t left = n - (batch * (RPW * Q) + gin);  // rows of this group's, every RPW-th
        for (int64_t k = 0; k < steps; ++k) {
            const int64_t c = k * SP + sub;
            uint32_t y[Q][C::NR];
            const bool more = k + 1 < steps;
            if (more || batch >= nwarps) load(more ? batch : batch - nwarps, more ? c + SP : sub, y);
            if (steps > 1 && c < chunks) tables(c);
            if (c < chunks) {
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    if (q * RPW < left) {
                        if constexpr (T > 1) {
#pragma unroll
                            for (int i = 0; i < C::NR; ++i) x[q][i] ^= b[i];
#pragma unroll
                            for (int t = 0; t < T; ++t) {
                                auto e = [&](int i) { return x[q][i] & m[t][i]; };
                                if (PACK && (t & 1))
                                    C::template matched<16>(f[q * S + t / 2], e, pc[t], one);
                                else
                                    C::matched(f[q * S + (PACK ? t / 2 : t)], e, pc[t], one);
                            }
                        } else {
                            C::matched(f[q], [&](int i) { return (x[q][i] & m[0][i]) ^ b[i]; },
                                       pc[0], one);
                        }
                    }
                }
            }
#pragma unroll
            for (int q = 0; q < Q; ++q)
#pragma unroll
                for (int i = 0; i < C::NR; ++i) x[q][i] = y[q][i];
        }
        group_sums<Q * S, G>(f, one);
#pragma unroll
        for (int l = 0; l < L; ++l) {
            if constexpr (PACK) {
                const uint32_t lo = f[l] & 0xffffu, hi = f[l] >> 16;
                if (lo > (uint64_t)v) acc[l][0] += lo - (uint32_t)v;
                if (hi > (uint64_t)v) acc[l][1] += hi - (uint32_t)v;
            } else {
                if (f[l] > (uint64_t)v) acc[l][0] += f[l] - (uint64_t)v;
            }
        }
    }
    if ((sub & (group_sums_copies<Q * S, G>() - 1)) == 0) {
        const int first = group_sums_value<Q * S, G>(sub);
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const int t = (first + l) % S;
            if constexpr (PACK) {
                if (acc[l][0]) atomicAdd(&blk[2 * t], acc[l][0]);
                if (acc[l][1]) atomicAdd(&blk[2 * t + 1], acc[l][1]);
            } else {
                if (acc[l][0]) atomicAdd(&blk[t], acc[l][0]);
            }
        }
    }
    __syncthreads();
    if (threadIdx.x < nthr && blk[threadIdx.x]) atomicAdd(&saved[threadIdx.x], blk[threadIdx.x]);
}

// The sweep over rows of at most 512 bytes in whole 16-byte pieces (32- and 64-bit words): the
// masks being nested, a bit has a level, the number of masks it is in, and a word matches the
// thresholds from the highest level among its mismatching bits on.  Levels are three bit planes,
// so that highest level is found by three tests from the top (the mismatches with the plane's
// bit, if there are any, are the ones that go on), and the word's set bits for each threshold
// from there on, packed into 16 bytes, come out of a shared table: about 18 integer operations
// a 64-bit word where seven compares take 31, and a third of the table registers.
// 600k rows of 64 64-bit words: check_saved_kernel 100 us, this 82 (88 with generic addresses
// for the table).
template <typename U, int G>
__global__ void __launch_bounds__(256, 2)
check_sweep_kernel(const U *__restrict__ data, int64_t n, int v, int nthr,
                   const U *__restrict__ masks, const U *__restrict__ bitvals,
                   unsigned long long *__restrict__ saved, uint32_t one) {
    using C = Chunk<U, 16, G>;
    constexpr int WPP = 16 / sizeof(U), H = sizeof(U) / 4;  // words of a piece, registers of a word
    constexpr int RPW = 32 / G, Q = 4, S = 4, L = Q * S > G ? Q * S / G : 1;
    extern __shared__ __align__(16) uint4 bits_from[];  // [level][word of piece][piece]
    __shared__ unsigned long long blk[kMaxThresholds];
    if (threadIdx.x < kMaxThresholds) blk[threadIdx.x] = 0;
    grid_dep_wait();
    grid_dep_release();
    const int lane = threadIdx.x & 31, sub = lane & (G - 1), gin = lane / G;
    const int pieces = v / WPP;
    const int stride = (v + 7) & ~7;  // whole rows of banks, so that levels do not meet
    for (int e = threadIdx.x; e < 8 * v; e += blockDim.x) {
        const int from = e / v, w = e % v;
        uint32_t pc[8] = {};
        for (int t = from; t < nthr; ++t) pc[t] = popc_w(masks[(int64_t)t * v + w]);
        bits_from[from * stride + (w % WPP) * pieces + w / WPP] =
            make_uint4(pc[0] | pc[1] << 16, pc[2] | pc[3] << 16, pc[4] | pc[5] << 16, pc[6]);
    }
    uint32_t b[4] = {}, p0[4] = {}, p1[4] = {}, p2[4] = {};
    if (sub < pieces) {
        C::load_words(bitvals, sub, pieces, b);
        uint32_t m[7][4];
#pragma unroll
        for (int t = 0; t < 7; ++t) {
            if (t < nthr) {
                C::load_words(masks + (int64_t)t * v, sub, pieces, m[t]);
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) m[t][i] = 0;
            }
        }
#pragma unroll
        for (int i = 0; i < 4; ++i) {  // masks a bit is in, as a three-bit number
            uint32_t s0, s1, c0, c1, c2;
            carry_save(c0, s0, m[0][i], m[1][i], m[2][i]);
            carry_save(c1, s1, m[3][i], m[4][i], m[5][i]);
            carry_save(c2, p0[i], s0, s1, m[6][i]);
            carry_save(p2[i], p1[i], c0, c1, c2);
        }
    }
    __syncthreads();
    const int64_t row_bytes = (int64_t)v * (int)sizeof(U);
    const int64_t warp = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    const int64_t batches = (n + RPW * Q - 1) / (RPW * Q);
    auto load = [&](int64_t batch, uint32_t (&x)[Q][4]) {
        const int64_t r0 = batch * (RPW * Q) + gin;
        const char *p = reinterpret_cast<const char *>(data) + r0 * row_bytes;
#pragma unroll
        for (int q = 0; q < Q; ++q)
            C::load(p + q * RPW * row_bytes, sub, r0 + q * RPW < n ? pieces : 0, x[q]);
    };
    const uint32_t at = (uint32_t)__cvta_generic_to_shared(bits_from) + sub * 16, step = stride * 16;
    unsigned long long acc[L][2] = {};
    uint32_t x[Q][4];
    // from the last rows to the first, as in check_saved_kernel
    int64_t batch = batches - 1 - warp;
    if (batch >= 0) load(batch, x);
    for (; batch >= 0; batch -= nwarps) {
        uint32_t y[Q][4], f[Q * S] = {};
        if (batch >= nwarps) load(batch - nwarps, y);
        const int64_t left = n - (batch * (RPW * Q) + gin);
        if (sub < pieces) {
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                if (q * RPW >= left) continue;
#pragma unroll
                for (int w = 0; w < WPP; ++w) {
                    uint32_t e[H];
                    uint32_t top = 0, mid = 0, low = 0;
#pragma unroll
                    for (int h = 0; h < H; ++h) {
                        e[h] = x[q][w * H + h] ^ b[w * H + h];
                        top |= e[h] & p2[w * H + h];
                    }
                    if (top) {
#pragma unroll
                        for (int h = 0; h < H; ++h) e[h] &= p2[w * H + h];
                    }
#pragma unroll
                    for (int h = 0; h < H; ++h) mid |= e[h] & p1[w * H + h];
                    if (mid) {
#pragma unroll
                        for (int h = 0; h < H; ++h) e[h] &= p1[w * H + h];
                    }
#pragma unroll
                    for (int h = 0; h < H; ++h) low |= e[h] & p0[w * H + h];
                    uint32_t from = at + w * pieces * 16, z[4];
                    if (top) from += 4 * step;
                    if (mid) from += 2 * step;
                    if (low) from += step;
                    // volatile, and a memory clobber: the barrier after the table's stores is
                    // all that orders them before this read
                    asm volatile("ld.shared.v4.u32 {%0,%1,%2,%3}, [%4];"
                                 : "=r"(z[0]), "=r"(z[1]), "=r"(z[2]), "=r"(z[3])
                                 : "r"(from)
                                 : "memory");
#pragma unroll
                    for (int i = 0; i < 4; ++i) f[q * S + i] = z[i] * one + f[q * S + i];
                }
            }
        }
#pragma unroll
        for (int q = 0; q < Q; ++q)
#pragma unroll
            for (int i = 0; i < 4; ++i) x[q][i] = y[q][i];
        group_sums<Q * S, G>(f, one);
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const uint32_t lo = f[l] & 0xffffu, hi = f[l] >> 16;
            if (lo > (uint32_t)v) acc[l][0] += lo - (uint32_t)v;
            if (hi > (uint32_t)v) acc[l][1] += hi - (uint32_t)v;
        }
    }
    if ((sub & (group_sums_copies<Q * S, G>() - 1)) == 0) {
        const int first = group_sums_value<Q * S, G>(sub);
#pragma unroll
        for (int l = 0; l < L; ++l) {
            const int t = 2 * ((first + l) % S);
            if (acc[l][0]) atomicAdd(&blk[t], acc[l][0]);
            if (acc[l][1]) atomicAdd(&blk[t + 1], acc[l][1]);
        }
    }
    __syncthreads();
    if (threadIdx.x < nthr && blk[threadIdx.x]) atomicAdd(&saved[threadIdx.x], blk[threadIdx.x]);
}

template <typename U>
static ibp_status launch_check_sweep(const U *data, int64_t n, int64_t v, int nthr, const U *masks,
                                     const U *bitvals, unsigned long long *saved,
                                     cudaStream_t st) {
    const bool narrow = v * (int64_t)sizeof(U) <= 128;
    auto kern = narrow ? check_sweep_kernel<U, 8> : check_sweep_kernel<U, 32>;
    const size_t smem = sizeof(uint4) * 8 * (size_t)((v + 7) & ~(int64_t)7);
    const int64_t per_block = 8 * 4 * (narrow ? 4 : 1);
    int per_sm = 0;
    IBP_RET(kernel_blocks_per_sm((const void *)kern, 256, smem, &per_sm));
    const int64_t blocks =
        std::min<int64_t>((n + per_block - 1) / per_block, (int64_t)device_sm_count() * per_sm);
    IBP_CUDA(launch_dependent(kern, (unsigned)blocks, 256, smem, st, data, n, (int)v, nthr, masks,
                              bitvals, saved, 1u));
    IBP_LAUNCHED("check_sweep_kernel");
    return IBP_OK;
}

template <typename U, int A>
static ibp_status launch_check(const U *data, int64_t n, int64_t v, int nthr, const U *masks,
                               const U *bitvals, unsigned long long *saved, cudaStream_t st) {
    // a sweep over rows that one warp covers with a 16-byte piece a lane: 100 us there, 82 here
    constexpr bool has_sweep = A == 16 && sizeof(U) >= 4;
    static_assert(!has_sweep || 8 * A * Chunk<U, A, 8>::NS <= 512);
    if constexpr (has_sweep)
        if (nthr > 1 && v * (int64_t)sizeof(U) <= 512)
            return launch_check_sweep<U>(data, n, v, nthr, masks, bitvals, saved, st);
    const bool narrow = v * (int64_t)sizeof(U) <= 8 * A * Chunk<U, A, 8>::NS;
    const bool pack = v * 8 * (int64_t)sizeof(U) < 65536;
    auto kern = nthr == 1 ? (narrow ? check_saved_kernel<U, A, 8, 1, false>
                                    : check_saved_kernel<U, A, 32, 1, false>)
                          : (narrow ? check_saved_kernel<U, A, has_sweep ? 32 : 8, 7, true>
                                    : (pack ? check_saved_kernel<U, A, 32, 7, true>
                                            : check_saved_kernel<U, A, 32, 7, false>));
    const int64_t per_block = 8 * (nthr == 1 ? 8 : 4) * (narrow ? 4 : 1);
    int per_sm = 0;
    IBP_RET(kernel_blocks_per_sm((const void *)kern, 256, 0, &per_sm));
    const int64_t blocks =
        std::min<int64_t>((n + per_block - 1) / per_block, (int64_t)device_sm_count() * per_sm);
    IBP_CUDA(launch_dependent(kern, (unsigned)blocks, 256, 0, st, data, n, v, nthr, masks, bitvals,
                              saved, 1u));
    IBP_LAUNCHED("check_saved_kernel");
    return IBP_OK;
}

// First threshold with strictly more saved bits than every earlier one (and > 0) wins;
// its mask/bitval go to the outputs, which are zero when none saves anything
// (include/preproc/ibp_preproc_host.cuh:91-99, src/preprocess.cu:46-47).
template <typename U>
__global__ void select_mask_kernel(const unsigned long long *__restrict__ saved, int nthr,
                                   int64_t v, const U *__restrict__ masks,
                                   const U *__restrict__ bitvals, U *__restrict__ mask_out,
                                   U *__restrict__ bitval_out, int32_t *__restrict__ selected) {
    grid_dep_wait();
    int sel = -1;
    double best = 0.0;
    for (int t = 0; t < nthr; ++t) {
        if ((double)saved[t] > best) {
            best = (double)saved[t];
            sel = t;
        }
    }
    if (threadIdx.x == 0 && blockIdx.x == 0 && selected) *selected = sel;
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < v;
         j += (int64_t)gridDim.x * blockDim.x) {
        mask_out[j] = sel >= 0 ? masks[sel * v + j] : (U)0;
        bitval_out[j] = sel >= 0 ? bitvals[sel * v + j] : (U)0;
    }
}

ThrList sweep_thresholds(float threshold) {
    // include/preproc/ibp_preproc_host.cuh:61-67: float loop variable, `+= 0.05` in double
    ThrList l{};
    l.count = 0;
    const float lo = threshold < 0 ? (float)0.7 : threshold;
    const float hi = threshold < 0 ? (float)1.0 : threshold;
    for (float t = lo; t <= hi && l.count < kMaxThresholds; t = (float)((double)t + 0.05))
        l.v[l.count++] = t;
    return l;
}

// Counts of the whole dataset: 16-byte pieces in groups of k rows' bytes, then the words left over
// at its ends.  `stage` (or null) starts on a 16-byte boundary, and with it `data`.
template <typename U>
static ibp_status launch_census(const U *data, int64_t n, int64_t v, uint32_t *counts, U *stage,
                                cudaStream_t st) {
    const int64_t row_bytes = v * (int64_t)sizeof(U);
    int64_t k = 1;
    while (k * row_bytes % 16) k *= 2;
    // Pieces from the first 16-byte boundary on, wherever the dataset starts: the bits of a group
    // are then those of k rows turned by the words before it.  192 MiB of 64-bit words 8 bytes off
    // a boundary take as long as on one (rows of 64 words 35 us, of one word 61); a thread per
    // word and 32 rows with an atomic per set bit, for such data before, took 1098 and 30561 us.
    const int64_t head = (int64_t)(-(uintptr_t)data & 15) / (int64_t)sizeof(U);
    const int64_t groups = std::max<int64_t>(0, (n * v - head) / (k * v));
    const int64_t tail = groups > 0 ? head + groups * k * v : 0;
    const int sms = device_sm_count();
    if (groups > 0) {
        const int64_t pieces = k * row_bytes / 16;
        const int cpb = (int)std::min<int64_t>(pieces, kCensusCols);
        const int R = kCensusThreads / cpb;
        const size_t smem = sizeof(uint32_t) * 128 * (size_t)(cpb | 1);
        int per_sm = 0;
        IBP_RET(kernel_blocks_per_sm((const void *)census_kernel, kCensusThreads, smem, &per_sm));
        const int64_t tiles = (pieces + cpb - 1) / cpb;
        // at least 32 groups per row slot (a block's counters cost 128 x cpb global atomics)
        const int64_t gx = std::max<int64_t>(
            1, std::min<int64_t>((groups + R * 32 - 1) / (R * 32), (int64_t)sms * per_sm / tiles));
        census_kernel<<<(unsigned)(gx * tiles), kCensusThreads, smem, st>>>(
            reinterpret_cast<const uint4 *>(data + head), groups, pieces, cpb, (int)tiles,
            row_bytes * 8, (int)(head * 8 * (int64_t)sizeof(U)), k > 1 || head > 0, counts,
            reinterpret_cast<uint4 *>(stage));
        IBP_LAUNCHED("census_kernel");
    }
    const int64_t first = groups > 0 ? head : 0;
    if (first > 0 || tail < n * v) {
        const int64_t blocks =
            std::min<int64_t>((v + kCensusThreads - 1) / kCensusThreads, (int64_t)sms * 8);
        census_rest_kernel<U><<<(unsigned)blocks, kCensusThreads, 0, st>>>(data, n * v, v, first,
                                                                           tail, counts, stage);
        IBP_LAUNCHED("census_rest_kernel");
    }
    return IBP_OK;
}

size_t preprocess_workspace(int64_t n, int64_t v, int wb, float threshold, bool staged) {
    Sizer s;
    s.take<char>(kStatusBytes);
    const ThrList l = sweep_thresholds(threshold);
    s.take<unsigned long long>(kMaxThresholds);          // saved bits
    s.take<uint32_t>((size_t)(v * 8 * wb));              // counts
    s.take<char>((size_t)(l.count > 0 ? l.count : 1) * v * wb);  // masks
    s.take<char>((size_t)(l.count > 0 ? l.count : 1) * v * wb);  // bitvals
    s.take<int32_t>(4);                                  // selected step
    if (staged) s.take<char>((size_t)(n * v * wb));
    return s.total();
}

template <typename U>
ibp_status preprocess_impl(const U *data, int64_t n, int64_t v, float threshold, U *mask,
                           U *bitval, void *ws, size_t ws_bytes, bool data_on_host,
                           cudaStream_t st) {
    constexpr int wb = sizeof(U);
    const ThrList thr = sweep_thresholds(threshold);
    Carver c{(char *)ws, 0, ws_bytes};
    c.take<char>(kStatusBytes);
    unsigned long long *saved = c.take<unsigned long long>(kMaxThresholds);
    uint32_t *counts = c.take<uint32_t>((size_t)(v * 8 * wb));
    U *masks = c.take<U>((size_t)(thr.count > 0 ? thr.count : 1) * v);
    U *bitvals = c.take<U>((size_t)(thr.count > 0 ? thr.count : 1) * v);
    int32_t *selected = c.take<int32_t>(4);
    if (!selected) {
        set_error("preprocess: workspace of %zu bytes is below the required %zu", ws_bytes,
                  preprocess_workspace(n, v, wb, threshold, false));
        return IBP_ERR_WORKSPACE;
    }
    U *stage = nullptr;
    if (data_on_host && thr.count > 0) stage = c.take<U>((size_t)(n * v));  // null if it does not fit
    if (stage && (((uintptr_t)data | (uintptr_t)stage) & 15) && n > 0 && v > 0) {
        // host rows off a 16-byte boundary: the copy engine stages them, the census reads the copy
        IBP_CUDA(cudaMemcpyAsync(stage, data, (size_t)(n * v) * wb, cudaMemcpyDefault, st));
        data = stage;
        stage = nullptr;
    }
    // the saved bits and the counts follow one another
    IBP_CUDA(cudaMemsetAsync(saved, 0, (size_t)((char *)(counts + v * 8 * wb) - (char *)saved), st));
    if (n > 0 && v > 0) IBP_RET(launch_census<U>(data, n, v, counts, stage, st));
    if (thr.count > 0 && v > 0) {
        const int64_t warps = (v * 8 * wb + 31) / 32;
        const unsigned blocks = (unsigned)std::min<int64_t>((warps + 7) / 8, 4096);
        IBP_CUDA(launch_dependent(masks_from_counts_kernel<U>, blocks, 256, 0, st, counts, n, v,
                                  thr, masks, bitvals));
        IBP_LAUNCHED("masks_from_counts_kernel");
        if (n > 0) {
            const U *rows = stage ? stage : data;
            const int a = row_piece_bytes(rows, v, wb);
            if (a == 16)
                IBP_RET((launch_check<U, 16>(rows, n, v, thr.count, masks, bitvals, saved, st)));
            else if (a == 4 && wb < 4)
                IBP_RET((launch_check<U, wb < 4 ? 4 : 16>(rows, n, v, thr.count, masks, bitvals,
                                                          saved, st)));
            else
                IBP_RET((launch_check<U, wb>(rows, n, v, thr.count, masks, bitvals, saved, st)));
        }
    }
    if (v > 0) {
        const int blocks = (int)((v + 255) / 256 < 1024 ? (v + 255) / 256 : 1024);
        IBP_CUDA(launch_dependent(select_mask_kernel<U>, (unsigned)blocks, 256, 0, st, saved,
                                  thr.count, v, masks, bitvals, mask, bitval, selected));
        IBP_LAUNCHED("select_mask_kernel");
    }
    return IBP_OK;
}

template ibp_status preprocess_impl<uint8_t>(const uint8_t *, int64_t, int64_t, float, uint8_t *,
                                             uint8_t *, void *, size_t, bool, cudaStream_t);
template ibp_status preprocess_impl<uint16_t>(const uint16_t *, int64_t, int64_t, float,
                                              uint16_t *, uint16_t *, void *, size_t, bool,
                                              cudaStream_t);
template ibp_status preprocess_impl<uint32_t>(const uint32_t *, int64_t, int64_t, float,
                                              uint32_t *, uint32_t *, void *, size_t, bool,
                                              cudaStream_t);
template ibp_status preprocess_impl<uint64_t>(const uint64_t *, int64_t, int64_t, float,
                                              uint64_t *, uint64_t *, void *, size_t, bool,
                                              cudaStream_t);

}  // namespace ibp200
