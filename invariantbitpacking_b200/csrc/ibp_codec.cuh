// ibp_codec.cuh -- device building blocks of the compressed row format.
//
// Row format (include/compress/ibp_compress_dev.cuh:7-97, restated):
//   words [0, Mw): bitmap, bit j (LSB-first in 32-bit units) = word j is compressible,
//                  Mw = ceil(ceil(v/8) / wb) words;
//   from word Mw : an MSB-first bit stream; word j contributes its non-invariant bits
//                  (the bits where mask_j is 0, highest first) when compressible, else
//                  all W bits;
//   then zeros up to v words.
//
// Bit gather/scatter (x -> bits of x under `sel`, packed; and the inverse) uses the
// parallel-suffix method of H. S. Warren, "Hacker's Delight", 2nd ed., sections 7-4
// (compress) and 7-5 (expand): five steps per 32-bit half, each moving bits by 2^i under a
// per-column "move" mask.  The move masks depend only on the column's mask, so they are
// built once per call (build_tables_kernel) and every word then costs a few branch-free
// steps instead of a data-dependent loop over mask runs.  64-bit words are moved as two
// 32-bit halves: five steps of one shift each (which can run as a multiplication on the other
// pipe) in place of six of two.
#pragma once

#include <type_traits>

#include "ibp_common.cuh"

namespace ibp200 {

template <typename U>
struct LogW { static constexpr int value = sizeof(U) == 8 ? 6 : 5; };

constexpr int kMoves = 5;  // move masks per 32-bit half

// Kept bits of a column: of the word (low byte) and, for 64-bit words, of its low half (high
// byte).
template <typename U>
using KeptBits = typename std::conditional<sizeof(U) == 8, uint16_t, uint8_t>::type;

template <typename U>
__device__ __forceinline__ KeptBits<U> kept_bits(U mask) {
    const int nb = 8 * (int)sizeof(U) - popc_w(mask);
    if constexpr (sizeof(U) == 8)
        return (KeptBits<U>)(nb | (32 - __popc((uint32_t)mask)) << 8);
    else
        return (KeptBits<U>)nb;
}

// Per-column decode/encode tables, structure-of-arrays in a workspace buffer.
template <typename U>
struct ColTables {
    U *mask;          // [v]
    U *bitval;        // [v]
    U *mv;            // [kMoves][v] move masks of sel = ~mask, each half's in its own half
    KeptBits<U> *nb;  // [v] bits a compressible word keeps
};

template <typename U>
size_t tables_bytes(int64_t v) {
    return align_up((size_t)v * sizeof(U), kAlign) * (2 + kMoves) +
           align_up((size_t)v * sizeof(KeptBits<U>), kAlign);
}

template <typename U>
ColTables<U> carve_tables(Carver &c, int64_t v) {
    ColTables<U> t;
    t.mask = c.take<U>(v);
    t.bitval = c.take<U>(v);
    t.mv = c.take<U>((size_t)v * kMoves);
    t.nb = c.take<KeptBits<U>>(v);
    return t;
}

// A shift that is well defined for every amount in [0, W].
template <typename U>
__device__ __forceinline__ U shr_w(U x, int s) {
    return s >= (int)(8 * sizeof(U)) ? (U)0 : (U)(x >> s);
}

// Move masks for scattering to (RIGHT: gathering from, packed right) the bits of `sel`
// (Hacker's Delight 7-4 / 7-5), or, mirrored, for gathering them packed left.
template <bool RIGHT>
__device__ __forceinline__ void move_masks(uint32_t sel, uint32_t (&mv)[kMoves]) {
    uint32_t m = sel;
    uint32_t mk = RIGHT ? ~m << 1 : ~m >> 1;
#pragma unroll
    for (int i = 0; i < kMoves; ++i) {
        uint32_t mp = mk;
#pragma unroll
        for (int k = 0; k < kMoves; ++k) mp ^= RIGHT ? mp << (1 << k) : mp >> (1 << k);
        const uint32_t v = mp & m;
        mv[i] = v;
        m = (m ^ v) | (RIGHT ? v >> (1 << i) : v << (1 << i));
        mk &= ~mp;
    }
}

// Bits of x at the set positions of ~mask, packed to the left (pext, left-aligned), with the
// first LEVELS moves: the later masks are all zero where no kept bit has 2^LEVELS or more
// dropped bits above it.
template <int LEVELS>
__device__ __forceinline__ uint32_t gather_left(uint32_t x, uint32_t mask,
                                                const uint32_t (&mv)[kMoves]) {
    x &= ~mask;
#pragma unroll
    for (int i = 0; i < LEVELS; ++i) {
        const uint32_t t = x & mv[i];
        x = (x ^ t) | (t << (1 << i));
    }
    return x;
}

// The low bits of y placed at the set positions of sel (pdep), for move masks of
// move_masks<true>; `keep` is the value outside sel.
__device__ __forceinline__ uint32_t scatter_half(uint32_t y, uint32_t sel, uint32_t keep,
                                                 const uint32_t (&mv)[kMoves]) {
#pragma unroll
    for (int i = kMoves - 1; i >= 0; --i) y = (y & ~mv[i]) | ((y << (1 << i)) & mv[i]);
    return (y & sel) | keep;
}

// The word whose kept bits are the low bits of y: scattered per half (the low half takes the
// last nbl of them), with the invariant bits bv.
template <typename U>
__device__ __forceinline__ U scatter_word(U y, U mask, U bv, int nbl, const U (&mv)[kMoves]) {
    uint32_t lo[kMoves];
#pragma unroll
    for (int i = 0; i < kMoves; ++i) lo[i] = (uint32_t)mv[i];
    const uint32_t l = scatter_half((uint32_t)y, ~(uint32_t)mask, (uint32_t)bv, lo);
    if constexpr (sizeof(U) == 8) {
        uint32_t hi[kMoves];
#pragma unroll
        for (int i = 0; i < kMoves; ++i) hi[i] = (uint32_t)(mv[i] >> 32);
        const uint32_t yh = __funnelshift_rc((uint32_t)y, (uint32_t)(y >> 32), nbl);
        const uint32_t h = scatter_half(yh, ~(uint32_t)(mask >> 32), (uint32_t)(bv >> 32), hi);
        return (uint64_t)h << 32 | l;
    } else {
        return l;
    }
}

// The top bits of y placed at the set positions of sel, for the first LEVELS masks of
// move_masks<false> (all of them, or the only ones that are not zero: see moves_left).
template <int LEVELS>
__device__ __forceinline__ uint32_t scatter_top(uint32_t y, uint32_t sel, uint32_t keep,
                                                const uint32_t *mv) {
#pragma unroll
    for (int i = LEVELS - 1; i >= 0; --i) y = (y & ~mv[i]) | ((y >> (1 << i)) & mv[i]);
    return (y & sel) | keep;
}

// Dropped bits above the lowest kept bit of sel: how far the farthest kept bit is from its place
// when they are packed left, so that moves of 1, 2, ... up to this many places suffice.
__device__ __forceinline__ int moves_left(uint32_t sel) {
    return sel ? 33 - __ffs((int)sel) - __popc(sel) : 0;
}

// Column j of the tables (RIGHT: for decoding; else for packing).
template <typename U, bool RIGHT = true>
__device__ __forceinline__ void build_table_column(const U *__restrict__ mask,
                                                   const U *__restrict__ bitval, int64_t v,
                                                   const ColTables<U> &t, int64_t j) {
    const U m = mask[j];
    t.mask[j] = m;
    t.bitval[j] = bitval[j];
    t.nb[j] = kept_bits<U>(m);
    uint32_t mv[kMoves];
    move_masks<RIGHT>(~(uint32_t)m, mv);
    if constexpr (sizeof(U) == 8) {
        uint32_t hv[kMoves];
        move_masks<RIGHT>(~(uint32_t)(m >> 32), hv);
#pragma unroll
        for (int i = 0; i < kMoves; ++i) t.mv[i * v + j] = (uint64_t)hv[i] << 32 | mv[i];
    } else {
#pragma unroll
        for (int i = 0; i < kMoves; ++i) t.mv[i * v + j] = mv[i];
    }
}

template <typename U, bool RIGHT>
__global__ void build_tables_kernel(const U *__restrict__ mask, const U *__restrict__ bitval,
                                    int64_t v, ColTables<U> t) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < v;
         j += (int64_t)gridDim.x * blockDim.x)
        build_table_column<U, RIGHT>(mask, bitval, v, t, j);
}

template <typename U, bool RIGHT = true>
inline ibp_status build_tables(const U *mask, const U *bitval, int64_t v, ColTables<U> t,
                               cudaStream_t st) {
    if (v <= 0) return IBP_OK;
    int blocks = (int)((v + 255) / 256);
    if (blocks > 1024) blocks = 1024;
    build_tables_kernel<U, RIGHT><<<blocks, 256, 0, st>>>(mask, bitval, v, t);
    IBP_LAUNCHED("build_tables_kernel");
    return IBP_OK;
}

// ---- MSB-first stream access on 32-bit units.  Stream bit s of a W-bit word stream
// lives in 32-bit unit s/32 of the stream when W == 32, and in unit (s/32) ^ 1 when
// W == 64 (the high half of a little-endian 64-bit word comes second in memory).

// OR up to 64 bits (left-aligned in hi:lo, the rest zero) into a shared-memory image at bit s.
// The image's units are in stream order; units of no bits are ORed too (a test costs more).
__device__ __forceinline__ void or_shared(uint32_t addr, uint32_t x) {
    asm volatile("red.shared.or.b32 [%0], %1;" ::"r"(addr), "r"(x) : "memory");
}
__device__ __forceinline__ void put_bits(uint32_t image, uint32_t s, uint32_t hi, uint32_t lo) {
    const uint32_t at = image + ((s >> 3) & ~3u), off = s & 31;
    or_shared(at, hi >> off);
    or_shared(at + 4, __funnelshift_r(lo, hi, off));
    or_shared(at + 8, __funnelshift_r(0, lo, off));
}

// Read L (0..W) bits at stream offset s from W-bit words (MSB-first); needs word s/W + 1.
template <typename U>
__device__ __forceinline__ U get_bits(const U *words, int64_t s, int L) {
    constexpr int W = 8 * sizeof(U);
    const int64_t q = s / W;
    const int r = (int)(s % W);
    const U hi = words[q], lo = words[q + 1];
    const U win = r == 0 ? hi : (U)((hi << r) | (lo >> (W - r)));
    return shr_w<U>(win, W - L);
}

// The W stream bits that end at stream bit e (e >= 1) of `words`, right-aligned: the word
// whose bits end there, with whatever precedes them above.  Read from 32-bit units with two
// funnel shifts (stream unit t is memory unit t ^ 1 for 64-bit words, whose high half comes
// second in memory, and unit t for 32-bit words).  A compressible word's L kept bits come out
// in the low bits; its scatter never moves the bits above them to a kept position (each kept
// position takes exactly one of the low L bits), so they need no masking, and neither the
// kept-bit count nor a variable shift enters the read.  For e < W the window starts before
// `words`, in the W bits before it, which the caller's buffer holds (a row's bitmap, or the
// stream's earlier words).
template <typename U>
__device__ __forceinline__ U stream_bits_ending(const U *words, int32_t e) {
    const uint32_t *u = reinterpret_cast<const uint32_t *>(words);
    const int32_t s = e - 8 * (int32_t)sizeof(U);
    const int32_t t = s >> 5;  // may be -2 or -1
    const uint32_t r = (uint32_t)s & 31u;
    if constexpr (sizeof(U) == 8) {
        const uint32_t a = u[t ^ 1], b = u[(t + 1) ^ 1], c = u[(t + 2) ^ 1];
        return ((uint64_t)__funnelshift_l(b, a, r) << 32) | __funnelshift_l(c, b, r);
    } else {
        return __funnelshift_l(u[t + 1], u[t], r);
    }
}

// Copy `words` W-bit words between global buffers with a warp; 16-byte accesses when both
// sides are 16-byte aligned.
template <typename U>
__device__ __forceinline__ void warp_copy(U *__restrict__ dst, const U *__restrict__ src,
                                          int64_t words) {
    const int lane = threadIdx.x & 31;
    const int64_t bytes = words * (int64_t)sizeof(U);
    if ((((uintptr_t)dst | (uintptr_t)src) & 15) == 0) {
        const int64_t n16 = bytes >> 4;
        const uint4 *s4 = reinterpret_cast<const uint4 *>(src);
        uint4 *d4 = reinterpret_cast<uint4 *>(dst);
        for (int64_t k = lane; k < n16; k += 32) d4[k] = s4[k];
        for (int64_t k = (n16 << 4) / (int64_t)sizeof(U) + lane; k < words; k += 32) dst[k] = src[k];
    } else {
        for (int64_t k = lane; k < words; k += 32) dst[k] = src[k];
    }
}

}  // namespace ibp200
