// ibp_bitcount.cuh -- set-bit counts per bit position over many words, in bit planes: plane d
// of a word holds bit d of the 32 positions' counts.  Eight words go in at a time through a
// tree of carry-save adders (7 of them, two logic operations each; the tree of W. Mula, N. Kurz and
// D. Lemire, "Faster population counts using AVX2 instructions", The Computer Journal 61(1),
// 2018, kept per bit position), so a 32-bit word costs ~3 logic operations where a ripple-carry
// add into eight planes costs 16.
#pragma once

#include "ibp_common.cuh"

namespace ibp200 {

// (h, l) = a + b + c in every bit position
__device__ __forceinline__ void carry_save(uint32_t &h, uint32_t &l, uint32_t a, uint32_t b,
                                           uint32_t c) {
    const uint32_t hh = (a & b) | (a & c) | (b & c);
    l = a ^ b ^ c;
    h = hh;
}

// Counts of up to 255 words of VEC 32-bit units.
template <int VEC>
struct BitPlanes {
    uint32_t p[8][VEC];

    __device__ __forceinline__ void clear() {
#pragma unroll
        for (int d = 0; d < 8; ++d)
#pragma unroll
            for (int w = 0; w < VEC; ++w) p[d][w] = 0;
    }

    __device__ __forceinline__ void add8(const uint32_t (&x)[8][VEC]) {
#pragma unroll
        for (int w = 0; w < VEC; ++w) {
            uint32_t t0, t1, f0, f1, e;
            carry_save(t0, p[0][w], p[0][w], x[0][w], x[1][w]);
            carry_save(t1, p[0][w], p[0][w], x[2][w], x[3][w]);
            carry_save(f0, p[1][w], p[1][w], t0, t1);
            carry_save(t0, p[0][w], p[0][w], x[4][w], x[5][w]);
            carry_save(t1, p[0][w], p[0][w], x[6][w], x[7][w]);
            carry_save(f1, p[1][w], p[1][w], t0, t1);
            carry_save(e, p[2][w], p[2][w], f0, f1);
#pragma unroll
            for (int d = 3; d < 8; ++d) {
                const uint32_t c = p[d][w] & e;
                p[d][w] ^= e;
                e = c;
            }
        }
    }

    // counts of bits s, s + 8, s + 16, s + 24 of unit w, in bytes 0..3
    __device__ __forceinline__ uint32_t bytes(int w, int s) const {
        uint32_t r = 0;
#pragma unroll
        for (int d = 0; d < 8; ++d) r += ((p[d][w] >> s) & 0x01010101u) << d;
        return r;
    }
};

}  // namespace ibp200
