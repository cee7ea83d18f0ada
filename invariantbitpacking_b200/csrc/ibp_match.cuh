// ibp_match.cuh -- which words of a row match the invariant bits, and how many bits that
// saves: the inner loop of the size pass and of the threshold check.
//
// A lane takes pieces of A bytes of a row (16 where rows allow it, else several smaller ones,
// each G pieces after the last) and keeps the mask, the values and the masks' set bits of those
// columns in registers while several rows pass by.
// Words of 1 and 2 bytes are compared four and two to a register: a byte (or half) of
// e = (x & mask) ^ value is zero exactly where its top bit stays clear in
// ((e & 0x7f..) + 0x7f..) | e, and a byte dot product adds up the set bits of the matches.
#pragma once

#include "ibp_common.cuh"

namespace ibp200 {

// s += pc where d is 0, as a predicated multiply-add by `one` (1, not known at compile time):
// logic, compares and adds share the integer pipe, which bounds these loops, and a multiply-add
// runs on the other one.
__device__ __forceinline__ void add_if_zero(uint32_t &s, uint32_t d, uint32_t pc, uint32_t one) {
    asm("{\n\t.reg .pred p;\n\tsetp.eq.u32 p, %1, 0;\n\t@p mad.lo.u32 %0, %2, %3, %0;\n\t}"
        : "+r"(s)
        : "r"(d), "r"(pc), "r"(one));
}

template <typename U, int A, int G>
struct Chunk {
    static constexpr int WB = sizeof(U);
    static constexpr int NS = A == 16 ? 1 : (A == 8 ? 2 : 4);  // pieces
    static constexpr int PR = A >= 4 ? A / 4 : 1;              // registers of a piece
    static constexpr int NR = NS * PR;
    static constexpr int NW = WB == 8 ? NR / 2 : NR;  // set-bit counts (bytes of one for WB < 4)
    static_assert(A >= WB && (A & (A - 1)) == 0 && A <= 16, "piece size");

    // Pieces c, c + G, ... of a row of `pieces`; those past the end are zero.
    static __device__ __forceinline__ void load(const char *row, int64_t c, int64_t pieces,
                                                uint32_t (&x)[NR]) {
        const char *p = row + c * A;
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            uint32_t *y = x + k * PR;
#pragma unroll
            for (int i = 0; i < PR; ++i) y[i] = 0;
            if (c + k * G < pieces) {
                if constexpr (A == 16) {
                    const uint4 z = *reinterpret_cast<const uint4 *>(p);
                    y[0] = z.x, y[1] = z.y, y[2] = z.z, y[3] = z.w;
                } else if constexpr (A == 8) {
                    const uint2 z = *reinterpret_cast<const uint2 *>(p + k * G * A);
                    y[0] = z.x, y[1] = z.y;
                } else if constexpr (A == 4) {
                    y[0] = *reinterpret_cast<const uint32_t *>(p + k * G * A);
                } else if constexpr (A == 2) {
                    y[0] = *reinterpret_cast<const uint16_t *>(p + k * G * A);
                } else {
                    y[0] = *reinterpret_cast<const uint8_t *>(p + k * G * A);
                }
            }
        }
    }

    // the same columns' masks or values, which start at any multiple of the word size
    static __device__ __forceinline__ void load_words(const U *p, int64_t c, int64_t pieces,
                                                      uint32_t (&x)[NR]) {
#pragma unroll
        for (int k = 0; k < NS; ++k) {
            uint32_t *y = x + k * PR;
#pragma unroll
            for (int i = 0; i < PR; ++i) y[i] = 0;
            if (c + k * G < pieces) {
#pragma unroll
                for (int j = 0; j < A / WB; ++j) {
                    const U w = __ldg(p + (c + k * G) * (A / WB) + j);
                    if constexpr (WB == 8) {
                        y[2 * j] = (uint32_t)w;
                        y[2 * j + 1] = (uint32_t)(w >> 32);
                    } else {
                        y[j * WB / 4] |= (uint32_t)w << (8 * (j * WB % 4));
                    }
                }
            }
        }
    }

    // set bits of each masked word, in the form matched<SHIFT>() adds them
    template <int SHIFT = 0>
    static __device__ __forceinline__ void set_bits(const uint32_t (&m)[NR], uint32_t (&pc)[NW]) {
#pragma unroll
        for (int i = 0; i < NW; ++i) {
            if constexpr (WB == 8) {
                pc[i] = (__popc(m[2 * i]) + __popc(m[2 * i + 1])) << SHIFT;
            } else if constexpr (WB == 4) {
                pc[i] = __popc(m[i]) << SHIFT;
            } else {
                uint32_t c = m[i] - ((m[i] >> 1) & 0x55555555u);
                c = (c & 0x33333333u) + ((c >> 2) & 0x33333333u);
                c = (c + (c >> 4)) & 0x0f0f0f0fu;  // per byte
                if constexpr (WB == 2) c = ((c << 8) + c) & 0xff00ff00u;  // per half, in its top byte
                pc[i] = c;
            }
        }
    }

    // s += set bits saved by the words whose mismatch bits e are all zero, shifted left by
    // SHIFT; e(i) is register i's, `one` is 1
    template <int SHIFT = 0, typename E>
    static __device__ __forceinline__ void matched(uint32_t &s, E e, const uint32_t (&pc)[NW],
                                                   uint32_t one) {
        if constexpr (WB >= 4) {
#pragma unroll
            for (int i = 0; i < NW; ++i)
                add_if_zero(s, WB == 8 ? (e(2 * i) | e(2 * i + 1)) : e(i), pc[i], one);
        } else {
            constexpr uint32_t low = WB == 1 ? 0x7f7f7f7fu : 0x7fff7fffu;
            uint32_t dot = 0;
#pragma unroll
            for (int i = 0; i < NW; ++i) {
                const uint32_t d = e(i);
                const uint32_t z = ~(((d & low) + low) | d | low);  // 0x80 in a match's top byte
                dot = __dp4a(z, pc[i], dot);
            }
            s += SHIFT ? (dot >> 7) << SHIFT : dot >> 7;
        }
    }
};

// Sums of N values over the G lanes of a group: every halving step sends one half of the
// values and keeps the other, so the lanes end up with N / G values each (or, once one is
// left, with the same one).  value_of(lane) is the first of the values a lane ends with.
template <int N, int G>
__device__ __forceinline__ void group_sums(uint32_t (&v)[N], uint32_t one) {
    const int lane = threadIdx.x & 31;
    int n = N;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        if (n > 1) {
            n >>= 1;
            const bool up = lane & o;
#pragma unroll
            for (int i = 0; i < N / 2; ++i) {
                if (i < n) {
                    const uint32_t send = up ? v[i] : v[i + n];
                    const uint32_t keep = up ? v[i + n] : v[i];
                    v[i] = __shfl_xor_sync(0xffffffffu, send, o) * one + keep;
                }
            }
        } else {
            v[0] = __shfl_xor_sync(0xffffffffu, v[0], o) * one + v[0];
        }
    }
}

// The first value that lane `sub` of its group holds after group_sums<N, G>.
template <int N, int G>
__device__ __forceinline__ int group_sums_value(int sub) {
    int n = N, first = 0;
#pragma unroll
    for (int o = G / 2; o > 0; o >>= 1) {
        if (n > 1) {
            n >>= 1;
            if (sub & o) first += n;
        }
    }
    return first;
}

// Lanes of a group that end with the same value: the low bits of the lane number.
template <int N, int G>
constexpr int group_sums_copies() {
    return G > N ? G / N : 1;
}

// Largest piece (16, 4 or the word itself; 8 for 64-bit words) that divides every row's start.
inline int row_piece_bytes(const void *base, int64_t v, int wb) {
    const uint64_t a = (uint64_t)(uintptr_t)base | (uint64_t)(v * wb);
    if ((a & 15) == 0) return 16;
    if (wb == 8) return (a & 7) == 0 ? 8 : 0;
    if ((a & 3) == 0) return 4;
    return wb;
}

}  // namespace ibp200
