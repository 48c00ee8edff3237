// Register lookups of 16-bit values by codes of up to four bits, shared by the kernels that expand or consume such codes.
#pragma once
#include "common.cuh"

namespace dd {

template <bool V> struct IsRagged { static constexpr bool value = V; };     // compile-time argument of a generic lambda

// Up to four plane words, regrouped: nibble position 4t of result ph, rotated left by B - 1 - ph, starts the field of the bits
// that planes P[0..B-1] carry at position 4t + ph, most significant plane first.
template <int B>
__device__ __forceinline__ void ap_merge(const uint32_t* P, uint32_t (&M)[4]) {
    uint32_t R[B];
#pragma unroll
    for (int i = 0; i < B; ++i) R[i] = i ? __funnelshift_r(P[i], P[i], i) : P[0];
#pragma unroll
    for (int ph = 0; ph < 4; ++ph) {
        M[ph] = 0u;
#pragma unroll
        for (int i = 0; i < B; ++i) M[ph] |= R[i] & (0x11111111u << ((ph - i) & 3));
    }
}
__device__ __forceinline__ uint32_t rotate_left(uint32_t v, int by) { return (by & 31) ? __funnelshift_l(v, v, by & 31) : v; }

// 4-bit fields: field t (bits 4t..4t+3) of result ph holds the code bits of position 4t + ph.
template <int B>
__device__ __forceinline__ void ap_fields(const uint32_t* P, uint32_t (&V)[4]) {
    ap_merge<B>(P, V);
#pragma unroll
    for (int ph = 0; ph < 4; ++ph) V[ph] = rotate_left(V[ph], B - 1 - ph);
}

// A table of 2^BITS 16-bit values in registers, split into low and high bytes so that one byte permute looks up the low (or
// high) bytes of four codes.  BITS <= 3 fits one permute; 4 bits take two and a permute that picks by the codes' top bit.
template <int BITS>
struct LutBytes {
    static constexpr int kEntries = 1 << BITS;
    static constexpr int kRegs = BITS == 4 ? 4 : 2;
    uint32_t lo[kRegs], hi[kRegs];      // entries 4i .. 4i+3

    // pairs[i] = entries 2i and 2i + 1, as a row of the table lies in memory
    __device__ __forceinline__ void fill_pairs(const uint32_t* pairs) {
#pragma unroll
        for (int r = 0; r < kRegs; ++r) {
            const uint32_t a = 4 * r < kEntries ? pairs[2 * r < kEntries / 2 ? 2 * r : 0] : 0u;
            const uint32_t b = 4 * r + 2 < kEntries ? pairs[2 * r + 1 < kEntries / 2 ? 2 * r + 1 : 0] : 0u;
            lo[r] = __byte_perm(a, b, 0x6420);
            hi[r] = __byte_perm(a, b, 0x7531);
        }
    }
    template <typename T>
    __device__ __forceinline__ void fill(const T* v) {
        uint32_t pairs[kEntries / 2];
#pragma unroll
        for (int i = 0; i < kEntries / 2; ++i) {
            T e[2] = {v[2 * i], v[2 * i + 1]};
            pairs[i] = (uint32_t)reinterpret_cast<const uint16_t*>(e)[0] | ((uint32_t)reinterpret_cast<const uint16_t*>(e)[1] << 16);
        }
        fill_pairs(pairs);
    }
    // values of the codes in nibbles 0..3 of v: e01 = {code 0, code 1}, e23 = {code 2, code 3}
    __device__ __forceinline__ void lookup(uint32_t v, uint32_t& e01, uint32_t& e23) const {
        uint32_t l, h;
        if constexpr (BITS < 4) {
            l = __byte_perm(lo[0], lo[1], v);       // nibbles hold codes below 8: no sign replication
            h = __byte_perm(hi[0], hi[1], v);
        } else {
            const uint32_t s = v & 0x7777u;
            const uint32_t top = ((v >> 1) & 0x4444u) | 0x3210u;
            l = __byte_perm(__byte_perm(lo[0], lo[1], s), __byte_perm(lo[2], lo[3], s), top);
            h = __byte_perm(__byte_perm(hi[0], hi[1], s), __byte_perm(hi[2], hi[3], s), top);
        }
        e01 = __byte_perm(l, h, 0x5140);
        e23 = __byte_perm(l, h, 0x7362);
    }
};

}  // namespace dd
