#pragma once
// Dot products of 32-element weight blocks with an input split into int8 digits (xsplit.cuh), on the tensor cores' integer path: the inner step of the
// short decode GEMV (gemv_short.cu) for the three formats whose blocks are 32 elements with one scale.
#include <cuda_fp16.h>

#include <cstdint>

#include "ptx.cuh"
#include "quant.cuh"

namespace dooms {
namespace dev {

// The A operand of one row of a block: elements 4 t .. 4 t + 3 (lo) and 16 + 4 t .. (hi) as int8. Rows and chunks
// hold an even number of blocks, so a pair starts 4-byte aligned: the even block's quants straddle two words, the odd block's are whole words. The input's factors
// assume weights times 16 (the q4_0 operand); kFactor makes up for what the format's operand carries instead.
template <int DT> struct PairFormat;

template <> struct PairFormat<kQ4_0> {
    static constexpr float kFactor = 1.f;            // 16 (q - 8)
    // base: the pair's first byte
    static __device__ __forceinline__ void even(uint32_t base, uint32_t t, uint32_t & lo, uint32_t & hi) {
        const uint32_t q = __byte_perm(lds32<0>(base + 4u * t), lds32<4>(base + 4u * t), 0x5432);
        lo = lop3_and_xor(q << 4, 0xF0F0F0F0u, 0x80808080u);
        hi = lop3_and_xor(q, 0xF0F0F0F0u, 0x80808080u);
    }
    static __device__ __forceinline__ void odd(uint32_t base, uint32_t t, uint32_t & lo, uint32_t & hi) {
        const uint32_t q = lds32<20>(base + 4u * t);
        lo = lop3_and_xor(q << 4, 0xF0F0F0F0u, 0x80808080u);
        hi = lop3_and_xor(q, 0xF0F0F0F0u, 0x80808080u);
    }
};

// q5_0: the fifth bits are the bits 4 t .. 4 t + 3 and 16 + 4 t .. of one word; multiplying four bits by 1 + 2^7 + 2^14 + 2^21 puts bit i at bit 8 i (the
// sixteen products fall on different bits, so nothing carries). 8 (v - 16) = (v << 3) with the top bit flipped.
template <> struct PairFormat<kQ5_0> {
    static constexpr float kFactor = 2.f;            // 8 (v - 16)
    static __device__ __forceinline__ uint32_t fifth(uint32_t bits) { return (((bits & 15u) * 0x00204081u) & 0x01010101u) << 7; }
    static __device__ __forceinline__ void combine(uint32_t q, uint32_t qh, uint32_t t, uint32_t & lo, uint32_t & hi) {
        lo = ((q << 3) & 0x78787878u) | (fifth(qh >> (4u * t)) ^ 0x80808080u);
        hi = ((q >> 1) & 0x78787878u) | (fifth(qh >> (16u + 4u * t)) ^ 0x80808080u);
    }
    static __device__ __forceinline__ void even(uint32_t base, uint32_t t, uint32_t & lo, uint32_t & hi) {
        const uint32_t qh = __byte_perm(lds32<0>(base), lds32<4>(base), 0x5432);
        combine(__byte_perm(lds32<4>(base + 4u * t), lds32<8>(base + 4u * t), 0x5432), qh, t, lo, hi);
    }
    static __device__ __forceinline__ void odd(uint32_t base, uint32_t t, uint32_t & lo, uint32_t & hi) {
        combine(lds32<28>(base + 4u * t), lds32<24>(base), t, lo, hi);
    }
};

template <> struct PairFormat<kQ8_0> {
    static constexpr float kFactor = 16.f;           // q
    static __device__ __forceinline__ void even(uint32_t base, uint32_t t, uint32_t & lo, uint32_t & hi) {
        lo = __byte_perm(lds32<0>(base + 4u * t), lds32<4>(base + 4u * t), 0x5432);
        hi = __byte_perm(lds32<16>(base + 4u * t), lds32<20>(base + 4u * t), 0x5432);
    }
    static __device__ __forceinline__ void odd(uint32_t base, uint32_t t, uint32_t & lo, uint32_t & hi) {
        lo = lds32<36>(base + 4u * t);
        hi = lds32<52>(base + 4u * t);
    }
};

// One pair of blocks of the lane's rows g and g + 8 (base0 / base1: the pair's first byte): both blocks go into one 8-column fragment, columns 0..3 the even block's
// four digits and 4..7 the odd block's, so that every lane has one (row, block, digit pair) to scale. ba / sa: the lane's digits and factor of the pair's input.
template <int DT>
__device__ __forceinline__ void pair_step_of(uint32_t base0, uint32_t base1, uint32_t ba, uint32_t sa, uint32_t t, bool first, float & acc0, float & acc1) {
    using F = PairFormat<DT>;
    constexpr uint32_t BB = BlockInfo<DT>::bytes;
    const uint2 bv = lds64<0>(ba);
    const float sx = ldsf<0>(sa) * F::kFactor;
    const uint32_t od = (t >> 1) * BB;                // which block of the pair this lane scales
    const float d0 = half_bits_to_float(lds16<0>(base0 + od)), d1 = half_bits_to_float(lds16<0>(base1 + od));
    uint32_t l0, h0, l1, h1;
    int c[4];
    F::even(base0, t, l0, h0);
    F::even(base1, t, l1, h1);
    mma_s8_16832_zero(c, l0, l1, h0, h1, first ? bv.x : 0u, first ? bv.y : 0u);
    F::odd(base0, t, l0, h0);
    F::odd(base1, t, l1, h1);
    mma_s8_16832(c, l0, l1, h0, h1, first ? 0u : bv.x, first ? 0u : bv.y);
    acc0 = fmaf(float(c[0] + 128 * c[1]), d0 * sx, acc0);
    acc1 = fmaf(float(c[2] + 128 * c[3]), d1 * sx, acc1);
}

}  // namespace dev
}  // namespace dooms
