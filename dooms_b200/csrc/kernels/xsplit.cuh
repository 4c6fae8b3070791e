#pragma once
// The input-vector format of the staged q4_0 GEMV (gemv_q4_0.cu): per 32-element block a power-of-two scale s and, for every element, the fixed-point
// value X = rint(x / s * 2^26) cut into four balanced base-128 digits (int8). Layout of xq for a vector of nb blocks: nb x 128 digit bytes
// ([digit 0..3][32 bytes], a lane t of an MMA fragment finding its 8 bytes of a digit contiguous at 8 t), then nb x 2 floats (the factors that turn the
// integer sums of the lower and the upper digit pair back into values).
#include <cstdint>

namespace dooms {
namespace dev {

// One warp, one block: lane holds element `lane` of block blk.
__device__ __forceinline__ void split_block(float v, int lane, int blk, int nb, uint8_t * xq) {
    const uint32_t amax = __reduce_max_sync(0xffffffffu, __float_as_uint(v) & 0x7FFFFFFFu);      // magnitudes order like their bits, infinities and NaN on top
    uint32_t eb = amax >> 23;                                  // biased exponent of the largest magnitude
    eb = max(eb, 30u);                                         // blocks below 2^-97 are treated as that small: their digits come out zero
    eb = min(eb, 250u);
    const float inv = __uint_as_float((279u - eb) << 23);      // 2^26 / s with s = 2^(eb - 126) > amax
    // Within 2^26 for a finite block (of values below 2^124), so the bounds touch infinities alone: they become +-(33 * 128^3 + 128), the digits +-33 and +-1 at the top of either pair, and their
    // neighbours (below 2^97) zero.
    int X = min(max(__float2int_rn(v * inv), -69206144), 69206144);
    int l[4];
    #pragma unroll
    for (int i = 0; i < 3; i++) { l[i] = ((X + 64) & 127) - 64; X = (X - l[i]) >> 7; }
    l[3] = X;
    const int pos = ((lane & 15) >> 2) * 8 + (lane >> 4) * 4 + (lane & 3);
    uint8_t * dst = xq + size_t(blk) * 128;
    #pragma unroll
    for (int i = 0; i < 4; i++) dst[i * 32 + pos] = uint8_t(int8_t(l[i]));
    if (lane == 0) {
        float * sx = reinterpret_cast<float *>(xq + size_t(nb) * 128) + blk * 2;
        // A block that is not finite has its largest magnitude itself for a factor. An infinity: a row's sum is what the product with its weight is in f32, an infinity or
        // (weight zero) NaN; of several in one block, the sign of their sum's. A NaN: every sum the block enters is NaN.
        const bool finite = amax < 0x7F800000u;
        sx[0] = __uint_as_float(finite ? (eb - 29u) << 23 : amax);      // s * 2^-26 / 16: the weights carry a factor 16
        sx[1] = __uint_as_float(finite ? (eb - 15u) << 23 : amax);      // the same for the upper digit pair (x 2^14)
    }
}

}  // namespace dev
}  // namespace dooms
