// Decode GEMV for matrices small enough that a block's whole share of the weights fits in a fraction of an SM's shared memory (the layers of a 0.5B model:
// 0.45 to 5 MB a matrix at four to eight bits, up to 17 MB as f16).
//
// Such a projection moves its bytes in well under a microsecond; what it costs is the chain of latencies from its predecessor's end to its own. So:
//   * Small blocks (8 warps, at most kSmemLimit of shared memory, no ring): the blocks of this kernel and of the ones after it sit on an SM together. Launched
//     early (launch.cuh), a block has asked for ALL of its weights, and mostly has them, before the kernel in front of it is done; after the wait only the
//     input vector is fetched. The ring kernels (gemv_q4_0.cu, gemv_blocks.cu) take most of an SM, so their first copy starts when the block before leaves.
//   * The block normalizes and splits a row of up to kOwnNorm elements itself: for 896 that is a handful of loads per thread, where the producer-side split of the
//     wide shapes (GemvNormLink) costs a fence, an atomic and a second trip through L2 at the end of the producer. Wider rows come through the link (the 8B
//     shape's qkv projection: 5.5 us on the ring kernel, 8.3 with the norm in every block here).
//   * A gate / up block owns whole 32-row groups, so it splits its results for ffn_down out of registers, without counting rows across blocks.
//   * The matrices of a q / k / v projection are parts of one launch, also when their formats differ.
//   * q4_0, q5_0 and q8_0 on the tensor cores' integer path (pair_mma.cuh): exact digit products, f32 sums over blocks; f16 rows as f32 dot products. Against f64 the
//     digits (27 bits below the largest of a block's 32 inputs) are closer than f32 dot products for q5_0 and q8_0 too, where they took those's place: 7.3e-8 against
//     2.9e-7 (1152 x 896) and 8.0e-8 against 1.2e-7 (151936 x 896) on normal inputs, 8.0e-8 against 3.0e-7 and 8.8e-8 against 1.4e-7 with one input in 97 a thousand
//     times its neighbours. Only q8_0 rows whose weights are zero at every such input see f32 ahead (1.2e-7 against 2.4e-6).
// Units of work are (16-row tile, matrix, chunk of the row); a warp adds what it computed for a (tile, matrix) into its own slot of a table whose slots are
// summed in a fixed order: results do not depend on timing.
// Replaces matvec1q / gate_up1q (llama_kernels.h:1197-1269) and norm_vec (:1272-1286) for these shapes.
#include <cuda_fp16.h>

#include <algorithm>

#include "kernels.h"
#include "launch.cuh"
#include "pair_mma.cuh"
#include "ptx.cuh"
#include "quant.cuh"
#include "xsplit.cuh"

namespace dooms {
namespace cuda {

using namespace dooms::dev;

namespace {

constexpr int kWarps = 8, kThreads = kWarps * 32;
constexpr int kTileRows = 16;
constexpr int kHeld = 8;                       // input blocks a warp keeps in registers while it normalizes: rows of up to 2048 make one pass
constexpr int64_t kOwnNorm = int64_t(kHeld) * kWarps * 32;
constexpr int kMaxRows = 64;                   // rows per block
template <bool HALF> constexpr int kPerSm = HALF ? 3 : 2;      // blocks per SM that the registers are to allow (72 and 90 a thread)
constexpr size_t kSmemLimit = 92 * 1024;       // two blocks per SM always fit, whatever kernel they belong to; the 8B attn_output's share (see plan_for)

struct Input {
    const uint8_t * xq;      // the split input, or
    const float * x;         // the input as f32,
    const float * gamma;     // RMS-normalized first when given
    float eps;
    int cols;
    const float * ss;        // optional, with xq: the producer's sums of squares (GemvNormLink), n_ss of them; the results are scaled by the norm's factor
    int n_ss;
};
struct Part {
    const uint8_t * W;
    const uint8_t * W2;      // gate/up: the second matrix (up)
    float * y;
    const float * bias;
    int rows, dt;
    int block0;              // its first block
    int rpb;                 // rows per block
    int cbk, nchunks;        // blocks per chunk, chunks per row
    int stride, upr;         // bytes between the rows of a unit; 16-byte pieces copied per row (the aligned cover of a chunk)
    uint32_t inv_upr, inv_nchunks;   // 65536 / d + 1: (j * inv) >> 16 = j / d for the small j divided here
};
struct ShortParams {
    Part part[kShortParts];
    int n_parts;
    Input in;
    uint8_t * xq_out;        // optional (one part, blocks of whole 32-row groups): the results split for the next projection
    uint32_t flags;
    int x_bytes;             // shared memory in front of the units
};

__device__ __forceinline__ void cp_async16(uint32_t dst, const void * src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(dst), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N> __device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// The input row in shared memory, as digits and factors (xsplit.cuh) or, HALF, as f32. load_gains before the wait for the kernel in front, prepare_input after
// it; the copies prepare_input starts are complete after the caller's cp_async_wait<0>() and block barrier.
template <int WARPS>
__device__ __forceinline__ void load_gains(const Input & in, float (&gm)[kHeld]) {
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, nb = in.cols / 32;
    if (in.gamma) {
        #pragma unroll
        for (int j = 0; j < kHeld; j++) {
            const int blk = warp + j * WARPS;
            gm[j] = blk < nb ? __ldg(in.gamma + blk * 32 + lane) : 0.f;
        }
    }
}
template <bool HALF, int WARPS>
__device__ __forceinline__ void prepare_input(const Input & in, float (&gm)[kHeld], uint8_t * smem, float * red) {
    constexpr int THREADS = WARPS * 32;
    const int tid = threadIdx.x, warp = tid / 32, lane = tid % 32, nb = in.cols / 32;
    const uint32_t smem0 = smem_u32(smem);
    if (!HALF && in.xq) {
        for (uint32_t i = tid; i < uint32_t(nb) * 136u / 16u; i += THREADS) cp_async16(smem0 + i * 16u, in.xq + size_t(i) * 16);
        cp_async_commit();
        return;
    }
    if (HALF && !in.gamma) {
        for (uint32_t i = tid; i < uint32_t(in.cols) / 4u; i += THREADS) cp_async16(smem0 + i * 16u, in.x + size_t(i) * 4);
        cp_async_commit();
        return;
    }
    // The norm's factor waits until after the product, W (s u) = s (W u): the row goes into shared memory with its gains alone, and the sums of squares meet the
    // other warps' at the barrier that the row needs anyway (input_scale).
    auto put = [&](float e, int blk) {
        if constexpr (HALF) reinterpret_cast<float *>(smem)[blk * 32 + lane] = e;
        else split_block(e, lane, blk, nb, smem);
    };
    float ss = 0.f;
    for (int blk0 = warp; blk0 < nb; blk0 += WARPS * kHeld) {      // kHeld loads on their way before the first block is used
        float v[kHeld];
        #pragma unroll
        for (int j = 0; j < kHeld; j++) {
            const int blk = blk0 + j * WARPS;
            v[j] = blk < nb ? __ldcg(in.x + blk * 32 + lane) : 0.f;
            if (blk0 != warp) gm[j] = (in.gamma && blk < nb) ? __ldg(in.gamma + blk * 32 + lane) : 0.f;
        }
        #pragma unroll
        for (int j = 0; j < kHeld; j++) {
            const int blk = blk0 + j * WARPS;
            ss += v[j] * v[j];
            if (blk < nb) put(in.gamma ? v[j] * gm[j] : v[j], blk);
        }
    }
    if (in.gamma) {
        #pragma unroll
        for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
        if (lane == 0) red[warp] = ss;
    }
}
// After the barrier: what the results are multiplied by. norm_scale: link_scale's, when the producer made the sums.
template <int WARPS>
__device__ __forceinline__ float input_scale(const Input & in, const float * red, float norm_scale) {
    if (in.ss) return norm_scale;
    if (!in.gamma) return 1.f;
    float total = 0.f;
    #pragma unroll
    for (int w = 0; w < WARPS; w++) total += red[w];
    return rsqrtf(total / float(in.cols) + in.eps);
}

// The factor of a norm whose gains the producer of the split applied: its per-block sums, added in a fixed order by one warp.
__device__ __forceinline__ float link_scale(const Input & in, int lane) {
    float ss = 0.f;
    for (int i = lane; i < in.n_ss; i += 32) ss += __ldcg(in.ss + i);
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) ss += __shfl_xor_sync(0xffffffffu, ss, o);
    return rsqrtf(ss / float(in.cols) + in.eps);
}

// Copies a unit (rows x the aligned cover of a chunk) into its stage, the pieces dealt to the warp's lanes. base: the unit's first byte.
__device__ __forceinline__ void fetch_unit(const uint8_t * base, uint32_t dst, int rows, int upr, uint32_t inv_upr, uint32_t stride, uint32_t RB, uint32_t CB, int lane) {
    const int pieces = rows * upr;
    for (int j = lane; j < pieces; j += 32) {
        const uint32_t row = (uint32_t(j) * inv_upr) >> 16, off = (uint32_t(j) - row * uint32_t(upr)) * 16u;
        const uint8_t * src = base + row * RB;
        const uint32_t shift = uint32_t(reinterpret_cast<uintptr_t>(src)) & 15u;
        if (off < CB + shift) cp_async16(dst + row * stride + off, src - shift + off);
    }
}

// The chunk's pairs of blocks for the lane's rows.
template <int DT>
__device__ __forceinline__ void unit_pairs(uint32_t base0, uint32_t base1, uint32_t ba, uint32_t sa, uint32_t t, bool first, int npairs, float & acc0, float & acc1) {
    #pragma unroll 4      // (a warp's pairs are one chain of loads, MMAs and conversions after another; two at a time: 70.3 instead of 65.0 ms for 512 + 128 tokens of 0.5B)
    for (int pr = 0; pr < npairs; pr++) {
        pair_step_of<DT>(base0, base1, ba, sa, t, first, acc0, acc1);
        base0 += 2 * BlockInfo<DT>::bytes;
        base1 += 2 * BlockInfo<DT>::bytes;
        ba += 256;
        sa += 16;
    }
}

// Adds a staged unit to the lane's sums: blocks blk0 .. blk0 + cbk - 1 of rows 0 .. last. st: the stage; lo: the low address bits of the unit's first byte.
// Block formats: acc0 / acc1 are the lane quad's shares of rows g and g + 8. HALF: acc0 is the lane's share of row lane % (32 >> parts_log).
template <bool HALF>
__device__ __forceinline__ void unit_dot(int dt, const uint8_t * smem, uint32_t smem0, uint32_t st, uint32_t lo, uint32_t RB, uint32_t stride, int last, int parts_log,
                                         int blk0, int cbk, int nb, int lane, float & acc0, float & acc1) {
    if constexpr (HALF) {
        const int row = min(lane & ((32 >> parts_log) - 1), last);      // (lanes of rows that do not exist repeat the last one; their sums are not used)
        const uint4 * w = reinterpret_cast<const uint4 *>(smem + (st - smem0) + uint32_t(row) * stride);
        const float4 * xs = reinterpret_cast<const float4 *>(smem) + size_t(blk0) * 8;
        for (int gq = lane >> (5 - parts_log); gq < cbk; gq += 1 << parts_log) {
            #pragma unroll
            for (int i = 0; i < 4; i++) {
                const uint4 h = w[gq * 4 + i];
                const float4 x0 = xs[gq * 8 + 2 * i], x1 = xs[gq * 8 + 2 * i + 1];
                const float2 a = __half22float2(*reinterpret_cast<const __half2 *>(&h.x)), b = __half22float2(*reinterpret_cast<const __half2 *>(&h.y));
                const float2 c = __half22float2(*reinterpret_cast<const __half2 *>(&h.z)), d = __half22float2(*reinterpret_cast<const __half2 *>(&h.w));
                acc0 = fmaf(a.x, x0.x, acc0); acc1 = fmaf(a.y, x0.y, acc1);
                acc0 = fmaf(b.x, x0.z, acc0); acc1 = fmaf(b.y, x0.w, acc1);
                acc0 = fmaf(c.x, x1.x, acc0); acc1 = fmaf(c.y, x1.y, acc1);
                acc0 = fmaf(d.x, x1.z, acc0); acc1 = fmaf(d.y, x1.w, acc1);
            }
        }
        acc0 += acc1;
        acc1 = 0.f;
    } else {
        const int g = lane >> 2, t = lane & 3;
        const int r0 = min(g, last), r1 = min(g + 8, last);
        const uint32_t base0 = st + uint32_t(r0) * stride + ((lo + uint32_t(r0) * RB) & 15u), base1 = st + uint32_t(r1) * stride + ((lo + uint32_t(r1) * RB) & 15u);
        const uint32_t ba = smem0 + uint32_t(blk0) * 128u + uint32_t(g >> 2) * 128u + uint32_t(g & 3) * 32u + uint32_t(t) * 8u;
        const uint32_t sa = smem0 + uint32_t(nb) * 128u + uint32_t(blk0) * 8u + uint32_t(t >> 1) * 8u + uint32_t(t & 1) * 4u;
        const int np = cbk / 2;
        if (dt == kQ4_0) unit_pairs<kQ4_0>(base0, base1, ba, sa, uint32_t(t), g < 4, np, acc0, acc1);
        else if (dt == kQ5_0) unit_pairs<kQ5_0>(base0, base1, ba, sa, uint32_t(t), g < 4, np, acc0, acc1);
        else unit_pairs<kQ8_0>(base0, base1, ba, sa, uint32_t(t), g < 4, np, acc0, acc1);
    }
}

// HALF: f16 weights, the input as f32 in shared memory; otherwise block formats and the input as digits.
template <bool HALF>
__global__ void __launch_bounds__(kThreads, kPerSm<HALF>) k_gemv_short(const __grid_constant__ ShortParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float red[kWarps];
    __shared__ float norm_scale;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32, tid = threadIdx.x;
    int which = 0;
    while (which + 1 < p.n_parts && int(blockIdx.x) >= p.part[which + 1].block0) which++;
    const Part & q = p.part[which];
    const int nb = p.in.cols / 32, nmat = q.W2 ? 2 : 1;
    const uint32_t RB = uint32_t(row_bytes_of(q.dt, p.in.cols)), CB = uint32_t(row_bytes_of(q.dt, q.cbk * 32));
    const int R0 = (int(blockIdx.x) - q.block0) * q.rpb;
    const int nrows = min(q.rpb, q.rows - R0);
    const int ntm = (nrows + kTileRows - 1) / kTileRows * nmat;
    const int units = ntm * q.nchunks;
    const uint32_t stride = uint32_t(q.stride), unit_bytes = uint32_t(min(q.rpb, kTileRows)) * stride;
    const uint32_t smem0 = smem_u32(smem), unit0 = smem0 + uint32_t(p.x_bytes);
    // [tile, matrix][warp][16], after the units of the largest block
    float * partial = reinterpret_cast<float *>(smem + p.x_bytes + size_t((q.rpb + kTileRows - 1) / kTileRows * nmat * q.nchunks) * unit_bytes);

    if (!(p.flags & kFlagLateDependents)) pdl_trigger();
    // all of this warp's weights, before the kernel in front is waited for
    for (int u = warp; u < units; u += kWarps) {
        const int tm = int((uint32_t(u) * q.inv_nchunks) >> 16), chunk = u - tm * q.nchunks;
        const int tile = nmat == 2 ? tm >> 1 : tm;
        const uint8_t * base = ((nmat == 2 && (tm & 1)) ? q.W2 : q.W) + int64_t(R0 + tile * kTileRows) * RB + uint32_t(chunk) * CB;
        fetch_unit(base, unit0 + uint32_t(u) * unit_bytes, min(kTileRows, nrows - tile * kTileRows), q.upr, q.inv_upr, stride, RB, CB, lane);
    }
    cp_async_commit();
    for (int i = tid; i < ntm * kWarps * kTileRows; i += kThreads) partial[i] = 0.f;
    float gm[kHeld];
    load_gains<kWarps>(p.in, gm);
    pdl_wait();
    // The bias is a buffer of the caller's like x and y: the kernel in front may be the one that writes it.
    const float bias = ((p.flags & kFlagBias) && tid < nrows) ? __ldcg(q.bias + R0 + tid) : 0.f;
    const float old = ((p.flags & kFlagAccumulate) && tid < nrows) ? __ldcg(q.y + R0 + tid) : 0.f;      // y is final here too: nobody else writes these rows
    prepare_input<HALF, kWarps>(p.in, gm, smem, red);
    if (p.in.ss && warp == 0) {
        const float f = link_scale(p.in, lane);
        if (lane == 0) norm_scale = f;
    }
    cp_async_wait<0>();
    __syncthreads();

    int acc_tm = -1;
    float acc0 = 0.f, acc1 = 0.f;
    const int g = lane >> 2, t = lane & 3;
    const int parts_log = min(q.rpb, kTileRows) <= 8 ? 2 : 1;      // f16: a tile of 8 rows gives each row four lanes, one of 16 two
    auto flush = [&]() {
        float * dst = partial + (acc_tm * kWarps + warp) * kTileRows;
        if constexpr (HALF) {
            float s = acc0 + __shfl_xor_sync(0xffffffffu, acc0, 16);
            if (parts_log == 2) s += __shfl_xor_sync(0xffffffffu, s, 8);
            if (lane < (32 >> parts_log)) dst[lane] += s;
        } else {
            float s0 = acc0, s1 = acc1;
            s0 += __shfl_xor_sync(0xffffffffu, s0, 1); s0 += __shfl_xor_sync(0xffffffffu, s0, 2);
            s1 += __shfl_xor_sync(0xffffffffu, s1, 1); s1 += __shfl_xor_sync(0xffffffffu, s1, 2);
            if (t == 0) { dst[g] += s0; dst[g + 8] += s1; }
        }
        acc0 = 0.f;
        acc1 = 0.f;
    };
    for (int u = warp; u < units; u += kWarps) {
        const int tm = int((uint32_t(u) * q.inv_nchunks) >> 16), chunk = u - tm * q.nchunks;
        if (tm != acc_tm) { if (acc_tm >= 0) flush(); acc_tm = tm; }
        const int tile = nmat == 2 ? tm >> 1 : tm;
        const int last = min(kTileRows, nrows - tile * kTileRows) - 1;
        const uint32_t lo = uint32_t(reinterpret_cast<uintptr_t>((nmat == 2 && (tm & 1)) ? q.W2 : q.W)) + uint32_t(R0 + tile * kTileRows) * RB + uint32_t(chunk) * CB;
        const uint32_t st = unit0 + uint32_t(u) * unit_bytes;
        unit_dot<HALF>(q.dt, smem, smem0, st, lo, RB, stride, last, parts_log, chunk * q.cbk, q.cbk, nb, lane, acc0, acc1);
    }
    if (acc_tm >= 0) flush();
    __syncthreads();
    if (tid < nrows) {
        const float * src = partial + (tid / kTileRows) * nmat * kWarps * kTileRows + (tid % kTileRows);
        float s = 0.f;
        #pragma unroll
        for (int w = 0; w < kWarps; w++) s += src[w * kTileRows];
        const float scale = input_scale<kWarps>(p.in, red, norm_scale);
        s *= scale;
        if (nmat == 2) {
            float s2 = 0.f;
            #pragma unroll
            for (int w = 0; w < kWarps; w++) s2 += src[(kWarps + w) * kTileRows];
            s = s / (1.f + expf(-s)) * (s2 * scale);
        }
        s += bias;
        const float out = (p.flags & kFlagAccumulate) ? accumulate_base(old, p.flags) + s : s;
        q.y[R0 + tid] = out;
        if (p.xq_out) split_block(out, lane, (R0 + tid) / 32, q.rows / 32, p.xq_out);      // (whole warps: nrows and R0 are multiples of 32)
    }
}

// Tall matrices (an output matrix: five times as many rows as fit one wave of the kernel above, or of the ring kernels, whose blocks then prepare the input again
// every 114 rows: 57 us for the 77 MB of 151936 x 896 at 4.5 bits). One block per SM prepares the input once and stays; a warp takes whole 16-row tiles, every
// kTallWarps-th of its block's, streams their chunks through its own ring of stages and writes the 16 results itself, so there is no table and no barrier after
// the first.
constexpr int kTallWarps = 16;
constexpr size_t kTallSmem = 208 * 1024;
struct TallParams {
    const uint8_t * W;
    float * y;
    const float * bias;
    Input in;
    int64_t rows;
    int dt, tiles;           // tiles: 16-row tiles of the matrix; block b takes tiles b * tiles / gridDim.x ..
    uint32_t flags;
    int cbk, nchunks, stride, upr;
    uint32_t inv_upr;
    int x_bytes;
};

template <bool HALF, int STAGES>
__global__ void __launch_bounds__(kTallWarps * 32, 1) k_gemv_tall(const __grid_constant__ TallParams p) {
    extern __shared__ __align__(128) uint8_t smem[];
    __shared__ float red[kTallWarps];
    __shared__ float norm_scale;
    const int warp = threadIdx.x / 32, lane = threadIdx.x % 32;
    const int nb = p.in.cols / 32;
    const uint32_t RB = uint32_t(row_bytes_of(p.dt, p.in.cols)), CB = uint32_t(row_bytes_of(p.dt, p.cbk * 32)), stride = uint32_t(p.stride);
    const uint32_t smem0 = smem_u32(smem), stage_bytes = kTileRows * stride, my_stages = smem0 + uint32_t(p.x_bytes) + uint32_t(warp) * STAGES * stage_bytes;
    const int tile_end = int(int64_t(blockIdx.x + 1) * p.tiles / gridDim.x);
    int f_tile = int(int64_t(blockIdx.x) * p.tiles / gridDim.x) + warp, f_chunk = 0, f_slot = 0;      // the unit being fetched
    int tile = f_tile, slot = 0;                                                                     // the unit being used
    auto fetch = [&]() {
        if (f_tile < tile_end) {
            const int64_t row0 = int64_t(f_tile) * kTileRows;
            fetch_unit(p.W + row0 * RB + uint32_t(f_chunk) * CB, my_stages + uint32_t(f_slot) * stage_bytes, int(min(int64_t(kTileRows), p.rows - row0)), p.upr, p.inv_upr,
                       stride, RB, CB, lane);
            if (++f_chunk == p.nchunks) { f_chunk = 0; f_tile += kTallWarps; }
            if (++f_slot == STAGES) f_slot = 0;
        }
        cp_async_commit();
    };
    if (!(p.flags & kFlagLateDependents)) pdl_trigger();
    #pragma unroll
    for (int i = 0; i < STAGES - 1; i++) fetch();
    float gm[kHeld];
    load_gains<kTallWarps>(p.in, gm);
    pdl_wait();
    prepare_input<HALF, kTallWarps>(p.in, gm, smem, red);
    if (p.in.ss && warp == 0) {
        const float f = link_scale(p.in, lane);
        if (lane == 0) norm_scale = f;
    }
    cp_async_wait<0>();
    __syncthreads();
    const float scale = input_scale<kTallWarps>(p.in, red, norm_scale);
    const int g = lane >> 2, t = lane & 3;
    for (; tile < tile_end; tile += kTallWarps) {
        const int64_t row0 = int64_t(tile) * kTileRows;
        const int last = int(min(int64_t(kTileRows), p.rows - row0)) - 1;
        const uint32_t tile_lo = uint32_t(reinterpret_cast<uintptr_t>(p.W + row0 * RB));
        float acc0 = 0.f, acc1 = 0.f;
        for (int chunk = 0; chunk < p.nchunks; chunk++) {
            cp_async_wait<STAGES - 2>();      // this unit has landed (this lane's pieces) ...
            __syncwarp();                     // ... and every lane's; also: every lane is done with the stage refilled next
            fetch();
            unit_dot<HALF>(p.dt, smem, smem0, my_stages + uint32_t(slot) * stage_bytes, tile_lo + uint32_t(chunk) * CB, RB, stride, last, 1, chunk * p.cbk, p.cbk, nb, lane,
                           acc0, acc1);
            if (++slot == STAGES) slot = 0;
        }
        auto put = [&](int r, float s) {
            if (r > last) return;
            const int64_t row = row0 + r;
            s *= scale;
            if (p.flags & kFlagBias) s += p.bias[row];
            p.y[row] = (p.flags & kFlagAccumulate) ? accumulate_base(__ldcg(p.y + row), p.flags) + s : s;
        };
        if constexpr (HALF) {
            const float s = acc0 + __shfl_xor_sync(0xffffffffu, acc0, 16);
            if (lane < 16) put(lane, s);
        } else {
            acc0 += __shfl_xor_sync(0xffffffffu, acc0, 1); acc0 += __shfl_xor_sync(0xffffffffu, acc0, 2);
            acc1 += __shfl_xor_sync(0xffffffffu, acc1, 1); acc1 += __shfl_xor_sync(0xffffffffu, acc1, 2);
            if (t == 0) { put(g, acc0); put(g + 8, acc1); }
        }
    }
    cp_async_wait<0>();
}

struct TallPlan { int cbk, nchunks, stride, upr, stages; size_t smem; bool ok; };

struct Plan { int rpb, cbk, nchunks, stride, upr, blocks; size_t smem; bool ok; };

bool takes_type(int dt) { return dt == kQ4_0 || dt == kQ5_0 || dt == kQ8_0 || dt == kF16; }
size_t x_bytes_of(int dt, int64_t cols) { return (size_t(cols / 32) * (dt == kF16 ? 128 : 136) + 127) & ~size_t(127); }

// How a matrix (pair) is cut, with rpb rows per block: the chunk length that leaves the busiest warp the least to do, the longer one on ties.
Plan plan_rows(int dt, int64_t rows, int64_t cols, int nmat, int rpb) {
    Plan best{};
    const int nb = int(cols / 32), block_bytes = int(row_bytes_of(dt, 32));
    const int trows = std::min(rpb, kTileRows), ntm = (rpb + kTileRows - 1) / kTileRows * nmat;
    const int grain = dt == kF16 ? (trows <= 8 ? 4 : 2) : 2;      // blocks a warp's step covers
    int64_t best_cost = -1;
    for (int cbk = 2; cbk <= nb; cbk += 2) {
        if (nb % cbk) continue;
        const int64_t chunk = int64_t(cbk) * block_bytes;
        const bool exact = chunk % 16 == 0 && (int64_t(nb) * block_bytes) % 16 == 0;
        const int upr = int(exact ? chunk / 16 : (chunk + 30) / 16);
        const int units = ntm * (nb / cbk);
        // the reciprocals are exact while these products stay below 2^16
        if (int64_t(kTileRows) * upr * upr >= 65536 || int64_t(units) * (nb / cbk) >= 65536) continue;
        const int stride = upr * 16 + (upr % 2 == 0 ? 16 : 0);      // an odd number of 16-byte pieces: the rows of a fragment lie on different banks
        const size_t smem = x_bytes_of(dt, cols) + size_t(units) * trows * stride + size_t(ntm) * kWarps * kTileRows * sizeof(float);
        if (smem > kSmemLimit) continue;
        const int64_t cost = int64_t((units + kWarps - 1) / kWarps) * ((cbk + grain - 1) / grain);
        if (best_cost < 0 || cost <= best_cost) {
            best_cost = cost;
            best = Plan{rpb, cbk, nb / cbk, stride, upr, int((rows + rpb - 1) / rpb), smem, true};
        }
    }
    return best;
}

// Every block has to be resident at once with room beside it (the early start is the point), so a matrix is short when its share per SM, in one to three
// blocks, fits. Rows per block: an equal share per SM, in whole 16-row tiles above 8 rows; whole 32-row groups when the results are to be split. A gate / up
// pair that does not fit so is halved until it does, and a half need not be whole tiles: 4864 x 896 in f16 goes from 48 rows to 24 and 12, at most 36 an SM,
// where blocks of 16 would make it 48.
// all_rows: the rows of all parts of the launch.
Plan plan_for(int dt, int64_t rows, int64_t all_rows, int64_t cols, int nmat, bool split_out) {
    if (!takes_type(dt) || rows < 1 || cols < 64 || cols % 64 != 0 || cols > 65536 || all_rows > int64_t(3) * sm_count() * kMaxRows) return Plan{};
    if (split_out) return rows % 32 == 0 ? plan_rows(dt, rows, cols, nmat, 32) : Plan{};
    const int sms = sm_count();
    int rpb = int((all_rows + sms - 1) / sms);
    if (rpb > 8) rpb = std::min(kMaxRows, (rpb + kTileRows - 1) / kTileRows * kTileRows);
    // A gate / up pair may take up to three smaller blocks per SM. A plain projection that does not fit one per SM is left to the ring kernels (the 8B shape's qkv: two
    // and three blocks per SM here made no difference after a prompt of 2048 tokens and cost 0.8 of 84.0 ms at a short one). The 8B attn_output does fit: 32 rows of
    // 4096 in q4_0 and their input are kSmemLimit to the byte. Its gate / up then normalizes the residual row in every block, where a ring kernel would have left it
    // normalized and split (GemvNormLink): 37 + 48 tokens take 80.4 ms either way.
    for (;; rpb /= 2) {
        const Plan pl = plan_rows(dt, rows, cols, nmat, rpb);
        if (pl.ok || rpb <= 8 || nmat == 1) return pl;
    }
}
// All blocks of the launch on the GPU at once, by shared memory and by registers.
bool fits(int dt, const Plan & pl) {
    const int64_t per_sm = std::min<int64_t>(dt == kF16 ? kPerSm<true> : kPerSm<false>, int64_t((224 * 1024) / (pl.smem + 1024)));
    return pl.ok && int64_t(pl.blocks) <= int64_t(sm_count()) * per_sm;
}

// The longest chunk that leaves three stages a warp (two where no chunk does): fewer, longer copies per unit, and 2 x 16 of them in flight per SM.
TallPlan tall_plan(int dt, int64_t rows, int64_t cols) {
    TallPlan best{};
    if (!takes_type(dt) || cols < 64 || cols % 64 != 0 || cols > 65536 || rows <= int64_t(sm_count()) * 8 * kTileRows || rows >= (int64_t(1) << 31)) return best;
    const int nb = int(cols / 32), block_bytes = int(row_bytes_of(dt, 32));
    for (int cbk = 2; cbk <= nb; cbk += 2) {
        if (nb % cbk) continue;
        const int64_t chunk = int64_t(cbk) * block_bytes;
        const bool exact = chunk % 16 == 0 && (int64_t(nb) * block_bytes) % 16 == 0;
        const int upr = int(exact ? chunk / 16 : (chunk + 30) / 16);
        if (int64_t(kTileRows) * upr * upr >= 65536) continue;
        const int stride = upr * 16 + (upr % 2 == 0 ? 16 : 0);
        for (int stages = 4; stages >= 2; stages--) {
            const size_t smem = x_bytes_of(dt, cols) + size_t(kTallWarps) * stages * kTileRows * stride;
            if (smem > kTallSmem) continue;
            if (std::min(stages, 3) >= std::min(best.stages, 3)) best = TallPlan{cbk, nb / cbk, stride, upr, stages, smem, true};
            break;
        }
    }
    return best;
}

}  // namespace

bool gemv_short_own_norm(int64_t cols) { return cols <= kOwnNorm; }
bool gemv_short_supported(int dt, const void * W, int64_t rows, int64_t cols, int nmat, bool split_out, int64_t all_rows) {
    return (reinterpret_cast<uintptr_t>(W) & 15u) == 0 && fits(dt, plan_for(dt, rows, all_rows > 0 ? all_rows : rows, cols, nmat, split_out));
}

cudaError_t launch_gemv_short(const ShortMatrix * mats, int n, const void * xq, const float * x, const float * gamma, float eps, int64_t cols, uint32_t flags,
                              cudaStream_t stream, void * xq_out, const GemvNormLink * link) {
    if (link && link->ss_in && !xq) return cudaErrorInvalidValue;
    if (n < 1 || n > kShortParts || (!xq && !x) || (xq && gamma) || (xq_out && n != 1)) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(xq) & 15u) || (reinterpret_cast<uintptr_t>(x) & 15u)) return cudaErrorInvalidValue;
    ShortParams p{};
    const bool half = mats[0].dt == kF16;
    size_t smem = 0;
    int blocks = 0;
    int64_t all_rows = 0;
    for (int i = 0; i < n; i++) all_rows += mats[i].rows;
    for (int i = 0; i < n; i++) {
        const ShortMatrix & m = mats[i];
        if ((m.dt == kF16) != half || !m.W || !m.y || ((flags & kFlagBias) && !m.bias) || (half && !x)) return cudaErrorInvalidValue;
        if ((reinterpret_cast<uintptr_t>(m.W) & 15u) || (reinterpret_cast<uintptr_t>(m.W2) & 15u)) return cudaErrorInvalidValue;
        const Plan pl = plan_for(m.dt, m.rows, all_rows, cols, m.W2 ? 2 : 1, xq_out != nullptr);
        if (!pl.ok) return cudaErrorInvalidValue;
        p.part[i] = Part{static_cast<const uint8_t *>(m.W), static_cast<const uint8_t *>(m.W2), m.y, m.bias, int(m.rows), m.dt, blocks, pl.rpb, pl.cbk, pl.nchunks, pl.stride,
                         pl.upr, 65536u / uint32_t(pl.upr) + 1u, 65536u / uint32_t(pl.nchunks) + 1u};
        blocks += pl.blocks;
        smem = std::max(smem, pl.smem);
    }
    p.n_parts = n;
    p.in = Input{half ? nullptr : static_cast<const uint8_t *>(xq), x, gamma, eps, int(cols), link ? link->ss_in : nullptr, link ? link->ss_n : 0};
    p.xq_out = static_cast<uint8_t *>(xq_out);
    p.flags = flags;
    p.x_bytes = int(x_bytes_of(mats[0].dt, cols));
    auto go = [&](auto kernel, std::atomic<uint64_t> & configured) -> cudaError_t {
        if (const cudaError_t e = allow_dynamic_smem(kernel, int(kSmemLimit), configured); e != cudaSuccess) return e;
        return launch_pdl(kernel, dim3(unsigned(blocks)), dim3(kThreads), smem, stream, p);
    };
    static std::atomic<uint64_t> done_int{0}, done_half{0};
    return half ? go(k_gemv_short<true>, done_half) : go(k_gemv_short<false>, done_int);
}

// Rows enough for more than one wave of the ring kernels' blocks (128 rows a block).
bool gemv_tall_supported(int dt, const void * W, int64_t rows, int64_t cols) { return (reinterpret_cast<uintptr_t>(W) & 15u) == 0 && tall_plan(dt, rows, cols).ok; }

cudaError_t launch_gemv_tall(int dt, const void * W, const void * xq, const float * x, const float * gamma, float eps, float * y, const float * bias, int64_t rows, int64_t cols,
                             uint32_t flags, cudaStream_t stream, const GemvNormLink * link) {
    const bool half = dt == kF16;
    if (!W || !y || (!xq && !x) || (xq && gamma) || (half && !x) || ((flags & kFlagBias) && !bias) || (link && link->ss_in && (half || !xq))) return cudaErrorInvalidValue;
    if ((reinterpret_cast<uintptr_t>(W) & 15u) || (reinterpret_cast<uintptr_t>(xq) & 15u) || (reinterpret_cast<uintptr_t>(x) & 15u)) return cudaErrorInvalidValue;
    const TallPlan pl = tall_plan(dt, rows, cols);
    if (!pl.ok) return cudaErrorInvalidValue;
    const TallParams p{static_cast<const uint8_t *>(W), y, bias, Input{half ? nullptr : static_cast<const uint8_t *>(xq), x, gamma, eps, int(cols), link ? link->ss_in : nullptr,
                       link ? link->ss_n : 0}, rows, dt, int((rows + kTileRows - 1) / kTileRows), flags, pl.cbk, pl.nchunks, pl.stride, pl.upr, 65536u / uint32_t(pl.upr) + 1u,
                       int(x_bytes_of(dt, cols))};
    auto go = [&](auto kernel, std::atomic<uint64_t> & configured) -> cudaError_t {
        if (const cudaError_t e = allow_dynamic_smem(kernel, int(kTallSmem), configured); e != cudaSuccess) return e;
        return launch_pdl(kernel, dim3(unsigned(sm_count())), dim3(kTallWarps * 32), pl.smem, stream, p);
    };
    static std::atomic<uint64_t> done[6];
    switch (pl.stages) {
        case 4: return half ? go(k_gemv_tall<true, 4>, done[0]) : go(k_gemv_tall<false, 4>, done[1]);
        case 3: return half ? go(k_gemv_tall<true, 3>, done[2]) : go(k_gemv_tall<false, 3>, done[3]);
        default: return half ? go(k_gemv_tall<true, 2>, done[4]) : go(k_gemv_tall<false, 2>, done[5]);
    }
}

}  // namespace cuda
}  // namespace dooms
