// Decode attention for one new token, grouped-query aware: the query heads that share a key/value head are processed together, so every cached key and value
// row is read from device memory once per step, in 16-byte coalesced asynchronous copies, by a grid of (key/value head, range of positions) blocks that
// covers all SMs. The kernel also does what used to be a launch of its own before it: it rotates the new token's query and key (rope_store,
// src/backend/metal/llama_kernels.h:521-545), writes the rotated key and the value into the f16 cache, and uses them from shared memory in the same pass.
// Only ranges that hold keys run. One range writes the row itself; ranges that form one cluster merge out of one another's shared memory; otherwise each block
// leaves an unnormalised partial result (max, sum, values) per query head, and the block that finishes a key/value head's last range merges the
// ranges of its query heads itself (attention_split / attention_combine, llama_kernels.h:860-929), or k_attention_combine does when no counters are given.
// The scores and the weighted sums run on the tensor cores (attention_decode_body.cuh).
#include <cuda_fp16.h>
#include <math_constants.h>

#include <algorithm>

#include "attention_decode_body.cuh"
#include "kernels.h"
#include "launch.cuh"
#include "ptx.cuh"
#include "xsplit.cuh"


namespace dooms {
namespace cuda {

using namespace dooms::dev;
using namespace dooms::cuda::attn_decode;

namespace {

template <int D, int GP, int STAGES>
__global__ void __launch_bounds__(kThreads) k_attention_decode(const AttnDecodeParams pp) {
    extern __shared__ __align__(128) uint8_t smem[];
    pdl_trigger();
    if (!pp.cache_ready) pdl_wait();
    attention_decode_body<D, GP, true, STAGES>(pp, int(blockIdx.x), int(blockIdx.y), int(blockIdx.z), smem);
}

// Heads of 128 on a context of which a range holds two pairs of tiles at most: two stages, and 74 KB instead of 143, leave a block room beside the projection in
// front, so that its fetches are early (the 8B shape at 60 keys: 10.3 us to 6.0). Longer ranges want the second pair on its way (the 32B shape
// at 8200 keys, ranges of four pairs: 24.1 us with four stages, 28.4 with two, also with twice as many blocks). What counts is the context the decoder was created
// with: a captured step serves all of its positions.
template <int D, int GP, int STAGES>
cudaError_t launch_staged(const AttnDecodeParams & p, cudaStream_t stream) {
    constexpr size_t smem = attention_decode_smem_bytes<D, GP, STAGES>();
    static std::atomic<uint64_t> configured{0};
    if (const cudaError_t e = allow_dynamic_smem(k_attention_decode<D, GP, STAGES>, int(smem), configured); e != cudaSuccess) return e;
    if (!p.cluster) return launch_pdl(k_attention_decode<D, GP, STAGES>, dim3(p.s.n_head_kv, p.splits, p.b_slot ? unsigned(p.b_rows) : 1u), dim3(kThreads), smem, stream, p);
    // clusters of kCluster consecutive ranges; the grid is rounded up to whole clusters, blocks past the last range leave at once
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(p.s.n_head_kv, (p.splits + kCluster - 1) / kCluster * kCluster, 1);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = smem;
    cfg.stream = stream;
    cudaLaunchAttribute attr[2];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1;
    attr[0].val.clusterDim.y = kCluster;
    attr[0].val.clusterDim.z = 1;
    attr[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = attr;
    cfg.numAttrs = pdl_enabled() ? 2 : 1;
    return cudaLaunchKernelEx(&cfg, k_attention_decode<D, GP, STAGES>, p);
}

template <int D, int GP>
cudaError_t launch_one(const AttnDecodeParams & p, cudaStream_t stream) {
    if constexpr (D > 64) {
        if (p.cache_ready && p.cache_ready <= p.splits * 4 * kTileKeys) return launch_staged<D, GP, 2>(p, stream);
    }
    return launch_staged<D, GP, kStagesFull>(p, stream);
}

template <int D>
cudaError_t launch_group(const AttnDecodeParams & p, int G, cudaStream_t stream) {
    if (G == 1) return launch_one<D, 1>(p, stream);
    if (G == 2) return launch_one<D, 2>(p, stream);
    if (G <= 4) return launch_one<D, 4>(p, stream);
    return launch_one<D, 8>(p, stream);
}

}  // namespace

bool attention_gqa_supported(const AttnShape & s) {
    return (s.head_dim == 64 || s.head_dim == 128) && s.n_head % s.n_head_kv == 0 && s.n_head / s.n_head_kv <= 8 && s.kv_stride % 8 == 0;
}

int attention_gqa_splits(int n_head_kv, int n_ctx) {
    // about one block per SM, and no more ranges than the context has tiles
    static const int per_sm = [] { const char * e = getenv("DOOMS_GQA_PER_SM"); return e ? std::max(1, atoi(e)) : 1; }();
    const int want = std::max(1, (sm_count() * per_sm + n_head_kv - 1) / n_head_kv);
    static const int fixed = [] { const char * e = getenv("DOOMS_GQA_SPLITS"); return e ? atoi(e) : 0; }();
    if (fixed > 0) return std::max(1, std::min(fixed, (n_ctx + kTileKeys - 1) / kTileKeys));
    return std::max(1, std::min(want, (n_ctx + kTileKeys - 1) / kTileKeys));
}

cudaError_t launch_attention_gqa(const float * qkv, void * kc, void * vc, float * part, const DevState * st, const double * inv_freq, int n_keys_fixed,
                                 int splits, const AttnShape & s, int * counters, float * out, void * xq, cudaStream_t stream, const void * rope_cs, int cache_keys, bool clusters) {
    if (!attention_gqa_supported(s) || (!inv_freq && n_keys_fixed < 1) || (counters && !out) || (xq && !counters) || cache_keys < 0 || (cache_keys && (!st || !inv_freq))) return cudaErrorInvalidValue;
    AttnDecodeParams p{qkv, static_cast<__half *>(kc), static_cast<__half *>(vc), part, st, inv_freq, n_keys_fixed, splits, s, counters, out,
                       static_cast<uint8_t *>(xq), static_cast<const float2 *>(rope_cs), nullptr, nullptr, 0, 0, 0, nullptr, 0};
    p.cache_ready = cache_keys;
    static const bool off = [] { const char * e = getenv("DOOMS_ATTN_CLUSTER"); return e && *e == '0'; }();
    p.cluster = clusters && !off && counters && splits > 1 ? 1 : 0;
    return s.head_dim == 64 ? launch_group<64>(p, s.n_head / s.n_head_kv, stream) : launch_group<128>(p, s.n_head / s.n_head_kv, stream);
}

cudaError_t launch_attention_gqa_rows(const float * qkv, void * kc, void * vc, float * part, const double * inv_freq, int splits, const AttnShape & s, int * counters,
                                      float * out, void * out16, const BatchRows & rows, int n_rows, cudaStream_t stream) {
    if (!attention_gqa_supported(s) || !inv_freq || !counters || !out || n_rows < 1 || splits < 1) return cudaErrorInvalidValue;
    const AttnDecodeParams p{qkv, static_cast<__half *>(kc), static_cast<__half *>(vc), part, nullptr, inv_freq, 0, splits, s, counters, out, nullptr, nullptr,
                             rows.slot, rows.pos, n_rows, rows.slot_elems, int64_t(splits) * s.n_head * (2 + s.head_dim), static_cast<__half *>(out16)};
    return s.head_dim == 64 ? launch_group<64>(p, s.n_head / s.n_head_kv, stream) : launch_group<128>(p, s.n_head / s.n_head_kv, stream);
}

}  // namespace cuda
}  // namespace dooms
