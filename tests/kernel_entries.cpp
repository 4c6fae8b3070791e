// C entries of internal launchers, for the tests: what the library reaches only through a decoder (a product whose reduction is dealt over blocks, the norm that
// adds its shares, prefill attention on its own). Linked from the library's own object files.
#include "kernels/kernels.h"

using namespace dooms;
using namespace dooms::cuda;

#pragma GCC visibility push(default)
extern "C" {

int kernel_gemm_splits(int dt, const void * W, int M, long long N, long long K, long long w16_bytes, int most) { return gemm_tc_k_splits(dt, W, M, N, K, size_t(w16_bytes), most); }
int kernel_rows16_splits(int M, long long N, long long K, int most) { return gemm_tc_rows16_k_splits(M, N, K, most); }

// shares[z][m][n], k_splits of them (1: the whole product)
int kernel_gemm(int dt, const void * W, const void * X16, float * shares, int M, long long N, long long K, int * error, void * w16, long long w16_bytes, int k_splits) {
    TensorMap map;
    const cudaError_t e = make_activation_map(&map, X16, M, K);
    if (e != cudaSuccess) return int(e);
    return int(launch_gemm_tc(dt, W, nullptr, &map, shares, nullptr, nullptr, M, N, K, N, 0, 0u, error, nullptr, w16, size_t(w16_bytes), k_splits, int64_t(M) * N));
}
int kernel_gemm_rows16(const void * W16, const void * X16, float * shares, int M, long long N, long long K, int * error, int k_splits) {
    TensorMap map;
    const cudaError_t e = make_activation_map(&map, X16, M, K);
    if (e != cudaSuccess) return int(e);
    return int(launch_gemm_tc_rows16(W16, nullptr, &map, shares, nullptr, nullptr, M, N, K, N, 0, 0u, error, nullptr, k_splits, int64_t(M) * N));
}
// The refusals alone: no product is launched for a count of shares that the reduction does not divide into.
int kernel_gemm_refuses(int dt, int rows16, long long N, long long K, int k_splits) {
    alignas(64) static char dummy[64];
    TensorMap map{};
    float y = 0.f;
    int error = 0;
    const cudaError_t e = rows16 ? launch_gemm_tc_rows16(dummy, nullptr, &map, &y, nullptr, nullptr, 1, N, K, N, 0, 0u, &error, nullptr, k_splits, N)
                                 : launch_gemm_tc(dt, dummy, nullptr, &map, &y, nullptr, nullptr, 1, N, K, N, 0, 0u, &error, nullptr, nullptr, 0, k_splits, N);
    return e == cudaErrorInvalidValue;
}
int kernel_rms_norm(float * x, const float * gamma, float * out, void * out16, int rows, int E, float eps, const float * shares, int n_shares) {
    return int(launch_rms_norm(x, gamma, out, out16, nullptr, rows, E, eps, nullptr, shares, n_shares, int64_t(rows) * E));
}
int kernel_add_shares(float * x, const float * shares, int n_shares, long long n) { return int(launch_add_shares(x, shares, n_shares, n, n, nullptr)); }

// qkv: M rows of (n_head + 2 n_head_kv) * head_dim, rotated; pos: device int, the first row's position
int kernel_flash(const float * qkv, const void * kc, const void * vc, float * out, const void * pos, int M, int n_head, int n_head_kv, int head_dim, int keys) {
    const AttnShape s{n_head, n_head_kv, head_dim, (n_head + 2 * n_head_kv) * head_dim, n_head_kv * head_dim, n_head * head_dim, 1, 1e6f};
    return int(launch_attention_flash(qkv, kc, vc, out, nullptr, static_cast<const DevState *>(pos), M, s, keys, nullptr));
}
}
#pragma GCC visibility pop
