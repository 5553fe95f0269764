// C ABI of the compression kernels: argument validation and launches.  See include/cobalt_b200.h.
#include "compress_kernels.cuh"

using namespace cb;

namespace {

int check_shape(int K, int N) {
    if (K <= 0 || N <= 0 || N % GROUP != 0 || (unsigned long long)K * (unsigned)N >= (1ull << 34)) return COBALT_EINVAL;
    return COBALT_OK;
}
// scoring: counts, ranks and the element index of score_columns_kernel are 32-bit words
int check_scores(int K, int N) {
    const int rc = check_shape(K, N);
    if (rc) return rc;
    return (unsigned long long)K * (unsigned)N < (1ull << 32) ? COBALT_OK : COBALT_ETOOBIG;
}
int check_tiling(int K, int N) {
    const int rc = check_shape(K, N);
    if (rc) return rc;
    return (K + TILE_ROWS - 1) / TILE_ROWS <= 65535 ? COBALT_OK : COBALT_ETOOBIG;             // row blocks are a grid dimension
}
int sm_count(int* n) {
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return COBALT_ELAUNCH;
    return cudaDeviceGetAttribute(n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess ? COBALT_OK : COBALT_ELAUNCH;
}
int launched() { return cudaGetLastError() == cudaSuccess ? COBALT_OK : COBALT_ELAUNCH; }
bool aligned16(const void* p) { return p && ((uintptr_t)p & 15) == 0; }

}  // namespace

extern "C" {

size_t cobalt_compress_state_bytes(void) { return sizeof(CompressState); }

int cobalt_score_rows(const void* W, int w_type, const float* norm, int K, int N, int n_row, int n_col, uint32_t k_keep, float* scores,
                      float* col_kth, void* state, void* stream) {
    int rc = check_scores(K, N);
    if (rc) return rc;
    if (!aligned16(W) || !aligned16(norm) || !aligned16(scores) || !aligned16(state) || w_type < 0 || w_type > 2) return COBALT_EINVAL;
    if (n_row < 0 || n_row > N || n_col < 0 || n_col > K || (n_col > 0 && !col_kth) || k_keep < 1 || k_keep > (unsigned long long)K * (unsigned)N) return COBALT_EINVAL;
    cudaStream_t st = (cudaStream_t)stream;
    CompressState* S = (CompressState*)state;
    compress_state_init_kernel<<<1, 512, 0, st>>>(S, k_keep);
    switch (w_type) {
        case 0: score_rows_kernel<<<K, ROW_THREADS, 0, st>>>((const float*)W, norm, scores, S, N, n_row); break;
        case 1: score_rows_kernel<<<K, ROW_THREADS, 0, st>>>((const __half*)W, norm, scores, S, N, n_row); break;
        default: score_rows_kernel<<<K, ROW_THREADS, 0, st>>>((const __nv_bfloat16*)W, norm, scores, S, N, n_row); break;
    }
    if (n_col > 0) column_kth_kernel<<<(N + 31) / 32, COL_THREADS, 0, st>>>(scores, S, col_kth, K, N, n_col, n_row > 0 ? 1 : 0);
    return launched();
}

int cobalt_keep_from_scores(float* scores, const float* col_div, int K, int N, int rows_normalised, int bracketed, void* state,
                            uint8_t* keep, void* stream) {
    int rc = check_scores(K, N);
    if (rc) return rc;
    if (!aligned16(scores) || !aligned16(state) || !aligned16(keep)) return COBALT_EINVAL;
    int sms = 0;
    rc = sm_count(&sms);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    CompressState* S = (CompressState*)state;
    const size_t n = (size_t)K * N;
    const int cols = col_div ? 1 : 0;
    auto blocks = [&](int per_sm, size_t work) { return (unsigned)(work < (size_t)per_sm * sms ? (work ? work : 1) : (size_t)per_sm * sms); };
    if (rows_normalised || cols) score_columns_kernel<<<blocks(8, (n / 4 + 255) / 256), 256, 0, st>>>(scores, S, col_div, n, N, rows_normalised);
    const unsigned gd = blocks(2, (n / 4 + 511) / 512);
    global_digit_kernel<<<gd, 512, 0, st>>>(scores, S, n, 21, 11, cols);
    global_digit_kernel<<<gd, 512, 0, st>>>(scores, S, n, 10, 11, cols);
    global_digit_kernel<<<gd, 512, 0, st>>>(scores, S, n, 0, 10, cols);
    if (bracketed) {
        score_range_kernel<<<gd, 512, 0, st>>>(scores, S, n, cols);
        below_bracket_kernel<<<gd, 512, 0, st>>>(scores, S, n, cols);
    }
    keep_compare_kernel<<<blocks(8, (n / 4 + 255) / 256), 256, 0, st>>>(scores, S, keep, n, cols, bracketed);
    return launched();
}

int cobalt_quantize_groups(const void* W, int w_type, const uint8_t* keep, int K, int N, int bits, uint8_t* q, void* scale, void* zero,
                           void* stream) {
    int rc = check_shape(K, N);
    if (rc) return rc;
    if (!aligned16(W) || !aligned16(keep) || !aligned16(q) || !scale || !zero || w_type < 0 || w_type > 2 || bits < 1 || bits > 8) return COBALT_EINVAL;
    const size_t groups = (size_t)K * (N / GROUP);
    const unsigned grid = (unsigned)((groups + 7) / 8);
    cudaStream_t st = (cudaStream_t)stream;
    switch (w_type) {
        case 0: quantize_groups_kernel<<<grid, 256, 0, st>>>((const float*)W, keep, q, (__half*)scale, (__half*)zero, groups, bits); break;
        case 1: quantize_groups_kernel<<<grid, 256, 0, st>>>((const __half*)W, keep, q, (__half*)scale, (__half*)zero, groups, bits); break;
        default: quantize_groups_kernel<<<grid, 256, 0, st>>>((const __nv_bfloat16*)W, keep, q, (__half*)scale, (__half*)zero, groups, bits); break;
    }
    return launched();
}

int cobalt_pack_plan(const uint8_t* keep, const uint8_t* q, int K, int N, int bits, uint32_t* tile_nnz, uint32_t* tile_off, void* info,
                     void* stream) {
    int rc = check_tiling(K, N);
    if (rc) return rc;
    if (!aligned16(keep) || !aligned16(q) || !tile_nnz || !tile_off || !aligned16(info) || bits < 2 || bits > 4) return COBALT_EINVAL;
    const int RB = (K + TILE_ROWS - 1) / TILE_ROWS, CT = (N / GROUP + TILE_GROUPS - 1) / TILE_GROUPS;
    cudaStream_t st = (cudaStream_t)stream;
    if (cudaMemsetAsync(info, 0, sizeof(PackInfo), st) != cudaSuccess) return COBALT_ELAUNCH;
    pack_count_kernel<<<dim3(CT, RB), 256, 0, st>>>(keep, q, K, N, CT, bits, tile_nnz, (PackInfo*)info);
    pack_scan_kernel<<<1, 1024, 0, st>>>(tile_nnz, tile_off, (PackInfo*)info, RB * CT, N, CT, bits);
    return launched();
}

int cobalt_pack_tiles(const uint8_t* keep, const uint8_t* q, const void* scale, const void* zero, int K, int N, int bits,
                      const uint32_t* tile_off, void* tiles, void* stream) {
    int rc = check_tiling(K, N);
    if (rc) return rc;
    if (!aligned16(keep) || !aligned16(q) || !scale || !zero || !tile_off || !aligned16(tiles) || bits < 2 || bits > 4) return COBALT_EINVAL;
    const int RB = (K + TILE_ROWS - 1) / TILE_ROWS, CT = (N / GROUP + TILE_GROUPS - 1) / TILE_GROUPS;
    pack_tiles_kernel<<<dim3(CT, RB), 256, 0, (cudaStream_t)stream>>>(keep, q, (const uint16_t*)scale, (const uint16_t*)zero, K, N, CT, bits,
                                                                      tile_off, (uint8_t*)tiles);
    return launched();
}

}  // extern "C"
