// Compression of a dense weight on the GPU: keep mask, group rounding, packing into the tile image.
//
// The recipe is the one of cobalt_b200/compress.py (reference: src/cobaltkernel/cobalt_math.py:15-32, 144-168) and every value
// is the one its torch form computes, bit for bit: fp32 products and IEEE divisions in the same order, order statistics exact.
//
//   score = |W| * norm;  row step: score /= k-th smallest of the row;  score /= max(score)
//                        column step: score /= (k-th smallest of the column)^beta;  score /= max(score)
//   keep  = score > k-th smallest of all scores
//
// Order statistics are radix selections on order-preserving 32-bit keys (NaN sorts last, as torch's kthvalue has it).  Dividing
// by a positive constant rounds monotonically, so the k-th smallest of score / max is (k-th smallest of score) / max: selections
// run on the undivided scores.  torch selects the global threshold of a 4096 x 4096 matrix with ONE block (96 ms on a B200);
// here every SM histograms its share of the scores.
#pragma once
#include <cuda_fp16.h>
#include "common.cuh"

namespace cb {

constexpr int SEL_BINS = 2048;                  // global selection: 11 + 11 + 10 key bits
constexpr int SEL_REPLICAS = 4;

// scratch words of one compression (device memory, zeroed by the first kernel that needs them)
struct CompressState {
    uint32_t top[2];                            // keys of the two maxima
    uint32_t prefix, rank;                      // global selection: key bits found so far, rank left within them
    float kth;                                  // k-th smallest of all scores
    float threshold;                            // what `keep` compares with
    uint32_t minmax[2];                         // keys of the smallest / largest score
    uint32_t below;                             // key of the largest score <= the bisection's bracket
    uint32_t done;                              // blocks that have added their histogram
    uint32_t hist[SEL_BINS];
};

__device__ __forceinline__ uint32_t order_key(float v) {
    const uint32_t u = __float_as_uint(v);
    return v != v ? 0xFFFFFFFFu : u ^ ((u & 0x80000000u) ? 0xFFFFFFFFu : 0x80000000u);
}
__device__ __forceinline__ float key_value(uint32_t k) {
    if (k == 0xFFFFFFFFu) return __uint_as_float(0x7FC00000u);
    return __uint_as_float((k & 0x80000000u) ? k ^ 0x80000000u : ~k);
}
// four consecutive weights as fp32
__device__ __forceinline__ void load4(const float* p, size_t i4, float (&f)[4]) {
    const float4 v = __ldg(reinterpret_cast<const float4*>(p) + i4);
    f[0] = v.x; f[1] = v.y; f[2] = v.z; f[3] = v.w;
}
__device__ __forceinline__ void load4(const __half* p, size_t i4, float (&f)[4]) {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(p) + i4);
    f[0] = half_bits_to_float(v.x); f[1] = half_bits_to_float(v.x >> 16); f[2] = half_bits_to_float(v.y); f[3] = half_bits_to_float(v.y >> 16);
}
__device__ __forceinline__ void load4(const __nv_bfloat16* p, size_t i4, float (&f)[4]) {
    const uint2 v = __ldg(reinterpret_cast<const uint2*>(p) + i4);
    f[0] = __uint_as_float(v.x << 16); f[1] = __uint_as_float(v.x & 0xFFFF0000u); f[2] = __uint_as_float(v.y << 16); f[3] = __uint_as_float(v.y & 0xFFFF0000u);
}

// score / top when top is finite and positive, else the score with its non-finite values zeroed
__device__ __forceinline__ bool top_divides(float top) { return top > 0.0f && top <= 3.402823466e38f; }
__device__ __forceinline__ float without_nonfinite(float v) { return fabsf(v) <= 3.402823466e38f ? v : 0.0f; }
__device__ __forceinline__ float over_top(float v, float top) { return top_divides(top) ? __fdiv_rn(v, top) : without_nonfinite(v); }
// what a selection looks at instead (same order as over_top; divided after the selection)
__device__ __forceinline__ float before_top(float v, bool divides) { return divides ? v : without_nonfinite(v); }

// Largest key of a block -> *out (which starts at 0).  All threads of the block call.
__device__ __forceinline__ void block_max_key(uint32_t k, uint32_t* out) {
    k = __reduce_max_sync(0xFFFFFFFFu, k);
    if ((threadIdx.x & 31) == 0) atomicMax(out, k);
}

// ---- k-th smallest score of every row, the scores over it, and their maximum.  One block per row; 8-bit digits, histogram
// replicated eight times (neighbouring lanes count into different words: the leading digit of a row's scores has few values).
// A row is read five times, from L1 after the first; issue-bound (order keys and shared-memory counting).  4096 x 4096 bf16: 88 us
// for selection and division; torch took 640 us for the selection alone.
constexpr int ROW_THREADS = 256, ROW_REPLICAS = 8;
template <class T>
__global__ void __launch_bounds__(ROW_THREADS) score_rows_kernel(const T* W, const float* norm, float* S, CompressState* st, int N, int k) {
    __shared__ uint32_t hist[256 * ROW_REPLICAS], warp_tot[ROW_THREADS / 32], sel[2];
    const T* w = W + (size_t)blockIdx.x * N;
    float* s = S + (size_t)blockIdx.x * N;
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    float rq = 1.0f;
    if (k > 0) {
        uint32_t prefix = 0, rank = (uint32_t)k - 1u;                  // 0-based rank within the keys that share the prefix
        for (int shift = 24; shift >= 0; shift -= 8) {
            for (int i = t; i < 256 * ROW_REPLICAS; i += ROW_THREADS) hist[i] = 0;
            __syncthreads();
            for (int i = t; i < N / 4; i += ROW_THREADS) {
                float f[4], nf[4];
                load4(w, i, f);
                load4(norm, i, nf);
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t key = order_key(__fmul_rn(fabsf(f[q]), nf[q]));
                    if (shift == 24 || (key >> (shift + 8)) == prefix) atomicAdd(&hist[((key >> shift) & 255u) * ROW_REPLICAS + (lane & (ROW_REPLICAS - 1))], 1u);
                }
            }
            __syncthreads();
            uint32_t cnt = 0;
#pragma unroll
            for (int r = 0; r < ROW_REPLICAS; ++r) cnt += hist[t * ROW_REPLICAS + ((r + t) & (ROW_REPLICAS - 1))];
            uint32_t inc = cnt;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) { const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, inc, d); if (lane >= d) inc += up; }
            if (lane == 31) warp_tot[warp] = inc;
            __syncthreads();
            uint32_t before = inc - cnt;
            for (int q = 0; q < warp; ++q) before += warp_tot[q];
            if (rank >= before && rank < before + cnt) { sel[0] = (uint32_t)t; sel[1] = rank - before; }
            __syncthreads();
            prefix = (prefix << 8) | sel[0];
            rank = sel[1];
        }
        rq = key_value(prefix);
        if (rq < 1e-30f) rq = 1e-30f;
    }
    uint32_t best = 0;
    for (int i = t; i < N / 4; i += ROW_THREADS) {
        float f[4], nf[4];
        load4(w, i, f);
        load4(norm, i, nf);
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            f[q] = __fmul_rn(fabsf(f[q]), nf[q]);
            if (k > 0) f[q] = __fdiv_rn(f[q], rq);
            const uint32_t key = order_key(f[q]);
            best = key > best ? key : best;
        }
        reinterpret_cast<float4*>(s)[i] = make_float4(f[0], f[1], f[2], f[3]);
    }
    if (k > 0) block_max_key(best, &st->top[0]);
}

// ---- k-th smallest of every column of S (over the first maximum).  A block takes 32 columns, lane = column, so that reads are
// whole lines and every lane counts into a bank of its own.  4096 x 4096: 73 us, four passes over the scores out of L2.
constexpr int COL_THREADS = 1024;
__global__ void __launch_bounds__(COL_THREADS) column_kth_kernel(const float* S, const CompressState* st, float* colq, int K, int N, int k, int rows_normalised) {
    __shared__ uint32_t hist[256 * 32];
    __shared__ uint32_t part[8][32];
    __shared__ uint32_t s_prefix[32], s_rank[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    const int col = blockIdx.x * 32 + lane;
    const float top = rows_normalised ? key_value(st->top[0]) : 1.0f;
    const bool div = rows_normalised ? top_divides(top) : true;
    if (warp == 0) { s_prefix[lane] = 0; s_rank[lane] = (uint32_t)k - 1u; }
    for (int shift = 24; shift >= 0; shift -= 8) {
        for (int i = t; i < 256 * 32; i += COL_THREADS) hist[i] = 0;
        __syncthreads();
        const uint32_t prefix = s_prefix[lane];
        if (col < N) {
#pragma unroll 4
            for (int r = warp; r < K; r += COL_THREADS / 32) {
                const uint32_t key = order_key(before_top(__ldg(S + (size_t)r * N + col), div));
                if (shift == 24 || (key >> (shift + 8)) == prefix) atomicAdd(&hist[((key >> shift) & 255u) * 32 + lane], 1u);
            }
        }
        __syncthreads();
        if (warp < 8) {                                                // warp q: counts of digits 32q .. 32q+31 of its lane's column
            uint32_t c = 0;
            for (int b = 0; b < 32; ++b) c += hist[(warp * 32 + b) * 32 + lane];
            part[warp][lane] = c;
        }
        __syncthreads();
        if (warp == 0) {
            uint32_t rank = s_rank[lane], q = 0;
            while (q < 7 && rank >= part[q][lane]) { rank -= part[q][lane]; ++q; }
            uint32_t b = 0;
            while (b < 31 && rank >= hist[(q * 32 + b) * 32 + lane]) { rank -= hist[(q * 32 + b) * 32 + lane]; ++b; }
            s_prefix[lane] = (prefix << 8) | (q * 32 + b);
            s_rank[lane] = rank;
        }
        __syncthreads();
    }
    if (warp == 0 && col < N) {
        float v = key_value(s_prefix[lane]);
        if (rows_normalised && div) v = __fdiv_rn(v, top);
        colq[col] = v;
    }
}

// ---- column step: S = over_top(S) / colq[column] and its maximum.  No column step: S = over_top(S) only.
__global__ void __launch_bounds__(256) score_columns_kernel(float* S, CompressState* st, const float* colq, size_t n, int N, int rows_normalised) {
    const float top = rows_normalised ? key_value(st->top[0]) : 1.0f;
    uint32_t best = 0;
    const uint32_t n4 = (uint32_t)(n / 4), row4 = (uint32_t)N / 4u;    // whole groups: N is a multiple of 4
    for (uint32_t i = blockIdx.x * 256 + threadIdx.x; i < n4; i += gridDim.x * 256) {
        const float4 v4 = reinterpret_cast<const float4*>(S)[i];
        float f[4] = {v4.x, v4.y, v4.z, v4.w};
        const uint32_t c = (i % row4) * 4u;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (rows_normalised) f[q] = over_top(f[q], top);
            if (colq) {
                f[q] = __fdiv_rn(f[q], colq[c + q]);
                const uint32_t key = order_key(f[q]);
                best = key > best ? key : best;
            }
        }
        reinterpret_cast<float4*>(S)[i] = make_float4(f[0], f[1], f[2], f[3]);
    }
    if (colq) block_max_key(best, &st->top[1]);
}

// ---- one digit of the global selection: histogram of the scores that share the prefix found so far; the block that finishes
// last picks the digit.  Bound by reading the scores (67 MB at 4096 x 4096: 21 us a digit, 3.3 TB/s).
__global__ void __launch_bounds__(512) global_digit_kernel(const float* S, CompressState* st, size_t n, int shift, int bits, int cols_normalised) {
    __shared__ uint32_t hist[SEL_BINS * SEL_REPLICAS];
    __shared__ uint32_t last;
    const int t = threadIdx.x;
    const uint32_t nb = 1u << bits;
    const bool div = cols_normalised ? top_divides(key_value(st->top[1])) : true;
    const uint32_t prefix = st->prefix;
    const int seen = shift + bits;                                     // key bits above this digit are fixed
    for (uint32_t i = t; i < nb * SEL_REPLICAS; i += 512) hist[i] = 0;
    __syncthreads();
    for (size_t i = (size_t)blockIdx.x * 512 + t; i < n / 4; i += (size_t)gridDim.x * 512) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(S) + i);
        const float f[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint32_t key = order_key(before_top(f[q], div));
            if (seen == 32 || (key >> seen) == prefix) atomicAdd(&hist[((key >> shift) & (nb - 1u)) * SEL_REPLICAS + (t & (SEL_REPLICAS - 1))], 1u);
        }
    }
    __syncthreads();
    for (uint32_t b = t; b < nb; b += 512) {
        uint32_t c = 0;
#pragma unroll
        for (int r = 0; r < SEL_REPLICAS; ++r) c += hist[b * SEL_REPLICAS + r];
        if (c) atomicAdd(&st->hist[b], c);
    }
    __threadfence();
    __syncthreads();
    if (t == 0) last = atomicAdd(&st->done, 1u) == gridDim.x - 1u ? 1u : 0u;
    __syncthreads();
    if (!last) return;
    __threadfence();
    const uint32_t per = nb / 512u;                                    // bins of a thread: 4 or 2
    uint32_t cnt[4] = {0, 0, 0, 0}, mine = 0;
    for (uint32_t q = 0; q < per; ++q) {
        cnt[q] = *reinterpret_cast<volatile uint32_t*>(&st->hist[t * per + q]);
        mine += cnt[q];
        st->hist[t * per + q] = 0;
    }
    uint32_t inc = mine;
    const int lane = t & 31, warp = t >> 5;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) { const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, inc, d); if (lane >= d) inc += up; }
    if (lane == 31) hist[warp] = inc;
    __syncthreads();
    uint32_t before = inc - mine;
    for (int q = 0; q < warp; ++q) before += hist[q];
    const uint32_t rank = st->rank;
    __syncthreads();
    if (rank >= before && rank < before + mine) {
        uint32_t left = rank - before, q = 0;
        while (left >= cnt[q]) { left -= cnt[q]; ++q; }
        st->prefix = (prefix << bits) | (t * per + q);
        st->rank = left;
        if (shift == 0) {
            const float v = key_value((prefix << bits) | (t * per + q));
            st->kth = cols_normalised ? over_top(v, key_value(st->top[1])) : v;
            st->threshold = st->kth;
        }
    }
    if (t == 0) st->done = 0;
}

// ---- matrices above 32 M elements: the reference brackets the threshold by at most 64 bisection steps on the value range and
// takes the largest score not above the bracket.  How many scores lie at or below a midpoint only matters against k, that is,
// whether the k-th smallest does: the bracket follows from it without counting.
__global__ void __launch_bounds__(512) score_range_kernel(const float* S, CompressState* st, size_t n, int cols_normalised) {
    const float top = cols_normalised ? key_value(st->top[1]) : 1.0f;
    uint32_t lo = 0xFFFFFFFFu, hi = 0;
    for (size_t i = (size_t)blockIdx.x * 512 + threadIdx.x; i < n; i += (size_t)gridDim.x * 512) {
        const uint32_t key = order_key(cols_normalised ? over_top(S[i], top) : S[i]);
        lo = key < lo ? key : lo;
        hi = key > hi ? key : hi;
    }
    lo = __reduce_min_sync(0xFFFFFFFFu, lo);
    hi = __reduce_max_sync(0xFFFFFFFFu, hi);
    if ((threadIdx.x & 31) == 0) { atomicMin(&st->minmax[0], lo); atomicMax(&st->minmax[1], hi); }
}
__global__ void __launch_bounds__(512) below_bracket_kernel(const float* S, CompressState* st, size_t n, int cols_normalised) {
    float lo = key_value(st->minmax[0]), hi = key_value(st->minmax[1]);
    const float kth = st->kth;
    for (int it = 0; it < 64; ++it) {
        const float mid = __fmul_rn(__fadd_rn(lo, hi), 0.5f);
        if (!(fabsf(mid) <= 3.402823466e38f) || mid <= lo || mid >= hi) break;
        if (kth <= mid) hi = mid; else lo = mid;
    }
    const float top = cols_normalised ? key_value(st->top[1]) : 1.0f;
    uint32_t best = 0;
    for (size_t i = (size_t)blockIdx.x * 512 + threadIdx.x; i < n; i += (size_t)gridDim.x * 512) {
        const float v = cols_normalised ? over_top(S[i], top) : S[i];
        if (v <= hi) { const uint32_t key = order_key(v); best = key > best ? key : best; }
    }
    block_max_key(best, &st->below);
    if (blockIdx.x == 0 && threadIdx.x == 0) st->threshold = hi;       // only if nothing lies at or below it; see keep_compare_kernel
}

// ---- keep = score > threshold
__global__ void __launch_bounds__(256) keep_compare_kernel(const float* S, const CompressState* st, uint8_t* keep, size_t n, int cols_normalised, int bracketed) {
    const float top = cols_normalised ? key_value(st->top[1]) : 1.0f;
    const float thr = bracketed && st->below != 0u ? key_value(st->below) : st->threshold;
    for (size_t i = (size_t)blockIdx.x * 256 + threadIdx.x; i < n / 4; i += (size_t)gridDim.x * 256) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(S) + i);
        const float f[4] = {v.x, v.y, v.z, v.w};
        uint32_t o = 0;
#pragma unroll
        for (int q = 0; q < 4; ++q) o |= ((cols_normalised ? over_top(f[q], top) : f[q]) > thr ? 1u : 0u) << (8 * q);
        reinterpret_cast<uint32_t*>(keep)[i] = o;
    }
}

__global__ void compress_state_init_kernel(CompressState* st, uint32_t k) {
    for (int i = threadIdx.x; i < SEL_BINS; i += blockDim.x) st->hist[i] = 0;
    if (threadIdx.x == 0) {
        st->top[0] = st->top[1] = 0; st->prefix = 0; st->rank = k - 1u; st->kth = st->threshold = 0.0f;
        st->minmax[0] = 0xFFFFFFFFu; st->minmax[1] = 0; st->below = 0; st->done = 0;
    }
}

// ---- group rounding over survivors: one warp per 128-wide group, four columns per lane (read once).  4096 x 4096 bf16: 29 us.
template <class T>
__global__ void __launch_bounds__(256) quantize_groups_kernel(const T* W, const uint8_t* keep, uint8_t* q, __half* scale, __half* zero, size_t groups, int bits) {
    const size_t g = (size_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    if (g >= groups) return;
    const int lane = threadIdx.x & 31;
    const size_t at = g * GROUP + 4 * lane;
    const uint32_t kp = *reinterpret_cast<const uint32_t*>(keep + at);
    constexpr float LIMIT = 3.402823466e38f;                            // what a pruned position counts as
    float w[4], lo = INFINITY, hi = -INFINITY;
    bool nan = false;                                                  // fminf and fmaxf drop a NaN; the hull carries it
    load4(W, at / 4, w);
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const bool kept = ((kp >> (8 * i)) & 0xFFu) != 0u;
        lo = fminf(lo, kept ? w[i] : LIMIT); hi = fmaxf(hi, kept ? w[i] : -LIMIT);
        nan = nan || (kept && w[i] != w[i]);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        lo = fminf(lo, __shfl_xor_sync(0xFFFFFFFFu, lo, o));
        hi = fmaxf(hi, __shfl_xor_sync(0xFFFFFFFFu, hi, o));
    }
    if (__any_sync(0xFFFFFFFFu, nan)) lo = hi = __uint_as_float(0x7FC00000u);
    if (!__any_sync(0xFFFFFFFFu, kp != 0u)) { lo = 0.0f; hi = 0.0f; }
    const float top = (float)((1 << bits) - 1);
    float span = __fsub_rn(hi, lo);
    if (span < 1e-4f) span = 1e-4f;
    const float s = __fdiv_rn(span, top), z = -rintf(__fdiv_rn(lo, s));
    uint32_t o = 0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const float c = fminf(fmaxf(rintf(__fadd_rn(__fdiv_rn(w[i], s), z)), 0.0f), top);
        if ((kp >> (8 * i)) & 0xFFu) o |= (uint32_t)c << (8 * i);
    }
    *reinterpret_cast<uint32_t*>(q + at) = o;
    if (lane == 0) { scale[g] = __float2half_rn(s); zero[g] = __float2half_rn(z); }
}

// ----------------------------------------------------------------------------- packing
struct PackInfo { uint64_t nnz; uint32_t total16, max_tile_bytes, max_tile_nnz, bad; };

__device__ __forceinline__ uint32_t nonzero_nibble(uint32_t k) {       // bit i: byte i is not zero
    return ((k & 0xFFu) ? 1u : 0u) | ((k & 0xFF00u) ? 2u : 0u) | ((k & 0xFF0000u) ? 4u : 0u) | ((k & 0xFF000000u) ? 8u : 0u);
}

// survivors of every tile, and whether a surviving code lies outside the grid.  One block of 8 warps per tile.
__global__ void __launch_bounds__(256) pack_count_kernel(const uint8_t* keep, const uint8_t* q, int K, int N, int CT, int bits, uint32_t* tile_nnz, PackInfo* info) {
    __shared__ uint32_t tot;
    const int ct = blockIdx.x, rb = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = min(TILE_GROUPS, N / GROUP - ct * TILE_GROUPS);
    if (threadIdx.x == 0) tot = 0;
    __syncthreads();
    uint32_t cnt = 0, bad = 0;
    for (int seg = warp; seg < TILE_ROWS * w; seg += 8) {
        const int row = rb * TILE_ROWS + seg / w;
        if (row >= K) continue;
        const size_t at = (size_t)row * N + (ct * TILE_GROUPS + seg % w) * GROUP + 4 * lane;
        const uint32_t nib = nonzero_nibble(__ldg(reinterpret_cast<const uint32_t*>(keep + at)));
        const uint32_t over = nonzero_nibble(__ldg(reinterpret_cast<const uint32_t*>(q + at)) & (0xFFu << bits & 0xFFu) * 0x01010101u);
        cnt += __popc(nib);
        bad |= nib & over;
    }
    cnt = __reduce_add_sync(0xFFFFFFFFu, cnt);
    bad = __reduce_or_sync(0xFFFFFFFFu, bad);
    if (lane == 0) { atomicAdd(&tot, cnt); if (bad) info->bad = 1u; }
    __syncthreads();
    if (threadIdx.x == 0) tile_nnz[rb * CT + ct] = tot;
}

// tile offsets (exclusive scan of the tiles' 16-byte sizes) and the totals the host needs.  One block: a few thousand tiles.
__global__ void __launch_bounds__(1024) pack_scan_kernel(const uint32_t* tile_nnz, uint32_t* tile_off, PackInfo* info, int n_tiles, int N, int CT, int bits) {
    __shared__ uint32_t wsum[32], wmaxb[32], wmaxn[32], carry_s;
    __shared__ unsigned long long wnnz[32];
    const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
    uint32_t carry = 0, maxb = 0, maxn = 0;
    unsigned long long nnz = 0;
    for (int base = 0; base < n_tiles; base += 1024) {
        const int i = base + t;
        uint32_t sz = 0;
        if (i < n_tiles) {
            const int w = min(TILE_GROUPS, N / GROUP - (i % CT) * TILE_GROUPS);
            const uint32_t c = tile_nnz[i], bytes = (TILE_ROWS * w * 20 + (c * bits + 7) / 8 + 15) / 16 * 16;
            sz = bytes / 16;
            maxb = max(maxb, bytes); maxn = max(maxn, c); nnz += c;
        }
        uint32_t inc = sz;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, inc, d); if (lane >= d) inc += up; }
        if (lane == 31) wsum[warp] = inc;
        __syncthreads();
        uint32_t off = carry + inc - sz;
        for (int q = 0; q < warp; ++q) off += wsum[q];
        if (i < n_tiles) tile_off[i] = off;
        if (t == 1023) carry_s = off + sz;
        __syncthreads();
        carry = carry_s;
    }
    maxb = __reduce_max_sync(0xFFFFFFFFu, maxb);
    maxn = __reduce_max_sync(0xFFFFFFFFu, maxn);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nnz += __shfl_xor_sync(0xFFFFFFFFu, nnz, o);
    if (lane == 0) { wmaxb[warp] = maxb; wmaxn[warp] = maxn; wnnz[warp] = nnz; }
    __syncthreads();
    if (t == 0) {
        for (int q = 1; q < 32; ++q) { maxb = max(maxb, wmaxb[q]); maxn = max(maxn, wmaxn[q]); nnz += wnnz[q]; }
        tile_off[n_tiles] = carry;
        info->total16 = carry; info->max_tile_bytes = maxb; info->max_tile_nnz = maxn; info->nnz = nnz;
    }
}

// One block of 8 warps per tile: a warp packs eight of the 64 segments (lane = four columns), the code stream is put together
// in shared memory and the tile leaves as whole 16-byte chunks.  4096 x 4096: 34 us;
// the torch form moved int64 words and took about 2 ms.
__global__ void __launch_bounds__(256) pack_tiles_kernel(const uint8_t* keep, const uint8_t* q, const uint16_t* scale, const uint16_t* zero, int K, int N, int CT,
                                                         int bits, const uint32_t* tile_off, uint8_t* tiles) {
    constexpr int SEGS = TILE_ROWS * TILE_GROUPS;
    constexpr int MAX_WORDS = SEGS * 5 + SEGS * GROUP * 4 / 32 + 4;
    __shared__ __align__(16) uint32_t buf[MAX_WORDS];
    __shared__ uint32_t seg_cnt[SEGS], seg_first[SEGS];
    const int ct = blockIdx.x, rb = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int G = N / GROUP, w = min(TILE_GROUPS, G - ct * TILE_GROUPS), nseg = TILE_ROWS * w;
    for (int i = threadIdx.x; i < MAX_WORDS; i += 256) buf[i] = 0;
    __syncthreads();
    uint32_t nib[SEGS / 8];
#pragma unroll
    for (int i = 0; i < SEGS / 8; ++i) {
        const int seg = warp + 8 * i;
        nib[i] = 0;
        if (seg >= nseg) continue;
        const int row = rb * TILE_ROWS + seg / w, grp = ct * TILE_GROUPS + seg % w;
        if (row < K) {
            nib[i] = nonzero_nibble(__ldg(reinterpret_cast<const uint32_t*>(keep + (size_t)row * N + grp * GROUP + 4 * lane)));
            if (lane == 0) buf[nseg * 4 + seg] = (uint32_t)scale[(size_t)row * G + grp] | ((uint32_t)zero[(size_t)row * G + grp] << 16);
        }
        uint32_t word = nib[i] << (4 * (lane & 7));
        word |= __shfl_xor_sync(0xFFFFFFFFu, word, 1); word |= __shfl_xor_sync(0xFFFFFFFFu, word, 2); word |= __shfl_xor_sync(0xFFFFFFFFu, word, 4);
        if ((lane & 7) == 0) buf[seg * 4 + (lane >> 3)] = word;
        const uint32_t c = __reduce_add_sync(0xFFFFFFFFu, __popc(nib[i]));
        if (lane == 0) seg_cnt[seg] = c;
    }
    __syncthreads();
    if (warp == 0) {                                                   // two segments per lane
        const uint32_t a = 2 * lane < nseg ? seg_cnt[2 * lane] : 0u, b = 2 * lane + 1 < nseg ? seg_cnt[2 * lane + 1] : 0u;
        uint32_t inc = a + b;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, inc, d); if (lane >= d) inc += up; }
        seg_first[2 * lane] = inc - a - b;
        seg_first[2 * lane + 1] = inc - b;
    }
    __syncthreads();
    uint32_t* codes = buf + nseg * 5;
#pragma unroll
    for (int i = 0; i < SEGS / 8; ++i) {
        const int seg = warp + 8 * i, row = rb * TILE_ROWS + seg / w;
        if (seg >= nseg) continue;
        const uint32_t c = __popc(nib[i]);
        uint32_t inc = c;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, inc, d); if (lane >= d) inc += up; }
        if (row >= K || c == 0) continue;
        const uint32_t qv = __ldg(reinterpret_cast<const uint32_t*>(q + (size_t)row * N + (ct * TILE_GROUPS + seg % w) * GROUP + 4 * lane));
        uint32_t v = 0, n = 0;
#pragma unroll
        for (int k = 0; k < 4; ++k)
            if ((nib[i] >> k) & 1u) { v |= ((qv >> (8 * k)) & 0xFFu) << (n * bits); ++n; }
        const uint32_t bit = (seg_first[seg] + inc - c) * bits, sh = bit & 31u;
        atomicOr(&codes[bit >> 5], v << sh);
        if (sh + n * bits > 32u) atomicOr(&codes[(bit >> 5) + 1], v >> (32u - sh));
    }
    __syncthreads();
    const uint32_t o0 = tile_off[rb * CT + ct], n16 = tile_off[rb * CT + ct + 1] - o0;
    for (uint32_t i = threadIdx.x; i < n16; i += 256) reinterpret_cast<uint4*>(tiles)[o0 + i] = reinterpret_cast<const uint4*>(buf)[i];
}

}  // namespace cb
