// Grouped-query attention of a prompt over the KV caches [n_kv][max_ctx][D], tcgen05.mma for both contractions.
//
// Same rounding points as the decode attention (glue_kernels.cuh) and the reference's executable spec
// (src/cobaltkernel/ref_llama.py:117-137): scores = bf16(q . k), times the scale rounded to bf16, softmax in fp32 over the
// allowed slots, probabilities rounded to bf16, context = bf16(sum p * v).  The probabilities need the row's maximum and
// sum before they are rounded, so a CTA walks its keys twice: pass A forms the scores and keeps the running maximum and
// sum of exp per row, pass B forms them again, turns them into probabilities and multiplies by V.  No score reaches memory.
//
// One CTA = 128 query rows of one KV head: (token, head) pairs, 128 / rep tokens of the rep query heads that share it.
//   warps 0-7  softmax: warp w owns TMEM lanes 32*(w%4).. (a thread = a row) and key columns 64*(w/4).. of every 128-key
//              tile; in pass B it writes its half of the probability tile (K-major, 128-byte swizzle) to shared memory
//   warp 8     TMA: the query tile once, then key and value tiles in the order the MMAs take them (no multicast)
//   warp 9     MMA: scores into one of two TMEM buffers, context into a third; the scores of tile j+1 are issued before
//              the context of tile j, so that the tensor pipe works under the softmax
// Key tiles outside the causal / sliding range of the CTA's rows are skipped; only tiles that cross its border are masked.
//
// The softmax is fp32 as in the decode attention: expf, and probabilities that are quotients.  At scores far apart it rounds 17 of
// a million probabilities to another bf16 value than an exact softmax, torch's fp32 softmax 15; a power of two of the
// product with log2(e) and a product with the reciprocal were 16 % faster and rounded 144.  The division itself takes
// 1.8 times as long as quotient() below (2048 tokens: 249 us), for the same bits.
//
// Bound: the element-wise work of the softmax warps.  A 128 x 128 tile holds 16384 scores that take about 30 operations over
// both passes (two roundings, scale, maximum, two exponentials, sum, quotient, packing), against 1570 cycles of tensor work.
// Hence eight softmax warps on one CTA per SM (two per scheduler, 32 independent values each) rather than four, and no third pass.
// Measured (1965 MHz, cold L2): 2048 tokens, 32 / 8 heads of 128: 139 us per layer, where batched matmuls with element-wise
// passes over the scores took 1490 us; 1024 tokens 50 us; 8 x 200 tokens, 32 / 16 heads 56 us.
#pragma once
#include "gemm_kernel.cuh"

namespace cb {

constexpr int PA_ROWS = 128;               // UMMA M: (token, head) rows per CTA
constexpr int PA_KEYS = 128;               // keys per tile
constexpr int PA_RING = 4;                 // key / value tiles in flight
constexpr int PA_SOFTMAX = 256;            // softmax threads
constexpr int PA_THREADS = PA_SOFTMAX + 64;
constexpr uint32_t PA_SUB = 128 * 128;     // bytes of 128 rows x 64 bf16: one swizzled sub-tile
constexpr uint32_t pa_tile_bytes(int D) { return PA_SUB * (uint32_t)(D / 64); }
constexpr uint32_t PA_P_BYTES = 2 * PA_SUB;
constexpr uint32_t PA_TAIL_BYTES = 160 + 2 * PA_ROWS * 6;     // barriers, then sum (fp32) and maximum (a bf16 value) of every row and half
constexpr uint32_t pa_smem_bytes(int D) {
    return pa_tile_bytes(D) * (1 + PA_RING) + 2 * PA_P_BYTES + PA_TAIL_BYTES + 1024;
}
static_assert(pa_smem_bytes(128) <= 227 * 1024, "the 128-wide head fills the shared memory of one SM");

struct PromptAttnParams {
    const long long* positions;            // [T], the same for every sequence (blockIdx.y)
    uint16_t* out;                         // [sequence][T][n_kv * rep * D]
    int T, n_kv, rep, tok_per_cta, S, window;
    float scale;
    uint32_t* status;                      // may be null
};

__device__ __forceinline__ void tma_load_4d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, int w, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.4d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5}], [%6];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(w), "r"(bar) : "memory");
}
__device__ __forceinline__ void tma_load_3d(uint32_t dst, const CUtensorMap* map, int x, int y, int z, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(z), "r"(bar) : "memory");
}
// N-major operand (value tile: 64 context columns per 128-byte row, one row per key), 128-byte swizzle: 8-key groups are
// 1024 bytes apart, 64-column blocks `block_bytes`
__device__ __forceinline__ uint64_t umma_smem_desc_mn(uint32_t smem_addr, uint32_t block_bytes) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);
    d |= (uint64_t)(block_bytes >> 4) << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}
// a / b with inv = 1.0f / b, which every probability of a row shares: the quotient by the reciprocal, put right by its remainder
// (Markstein, "Computation of elementary functions on the IBM RISC System/6000 processor", 1990).  Equal to the division
// for the sums met here (1 <= b < 2^25).
__device__ __forceinline__ float quotient(float a, float b, float inv) {
    const float q = a * inv;
    return fmaf(fmaf(-q, b, a), inv, q);
}
template <int D>
__global__ void __launch_bounds__(PA_THREADS, 1) prompt_attn_kernel(const PromptAttnParams P, const __grid_constant__ CUtensorMap qmap,
                                                                    const __grid_constant__ CUtensorMap kmap,
                                                                    const __grid_constant__ CUtensorMap vmap) {
    extern __shared__ __align__(1024) uint8_t smem[];
    constexpr uint32_t TILE = pa_tile_bytes(D);
    constexpr int SUBS = D / 64;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t full_mask = 0xFFFFFFFFu;
    const uint32_t s_raw = smem_u32(smem);
    const uint32_t s0 = (s_raw + 1023u) & ~1023u;
    const uint32_t q_base = s0, ring = q_base + TILE, p_base = ring + PA_RING * TILE, bar_base = p_base + 2 * PA_P_BYTES;
    const uint32_t bar_q = bar_base, bar_o = bar_base + 8u, tmem_slot = bar_base + 16u;
    auto bar_full = [&](int s) { return bar_base + 32u + 8u * s; };
    auto bar_empty = [&](int s) { return bar_base + 64u + 8u * s; };
    auto bar_sfull = [&](int s) { return bar_base + 96u + 8u * s; };
    auto bar_sempty = [&](int s) { return bar_base + 112u + 8u * s; };
    auto bar_pfull = [&](int s) { return bar_base + 128u + 8u * s; };
    auto bar_pempty = [&](int s) { return bar_base + 144u + 8u * s; };
    float* stat_l = reinterpret_cast<float*>(smem + (bar_base + 160u - s_raw));      // [half][row]
    uint16_t* stat_m = reinterpret_cast<uint16_t*>(stat_l + 2 * PA_ROWS);

    // the longest rows (last tokens of the prompt) first, so that the short ones fill the end of the grid
    const int kvh = blockIdx.x % P.n_kv;
    const int tok0 = ((int)(gridDim.x / P.n_kv) - 1 - (int)blockIdx.x / P.n_kv) * P.tok_per_cta;
    // range of positions of this CTA's tokens (every warp for itself: at most four loads per lane), hence of its key tiles
    int pmin = 0x7FFFFFFF, pmax = -1;
    for (int i = lane; i < P.tok_per_cta && tok0 + i < P.T; i += 32) {
        const long long pl = P.positions[tok0 + i];
        const int p = pl < 0 ? -1 : pl > 0x3FFFFFFF ? 0x3FFFFFFF : (int)pl;
        pmin = min(pmin, p); pmax = max(pmax, p);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        pmin = min(pmin, __shfl_xor_sync(full_mask, pmin, o));
        pmax = max(pmax, __shfl_xor_sync(full_mask, pmax, o));
    }
    const int last_key = max(0, min(pmax, P.S - 1));
    const int first_key = P.window > 0 ? max(0, min(pmin - P.window + 1, last_key)) : 0;
    const int t_lo = first_key / PA_KEYS, n = last_key / PA_KEYS - t_lo + 1;           // at least one tile

    if (threadIdx.x == 0) {
        mbar_init(bar_q, 1); mbar_init(bar_o, 1);
        for (int s = 0; s < PA_RING; ++s) { mbar_init(bar_full(s), 1); mbar_init(bar_empty(s), 1); }
        for (int s = 0; s < 2; ++s) {
            mbar_init(bar_sfull(s), 1); mbar_init(bar_sempty(s), PA_SOFTMAX);
            mbar_init(bar_pfull(s), PA_SOFTMAX); mbar_init(bar_pempty(s), 1);
        }
        mbar_fence_init();
        fence_proxy_async();
    }
    if (warp == 9) { tmem_alloc<false>(tmem_slot, 512); tmem_relinquish<false>(); }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = lds32(tmem_slot);
    const uint32_t tmem_o = tmem + 2 * PA_KEYS;

    if (warp < 8) {
        // =========================================================== softmax, epilogue
        const int half = warp >> 2, r = threadIdx.x & 127;
        const int tok = tok0 + r / P.rep, head = r % P.rep;
        const bool valid = r < P.rep * P.tok_per_cta && tok < P.T;
        int hi = -1, lo = 0;                                           // allowed keys of this row: lo <= key <= hi
        if (valid) {
            const long long pl = P.positions[tok];
            hi = (int)min(pl, (long long)(P.S - 1));
            if (P.window > 0) lo = (int)max(0ll, min(pl, 0x3FFFFFFFll) - P.window + 1);
        }
        const uint32_t my_lanes = (uint32_t)((warp & 3) * 32) << 16;
        bool healthy = true;

        // scaled, rounded and masked scores of this row's 64 keys of S tile `g` (key tile `jt`); frees the TMEM buffer
        auto scores = [&](int g, int jt, float (&x)[64]) {
            healthy = healthy && __all_sync(full_mask, mbar_wait_bounded(bar_sfull(g & 1), (uint32_t)(g >> 1) & 1u, P.status, DEV_TIMEOUT_ACC));
            if (!healthy) return;
            tc_fence_after();
            uint32_t v[2][32];
            tmem_ld32(tmem + my_lanes + (uint32_t)((g & 1) * PA_KEYS + half * 64), v[0]);
            tmem_ld32(tmem + my_lanes + (uint32_t)((g & 1) * PA_KEYS + half * 64 + 32), v[1]);
            tmem_ld_wait();
            tc_fence_before();
            mbar_arrive(bar_sempty(g & 1));
#pragma unroll
            for (int i = 0; i < 64; i += 2) {
                const uint32_t a = pack_bf16x2(__uint_as_float(v[i >> 5][i & 31]), __uint_as_float(v[i >> 5][(i & 31) + 1]));
                const uint32_t b = pack_bf16x2(__uint_as_float(a << 16) * P.scale, __uint_as_float(a & 0xFFFF0000u) * P.scale);
                x[i] = __uint_as_float(b << 16);
                x[i + 1] = __uint_as_float(b & 0xFFFF0000u);
            }
            const int k0 = jt * PA_KEYS;
            if (k0 + PA_KEYS - 1 > min(pmin, P.S - 1) || (P.window > 0 && k0 <= pmax - P.window)) {      // the border crosses this tile
                const int a = lo - k0 - half * 64, b = hi - k0 - half * 64;
#pragma unroll
                for (int i = 0; i < 64; ++i)
                    if (i < a || i > b) x[i] = -INFINITY;
            }
        };

        float m = -INFINITY, l = 0.0f;
        for (int j = 0; j < n && healthy; ++j) {                        // pass A
            float x[64];
            scores(j, t_lo + j, x);
            if (!healthy) break;
            float t[4] = {x[0], x[1], x[2], x[3]};
#pragma unroll
            for (int i = 4; i < 64; ++i) t[i & 3] = fmaxf(t[i & 3], x[i]);
            const float nm = fmaxf(m, fmaxf(fmaxf(t[0], t[1]), fmaxf(t[2], t[3])));
            const float base = nm == -INFINITY ? 0.0f : nm;             // nothing allowed so far: every exponential is zero
            float s[4] = {l * expf(m - base), 0.0f, 0.0f, 0.0f};
#pragma unroll
            for (int i = 0; i < 64; ++i) s[i & 3] += expf(x[i] - base);
            l = (s[0] + s[1]) + (s[2] + s[3]);
            m = nm;
        }
        stat_l[half * PA_ROWS + r] = l;
        stat_m[half * PA_ROWS + r] = (uint16_t)(__float_as_uint(m) >> 16);           // scores are bf16 values
        asm volatile("bar.sync 1, 256;" ::: "memory");                  // the eight softmax warps
        const float ol = stat_l[(half ^ 1) * PA_ROWS + r], om = bf16_to_float(stat_m[(half ^ 1) * PA_ROWS + r]);
        const float gm = fmaxf(m, om);
        const float base = gm == -INFINITY ? 0.0f : gm;
        // (a sum of two: both halves get the same bits)
        const float tot = l * expf(m - base) + ol * expf(om - base), inv = 1.0f / tot;

        for (int j = 0; j < n && healthy; ++j) {                        // pass B
            float x[64];
            scores(n + j, t_lo + j, x);
            if (!healthy) break;
            uint32_t p[32];
#pragma unroll
            for (int i = 0; i < 32; ++i)
                p[i] = pack_bf16x2(quotient(expf(x[2 * i] - base), tot, inv), quotient(expf(x[2 * i + 1] - base), tot, inv));
            healthy = __all_sync(full_mask, mbar_wait_bounded(bar_pempty(j & 1), ((uint32_t)(j >> 1) & 1u) ^ 1u, P.status, DEV_TIMEOUT_EMPTY));
            if (!healthy) break;
            const uint32_t row = p_base + (uint32_t)(j & 1) * PA_P_BYTES + (uint32_t)half * PA_SUB + (uint32_t)r * 128u;
#pragma unroll
            for (int c = 0; c < 8; ++c)
                sts128(row + (((uint32_t)c ^ (uint32_t)(r & 7)) << 4), p[4 * c], p[4 * c + 1], p[4 * c + 2], p[4 * c + 3]);
            fence_proxy_async();
            mbar_arrive(bar_pfull(j & 1));
        }
        if (healthy) healthy = __all_sync(full_mask, mbar_wait_bounded(bar_o, 0u, P.status, DEV_TIMEOUT_ACC));
        tc_fence_after();
        if (healthy) {
#pragma unroll
            for (int c0 = 0; c0 < D / 2; c0 += 32) {
                uint32_t v[32];
                const int col = half * (D / 2) + c0;
                tmem_ld32(tmem_o + my_lanes + (uint32_t)col, v);
                tmem_ld_wait();
                if (valid) {
                    uint4* dst = reinterpret_cast<uint4*>(P.out + (((size_t)blockIdx.y * P.T + tok) * P.n_kv * P.rep + (size_t)kvh * P.rep + head) * D + col);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        uint32_t o[4];
#pragma unroll
                        for (int e = 0; e < 4; ++e) o[e] = pack_bf16x2(__uint_as_float(v[8 * c + 2 * e]), __uint_as_float(v[8 * c + 2 * e + 1]));
                        dst[c] = make_uint4(o[0], o[1], o[2], o[3]);
                    }
                }
            }
        }
        tc_fence_before();
    } else if (warp == 8) {
        // =========================================================== TMA
        // (loops on the whole warp, the instructions elected: see elect_one())
        if (elect_one()) {
            mbar_arrive_expect_tx(bar_q, (uint32_t)(P.rep * P.tok_per_cta) * 128u * SUBS);
            for (int c = 0; c < SUBS; ++c) tma_load_3d(q_base + c * PA_SUB, &qmap, 64 * c, kvh * P.rep, (int)blockIdx.y * P.T + tok0, bar_q);
        }
        __syncwarp();
        bool healthy = true;
        uint32_t s = 0, ph = 0;
        auto load = [&](const CUtensorMap* map, int jt) {
            healthy = __all_sync(full_mask, healthy && mbar_wait_bounded(bar_empty(s), ph ^ 1u, P.status, DEV_TIMEOUT_EMPTY));
            if (!healthy) return;
            if (elect_one()) {
                mbar_arrive_expect_tx(bar_full(s), TILE);
#pragma unroll
                for (int c = 0; c < SUBS; ++c) tma_load_4d(ring + s * TILE + c * PA_SUB, map, 64 * c, jt * PA_KEYS, kvh, (int)blockIdx.y, bar_full(s));
            }
            __syncwarp();
            if (++s == PA_RING) { s = 0; ph ^= 1u; }
        };
        for (int j = 0; j < n && healthy; ++j) load(&kmap, t_lo + j);
        for (int j = 0; j <= n && healthy; ++j) {                       // K0, K1, V0, K2, V1, ..., V(n-1)
            if (j < n) load(&kmap, t_lo + j);
            if (j > 0) load(&vmap, t_lo + j - 1);
        }
    } else {
        // =========================================================== MMA
        const uint32_t idesc_s = umma_idesc(PA_KEYS);
        const uint32_t idesc_o = umma_idesc(D) | (1u << 16);            // B (= V) is N-major
        bool healthy = __all_sync(full_mask, mbar_wait_bounded(bar_q, 0u, P.status, DEV_TIMEOUT_STAGE));
        uint32_t s = 0, ph = 0;
        const uint64_t qd = umma_smem_desc(q_base);
        auto issue_scores = [&](int g) {
            healthy = healthy && mbar_wait_bounded(bar_full(s), ph, P.status, DEV_TIMEOUT_STAGE);
            healthy = __all_sync(full_mask, healthy && mbar_wait_bounded(bar_sempty(g & 1), ((uint32_t)(g >> 1) & 1u) ^ 1u, P.status, DEV_TIMEOUT_EMPTY));
            if (!healthy) return;
            tc_fence_after();
            const uint64_t kd = umma_smem_desc(ring + s * TILE);
            const uint32_t d = tmem + (uint32_t)((g & 1) * PA_KEYS);
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < D / 16; ++k) {
                    const uint64_t off = (uint64_t)((k / 4) * (PA_SUB >> 4) + (k % 4) * 2);
                    umma_bf16<false>(d, qd + off, kd + off, idesc_s, k > 0 ? 1u : 0u);
                }
                umma_commit<false>(bar_empty(s));
                umma_commit<false>(bar_sfull(g & 1));
            }
            __syncwarp();
            if (++s == PA_RING) { s = 0; ph ^= 1u; }
        };
        auto issue_context = [&](int j) {
            healthy = healthy && mbar_wait_bounded(bar_full(s), ph, P.status, DEV_TIMEOUT_STAGE);
            healthy = __all_sync(full_mask, healthy && mbar_wait_bounded(bar_pfull(j & 1), (uint32_t)(j >> 1) & 1u, P.status, DEV_TIMEOUT_FULL));
            if (!healthy) return;
            tc_fence_after();
            const uint64_t pd = umma_smem_desc(p_base + (uint32_t)(j & 1) * PA_P_BYTES), vd = umma_smem_desc_mn(ring + s * TILE, PA_SUB);
            if (elect_one()) {
#pragma unroll
                for (int k = 0; k < PA_KEYS / 16; ++k)
                    umma_bf16<false>(tmem_o, pd + (uint64_t)((k / 4) * (PA_SUB >> 4) + (k % 4) * 2), vd + (uint64_t)(k * (2048 >> 4)), idesc_o,
                                     (j > 0 || k > 0) ? 1u : 0u);
                umma_commit<false>(bar_empty(s));
                umma_commit<false>(bar_pempty(j & 1));
            }
            __syncwarp();
            if (++s == PA_RING) { s = 0; ph ^= 1u; }
        };
        for (int g = 0; g < n && healthy; ++g) issue_scores(g);
        for (int j = 0; j <= n && healthy; ++j) {
            if (j < n) issue_scores(n + j);
            if (j > 0) issue_context(j - 1);
        }
        if (healthy && elect_one()) umma_commit<false>(bar_o);
        __syncwarp();
    }
    tc_fence_before();
    __syncthreads();
    if (warp == 9) { tc_fence_after(); tmem_dealloc<false>(tmem, 512); }
}

}  // namespace cb
