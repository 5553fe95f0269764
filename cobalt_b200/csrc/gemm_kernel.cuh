// Prefill GEMM: Y[m, k] = sum_j bf16(W[k, j]) * X[m, j] with tcgen05.mma, accumulators in tensor memory.  Up to four
// matrices that read the same activations (q|k|v, gate|up) go out as one launch: their 128-row tiles form one list.
//
// A CTA owns 128 weight rows and one token tile and walks the 64-column stages of its range of 128-column groups:
//
//   decode     sets of eight warps: the first four take the first 64 columns of a group, the others the second; thread r of
//              either half owns weight row r.  It reads the row's bitmask words and code bits straight from the tile image
//              in global memory (the next group's codes are requested before the current one is expanded; whole tiles are
//              prefetched into the L2 two column tiles ahead), expands them to bf16 (decode_core.cuh) and writes eight
//              swizzled 16-byte chunks into the A stage.  One set per CTA of the single form, two (on alternate groups) in
//              a pair: 16 warps per SM, whose expansion is bound by latency more than by issue slots.  After the main
//              loop the same warps drain TMEM.
//   next warp  one elected lane issues the TMA loads of the activation stage (2-D tensor map, 128-byte swizzle, rows
//              beyond M zero-filled; no multicast).
//   last warp  one elected lane issues tcgen05.mma and tcgen05.commit.
//
// Two forms, picked per launch by a cost model (gemm_config() in cobalt_abi.cu):
//   single  up to 256 tokens in one accumulator, two CTAs per SM: one CTA's load latencies, start-up and epilogue hide
//           under the other's work.  Small and middling token counts, where expanding the weights is the cost.
//   pair    two CTAs of a cluster form one 256-row tile (tcgen05.mma.cta_group::2) of up to 512 tokens in two
//           accumulators.  With one CTA per tile the limit at many tokens was operand traffic through shared memory: per
//           stage 16 KB of A written and read twice, 64 KB of B written and read = 176 KB against 1024 cycles of MMA (128
//           bytes per cycle: 1375 cycles).  In a pair each SM holds and reads half of B: 112 KB, 875 cycles.
//
// Split-K (grids that leave SMs idle): the CTAs of a tile's column ranges form a cluster, park their fp32 sums in shared
// memory and each adds its share of the tokens over the cluster in split order (distributed shared memory): no partial
// sum goes through global memory and no CTA adds alone.
// Measured (1965 MHz, cold L2, one CTA per tile with 512 tokens and partial sums in global memory -> this kernel): 4096 x 14336, 3 bit,
// 2048 tokens 232 -> 172 us (1.40 PFLOP/s); 4096 x 4096, 2048 tokens 91 -> 68 us; 14336 x 4096, 2048 tokens 317 -> 238 us;
// 4096 x 4096, 100 tokens 33 -> 26 us; q|k|v of a 7B block (one launch instead of three), 2048 tokens 241 -> 123 us.
//
// Generic-proxy writes to A stages are published with fence.proxy.async before the mbarrier arrive.  In a pair the second CTA's half
// of A is read by MMAs that the first CTA issues: its decode warps release and the issuing warp acquires at cluster scope (an
// unqualified arrive or wait orders the threads of one CTA only), by the fences that cover shared memory alone: 4096 x
// 14336, 2048 tokens 169 -> 170.5 us.  release.cluster / acquire.cluster on the barrier operations themselves cover all memory, the
// decode warps' loads in flight with it, and cost 80 us at 4096 x 4096; the acquire after every wait of a pair cost 3.6 %
// and is not needed for completions of tcgen05.commit.  Every wait on an mbarrier is bounded: on expiry the kernel records a
// status code, stops issuing work, frees its tensor memory and returns.
//
// Behaviour replaced: cbk::gemm_tile (mma.sync m16n8k16, per-fragment bf16x2 dequantisation,
// src/cobaltkernel/csrc/cobalt_gemm.cuh:243-609) driven by gemm_phase
// (src/cobaltkernel/csrc/prefill_kernel.cu:103-150).
#pragma once
#include <cuda.h>
#include "common.cuh"
#include "gemv_kernel.cuh"   // finish_output

namespace cb {

constexpr int GEMM_ROWS = 128;            // weight rows per CTA
constexpr int GEMM_KS = 64;               // columns per stage = one 128-byte swizzle row of bf16
constexpr int GEMM_RB = GEMM_ROWS / TILE_ROWS;   // 8 row blocks per CTA
constexpr int GEMM_LUT_COPIES = 8;
constexpr int GEMM_MAX_STAGES = 8;
constexpr int GEMM_MAX_SPLITS = 8;        // CTAs of a cluster along the columns (portable cluster size)
constexpr int gemm_decode_warps(bool pair) { return pair ? 16 : 8; }     // 16 on an SM either way: singles come in twos
constexpr int gemm_threads(bool pair) { return gemm_decode_warps(pair) * 32 + 64; }
constexpr int gemm_red_tokens(bool pair) { return pair ? 256 : 128; }    // tokens per round of the split reduction
constexpr uint32_t GEMM_LUT_BYTES = LUT_ENTRIES * GEMM_LUT_COPIES * 8;   // 16 KB
constexpr uint32_t GEMM_A_BYTES = GEMM_ROWS * GEMM_KS * 2;               // 16 KB
constexpr uint32_t gemm_red_bytes(bool pair) { return (uint32_t)gemm_red_tokens(pair) * GEMM_ROWS * 4; }   // laid over the operand stages
constexpr uint32_t GEMM_BAR_BYTES = 4 * GEMM_MAX_STAGES * 8 + 64;
constexpr int GEMM_SINGLE_TOKENS = 256, GEMM_PAIR_TOKENS = 512;          // accumulator columns a CTA may hold

struct GemmMat {
    const uint8_t* tiles;
    const uint32_t* tile_off;
    uint16_t* y;
    float* y32;                 // when set, raw fp32 sums go here instead (no bias, no rounding)
    const uint16_t* bias;
    int64_t ldy;
    int K, RB;
    int rt_start;               // first row tile of this matrix in the launch's list
};

struct GemmParams {
    GemmMat mat[GEMV_MAX_MATS];
    int n_mats;
    int G, CT;
    const uint16_t* col_scale;  // fp16 bits; the SCALED instantiation only (single-matrix launches)
    bool literal_scale;         // not on a 16-byte boundary: read one value at a time, by the literal path
    int M;
    int tok_per_cta;            // tokens per token tile
    int acc_tokens;             // tokens per accumulator (tok_per_cta = one or two of these)
    int splits;                 // column ranges = CTAs of the cluster along z
    int a_stages, b_stages;     // operand stages in shared memory
    uint32_t b_acc_bytes;       // B bytes of one accumulator's tokens that this CTA holds per stage
    uint32_t b_stage_bytes;
    uint32_t* status;
};

// ---- tcgen05 / TMA / cluster wrappers
template <bool PAIR>
__device__ __forceinline__ void tmem_alloc(uint32_t smem_dst, uint32_t ncols) {
    if (PAIR) asm volatile("tcgen05.alloc.cta_group::2.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
    else asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_dst), "r"(ncols) : "memory");
}
template <bool PAIR>
__device__ __forceinline__ void tmem_relinquish() {
    if (PAIR) asm volatile("tcgen05.relinquish_alloc_permit.cta_group::2.sync.aligned;" ::: "memory");
    else asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
template <bool PAIR>
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    if (PAIR) asm volatile("tcgen05.dealloc.cta_group::2.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
    else asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
template <bool PAIR>
__device__ __forceinline__ void umma_bf16(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t accumulate) {
    if (PAIR)
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::2.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
    else
        asm volatile(
            "{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\t"
            "tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n\t}"
            ::"r"(tmem_d), "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate) : "memory");
}
// completion of the MMAs issued so far -> the barrier at this offset (pair: in both CTAs, `mask` = their cluster ranks)
template <bool PAIR>
__device__ __forceinline__ void umma_commit(uint32_t bar, uint16_t mask = 0) {
    if (PAIR)
        asm volatile("tcgen05.commit.cta_group::2.mbarrier::arrive::one.shared::cluster.multicast::cluster.b64 [%0], %1;" ::"r"(bar), "h"(mask) : "memory");
    else
        asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// One lane of a converged warp.  The loops around TMA and MMA instructions run on the whole warp and only the instruction
// itself is elected: their operands are then known to be warp-uniform and live in uniform registers.  With the loop inside
// "if (lane == 0)" every descriptor took moves to uniform registers and 64-bit adds in one thread's dependent chain, and issuing
// the four MMAs and two commits of a stage took 650 clocks, more than the stage's arithmetic.
__device__ __forceinline__ bool elect_one() {
    uint32_t e;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.b32 %0, 1, 0, p;\n\t}" : "=r"(e));
    return e != 0;
}
__device__ __forceinline__ uint32_t cluster_rank() { uint32_t r; asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r)); return r; }
__device__ __forceinline__ void cluster_sync_all() {       // every thread of every CTA of the cluster
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ uint32_t map_to_rank(uint32_t addr, uint32_t rank) {
    uint32_t r; asm("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank)); return r;
}
__device__ __forceinline__ float4 ld_cluster_f4(uint32_t addr) {
    float4 v;
    asm volatile("ld.shared::cluster.v4.f32 {%0,%1,%2,%3}, [%4];" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "r"(addr) : "memory");
    return v;
}
// arrival on a barrier of another CTA of the cluster; releases this thread's (and, after a __syncwarp, its warp's) writes to the shared
// memory of its own CTA
__device__ __forceinline__ void mbar_arrive_cluster(uint32_t cluster_addr) {
    asm volatile("fence.release.sync_restrict::shared::cta.cluster;\n\tmbarrier.arrive.relaxed.cluster.shared::cluster.b64 _, [%0];" ::"r"(cluster_addr) : "memory");
}
__device__ __forceinline__ void tmem_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr) : "memory");
}
__device__ __forceinline__ void tmem_ld_wait() { asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory"); }
// 2-D tiled TMA load (no multicast): box of the tensor map at (x = column, y = token) -> this CTA's shared memory; the pair
// form may count its bytes on a barrier of either CTA of the pair
template <bool PAIR>
__device__ __forceinline__ void tma_load_2d(uint32_t dst, const CUtensorMap* map, int x, int y, uint32_t bar) {
    if (PAIR)
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.cta_group::2 [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
    else
        asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                     ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}

// K-major, 128-byte swizzle, 8-row groups 1024 B apart; descriptor version 1 (sm_100)
__device__ __forceinline__ uint64_t umma_smem_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3FFFFu) >> 4);        // start address
    d |= (uint64_t)1 << 16;                               // leading byte offset (unused for swizzled K-major)
    d |= (uint64_t)(1024 >> 4) << 32;                     // stride byte offset
    d |= (uint64_t)1 << 46;                               // version
    d |= (uint64_t)2 << 61;                               // SWIZZLE_128B
    return d;
}
// D = f32, A = B = bf16, both K-major, M = m rows, N = n
__device__ __forceinline__ uint32_t umma_idesc(uint32_t n, uint32_t m = GEMM_ROWS) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((n >> 3) << 17) | ((m >> 4) << 24);
}

// What a thread needs to expand 64 columns of its row; requested one group ahead.  The rows of a warp lie about 128 bytes
// apart in the code stream, so every load touches 32 lines whatever its width: the up to 256 bits come in as aligned
// 16-byte chunks (only those that hold survivors of these columns) and the words are picked out of registers.  With one
// 4-byte load per word that lookup was the limit: ten loads = 320 lines per warp and stage, 1600 clocks a stage per SM.
template <int BITS>
struct GemmFetch {
    static constexpr int NC = BITS == 2 ? 2 : 3;          // 64 codes at any bit offset of the first chunk
    uint4 chunk[NC];
    uint32_t mask[2];
    uint32_t bit;                                         // offset of the first code in chunk[0]
    uint32_t sz;
};
// the N words from word `first` on, out of W words in registers (barrel shift: no indexed registers)
template <int W, int N, bool WIDE>
__device__ __forceinline__ void pick_words(const uint32_t (&c)[W], uint32_t first, uint32_t (&out)[N]) {
    uint32_t a[W];
#pragma unroll
    for (int i = 0; i < W; ++i) a[i] = c[i];
#pragma unroll
    for (int step = WIDE ? 4 : 2; step > 0; step >>= 1) {
        const bool on = (first & (uint32_t)step) != 0;
#pragma unroll
        for (int i = 0; i < W; ++i)
            if (i < N + step - 1) a[i] = on && i + step < W ? a[i + step] : a[i];
    }
#pragma unroll
    for (int i = 0; i < N; ++i) out[i] = i < W ? a[i] : 0u;
}

template <int BITS, bool PAIR, bool SCALED>
__global__ void __launch_bounds__(gemm_threads(PAIR), PAIR ? 1 : 2) gemm_tcgen05_kernel(const __grid_constant__ GemmParams P,
                                                                                  const __grid_constant__ CUtensorMap xmap) {
    extern __shared__ __align__(1024) uint8_t smem[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t full_mask = 0xFFFFFFFFu;
    constexpr int DW = gemm_decode_warps(PAIR);

    // ---- shared memory: A stages | B stages | expansion table | barriers.  The operand stages need 1024-byte alignment;
    // the dynamic window starts on it (two CTAs of 113 KB leave no room for slack).
    const uint32_t s0 = smem_u32(smem);
    if (s0 & 1023u) {
        if (threadIdx.x == 0 && P.status) atomicCAS(P.status, 0u, (uint32_t)DEV_TIMEOUT_STAGE);
        return;
    }
    const uint32_t a_base = s0;
    const uint32_t b_base = a_base + GEMM_A_BYTES * (uint32_t)P.a_stages;
    const uint32_t lut_addr = b_base + P.b_stage_bytes * (uint32_t)P.b_stages;
    const uint32_t bar_base = lut_addr + GEMM_LUT_BYTES;
    auto bar_afull = [&](uint32_t s) { return bar_base + 8u * s; };
    auto bar_aempty = [&](uint32_t s) { return bar_base + 8u * GEMM_MAX_STAGES + 8u * s; };
    auto bar_bfull = [&](uint32_t s) { return bar_base + 16u * GEMM_MAX_STAGES + 8u * s; };
    auto bar_bempty = [&](uint32_t s) { return bar_base + 24u * GEMM_MAX_STAGES + 8u * s; };
    const uint32_t bar_acc = bar_base + 32u * GEMM_MAX_STAGES;
    const uint32_t tmem_slot = bar_acc + 8u;

    LutEntry* const lut_s = reinterpret_cast<LutEntry*>(smem + (lut_addr - s0));
    const uint32_t rank = cluster_rank();
    const uint32_t leader = PAIR ? rank & ~1u : rank;                   // the CTA that issues the MMAs of a pair
    const uint32_t half_id = PAIR ? rank & 1u : 0u;
    const int m0 = blockIdx.y * P.tok_per_cta;
    int n_tok = P.M - m0;
    if (n_tok > P.tok_per_cta) n_tok = P.tok_per_cta;
    // tokens of the two accumulators, and the N of their MMAs (columns beyond n_tok are computed and never read)
    const int n_acc0 = n_tok < P.acc_tokens ? n_tok : P.acc_tokens, n_acc1 = n_tok - n_acc0;
    constexpr int N_STEP = PAIR ? 32 : 16;
    const uint32_t n_mma0 = (uint32_t)((n_acc0 + N_STEP - 1) / N_STEP * N_STEP), n_mma1 = (uint32_t)((n_acc1 + N_STEP - 1) / N_STEP * N_STEP);
    const int split = blockIdx.z;
    const int g_begin = (int)((long long)P.G * split / P.splits), g_end = (int)((long long)P.G * (split + 1) / P.splits);
    const int my_stages = 2 * (g_end - g_begin);

    // the matrix of this row tile, with compares over the (at most four) slots (see gemv_kernel.cuh)
    const int row_tile = blockIdx.x;
    int mi = 0;
#pragma unroll
    for (int k = 1; k < GEMV_MAX_MATS; ++k)
        if (k < P.n_mats && row_tile >= P.mat[k].rt_start) mi = k;
    const int local_rt = row_tile - MAT_FIELD(mi, rt_start);

    // ---- the decode warps' first requests fly during the block set-up (they touch nothing that it prepares)
    const int r = threadIdx.x & 127;                                    // weight row within the CTA tile
    const int row = local_rt * GEMM_ROWS + r;
    const uint32_t half = ((uint32_t)warp >> 2) & 1u;               // columns 64*half .. of a group
    constexpr int STEP = DW / 8;                                    // two sets of decode warps take alternate groups
    const int set = warp >> 3;
    const int rr = r & 15;
    const int rb = local_rt * GEMM_RB + (r >> 4);
    const bool have_rb = warp < DW && rb < MAT_FIELD(mi, RB);
    const uint8_t* const tiles = MAT_FIELD(mi, tiles);
    const uint32_t* const tile_off = MAT_FIELD(mi, tile_off) + (size_t)(have_rb ? rb : 0) * P.CT;
    const uint2* const lut_lane = reinterpret_cast<const uint2*>(lut_s) + (lane & (GEMM_LUT_COPIES - 1));
    const uint32_t x7 = (uint32_t)(r & 7);
    const uint32_t rowaddr = a_base + (uint32_t)(r >> 3) * 1024u + x7 * 128u;
    // Weight bytes are read by per-thread loads whose addresses depend on each other (tile offset -> masks -> codes), so
    // each is requested one step ahead of its use: offsets four column tiles ahead, a tile's masks when the last group of
    // the tile before has been taken, a group's codes while the group before is expanded.  One thread per row block
    // asks the L2 for whole tiles, two ahead of the one requested.
    const int ct_begin = g_begin / TILE_GROUPS, ct_end = (g_end + TILE_GROUPS - 1) / TILE_GROUPS;
    auto offset_of = [&](int ct) { return have_rb ? __ldg(tile_off + (ct < P.CT ? ct : P.CT)) : 0u; };
    auto prefetch_l2 = [&](int ct, uint32_t from, uint32_t to) {
        if (have_rb && rr == 0 && warp < 4 && ct < ct_end)
            asm volatile("cp.async.bulk.prefetch.L2.global [%0], %1;" ::"l"(tiles + (size_t)from * 16), "r"((to - from) * 16u) : "memory");
    };
    uint4 mk[TILE_GROUPS];                                          // masks and scale | zero of the tile's groups from `pos` on
    uint32_t szv[TILE_GROUPS];
    uint32_t o0 = offset_of(ct_begin), o1 = offset_of(ct_begin + 1), o2 = offset_of(ct_begin + 2), o3 = offset_of(ct_begin + 3);
    uint32_t codes = 0, codes_cur = 0;                              // code stream of the tile in mk / being taken from, 16-byte units
    uint32_t off = 0;                                               // rank of this row's next survivor within the tile
    int pos = 0;
    auto request_tile = [&](int ct) {
        int w = P.G - TILE_GROUPS * ct;
        if (w > TILE_GROUPS) w = TILE_GROUPS;
        const uint8_t* tile = tiles + (size_t)o0 * 16;
        codes = o0 + (uint32_t)(TILE_ROWS * 20 / 16) * (uint32_t)w;
#pragma unroll
        for (int gi = 0; gi < TILE_GROUPS; ++gi) {
            mk[gi] = make_uint4(0, 0, 0, 0);
            szv[gi] = 0;
            if (have_rb && gi < w) {
                mk[gi] = __ldg(reinterpret_cast<const uint4*>(tile) + rr * w + gi);
                szv[gi] = __ldg(reinterpret_cast<const uint32_t*>(tile + TILE_ROWS * w * 16) + rr * w + gi);
            }
        }
        prefetch_l2(ct + 2, o2, o3);
        o0 = o1; o1 = o2; o2 = o3;
        o3 = offset_of(ct + 4);
    };
    auto count = [&](const uint4& v) { return (uint32_t)(__popc(v.x) + __popc(v.y) + __popc(v.z) + __popc(v.w)); };
    auto settle_tile = [&]() {                                      // the masks are there: where this row's codes start
        uint32_t cnt = 0;
#pragma unroll
        for (int gi = 0; gi < TILE_GROUPS; ++gi) cnt += count(mk[gi]);
        uint32_t inc = cnt;
#pragma unroll
        for (int d = 1; d < 16; d <<= 1) {
            const uint32_t up = __shfl_up_sync(full_mask, inc, d, 16);
            if ((lane & 15) >= d) inc += up;
        }
        off = inc - cnt;
        codes_cur = codes;
        pos = 0;
    };
    auto skip = [&]() {                                             // the next group moves into slot 0
        off += count(mk[0]);
#pragma unroll
        for (int k2 = 0; k2 + 1 < TILE_GROUPS; ++k2) { mk[k2] = mk[k2 + 1]; szv[k2] = szv[k2 + 1]; }
        ++pos;
    };
    int ct_cur = -1;
    auto take = [&](GemmFetch<BITS>& f, int g) {                    // request the codes of group g (of the matrix)
        if (g / TILE_GROUPS != ct_cur) { ct_cur = g / TILE_GROUPS; settle_tile(); }
        while (pos < g % TILE_GROUPS) skip();
        f.mask[0] = half ? mk[0].z : mk[0].x;
        f.mask[1] = half ? mk[0].w : mk[0].y;
        f.sz = szv[0];
        const uint32_t first = (half ? off + __popc(mk[0].x) + __popc(mk[0].y) : off) * (uint32_t)BITS;
        f.bit = first & 127u;
        const uint32_t end = f.bit + (uint32_t)(__popc(f.mask[0]) + __popc(f.mask[1])) * (uint32_t)BITS;
        const uint4* p = reinterpret_cast<const uint4*>(tiles) + codes_cur + (first >> 7);
#pragma unroll
        for (int i = 0; i < GemmFetch<BITS>::NC; ++i)
            if (end > f.bit && end > 128u * i) f.chunk[i] = __ldg(p + i);
        skip();
        const int next = g + STEP;                                  // was this the last group taken from the tile?
        if (next < g_end && next / TILE_GROUPS != ct_cur) request_tile(next / TILE_GROUPS);
    };
    prefetch_l2(ct_begin + 1, o1, o2);
    request_tile(ct_begin);
    if ((g_begin + set) / TILE_GROUPS != ct_begin) request_tile(ct_begin + 1);          // a set that starts in the second tile

    if (threadIdx.x == 0) {
        for (uint32_t s = 0; s < GEMM_MAX_STAGES; ++s) {
            mbar_init(bar_afull(s), PAIR ? 8 : 4); mbar_init(bar_aempty(s), 1);      // afull: one arrival per decode warp
            mbar_init(bar_bfull(s), 1); mbar_init(bar_bempty(s), 1);
        }
        mbar_init(bar_acc, 1);
        mbar_fence_init();
        fence_proxy_async();
    }
    if (threadIdx.x < LUT_ENTRIES) {      // expansion table: .x = selector A | view selector << 16, .y = selector B | bits consumed << 16
        const uint4 e = gemv_lut_entry(threadIdx.x, BITS);
#pragma unroll
        for (int c = 0; c < GEMM_LUT_COPIES; ++c) lut_s[threadIdx.x * GEMM_LUT_COPIES + c] = LutEntry{e.x | (e.z << 16), e.y | (e.w << 16)};
    }
    constexpr uint32_t TMEM_COLS = PAIR ? GEMM_PAIR_TOKENS : GEMM_SINGLE_TOKENS;
    if (warp == DW + 1) { tmem_alloc<PAIR>(tmem_slot, TMEM_COLS); tmem_relinquish<PAIR>(); }
    tc_fence_before();
    __syncwarp();
    if (PAIR) cluster_sync_all();                                       // the other CTA's barriers are in place before anyone arrives on them
    else __syncthreads();
    tc_fence_after();
    const uint32_t tmem_d = lds32(tmem_slot);

    bool healthy = true;
    if (warp < DW) {
        // =========================================================== decode
        GemmFetch<BITS> cur = {};
        if (g_begin + set < g_end) take(cur, g_begin + set);
        uint32_t s = 2u * (uint32_t)set + half, ph = 0;                 // slot and phase of the stage: group n of the CTA is stages 2n, 2n + 1
#pragma unroll 1
        for (int g = g_begin + set; g < g_end; g += STEP) {
            GemmFetch<BITS> nxt = {};
            if (g + STEP < g_end) take(nxt, g + STEP);
            const SegParams sp = make_seg_params(cur.sz, BITS, SCALED && P.literal_scale);
            uint32_t words[4 * GemmFetch<BITS>::NC];
#pragma unroll
            for (int i = 0; i < GemmFetch<BITS>::NC; ++i) {
                words[4 * i] = cur.chunk[i].x; words[4 * i + 1] = cur.chunk[i].y;
                words[4 * i + 2] = cur.chunk[i].z; words[4 * i + 3] = cur.chunk[i].w;
            }
            const uint32_t bit1 = cur.bit + (uint32_t)__popc(cur.mask[0]) * (uint32_t)BITS;
            healthy = __all_sync(full_mask, mbar_wait_bounded<PAIR>(bar_aempty(s), ph ^ 1u, P.status, DEV_TIMEOUT_EMPTY));
            if (!healthy) break;
            const uint32_t dst = rowaddr + s * GEMM_A_BYTES;
            const int col = g * GROUP + (int)half * 64;
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                const uint32_t o = h ? bit1 : cur.bit;
                if (sp.fast) {
                    uint2 lut[4];                                       // table entries first: their latencies overlap
#pragma unroll
                    for (int c = 0; c < 4; ++c) lut[c] = lut_lane[((cur.mask[h] >> (8 * c)) & 0xFFu) * GEMM_LUT_COPIES];
                    uint32_t raw[BITS + 1], win[BITS];                  // codes of the word, first survivor in the low bits of win[0]
                    if (h) pick_words<4 * GemmFetch<BITS>::NC, BITS + 1, true>(words, o >> 5, raw);
                    else pick_words<4 * GemmFetch<BITS>::NC, BITS + 1, false>(words, o >> 5, raw);
#pragma unroll
                    for (int i = 0; i < BITS; ++i) win[i] = funnel_r(raw[i], raw[i + 1], o);
#pragma unroll
                    for (int c = 0; c < 4; ++c) {
                        const uint2 e = lut[c];
                        uint32_t out[4];
                        if (SCALED) {
                            const uint4 cv = __ldg(reinterpret_cast<const uint4*>(P.col_scale + col + 32 * h) + c);
                            const uint32_t cw[4] = {cv.x, cv.y, cv.z, cv.w};
                            float cs[8];
#pragma unroll
                            for (int i = 0; i < 4; ++i) { cs[2 * i] = half_bits_to_float(cw[i]); cs[2 * i + 1] = half_bits_to_float(cw[i] >> 16); }
                            decode8_scaled<BITS>((cur.mask[h] >> (8 * c)) & 0xFFu, win[0], e.x, e.y, e.x >> 16, sp, cs, out);
                        } else {
                            decode8<BITS>(win[0], e.x, e.y, e.x >> 16, sp, out);
                        }
                        sts128(dst + (((uint32_t)(4 * h + c) ^ x7) << 4), out[0], out[1], out[2], out[3]);
                        if (c < 3) {
                            const uint32_t amt = e.y >> 16;             // at most 32 bits
#pragma unroll
                            for (int i = 0; i + 1 < BITS; ++i) win[i] = funnel_rc(win[i], win[i + 1], amt);
                            win[BITS - 1] = funnel_rc(win[BITS - 1], 0u, amt);
                        }
                    }
                } else {                                                // literal fp32 path (off-grid zero point, scale not finite)
                    float cs[32];
                    if (SCALED)
                        for (int i = 0; i < 32; ++i) cs[i] = half_bits_to_float(P.col_scale[col + 32 * h + i]);
                    uint32_t e[16];
                    decode32_slow(cur.mask[h], [&](uint32_t k) { return words[k]; }, o, BITS, sp, SCALED ? cs : nullptr, e);
                    for (int c = 0; c < 4; ++c)
                        sts128(dst + (((uint32_t)(4 * h + c) ^ x7) << 4), e[4 * c], e[4 * c + 1], e[4 * c + 2], e[4 * c + 3]);
                }
            }
            fence_proxy_async();
            __syncwarp();
            if (lane == 0) {
                if (PAIR) mbar_arrive_cluster(map_to_rank(bar_afull(s), leader));
                else mbar_arrive(bar_afull(s));
            }
            s += 2 * STEP;                                              // a_stages >= 2 * STEP: at most one turn of the ring
            if (s >= (uint32_t)P.a_stages) { s -= (uint32_t)P.a_stages; ph ^= 1u; }
            cur = nxt;
        }
        if (healthy) healthy = __all_sync(full_mask, mbar_wait_bounded<PAIR>(bar_acc, 0u, P.status, DEV_TIMEOUT_ACC));
    } else if (warp == DW) {
        // =========================================================== activation loader (TMA)
        bool good = true;
        const uint32_t bytes = P.b_acc_bytes * (n_acc1 > 0 ? 2u : 1u);
        uint32_t s = 0, ph = 0;
        for (uint32_t q = 0; q < (uint32_t)my_stages; ++q) {
            good = mbar_wait_bounded<PAIR>(bar_bempty(s), ph ^ 1u, P.status, DEV_TIMEOUT_EMPTY);
            if (!__all_sync(full_mask, good)) break;
            const int col = g_begin * GROUP + (int)q * GEMM_KS;
            // pair: each CTA loads its half of every accumulator's tokens; both count on the leader's barrier
            const uint32_t bar = PAIR ? map_to_rank(bar_bfull(s), leader) : bar_bfull(s);
            const uint32_t dst = b_base + s * P.b_stage_bytes;
            if (elect_one()) {
                if (half_id == 0) mbar_arrive_expect_tx(bar_bfull(s), PAIR ? 2u * bytes : bytes);
                tma_load_2d<PAIR>(dst, &xmap, col, m0 + (int)(half_id * (n_mma0 / 2u)), bar);
                if (n_acc1 > 0) tma_load_2d<PAIR>(dst + P.b_acc_bytes, &xmap, col, m0 + P.acc_tokens + (int)(half_id * (n_mma1 / 2u)), bar);
            }
            __syncwarp();
            if (++s == (uint32_t)P.b_stages) { s = 0; ph ^= 1u; }
        }
    } else {
        // =========================================================== MMA issuer (pair: of the leader)
        if (half_id == 0) {
            const uint32_t idesc0 = umma_idesc(n_mma0, PAIR ? 2 * GEMM_ROWS : GEMM_ROWS), idesc1 = umma_idesc(n_mma1 ? n_mma1 : 32, PAIR ? 2 * GEMM_ROWS : GEMM_ROWS);
            const uint16_t both = (uint16_t)(3u << leader);
            const uint32_t d0 = tmem_d, d1 = tmem_d + (uint32_t)P.acc_tokens;
            bool good = true;
            uint32_t sa = 0, pa = 0, sb = 0, pb = 0;
            for (uint32_t q = 0; q < (uint32_t)my_stages; ++q) {
                good = mbar_wait_bounded<PAIR>(bar_bfull(sb), pb, P.status, DEV_TIMEOUT_STAGE);
                if (good) good = mbar_wait_bounded<PAIR>(bar_afull(sa), pa, P.status, DEV_TIMEOUT_FULL);
                good = __all_sync(full_mask, good);
                if (!good) break;
                if (PAIR) cluster_acquire();                            // the other CTA's half of A (and of B)
                tc_fence_after();
                const uint64_t ad = umma_smem_desc(a_base + sa * GEMM_A_BYTES);
                const uint64_t bd0 = umma_smem_desc(b_base + sb * P.b_stage_bytes);
                const uint64_t bd1 = umma_smem_desc(b_base + sb * P.b_stage_bytes + P.b_acc_bytes);
                if (elect_one()) {
#pragma unroll
                    for (int k = 0; k < GEMM_KS / 16; ++k)
                        umma_bf16<PAIR>(d0, ad + (uint64_t)(2 * k), bd0 + (uint64_t)(2 * k), idesc0, (q > 0 || k > 0) ? 1u : 0u);
                    if (PAIR && n_mma1) {
#pragma unroll
                        for (int k = 0; k < GEMM_KS / 16; ++k)
                            umma_bf16<PAIR>(d1, ad + (uint64_t)(2 * k), bd1 + (uint64_t)(2 * k), idesc1, (q > 0 || k > 0) ? 1u : 0u);
                    }
                    umma_commit<PAIR>(bar_aempty(sa), both);
                    umma_commit<PAIR>(bar_bempty(sb), both);
                }
                __syncwarp();
                if (++sa == (uint32_t)P.a_stages) { sa = 0; pa ^= 1u; }
                if (++sb == (uint32_t)P.b_stages) { sb = 0; pb ^= 1u; }
            }
            if (good && elect_one()) umma_commit<PAIR>(bar_acc, both);
            __syncwarp();
        }
    }

    // ---- epilogue: TMEM lane = weight row, column = token; decode warp w drains lanes 32*(w%4).., every (DW / 4)-th 32 tokens
    const uint32_t my_tmem = tmem_d + ((uint32_t)((warp & 3) * 32) << 16);
    const bool stores = warp < DW && healthy && row < MAT_FIELD(mi, K);
    uint16_t* const y = MAT_FIELD(mi, y);
    float* const y32 = MAT_FIELD(mi, y32);
    const uint16_t* const bias = MAT_FIELD(mi, bias);
    const int64_t ldy = MAT_FIELD(mi, ldy);
    if (P.splits == 1) {
        if (warp < DW && healthy) {
            tc_fence_after();
            for (int c0 = 32 * (warp >> 2); c0 < n_tok; c0 += 8 * DW) {
                uint32_t v[32];
                tmem_ld32(my_tmem + (uint32_t)c0, v);
                tmem_ld_wait();
                if (stores) {
                    if (y32) {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (c0 + i < n_tok) y32[(size_t)(m0 + c0 + i) * ldy + row] = __uint_as_float(v[i]);
                    } else {
#pragma unroll
                        for (int i = 0; i < 32; ++i)
                            if (c0 + i < n_tok) y[(size_t)(m0 + c0 + i) * ldy + row] = finish_output(__uint_as_float(v[i]), bias, row);
                    }
                }
            }
        }
    } else {
        // split-K, in rounds of RED tokens: every CTA of the cluster parks its sums (the operand stages are free by now) and adds
        // its share of the tokens over all splits, in split order
        constexpr int RED = gemm_red_tokens(PAIR);
        float* red = reinterpret_cast<float*>(smem);
        const int row0 = local_rt * GEMM_ROWS + 4 * lane, K = MAT_FIELD(mi, K);
        const bool wide = row0 + 3 < K && (ldy & 3) == 0 && ((uintptr_t)y & 7) == 0 && ((uintptr_t)y32 & 15) == 0;
        for (int t0 = 0; t0 < n_tok; t0 += RED) {
            const int nt = n_tok - t0 < RED ? n_tok - t0 : RED;
            if (warp < DW && healthy) {
                tc_fence_after();
                for (int c0 = 32 * (warp >> 2); c0 < nt; c0 += 8 * DW) {
                    uint32_t v[32];
                    tmem_ld32(my_tmem + (uint32_t)(t0 + c0), v);
                    tmem_ld_wait();
#pragma unroll
                    for (int i = 0; i < 32; ++i) red[(c0 + i) * GEMM_ROWS + r] = __uint_as_float(v[i]);
                }
            }
            __syncwarp();
            cluster_sync_all();
            if (warp < DW && healthy) {                                 // a lane takes four rows, a warp every DW-th token
                const int per = (nt + P.splits - 1) / P.splits;
                const int tk_end = min(nt, per * (split + 1));
                uint32_t src[GEMM_MAX_SPLITS];
#pragma unroll
                for (int s = 0; s < GEMM_MAX_SPLITS; ++s)
                    src[s] = map_to_rank(s0, s < P.splits ? (PAIR ? (rank & 1u) + 2u * s : (uint32_t)s) : rank) + (uint32_t)lane * 16u;
#pragma unroll 2
                for (int tk = per * split + warp; tk < tk_end; tk += DW) {
                    float4 v[GEMM_MAX_SPLITS];
#pragma unroll
                    for (int s = 0; s < GEMM_MAX_SPLITS; ++s)
                        if (s < P.splits) v[s] = ld_cluster_f4(src[s] + (uint32_t)tk * (GEMM_ROWS * 4u));
                    float sum[4] = {0.0f, 0.0f, 0.0f, 0.0f};
#pragma unroll
                    for (int s = 0; s < GEMM_MAX_SPLITS; ++s)
                        if (s < P.splits) { sum[0] += v[s].x; sum[1] += v[s].y; sum[2] += v[s].z; sum[3] += v[s].w; }
                    const size_t at = (size_t)(m0 + t0 + tk) * ldy + row0;
                    if (y32) {
                        if (wide) *reinterpret_cast<float4*>(y32 + at) = make_float4(sum[0], sum[1], sum[2], sum[3]);
                        else
                            for (int i = 0; i < 4; ++i)
                                if (row0 + i < K) y32[at + i] = sum[i];
                    } else if (wide) {
                        uint2 o;
                        o.x = finish_output(sum[0], bias, row0) | ((uint32_t)finish_output(sum[1], bias, row0 + 1) << 16);
                        o.y = finish_output(sum[2], bias, row0 + 2) | ((uint32_t)finish_output(sum[3], bias, row0 + 3) << 16);
                        *reinterpret_cast<uint2*>(y + at) = o;
                    } else {
                        for (int i = 0; i < 4; ++i)
                            if (row0 + i < K) y[at + i] = finish_output(sum[i], bias, row0 + i);
                    }
                }
            }
            __syncwarp();
            cluster_sync_all();                                         // nobody overwrites or leaves while a neighbour still reads
        }
    }
    tc_fence_before();
    __syncwarp();
    if (PAIR) cluster_sync_all();                                       // the pair frees its tensor memory together
    else __syncthreads();
    if (warp == DW + 1) { tc_fence_after(); tmem_dealloc<PAIR>(tmem_d, TMEM_COLS); }
}

}  // namespace cb
