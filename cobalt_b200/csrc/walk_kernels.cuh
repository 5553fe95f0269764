// One-thread-per-segment kernels: RAW recovery, dense dequantisation and a plain GEMV.
// They read the tile image straight from global memory and walk the 128 positions of a
// segment bit by bit; they are the simple, obviously-correct side of the library.
#pragma once
#include "common.cuh"

namespace cb {

// 64 threads per block = the 16 x 4 segments of one tile; thread t <-> (row r = t/4, group gi = t%4).
// Returns the index of the thread's first survivor code within the tile and the tile pointers.
struct SegCtx {
    const uint32_t* mask;      // 4 words, valid when active
    const uint32_t* stream;    // code stream of the tile
    uint32_t sz;               // {scale, zero} bits
    uint32_t first;            // rank of the first survivor of this segment within the tile
    bool active;
    int w;
};

__device__ __forceinline__ SegCtx open_segment(const MatView& W, int rb, int ct, uint32_t* sh_cnt /*[64]*/) {
    SegCtx c;
    const int t = threadIdx.x, r = t >> 2, gi = t & 3;
    c.w = tile_width(W, ct);
    c.active = gi < c.w;
    const uint8_t* tile = W.tiles + (size_t)W.tile_off[rb * W.CT + ct] * 16;
    const int seg = r * c.w + gi;
    c.mask = (const uint32_t*)tile + seg * 4;
    c.stream = (const uint32_t*)(tile + TILE_ROWS * c.w * 20);
    uint32_t cnt = 0;
    c.sz = 0;
    if (c.active) {
        cnt = __popc(c.mask[0]) + __popc(c.mask[1]) + __popc(c.mask[2]) + __popc(c.mask[3]);
        c.sz = ((const uint32_t*)(tile + TILE_ROWS * c.w * 16))[seg];
    }
    __syncthreads();                 // protect sh_cnt against the previous tile's readers
    sh_cnt[t] = cnt;
    __syncthreads();
    uint32_t first = 0;
    for (int i = 0; i < t; ++i) first += sh_cnt[i];     // thread order == segment order among active threads
    c.first = first;
    return c;
}

// codes u8[K,N] (0 at pruned), keep u8[K,N], dense bf16[K,N]; any output may be null.
// One block of 8 warps per tile, a warp per segment, a lane per four columns: a warp writes whole 128-byte lines (256 for the
// dense weight), which is what bounds it.  4096 x 4096: 31 us; a thread per segment with byte stores took 223.
constexpr int UNPACK_THREADS = 256;
__global__ void __launch_bounds__(UNPACK_THREADS) unpack_kernel(MatView W, uint8_t* codes, uint8_t* keep, uint16_t* dense, int wide) {
    __shared__ uint32_t first_s[TILE_ROWS * TILE_GROUPS];
    const int ct = blockIdx.x, rb = blockIdx.y, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int w = tile_width(W, ct), nseg = TILE_ROWS * w;
    const uint8_t* tile = W.tiles + (size_t)W.tile_off[(size_t)rb * W.CT + ct] * 16;
    if (warp == 0) {                                                   // rank of every segment's first survivor, two segments per lane
        uint32_t c[2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            c[k] = 0;
            if (2 * lane + k < nseg) {
                const uint4 m = __ldg(reinterpret_cast<const uint4*>(tile) + 2 * lane + k);
                c[k] = __popc(m.x) + __popc(m.y) + __popc(m.z) + __popc(m.w);
            }
        }
        uint32_t inc = c[0] + c[1];
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) { const uint32_t up = __shfl_up_sync(0xFFFFFFFFu, inc, d); if (lane >= d) inc += up; }
        first_s[2 * lane] = inc - c[0] - c[1];
        first_s[2 * lane + 1] = inc - c[1];
    }
    __syncthreads();
    const uint32_t* stream = reinterpret_cast<const uint32_t*>(tile + nseg * 20);
    for (int seg = warp; seg < nseg; seg += UNPACK_THREADS / 32) {
        const int row = rb * TILE_ROWS + seg / w;
        if (row >= W.K) continue;
        const int col = (ct * TILE_GROUPS + seg % w) * GROUP + 4 * lane;
        const uint4 m = __ldg(reinterpret_cast<const uint4*>(tile) + seg);
        const uint32_t sz = __ldg(reinterpret_cast<const uint32_t*>(tile + nseg * 16) + seg);
        const int j = lane >> 3, sh = 4 * (lane & 7);
        const uint32_t mj = j == 0 ? m.x : j == 1 ? m.y : j == 2 ? m.z : m.w;
        uint32_t rank = first_s[seg] + __popc(mj & ((1u << sh) - 1u));
        if (j > 0) rank += __popc(m.x);
        if (j > 1) rank += __popc(m.y);
        if (j > 2) rank += __popc(m.z);
        const uint32_t nib = (mj >> sh) & 15u, bit = rank * (uint32_t)W.bits, cmask = (1u << W.bits) - 1u;
        uint32_t v = funnel_r(__ldg(stream + (bit >> 5)), __ldg(stream + (bit >> 5) + 1), bit);       // the image ends in slack words
        const float s = half_bits_to_float(sz & 0xFFFFu), z = half_bits_to_float(sz >> 16);
        uint32_t code4 = 0, keep4 = 0, d[4];
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const uint32_t kept = (nib >> b) & 1u, code = kept ? v & cmask : 0u;
            if (kept) v >>= W.bits;
            code4 |= code << (8 * b);
            keep4 |= kept << (8 * b);
            if (dense) {
                const float cs = W.col_scale ? half_bits_to_float(W.col_scale[col + b]) : 1.0f;
                // literal reference order: ((q - z) * s) * col_scale, then * keep, then one cast
                d[b] = float_to_bf16(__fmul_rn(dequant_fp32((float)code, z, s, cs), (float)kept));
            }
        }
        const size_t o = (size_t)row * W.N + col;
        if (!wide) {                                                   // outputs at odd addresses: one element at a time
#pragma unroll
            for (int b = 0; b < 4; ++b) {
                if (codes) codes[o + b] = (uint8_t)(code4 >> (8 * b));
                if (keep) keep[o + b] = (uint8_t)(keep4 >> (8 * b));
                if (dense) dense[o + b] = (uint16_t)d[b];
            }
            continue;
        }
        if (codes) *reinterpret_cast<uint32_t*>(codes + o) = code4;
        if (keep) *reinterpret_cast<uint32_t*>(keep + o) = keep4;
        if (dense) *reinterpret_cast<uint2*>(dense + o) = make_uint2(d[0] | (d[1] << 16), d[2] | (d[3] << 16));
    }
}

// y[m,k] = bf16( sum_j bf16(W[k,j]) * x[m,j] + bias[k] ), one block of 64 threads per row block
template <int MM>
__global__ void __launch_bounds__(64) gemv_rowwalk_kernel(MatView W, const uint16_t* x, int64_t ldx, uint16_t* y,
                                                          int64_t ldy, const uint16_t* bias, int M) {
    __shared__ uint32_t sh_cnt[64];
    const int rb = blockIdx.x;
    const int r = threadIdx.x >> 2, gi = threadIdx.x & 3;
    const int row = rb * TILE_ROWS + r;
    float acc[MM];
#pragma unroll
    for (int m = 0; m < MM; ++m) acc[m] = 0.0f;
    for (int ct = 0; ct < W.CT; ++ct) {
        SegCtx c = open_segment(W, rb, ct, sh_cnt);
        if (!c.active) continue;
        const int col0 = (ct * TILE_GROUPS + gi) * GROUP;
        const float s = half_bits_to_float(c.sz & 0xFFFFu), z = half_bits_to_float(c.sz >> 16);
        uint32_t bitpos = c.first * (uint32_t)W.bits;
        for (int j = 0; j < 4; ++j) {
            uint32_t m = c.mask[j];
            while (m) {
                const int b = __ffs(m) - 1;
                m &= m - 1;
                const int col = col0 + 32 * j + b;
                const uint32_t code = extract_code(c.stream, bitpos, W.bits);
                bitpos += W.bits;
                const float cs = W.col_scale ? half_bits_to_float(W.col_scale[col]) : 1.0f;
                const float wv = bf16_to_float(float_to_bf16(dequant_fp32((float)code, z, s, cs)));
#pragma unroll
                for (int mm = 0; mm < MM; ++mm)
                    if (mm < M) acc[mm] = fmaf(wv, bf16_to_float(x[(size_t)mm * ldx + col]), acc[mm]);
            }
        }
    }
#pragma unroll
    for (int mm = 0; mm < MM; ++mm) {
        float v = acc[mm];
        v += __shfl_xor_sync(0xFFFFFFFFu, v, 1);
        v += __shfl_xor_sync(0xFFFFFFFFu, v, 2);
        if (gi == 0 && mm < M && row < W.K) {
            if (bias) v += bf16_to_float(bias[row]);
            y[(size_t)mm * ldy + row] = float_to_bf16(v);
        }
    }
}

}  // namespace cb
