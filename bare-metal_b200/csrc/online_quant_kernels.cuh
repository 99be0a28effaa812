// online_quant_kernels.cuh — the quantisation step of the reference's FP16-in GEMMs
// (kernels/gemm/igemm/igemm_online_quant.cu and its _inplace / _bankfree / _bf_128x256 /
// warp_specialized variants), restated as two streaming kernels in front of the tcgen05 GEMM.
//
// What the reference computes (igemm_online_quant.cu:66-142,255,393): every thread block owns a
// 128 x 128 output tile (128 x 256 in _bf_128x256).  It takes max|A| over its 128 rows x the FIRST
// 32 columns of K and max|B| over the first 32 rows of K x its 128 (256) columns, sets
// inv = 127 / max (1 if max == 0), and quantises EVERY K tile with those two factors
// (QUANTIZE_TILE on tile 0, QUANTIZE_TILE_FAST afterwards): q = clamp(rint(x * inv), -128, 127).
// Each K tile's int32 sum is folded into an fp32 accumulator with tile_scale =
// (max_a / 127) * (max_b / 127).  So the scales are per 128-row block of A and per 128 (256)
// column block of B — a block-scaled W8A8 GEMM whose int32 sums can be kept exactly over all of K
// and multiplied by tile_scale once.
#pragma once
#include <cstdint>
#include <cuda_fp16.h>

#include "sm100_ptx.cuh"

namespace bm {

constexpr int kOqRowBlock = 128;
constexpr int kOqKTile = 32;

// One launch does both steps.  A CTA of 512 (256) threads owns a chunk of 32768 (16384) elements inside ONE scale block —
// 128 rows x 256 (128) columns of A, or 256 or 128 (128 or 64) rows x 128 or 256 columns of B.  It asks for its whole chunk
// first, 64 elements a thread in registers, then takes the block's maximum over the first K tile itself (4096 / 8192 elements, an
// L2 hit for all but the first CTA of a block) while those loads are under way, and converts: two
// 16-byte loads and one 16-byte store per 16 elements.  The CTAs of chunk 0 also publish the dequantisation scale
// max / 127 per row / column for the GEMM epilogue.
// K % 16 == 0 and N % 16 == 0, so a 16-element unit never straddles an edge.
// Bound by HBM: 3 bytes per element (the GEMM behind it takes the rest of the time at the larger sizes).  With both steps,
// before (256 threads, loads after the maximum, conversions of ~14 instructions an element) -> now: 256^3 10.2 ->
// 7.7 us, 512 x 512 x 4096 15.7 -> 13.3, 8192 x 512 x 512 14.8 -> 12.5, 4096^3 (the GEMM under the power cap) 73.4 -> 69.3.
//
// With 62 registers a thread an SM holds 1024 threads.  Chunks of 32768 are for what the SMs take in at once: beyond that,
// CTAs of 512 threads came in waves of which the last was partly empty, and the call was slower than with the 256 threads
// that loaded after the maximum.  Those, 512 threads, 256 threads now: 8192 x 512 x 8192 69.7, 72.7, 66.5 us; 3000 x 1024 x
// 8192 48.5, 50.0, 46.4; 8192 x 512 x 4096 39.1, 41.2, 37.1; 8192 x 1024 x 8192 92.6, 94.6, 89.1; 4096^3 73.4, 71.9, 69.3.
// Within one wave the larger chunks read the maximum's window less often: 4096 x 16 x 2048 15.7 against 17.3, 8192 x 16 x 1024
// 17.4 against 18.5.
constexpr int kOqUnits = 4;                                    // 16-element units a thread holds
constexpr int kOqResidentThreads = 1024;                       // of an SM, with the registers that takes
template <int THREADS>
struct OqCfg {
    static constexpr int CHUNK = THREADS * kOqUnits * 16;
    static constexpr int A_COLS = CHUNK / kOqRowBlock;
    static constexpr int A_UNITS_LOG = A_COLS == 256 ? 4 : 3;  // units of a chunk's row of A
    static_assert(A_COLS == 256 || A_COLS == 128, "chunk of A");
};

struct OqUnit {
    uint4 lo, hi;
};

__device__ __forceinline__ OqUnit oq_load(const __half* p) {
    return {__ldg(reinterpret_cast<const uint4*>(p)), __ldg(reinterpret_cast<const uint4*>(p) + 1)};
}

__device__ __forceinline__ float oq_unit_max(const OqUnit& u) {
    const uint32_t in[8] = {u.lo.x, u.lo.y, u.lo.z, u.lo.w, u.hi.x, u.hi.y, u.hi.z, u.hi.w};
    float m = 0.f;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const __half2 h = *reinterpret_cast<const __half2*>(&in[j]);
        m = fmaxf(m, fmaxf(fabsf(__low2float(h)), fabsf(__high2float(h))));
    }
    return m;
}

// q = clamp(rint(x * inv), -128, 127), NaN -> 0.  Rounding by adding 1.5 * 2^23: the sum's low byte is the integer,
// ties to even like rint; values beyond the type are clamped before, in a form that keeps NaNs, and a NaN shows in
// a bit that no sum has (a unit that holds one takes the conversions instead).
__device__ __forceinline__ uint4 oq_unit_convert(const OqUnit& u, float inv) {
    const uint32_t in[8] = {u.lo.x, u.lo.y, u.lo.z, u.lo.w, u.hi.x, u.hi.y, u.hi.z, u.hi.w};
    constexpr float kMagic = 12582912.f;
    uint32_t out[4], seen = 0;
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        uint32_t z[4];
#pragma unroll
        for (int j = 0; j < 2; ++j) {
            const float2 f = __half22float2(*reinterpret_cast<const __half2*>(&in[2 * g + j]));
            const float y0 = __fmul_rn(f.x, inv), y1 = __fmul_rn(f.y, inv);
            float c0, c1;
            asm("max.NaN.f32 %0, %1, 0fC3000000;" : "=f"(c0) : "f"(y0));          // -128
            asm("max.NaN.f32 %0, %1, 0fC3000000;" : "=f"(c1) : "f"(y1));
            asm("min.NaN.f32 %0, %1, 0f42FE0000;" : "=f"(c0) : "f"(c0));          // 127
            asm("min.NaN.f32 %0, %1, 0f42FE0000;" : "=f"(c1) : "f"(c1));
            z[2 * j] = __float_as_uint(__fadd_rn(c0, kMagic));
            z[2 * j + 1] = __float_as_uint(__fadd_rn(c1, kMagic));
        }
        seen |= z[0] | z[1] | z[2] | z[3];
        out[g] = __byte_perm(__byte_perm(z[0], z[1], 0x0040), __byte_perm(z[2], z[3], 0x0040), 0x5410);
    }
    if (seen & 0x10000000u) {                    // sums are 0x4B3FFF80 .. 0x4B40007F, a NaN is 0x7F......
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const __half h = __ushort_as_half(static_cast<unsigned short>((in[j >> 1] >> (16 * (j & 1))) & 0xFFFFu));
            const int q = max(-128, min(127, __float2int_rn(__fmul_rn(__half2float(h), inv))));
            out[j >> 2] = (out[j >> 2] & ~(0xFFu << (8 * (j & 3)))) | (static_cast<uint32_t>(q) & 0xFFu) << (8 * (j & 3));
        }
    }
    return make_uint4(out[0], out[1], out[2], out[3]);
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS, kOqResidentThreads / THREADS)
oq_quantize_kernel(const __half* __restrict__ A, const __half* __restrict__ B, int8_t* __restrict__ Aq,
                   int8_t* __restrict__ Bq, float* __restrict__ row_scale, float* __restrict__ col_scale, int M, int N,
                   int K, int col_block, int chunks_a, int a_chunks_per_block, int b_chunks_per_block) {
    using Cfg = OqCfg<THREADS>;
    __shared__ float warp_max[THREADS / 32];
    pdl_launch_dependents();      // the GEMM behind this kernel may start its own set-up
    const int kt = K < kOqKTile ? K : kOqKTile;
    const int tid = threadIdx.x;
    const bool is_a = static_cast<int>(blockIdx.x) < chunks_a;
    const int id = is_a ? blockIdx.x : blockIdx.x - chunks_a;
    const int per = is_a ? a_chunks_per_block : b_chunks_per_block;
    const int blk = id / per, chunk = id % per;
    // operand-independent view: `rows` x `cols` matrix, the chunk at (r0, c0) is ch_rows x 2^units_log units of 16
    // columns, the first-K-tile window at (w_r0, w_c0) is w_rows x w_cols
    const __half* X = is_a ? A : B;
    int8_t* Xq = is_a ? Aq : Bq;
    const int rows = is_a ? M : K, cols = is_a ? K : N;
    const int units_log = is_a ? Cfg::A_UNITS_LOG : col_block == 256 ? 4 : 3;
    const int ch_rows = (Cfg::CHUNK / 16) >> units_log;
    const int r0 = is_a ? blk * kOqRowBlock : chunk * ch_rows, c0 = is_a ? chunk * Cfg::A_COLS : blk * col_block;
    const int w_r0 = is_a ? r0 : 0, w_c0 = is_a ? 0 : c0;
    const int w_rows = is_a ? kOqRowBlock : kt, w_cols = is_a ? kt : col_block;

    // a thread's units lie below one another, `step` rows apart
    const int first_r = r0 + (tid >> units_log), my_c = c0 + (tid & ((1 << units_log) - 1)) * 16;
    const int step = THREADS >> units_log;
    const int mine = my_c < cols ? rows - first_r : 0;     // unit i exists if i * step < mine
    const size_t at = static_cast<size_t>(first_r) * cols + my_c, pitch = static_cast<size_t>(step) * cols;
    OqUnit held[kOqUnits];
#pragma unroll
    for (int i = 0; i < kOqUnits; ++i)
        if (i * step < mine) held[i] = oq_load(X + at + i * pitch);

    const int w_log = is_a ? 1 : units_log;               // window units per row: 2 (of which K < 32 has one) or those of the chunk
    float m = 0.f;
    for (int u = tid; u < w_rows << w_log; u += THREADS) {
        const int r = w_r0 + (u >> w_log), c = w_c0 + (u & ((1 << w_log) - 1)) * 16;
        if (r < rows && c < cols && c < w_c0 + w_cols) m = fmaxf(m, oq_unit_max(oq_load(X + static_cast<size_t>(r) * cols + c)));
    }
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) m = fmaxf(m, __shfl_xor_sync(0xFFFFFFFFu, m, off));
    if ((tid & 31) == 0) warp_max[tid >> 5] = m;
    __syncthreads();
    float bmax = warp_max[0];
#pragma unroll
    for (int w = 1; w < THREADS / 32; ++w) bmax = fmaxf(bmax, warp_max[w]);
    const float inv = bmax > 0.f ? __fdiv_rn(127.0f, bmax) : 1.0f;
    if (chunk == 0) {
        const float scale = __fdiv_rn(bmax, 127.0f);
        float* dst = is_a ? row_scale : col_scale;
        const int first = is_a ? r0 : c0, count = is_a ? kOqRowBlock : col_block, limit = is_a ? M : N;
        for (int i = tid; i < count; i += THREADS)
            if (first + i < limit) dst[first + i] = scale;
    }
#pragma unroll
    for (int i = 0; i < kOqUnits; ++i)
        if (i * step < mine) *reinterpret_cast<uint4*>(Xq + at + i * pitch) = oq_unit_convert(held[i], inv);
}

}  // namespace bm
