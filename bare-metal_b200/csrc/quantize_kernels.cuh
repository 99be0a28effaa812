// quantize_kernels.cuh — per-token dynamic quantisation fp16 -> int8, the step BEFORE the W8A8 GEMM.
//
// The reference's online-quant kernels (kernels/gemm/igemm/igemm_online_quant*.cu) take fp16 operands
// and quantise them tile by tile inside the GEMM with scale = max|x| / 127 (igemm_online_quant.cu:66-120).
// On B200 the W8A8 kernels want int8 operands with one fp32 scale per token, so the quantisation is
// its own HBM-bound pass with the arithmetic of the reference's host quantiser
// (kernels/gemm/igemm/bench.cu:28-51) applied per row:
//     scale[m] = max_k |x[m][k]| / 127   (1 if the row is all zero)
//     q[m][k]  = clamp((int)roundf(x[m][k] * (1 / scale[m])), -128, 127)
// The row is read once (16-byte loads, kept in registers while the maximum is reduced) and written once:
// 3 bytes of HBM traffic per element, which bound it from a few hundred rows up; below that it is one memory round
// trip plus a thread's own work.  Measured back to back on inputs beyond L2, against one warp per row with the row in its
// registers (16 warps an SM, rows beyond 4096 read twice): 8192 x 4096 21.0 -> 17.0 us (5.9 TB/s; 18.7 in bench.py), 8192 x
// 11008 70.2 -> 45, 777 x 11008 15.2 -> 7.3, 16 x 4096 3.8 -> 1.9, 16 x 11008 9.0 -> 2.4.
#pragma once
#include <cstdint>
#include <cuda_fp16.h>

#include "sm100_ptx.cuh"

namespace bm {

constexpr int kQuantMaxThreads = 1024;         // threads of a row group at most

// Largest |x| of 8 halves as the bits of a half, both 16-bit lanes at once: without their signs the bits of
// halves order like integers, infinities above every number and NaNs above those.
__device__ __forceinline__ uint32_t half_bits_max(uint32_t m, const uint4& d) {
    m = __vmaxu2(m, d.x & 0x7FFF7FFFu);
    m = __vmaxu2(m, d.y & 0x7FFF7FFFu);
    m = __vmaxu2(m, d.z & 0x7FFF7FFFu);
    return __vmaxu2(m, d.w & 0x7FFF7FFFu);
}

// Largest |x| that is not a NaN (what fmaxf leaves), for rows that hold infinities or NaNs.
__device__ __forceinline__ float half_max_skip_nan(float m, const uint4& d) {
    const __half2* h = reinterpret_cast<const __half2*>(&d);
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const float2 f = __half22float2(h[j]);
        m = fmaxf(m, fmaxf(fabsf(f.x), fabsf(f.y)));
    }
    return m;
}

// Four finite halves with |x * inv| < 128 (two words) -> four int8, rounded half away from zero.  With the unit of
// the last place of 2^15 at 2^-8, the truncating sum |y| + (2^15 + 1/2) carries floor(|y| + 1/2) in the
// second byte of its bits; the sign returns in all four bytes at once (two's complement without carries
// between bytes).  5 instructions an element instead of about 14 with roundf, a conversion and a clamp.
__device__ __forceinline__ uint32_t quant4_half_away(uint32_t w0, uint32_t w1, float inv) {
    const float2 a = __half22float2(*reinterpret_cast<const __half2*>(&w0));
    const float2 b = __half22float2(*reinterpret_cast<const __half2*>(&w1));
    constexpr float kBase = 32768.5f;
    const uint32_t z0 = __float_as_uint(__fadd_rz(fabsf(__fmul_rn(a.x, inv)), kBase));
    const uint32_t z1 = __float_as_uint(__fadd_rz(fabsf(__fmul_rn(a.y, inv)), kBase));
    const uint32_t z2 = __float_as_uint(__fadd_rz(fabsf(__fmul_rn(b.x, inv)), kBase));
    const uint32_t z3 = __float_as_uint(__fadd_rz(fabsf(__fmul_rn(b.y, inv)), kBase));
    const uint32_t mag = __byte_perm(__byte_perm(z0, z1, 0x0051), __byte_perm(z2, z3, 0x0051), 0x5410);
    uint32_t neg;                                                       // 0xFF in the bytes of negative inputs
    asm("prmt.b32 %0, %1, %2, 0xFDB9;" : "=r"(neg) : "r"(w0), "r"(w1));
    const uint32_t t = mag ^ neg;
    return ((t & 0x7F7F7F7Fu) + (neg & 0x01010101u)) ^ (t & 0x80808080u);
}

// The same for any input (NaN gives 0, as the conversion to int does).
__device__ __forceinline__ uint32_t quant4_any(uint32_t w0, uint32_t w1, float inv) {
    const uint32_t in[2] = {w0, w1};
    uint32_t packed = 0;
#pragma unroll
    for (int j = 0; j < 4; ++j) {
        const __half h = __ushort_as_half(static_cast<unsigned short>(in[j >> 1] >> (16 * (j & 1))));
        int r = static_cast<int>(roundf(__fmul_rn(__half2float(h), inv)));
        r = r > 127 ? 127 : (r < -128 ? -128 : r);
        packed |= (static_cast<uint32_t>(r) & 0xFFu) << (8 * j);
    }
    return packed;
}

// A group of blockDim.x threads per row, blockDim.y rows per CTA (more than one only where a group is one warp);
// each thread holds up to HELD 16-byte pieces of its row.
template <int HELD>
__global__ void __launch_bounds__(HELD == 4 ? 512 : kQuantMaxThreads)
quantize_rows_f16_kernel(const __half* __restrict__ x, int8_t* __restrict__ q, float* __restrict__ scale, int M, int K) {
    __shared__ uint32_t warp_bits[kQuantMaxThreads / 32];
    __shared__ float warp_max[kQuantMaxThreads / 32];
    const int row = blockIdx.x * blockDim.y + threadIdx.y;
    const int tid = threadIdx.x, group = blockDim.x;
    pdl_launch_dependents();      // the GEMM behind this kernel may start its own set-up
    if (row >= M) return;                          // whole warps: a CTA of several rows has one-warp groups
    const uint4* src = reinterpret_cast<const uint4*>(x + static_cast<size_t>(row) * K);
    const int vecs = K / 8;                        // K % 16 == 0

    uint4 held[HELD];
#pragma unroll
    for (int i = 0; i < HELD; ++i) {
        const int v = tid + i * group;
        held[i] = v < vecs ? __ldg(src + v) : make_uint4(0, 0, 0, 0);
    }
    uint32_t bits2 = 0;
#pragma unroll
    for (int i = 0; i < HELD; ++i) bits2 = half_bits_max(bits2, held[i]);
    for (int v = tid + HELD * group; v < vecs; v += group) bits2 = half_bits_max(bits2, __ldg(src + v));   // very long rows
    uint32_t bits = max(bits2 & 0xFFFFu, bits2 >> 16);
    bits = __reduce_max_sync(0xFFFFFFFFu, bits);
    if (group > 32) {
        if ((tid & 31) == 0) warp_bits[tid >> 5] = bits;
        __syncthreads();
        for (int w = 0; w < group / 32; ++w) bits = max(bits, warp_bits[w]);
    }
    const bool finite = bits < 0x7C00u;
    float mx = __half2float(__ushort_as_half(static_cast<unsigned short>(bits)));
    if (!finite) {                                 // uniform in the row group
        mx = 0.f;
#pragma unroll
        for (int i = 0; i < HELD; ++i) mx = half_max_skip_nan(mx, held[i]);
        for (int v = tid + HELD * group; v < vecs; v += group) mx = half_max_skip_nan(mx, __ldg(src + v));
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) mx = fmaxf(mx, __shfl_xor_sync(0xFFFFFFFFu, mx, o));
        if (group > 32) {
            if ((tid & 31) == 0) warp_max[tid >> 5] = mx;
            __syncthreads();
            for (int w = 0; w < group / 32; ++w) mx = fmaxf(mx, warp_max[w]);
        }
    }

    const float s = mx == 0.f ? 1.0f : __fdiv_rn(mx, 127.0f);
    const float inv = __fdiv_rn(1.0f, s);
    if (tid == 0) scale[row] = s;

    uint2* dst = reinterpret_cast<uint2*>(q + static_cast<size_t>(row) * K);
    auto emit = [&](const uint4& d, int v) {
        dst[v] = finite ? make_uint2(quant4_half_away(d.x, d.y, inv), quant4_half_away(d.z, d.w, inv))
                        : make_uint2(quant4_any(d.x, d.y, inv), quant4_any(d.z, d.w, inv));
    };
#pragma unroll
    for (int i = 0; i < HELD; ++i) {
        const int v = tid + i * group;
        if (v < vecs) emit(held[i], v);
    }
    for (int v = tid + HELD * group; v < vecs; v += group) emit(__ldg(src + v), v);   // second read hits L2
}

}  // namespace bm
