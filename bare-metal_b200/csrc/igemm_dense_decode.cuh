// igemm_dense_decode.cuh — dense INT8 GEMM for few tokens: D^T = W * X^T, weights in the MMA's A slot.
//
// With at most 256 tokens the weights are most of the bytes and every one of them is used once, so the time is
// that of streaming W[N x K] — if all SMs stream.  The tiles of igemm_dense.cuh put 64 to 256 output channels
// on the accumulator columns: N = 4096 is then 64 CTAs on 148 SMs, each fetching a token tile that is
// mostly padding.  Here the output channels are the accumulator LANES, and a tile holds as many of them as it
// takes to give every SM the same share: h channels, any multiple of 8 up to 128 (N = 4096: 32 channels on 128
// SMs; N = 12288: 88 on 140).  The MMA always spans 128 lanes; what it reads beyond the tile's h rows (other
// ring bytes) lands in lanes nobody stores.  Tokens are the accumulator columns, rounded up to 16.
//
// An MMA takes at least 57 clocks however few tokens it has (measured with the operands resident; half a clock per
// column where that is more), so K = 4096 in steps of 32 is 3.9 us of MMAs — more than
// the 2.6 us that 4096 x 4096 weights take from HBM.  Tiles of at most 64 channels therefore FOLD K: the
// stage's chunks lie in shared memory one after the other, [chunk][h rows][128 B], which is also a
// matrix of chunk * h rows; `fold` chunks of W stacked on the 128 lanes against `fold` chunks of X stacked on
// the columns are ONE MMA whose diagonal blocks — channels of chunk i against tokens of chunk i — are the
// partial sums of `fold` K ranges (the other blocks are never read).  The epilogue adds the `fold` partial
// sums, exact integers, through shared memory.  A folded CTA has one tile: more than one tile per SM means tiles of 72
// channels or more, which do not fold.
//
// A ring stage covers `chunks` K blocks of 128 bytes, a multiple of `fold`.  W and X are described to the TMA as
// [K / 128][rows][128 B], so one copy fetches all chunks of an operand's stage: a 32-row box of one chunk is only
// 4 KiB (chunks that do not exist arrive as zeros).  The ragged chunk of a K that is not a multiple of 128 is a stage of its
// own, the last of every tile: one copy per operand through a plain 2-D map, which zero-fills beyond K, and MMAs without
// folding, whose sums join those of the first K range.  (As part of the last stage it took a copy per chunk of that stage
// and operand and a folded MMA for the one chunk: 1024 x 1040 with 16 / 32 tokens 5.1 / 5.3 us against 4.3 / 4.7.)  All
// stage geometry is a launch parameter: one instantiation per epilogue.
//
// What bounds it: the weights' stream from HBM (28672 x 8192, 1 token: 35.5 us = 6.6 TB/s) plus ~3.2 us of launch, ramp and
// drain; with many tokens what one SM can take in of both operands.  16 tokens, before (wide tiles) -> without folding ->
// folded -> with copies and MMAs from an elected lane: 4096 x 4096 14.4 -> 10.3 -> 7.0 -> 5.9 us, 4096 x 11008 25.0 -> 22.4 ->
// 12.1 -> 9.9, 12288 x 4096 20.3 -> 12.5 -> 12.6 (88 channels a tile: no fold) -> 10.2, 512 x 4096 10.1 -> 8.3 -> 4.7 -> 3.9.
//
// Every CTA starts its K walk at another stage and wraps around (exact integer sums do not depend on the
// order), so the CTAs do not ask the L2 for the same activations at the same moment.
#pragma once
#include "epilogue.cuh"
#include "igemm_dense.cuh"
#include "sm100_ptx.cuh"

namespace bm {

constexpr int kDdMaxTokens = 256;
constexpr int kDdMaxStages = 12;
constexpr int kDdRingBytes = 176 * 1024;
constexpr int kDdPartInts = 8192;                         // partial sums of a folded tile: fold * h * padded tokens
constexpr int kDdThreads = 96 + 32 * kEpiWarps;           // W producer, MMA issuer, epilogue warps, X producer
constexpr int kDdBarOffset = kDdRingBytes;
constexpr int kDdStripOffset = kDdBarOffset + (2 * kDdMaxStages + 6) * 8 + 24;
constexpr int kDdPartOffset = (kDdStripOffset + kEpiWarps * kDdMaxTokens * 4 + 127) / 128 * 128;
constexpr int kDdSmemBytes = kDdPartOffset + kDdPartInts * 4 + 1024;
static_assert(kDdSmemBytes <= 227 * 1024, "shared memory over-subscribed");

struct DenseDecodeParams {
    EpilogueParams epi;                // out [rows = tokens x cols = channels]
    int tiles, tile_rows;              // channels per tile (h)
    int tokens_padded;                 // accumulator columns in use: tokens rounded up to 16
    int fold;                          // K blocks side by side in one MMA (1: none); above 1 only with tiles <= grid
    int acc_stride, tmem_cols;         // columns between the two accumulators; columns allocated
    int chunks, stages;                // K blocks of 128 bytes per ring stage; ring stages
    int full_chunks;                   // K blocks entirely inside K
    int full_stages, k_stages;         // stages that cover these; one more where K ends inside a block
    int* status;
};

template <int EPI>
__global__ void __launch_bounds__(kDdThreads, 1)
igemm_dense_decode_kernel(const __grid_constant__ CUtensorMap map_w3, const __grid_constant__ CUtensorMap map_w2,
                          const __grid_constant__ CUtensorMap map_x3, const __grid_constant__ CUtensorMap map_x2,
                          const DenseDecodeParams p) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem_base = (smem_u32(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem_gen = smem_raw + (smem_base - smem_u32(smem_raw));

    const uint32_t w_chunk = static_cast<uint32_t>(p.tile_rows) * 128u;          // multiples of 1 KiB
    const uint32_t x_chunk = static_cast<uint32_t>(p.tokens_padded) * 128u;
    const uint32_t w_stage = w_chunk * p.chunks, x_stage = x_chunk * p.chunks;
    const uint32_t w_smem0 = smem_base;
    const uint32_t x_smem0 = w_smem0 + w_stage * p.stages;
    const uint32_t bar0 = smem_base + kDdBarOffset;
    auto full_bar = [&](int s) { return bar0 + 8u * s; };
    auto empty_bar = [&](int s) { return bar0 + 8u * (kDdMaxStages + s); };
    auto acc_full_bar = [&](int a) { return bar0 + 8u * (2 * kDdMaxStages + a); };
    auto acc_empty_bar = [&](int a) { return bar0 + 8u * (2 * kDdMaxStages + 2 + a); };
    const uint32_t drain_bar = bar0 + 8u * (2 * kDdMaxStages + 4);
    const uint32_t parked_bar = bar0 + 8u * (2 * kDdMaxStages + 5);   // folded tile: partial sums written
    const uint32_t tmem_slot = bar0 + 8u * (2 * kDdMaxStages + 6);
    volatile uint32_t* tmem_slot_gen =
        reinterpret_cast<volatile uint32_t*>(smem_gen + kDdBarOffset + 8 * (2 * kDdMaxStages + 6));
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot_gen + 1);

    const int warp = __shfl_sync(0xFFFFFFFFu, threadIdx.x >> 5, 0);      // known to be the same in all lanes
    const int lane = threadIdx.x & 31;
    const uint32_t nstages = static_cast<uint32_t>(p.stages);
    const int rot = p.full_stages > 0 ? static_cast<int>((blockIdx.x * 7u) % static_cast<unsigned>(p.full_stages)) : 0;
    auto k_stage_of = [&](int i) { const int k = i + rot; return k < p.full_stages ? k : k - p.full_stages; };

    if (threadIdx.x == 0) {
        for (int s = 0; s < p.stages; ++s) {
            mbar_init(full_bar(s), 1);
            mbar_init(empty_bar(s), 1);
        }
        for (int a = 0; a < 2; ++a) {
            mbar_init(acc_full_bar(a), 1);
            mbar_init(acc_empty_bar(a), kEpiWarps);
        }
        mbar_init(drain_bar, 1);
        mbar_init(parked_bar, kEpiWarps);
        *abort_flag = 0;
        fence_mbar_init();
    }
    if (warp == 1) {
        tmem_alloc(tmem_slot, p.tmem_cols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = *tmem_slot_gen;
    pdl_launch_dependents();      // the next kernel of the stream may start its own set-up
    pdl_wait_prior_grid();        // nothing global is touched before the previous grid is complete

    if (warp == 0 || warp == 2 + kEpiWarps) {
        // ------------------------------------------------------------------ producers: weights, activations
        const bool is_w = warp == 0;
        const CUtensorMap* map3 = is_w ? &map_w3 : &map_x3;
        const CUtensorMap* map2 = is_w ? &map_w2 : &map_x2;
        prefetch_tensormap(map3);
        if (p.k_stages > p.full_stages) prefetch_tensormap(map2);
        const uint32_t base = is_w ? w_smem0 : x_smem0, stage_bytes = is_w ? w_stage : x_stage;
        uint32_t stage = 0, phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < p.tiles; tile += gridDim.x) {
            const int row0 = is_w ? tile * p.tile_rows : 0;
            for (int i = 0; i < p.k_stages; ++i) {
                if (!warp_bounded_wait(empty_bar(stage), phase ^ 1u, abort_flag, p.status,
                                  DEV_TIMEOUT_PRODUCER_EMPTY)) { ok = false; break; }
                const uint32_t bar = full_bar(stage);
                const uint32_t dst = base + stage * stage_bytes;
                if (elect_one()) {
                    if (i < p.full_stages) {
                        if (is_w) mbar_expect_tx(bar, w_stage + x_stage);   // both operands
                        tma_load_3d(dst, map3, bar, 0, row0, k_stage_of(i) * p.chunks);
                    } else {
                        if (is_w) mbar_expect_tx(bar, w_chunk + x_chunk);
                        tma_load_2d(dst, map2, bar, p.full_chunks * 128, row0);
                    }
                }
                __syncwarp();
                if (++stage == nstages) { stage = 0; phase ^= 1u; }
            }
        }
    } else if (warp == 1) {
        // ------------------------------------------------------------------ MMA issuer
        const uint32_t idesc = make_idesc_i8(kBM, p.tokens_padded * p.fold, false, false);
        const uint32_t idesc_ragged = make_idesc_i8(kBM, p.tokens_padded, false, false);
        const uint64_t w_desc0 = make_smem_desc(w_smem0, 0, 1024, SWIZZLE_128B_DESC);
        const uint64_t x_desc0 = make_smem_desc(x_smem0, 0, 1024, SWIZZLE_128B_DESC);
        uint32_t stage = 0, phase = 0, acc = 0, acc_phase = 0;
        bool ok = true;
        for (int tile = blockIdx.x; ok && tile < p.tiles; tile += gridDim.x) {
            if (!warp_bounded_wait(acc_empty_bar(acc), acc_phase ^ 1u, abort_flag, p.status,
                              DEV_TIMEOUT_MMA_ACC_EMPTY)) { ok = false; break; }
            tc_fence_after_sync();
            const uint32_t d_tmem = tmem_base + acc * p.acc_stride;
            uint32_t accumulate = 0u;
            for (int i = 0; i < p.full_stages; ++i) {
                if (!warp_bounded_wait(full_bar(stage), phase, abort_flag, p.status, DEV_TIMEOUT_MMA_FULL)) {
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                if (elect_one()) {
                    uint64_t a_desc = w_desc0 + ((stage * w_stage) >> 4);         // addresses are in units of 16 bytes
                    uint64_t b_desc = x_desc0 + ((stage * x_stage) >> 4);
                    for (int c = 0; c < p.chunks; c += p.fold) {
#pragma unroll
                        for (int s = 0; s < kBK / kUmmaK; ++s)
                            mma_i8(d_tmem, a_desc + s * (kUmmaK >> 4), b_desc + s * (kUmmaK >> 4), idesc,
                                   (c | s) != 0 ? 1u : accumulate);
                        a_desc += (w_chunk * p.fold) >> 4;
                        b_desc += (x_chunk * p.fold) >> 4;
                    }
                    tc_commit(empty_bar(stage));
                }
                __syncwarp();
                accumulate = 1u;
                if (++stage == nstages) { stage = 0; phase ^= 1u; }
            }
            if (!ok) break;
            if (p.k_stages > p.full_stages) {                        // the ragged chunk
                if (!warp_bounded_wait(full_bar(stage), phase, abort_flag, p.status, DEV_TIMEOUT_MMA_FULL)) {
                    ok = false;
                    break;
                }
                tc_fence_after_sync();
                if (elect_one()) {
                    const uint64_t a_desc = w_desc0 + ((stage * w_stage) >> 4), b_desc = x_desc0 + ((stage * x_stage) >> 4);
#pragma unroll
                    for (int s = 0; s < kBK / kUmmaK; ++s)
                        mma_i8(d_tmem, a_desc + s * (kUmmaK >> 4), b_desc + s * (kUmmaK >> 4), idesc_ragged,
                               s != 0 ? 1u : accumulate);
                    tc_commit(empty_bar(stage));
                }
                __syncwarp();
                if (++stage == nstages) { stage = 0; phase ^= 1u; }
            }
            if (elect_one()) tc_commit(acc_full_bar(acc));
            __syncwarp();
            acc ^= 1u;
            if (acc == 0) acc_phase ^= 1u;
        }
        if (!ok) {
            if (elect_one()) tc_commit(drain_bar);
            __syncwarp();
            uint64_t t0 = global_timer_ns();
            while (!mbar_try_wait(drain_bar, 0) && global_timer_ns() - t0 < 20000000ull) {}
        }
    } else {
        // ------------------------------------------------------------------ epilogue warps
        using T = typename OutType<EPI>::type;
        const int quarter = warp & 3;                        // lanes 32q .. 32q+31 = channels of the tile
        const int half = (warp - 2) >> 2;                    // even / odd 32-token chunks
        float* strip = reinterpret_cast<float*>(smem_gen + kDdStripOffset) + (warp - 2) * kDdMaxTokens;
        int32_t* parts = reinterpret_cast<int32_t*>(smem_gen + kDdPartOffset);
        const int tokens = p.epi.rows;
        if constexpr (EPI == EPI_F16_ROWCOL) {
            for (int t = lane; t < tokens; t += 32) strip[t] = __ldg(p.epi.row_scale + t);
            __syncwarp();
        }
        uint32_t acc = 0, acc_phase = 0;
        for (int tile = blockIdx.x; tile < p.tiles; tile += gridDim.x) {
            const int in_tile = quarter * 32 + lane;
            const int channel = tile * p.tile_rows + in_tile;
            const bool live = in_tile < p.tile_rows && channel < p.epi.cols;
            float lane_s = 0.f;
            int lane_z = 0;
            if constexpr (EPI == EPI_F16_ROWCOL || EPI == EPI_F32_CHANNEL) lane_s = live ? __ldg(p.epi.col_scale + channel) : 0.f;
            if constexpr (EPI == EPI_F32_CHANNEL) lane_z = live ? __ldg(p.epi.col_zero + channel) : 0;
            if (!bounded_wait(acc_full_bar(acc), acc_phase, abort_flag, p.status, DEV_TIMEOUT_EPI_ACC_FULL))
                break;
            tc_fence_after_sync();
            if (p.fold > 1) {
                // lane = (K range, channel); column block = K range: park the diagonal blocks, then add them up
                const int range = in_tile / p.tile_rows, row = in_tile - range * p.tile_rows;
                const int first = quarter * 32 / p.tile_rows, last = (quarter * 32 + 31) / p.tile_rows;   // warp-uniform
                for (int rg = first; rg <= last && rg < p.fold; ++rg) {
                    const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) +
                                           acc * p.acc_stride + rg * p.tokens_padded;
                    for (int t0 = half * 16; t0 < p.tokens_padded; t0 += 32) {
                        uint32_t r[16];
                        tmem_ld_32x16(taddr + t0, r);
                        tmem_ld_wait();
                        if (range == rg) {
                            int32_t* dst = parts + (rg * p.tokens_padded + t0) * p.tile_rows + row;
#pragma unroll
                            for (int k = 0; k < 16; ++k) dst[k * p.tile_rows] = static_cast<int32_t>(r[k]);
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(parked_bar);
                if (!bounded_wait(parked_bar, 0, abort_flag, p.status, DEV_TIMEOUT_EPI_ACC_FULL)) break;
                const int part = p.tokens_padded * p.tile_rows;
                for (int c = lane; c < p.tile_rows; c += 32) {
                    const int ch = tile * p.tile_rows + c;
                    if (ch >= p.epi.cols) break;
                    float s = 0.f;
                    int z = 0;
                    if constexpr (EPI == EPI_F16_ROWCOL || EPI == EPI_F32_CHANNEL) s = __ldg(p.epi.col_scale + ch);
                    if constexpr (EPI == EPI_F32_CHANNEL) z = __ldg(p.epi.col_zero + ch);
                    for (int t = warp - 2; t < tokens; t += kEpiWarps) {
                        const int32_t* src = parts + t * p.tile_rows + c;
                        int32_t sum = 0;
                        for (int i = 0; i < p.fold; ++i) sum += src[i * part];
                        reinterpret_cast<T*>(p.epi.out)[static_cast<long long>(t) * p.epi.ld + ch] =
                            convert_acc<EPI>(sum, p.epi.tensor_scale, s, EPI == EPI_F16_ROWCOL ? strip[t] : s, z);
                    }
                }
                break;                                       // the CTA's only tile
            }
            if (quarter * 32 < p.tile_rows) {                                    // warp-uniform
                const uint32_t taddr = tmem_base + (static_cast<uint32_t>(quarter * 32) << 16) + acc * p.acc_stride;
                for (int t0 = half * 32; t0 < tokens; t0 += 64) {
                    uint32_t r[32];
                    tmem_ld_32x32(taddr + t0, r);
                    tmem_ld_wait();
                    T v[32];
#pragma unroll
                    for (int k = 0; k < 32; ++k)
                        v[k] = convert_acc<EPI>(static_cast<int32_t>(r[k]), p.epi.tensor_scale, lane_s,
                                                EPI == EPI_F16_ROWCOL ? strip[t0 + k] : lane_s, lane_z);
                    if (live) {
                        T* dst = reinterpret_cast<T*>(p.epi.out) + static_cast<long long>(t0) * p.epi.ld + channel;
                        const int left = tokens - t0;
#pragma unroll
                        for (int k = 0; k < 32; ++k) {
                            if (k < left) *dst = v[k];
                            dst += p.epi.ld;
                        }
                    }
                }
            }
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(acc_empty_bar(acc));
            acc ^= 1u;
            if (acc == 0) acc_phase ^= 1u;
        }
    }

    // ---------------------------------------------------------------------- teardown
    tc_fence_before_sync();
    __syncthreads();
    if (*abort_flag && threadIdx.x == 0) {
        const uint64_t t0 = global_timer_ns();               // aborting: let copies in flight land
        while (global_timer_ns() - t0 < 200000ull) {}
    }
    __syncthreads();
    if (warp == 1) {
        __syncwarp();
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, p.tmem_cols);
    }
}

}  // namespace bm
