// LUT matvec (m = 1) fed by regular copies, sm_100a, and the any-shape fallback kernel.
//
// gemv_reg_kernel is gemv_tma_kernel (same table, lane mapping, ring, split-k finish and tensor-parallel links; see gemv_tma.cuh)
// for containers that tensor maps cannot describe: any N % 4 == 0 (rows of scales then begin on 8 bytes) and any group size that
// is a multiple of 32 (the scales' rows of a slab begin anywhere).  Four warps bring the stages with cp.async, 16 bytes of words
// and 8 of scales at a time, and each of their copies' completion counts on the stage's barrier.  The container's columns and K may
// end inside a stage: zeros come instead.
// Replaces _nqmv / _nqmv_bias (lutGEMM/src/cuda/kernels/mv_fp16.hpp:25-97, mv_fp16_bias.hpp:24-118).
//
// Measured, us, one row, this / four stages in registers of the consuming lanes, which is what it replaced: 11004 x 4128, q = 3, g = 96, 8.6
// / 11.2; 12284 x 12288, q = 3, g = 128, 17.7 / 22.9 (12288 x 12288 with tensor maps 16.8); 28672 x 8160, q = 4 + q_bias, g = 96, 34.9 / 53.0.
#pragma once
#include "gemv_tma.cuh"

namespace lg {

constexpr int kRegFeedWarps = 4;
constexpr int kRegThreads = (kConsWarps + kRegFeedWarps) * 32;

// Most scale groups of g that a slab of 512 k touches: it begins at a multiple of the largest power of two in g (up to 512) into one,
// the last of those at most, and its last word 480 further.
constexpr int reg_scale_rows(int g) {
    const int step = (g & -g) < kSlab2 ? g & -g : kSlab2;
    return (g - step + kSlab2 - 32) / g + 1;
}
constexpr bool reg_scale_rows_exact() {
    for (int g = 32; g <= 2 * kSlab2 + 32; g += 32) {
        int most = 0;
        for (int slab = 0; slab < g / 32; slab++) {               // 512 slab runs through all its remainders
            const int touched = (slab * kSlab2 + kSlab2 - 32) / g - slab * kSlab2 / g + 1;
            if (touched > most) most = touched;
        }
        if (most != reg_scale_rows(g)) return false;
    }
    return true;
}
static_assert(reg_scale_rows_exact(), "rows of scales for every slab, and none too many");

struct FeedCopies {
    static constexpr int kArrivals = kRegFeedWarps * 32;
    __device__ __forceinline__ void operator()(const Gemv2Params& p, unsigned char* smem, uint32_t bar_full, uint32_t bar_empty, int n_begin,
                                               int total_stages) const {
        const int tid = threadIdx.x - kConsWarps * 32;
        const int q = p.q, N = p.N, G = p.K / p.g, stage_bytes = gemv2_stage_bytes(p.a_rows), nstages = gemv2_num_stages(p.a_rows);
        const int chunk = tid & 63, row0 = tid >> 6;         // 64 chunks of four columns, two rows at a time
        const int kw0 = blockIdx.y * kSlabWords + row0, grp0 = (int)(blockIdx.y * kSlab2 / p.g) + row0;
        const int words = min(kSlabWords / 2, (p.K / 32 - kw0 + 1) / 2), scales = min((p.a_rows - row0 + 1) / 2, (G - grp0 + 1) / 2);
        const size_t step = 2 * (size_t)q * N;               // two rows on
        const uint32_t dst0 = smem_u32(smem + kStage0Off) + row0 * kRowPitch + chunk * 16;
        const uint32_t adst0 = smem_u32(smem + kStage0Off) + kWStageBytes + row0 * kARowPitch + chunk * 8;
        int slot = 0, round = 0, b = 0, col = n_begin + 4 * chunk;
        for (int t = 0; t < total_stages; t++) {
            if (round > 0) {
                if (!mbar_wait_bounded(bar_empty + 8 * slot, (round - 1) & 1)) {
                    atomicExch(p.status, kStatusProducerTimeout);
                    break;
                }
            }
            const bool ok = col < N;
            const uint32_t* src = p.bW + ((size_t)kw0 * q + b) * N + col;
            const __half* asrc = p.alpha + ((size_t)grp0 * q + b) * N + col;
            const uint32_t dst = dst0 + slot * stage_bytes, adst = adst0 + slot * stage_bytes;
#pragma unroll
            for (int i = 0; i < kSlabWords / 2; i++) cp_async16(dst + i * 2 * kRowPitch, src + i * step, ok && i < words ? 16u : 0u);
            for (int i = 0; 2 * i + row0 < p.a_rows; i++) cp_async8(adst + i * 2 * kARowPitch, asrc + i * step, ok && i < scales ? 8u : 0u);
            asm volatile("cp.async.mbarrier.arrive.noinc.shared::cta.b64 [%0];" ::"r"(bar_full + 8 * slot) : "memory");
            if (++slot == nstages) { slot = 0; round++; }
            if (++b == q) {
                b = 0;
                col += kStageCols;
            }
        }
    }
};

// p.a_rows: the most groups that a slab touches.
template <int WPG, bool BIAS>
__global__ void __launch_bounds__(kRegThreads, 1)
gemv_reg_kernel(const Gemv2Params p) {
    extern __shared__ __align__(1024) unsigned char smem[];
    gemv_body<WPG, BIAS, kRegThreads>(p, smem, FeedCopies{});
}

// Fallback for shapes the LUT kernel does not take (N % 4 != 0 or K % 256 != 0): one thread per
// column, activations staged in shared memory, signs applied bit by bit.  Correctness path only.
__global__ void __launch_bounds__(128)
gemv_generic_kernel(const uint32_t* __restrict__ bW, const __half* __restrict__ alpha,
                    const __half* __restrict__ q_bias, const __half* __restrict__ x,
                    __half* __restrict__ y16, float* __restrict__ y32, int N, int K, int q, int g) {
    __shared__ float xs[1024];
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    float acc = 0.f;
    for (int kt = 0; kt < K; kt += 1024) {
        const int klen = min(1024, K - kt);
        __syncthreads();
        for (int i = threadIdx.x; i < klen; i += blockDim.x) xs[i] = __half2float(x[kt + i]);
        __syncthreads();
        if (n < N) {
            for (int kw = 0; kw < klen / 32; kw++) {
                const int k = kt + kw * 32;
                const int grp = k / g;
                float xsum = 0.f;
                if (q_bias) {
                    for (int t = 0; t < 32; t++) xsum += xs[kw * 32 + t];
                    acc = fmaf(xsum, __half2float(q_bias[(size_t)grp * N + n]), acc);
                }
                for (int b = 0; b < q; b++) {
                    const uint32_t word = bW[((size_t)(k / 32) * q + b) * N + n];
                    float t_sum = 0.f;
#pragma unroll 8
                    for (int t = 0; t < 32; t++) t_sum += ((word >> t) & 1u) ? xs[kw * 32 + t] : -xs[kw * 32 + t];
                    acc = fmaf(t_sum, __half2float(alpha[((size_t)grp * q + b) * N + n]), acc);
                }
            }
        }
    }
    if (n < N) {
        if (y32) y32[n] = acc;
        if (y16) y16[n] = __float2half_rn(acc);
    }
}

}  // namespace lg
