// LUT matvec (m = 1) for shapes whose 512-k slabs do not share out evenly: one CTA per SM and one wave, whatever N and K are.
//
// gemv_tma_kernel gives a CTA whole column groups of one slab.  With many slabs that leaves SMs idle or takes a second wave, with a
// second start and a second table: 8192 x 28672, q = 4, is 56 slabs x 32 column groups, 280 CTAs of 7 groups on 148 SMs.  Here
// the stages (slab, column group, plane), slab by slab, are cut into as many equal runs as there are SMs.  A run goes through
// its column groups as gemv_tma_kernel does (same table, same lookups, same ring); where it crosses into the next slab it
// builds that slab's table while the ring keeps filling.  A run may begin or end inside a column group, between two planes.
//
// Result: fp32 reductions in L2 into one zeroed row.  Every column group has a counter of the planes that have arrived; the CTA
// that brings it to slabs * q rounds the group's columns and leaves row and counter zeroed.
//
// Bound like gemv_tma_kernel by lookups and staging in shared memory (some 860 cycles a stage; its loop takes 3.5 % more here).
// Measured, us, one row, this / gemv_tma_kernel: 8192 x 28672, q = 4 + q_bias, 30.4 / 34.4; 4096 x 28672, q = 3, 16.3 / 28.7; 8192 x
// 20480, q = 3, 19.8 / 22.5; where the shares are even 49152 x 12288, q = 4, on one weight 64.8 / 62.6.
#pragma once
#include "gemv_seq.cuh"

namespace lg {

// The lookups have the table's address in their instructions (lookup_word_seq) where dynamic shared memory begins at BASE, as it
// does for a kernel without static shared memory; elsewhere, as under a tool that takes some for itself, the same loop adds the address
// in a register, which is 2 to 7 % slower (8192 x 28672, q = 4, 31.0 and 32.3 us).
//
// The runs travel as a parameter: read at blockIdx.x they are in uniform registers and so are the loops' bounds.  (Worked out from
// blockIdx.x in the kernel, by divisions, they were not, and every loop reconverged its warp, as it does where
// one lane's failed wait may end it: hence the vote.  49152 x 12288, q = 4, 67.6 us without either, 64.8 with both.)
constexpr int kFlatMaxCtas = 160;
struct FlatRun {
    int stages;              // length
    int plane, group, slab;  // where it begins
};
struct FlatRuns {
    FlatRun run[kFlatMaxCtas];
};
constexpr int kFlatMaxPieces = kConsWarps * 16;             // column groups of a CTA's run: their list lies in the exchange area

// Stages (slab, group, plane) cut into `ctas` runs that differ by one stage at most.
inline void flat_plan(FlatRuns& runs, int nslabs, int groups, int q, int ctas) {
    const int total = nslabs * groups * q, base = total / ctas, longer = total % ctas;
    int unit = 0, plane = 0;                 // run i begins at stage i * base + min(i, longer)
    for (int i = 0; i < ctas; i++) {
        const int stages = base + (i < longer ? 1 : 0);
        runs.run[i] = {stages, plane, unit % groups, unit / groups};
        plane += stages;
        unit += plane / q;
        plane %= q;
    }
}

template <int WPG, bool BIAS, uint32_t BASE = kSeqSmemBase>
__global__ void __launch_bounds__(kGemv2Threads, 1)
gemv_flat_kernel(const __grid_constant__ CUtensorMap tmW, const __grid_constant__ CUtensorMap tmA, const Gemv2Params p,
                 const __grid_constant__ FlatRuns runs) {
    extern __shared__ __align__(1024) unsigned char smem[];
    unsigned char* lut = smem;
    const int stage_bytes = gemv2_stage_bytes(p.a_rows);
    const int nstages = gemv2_num_stages(p.a_rows);
    const uint32_t bar_full = smem_u32(smem + kBarOff);          // nstages x 8 B
    const uint32_t bar_empty = bar_full + 8 * kMaxStages;
    int* s_count = reinterpret_cast<int*>(smem + kBarOff + 16 * kMaxStages);

    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int N = p.N, q = p.q;
    const int groups = (N + kStageCols - 1) / kStageCols;
    const FlatRun run = runs.run[blockIdx.x];
    const int plane0 = run.plane, slab0 = run.slab, group0 = run.group;

    if (tid == 0) {
        for (int s = 0; s < nstages; s++) {
            mbar_init(bar_full + 8 * s, 1);
            mbar_init(bar_empty + 8 * s, kConsWarps);
        }
        mbar_fence_init();
        *s_count = 0;
    }
    __syncthreads();
    pdl_launch_dependents();

    if (warp == kConsWarps) {
        // ---------------- producer: one lane, two TMA loads per stage, ahead of the dependency wait (as in gemv_tma_kernel) ----
        if (lane == 0) {
            tma_prefetch_descriptor(&tmW);
            tma_prefetch_descriptor(&tmA);
            int b = plane0, cg = group0, slab = slab0, grp = slab0 * kSlab2 / p.g;
            int slot = 0, round = 0;
            for (int t = 0; t < run.stages; t++) {
                if (round > 0) {
                    if (!mbar_wait_bounded(bar_empty + 8 * slot, (round - 1) & 1)) {
                        atomicExch(p.status, kStatusProducerTimeout);
                        break;
                    }
                }
                const uint32_t dst = smem_u32(smem + kStage0Off + slot * stage_bytes);
                mbar_arrive_expect_tx(bar_full + 8 * slot, (uint32_t)stage_bytes);       // out-of-range parts are zero-filled and counted
                tma_load_3d(dst, &tmW, cg * kStageCols, b, slab * kSlabWords, bar_full + 8 * slot);
                tma_load_3d(dst + kWStageBytes, &tmA, cg * kStageCols, b, grp, bar_full + 8 * slot);
                if (++slot == nstages) { slot = 0; round++; }
                if (++b == q) {
                    b = 0;
                    if (++cg == groups) {
                        cg = 0;
                        slab++;
                        grp = slab * kSlab2 / p.g;
                    }
                }
            }
        }
        pdl_wait_prior_grids();
    } else {
        // ---------------- consumers ----------------
        const int c8 = lane & 7;                 // 16-byte column chunk inside the warp's 32 columns
        const int rr = lane >> 3;                // G: which 128-k run of the slab
        const int cb = warp & 7, h = warp >> 3;
        const int jp = (c8 & 1) ^ h;             // this lane's words in the slab: kw = 4 rr + jp + 2 u, u = 0, 1
        // everything that does not depend on the activations comes before the dependency wait
        uint32_t cs = 0, sel[4];
#pragma unroll
        for (int b = 0; b < 4; b++) cs |= (uint32_t)(32 * rr + 16 * jp + 4 * b) << (8 * b);
#pragma unroll
        for (int s = 0; s < 4; s++) {
            const uint32_t beta = (uint32_t)(s + (c8 >> 1)) & 3u;
            sel[s] = 0xCC00u | (beta << 4) | (4u + beta);     // -> {0, 0, word.byte[beta], cs.byte[beta]}
        }


        constexpr int NG = 2 / WPG;                              // alpha groups among the lane's 2 words
        int arow[NG];                                            // row of each group in the alpha box: the same in every slab
#pragma unroll
        for (int gi = 0; gi < NG; gi++) arow[gi] = 32 * (4 * rr + jp + 2 * gi * WPG) / p.g;
        float4* xchg = reinterpret_cast<float4*>(smem + kXchgOff) + cb * 8 + c8;
        const int col_in_stage = 32 * cb + 4 * c8;
        const uint32_t w_off = (uint32_t)(4 * rr + jp) * kRowPitch + (uint32_t)col_in_stage * 4u;
        bool aborted = false;
        int slot = 0, round = 0;
        int left = run.stages, b0 = plane0, cg = group0;
        pdl_wait_prior_grids();                  // the activations may come from the previous kernel
        auto consume = [&](auto known_base) {
        constexpr bool KNOWN = decltype(known_base)::value;
#pragma unroll 1
        for (int slab = slab0; left > 0; slab++, cg = 0) {
            const int k0 = slab * kSlab2;
            const uint4 raw = load_x_chunk(p.x, k0, p.K, tid);
            if (slab != slab0) asm volatile("bar.sync 1, %0;" ::"n"(kConsWarps * 32) : "memory");      // nobody looks up the last table any more
            build_lut_from_raw(lut, raw, tid);
            asm volatile("bar.sync 1, %0;" ::"n"(kConsWarps * 32) : "memory");
            float xsum[NG];
            const __half* bias[NG];              // this lane's rows of q_bias, at its columns of the first group; nullptr beyond K
            if (BIAS) {
                // sum of the activations under each group of words: entries idx = 255 (all signs +)
#pragma unroll
                for (int gi = 0; gi < NG; gi++) {
                    float s = 0.f;
#pragma unroll
                    for (int jj = 0; jj < WPG; jj++) {
                        const int u = gi * WPG + jj;
                        const unsigned char* e = lut + 255 * 256 + (32 * u + 8 * rr + 4 * jp) * 4;
                        s += *reinterpret_cast<const float*>(e) + *reinterpret_cast<const float*>(e + 4) +
                             *reinterpret_cast<const float*>(e + 8) + *reinterpret_cast<const float*>(e + 12);
                    }
                    xsum[gi] = s;
                    const int k = k0 + 32 * (4 * rr + jp + 2 * gi * WPG);
                    bias[gi] = k < p.K ? p.q_bias + (size_t)(k / p.g) * N + col_in_stage : nullptr;
                }
            }
#pragma unroll 1
            for (; cg < groups && left > 0; cg++) {
                const int col = cg * kStageCols + col_in_stage;
                const bool col_ok = col < N;
                const int nb = min(q - b0, left);
                float acc[4] = {0.f, 0.f, 0.f, 0.f};
                uint2 bv[NG];
                const bool first = b0 == 0;      // the piece with the group's first plane adds the offset term: 0 times an infinite sum is NaN
                if (BIAS) {
#pragma unroll
                    for (int gi = 0; gi < NG; gi++)
                        bv[gi] = (col_ok && first && bias[gi]) ? ldg_nc_v2(bias[gi] + cg * kStageCols) : make_uint2(0u, 0u);
                }
                for (int b = 0; b < nb && !aborted; b++) {
                    if (!__all_sync(0xffffffffu, mbar_wait_bounded(bar_full + 8 * slot, round & 1))) {
                        atomicExch(p.status, kStatusConsumerTimeout);
                        aborted = true;     // keep walking the loops (the barriers below must stay matched)
                        break;
                    }
                    const unsigned char* st = smem + kStage0Off + slot * stage_bytes + w_off;
                    const unsigned char* sa = smem + kStage0Off + slot * stage_bytes + kWStageBytes + col_in_stage * 2;
                    uint4 wv[2];
#pragma unroll
                    for (int u = 0; u < 2; u++) wv[u] = *reinterpret_cast<const uint4*>(st + u * 2 * kRowPitch);
                    uint2 av[NG];
#pragma unroll
                    for (int gi = 0; gi < NG; gi++) av[gi] = *reinterpret_cast<const uint2*>(sa + arow[gi] * kARowPitch);
                    __syncwarp();
                    if (lane == 0) mbar_arrive(bar_empty + 8 * slot);   // words are in registers: free the stage
                    if (++slot == nstages) { slot = 0; round++; }

#pragma unroll
                    for (int gi = 0; gi < NG; gi++) {
                        float2 s2[4];
#pragma unroll
                        for (int jj = 0; jj < WPG; jj++) {
                            const int u = gi * WPG + jj;
                            const uint32_t ww[4] = {wv[u].x, wv[u].y, wv[u].z, wv[u].w};
#pragma unroll
                            for (int c = 0; c < 4; c++) {
                                float2 v;
                                if constexpr (KNOWN) v = (u == 0) ? lookup_word_seq<0>(ww[c], cs, sel) : lookup_word_seq<128>(ww[c], cs, sel);
                                else v = (u == 0) ? lookup_word<0>(lut, ww[c], cs, sel) : lookup_word<128>(lut, ww[c], cs, sel);
                                s2[c] = (jj == 0) ? v : add_f32x2(s2[c], v);
                            }
                        }
                        const float2 a01 = half2_bits_to_float2(av[gi].x), a23 = half2_bits_to_float2(av[gi].y);
                        acc[0] = fmaf(s2[0].x + s2[0].y, a01.x, acc[0]);
                        acc[1] = fmaf(s2[1].x + s2[1].y, a01.y, acc[1]);
                        acc[2] = fmaf(s2[2].x + s2[2].y, a23.x, acc[2]);
                        acc[3] = fmaf(s2[3].x + s2[3].y, a23.y, acc[3]);
                    }
                }
                if (BIAS && first) {
#pragma unroll
                    for (int gi = 0; gi < NG; gi++) {
                        const float2 b01 = half2_bits_to_float2(bv[gi].x), b23 = half2_bits_to_float2(bv[gi].y);
                        acc[0] = fmaf(xsum[gi], b01.x, acc[0]);
                        acc[1] = fmaf(xsum[gi], b01.y, acc[1]);
                        acc[2] = fmaf(xsum[gi], b23.x, acc[2]);
                        acc[3] = fmaf(xsum[gi], b23.y, acc[3]);
                    }
                }
                // add the 4 lanes (128-k runs) that share a column quad, then the two warp halves through shared memory
#pragma unroll
                for (int off = 8; off < 32; off <<= 1) {
#pragma unroll
                    for (int c = 0; c < 4; c++) acc[c] += __shfl_xor_sync(0xffffffffu, acc[c], off);
                }
                if (h == 1 && rr == 0) *xchg = make_float4(acc[0], acc[1], acc[2], acc[3]);
                asm volatile("bar.sync %0, 64;" ::"r"(2 + cb) : "memory");
                if (h == 0 && rr == 0 && col_ok) {
                    const float4 o = *xchg;
                    red_add_v4(p.partial + col, make_float4(acc[0] + o.x, acc[1] + o.y, acc[2] + o.z, acc[3] + o.w));
                }
                asm volatile("bar.sync %0, 64;" ::"r"(2 + cb) : "memory");   // exchange slot free for the next column group
                left -= nb;
                b0 = 0;
            }
        }
        };
        if (smem_u32(smem) == BASE) consume(std::true_type{});
        else consume(std::false_type{});
    }

    // ---- finish: the column groups that this CTA's planes complete ----
    __syncthreads();
    const int pieces = (plane0 + run.stages + q - 1) / q;
    int* s_done = reinterpret_cast<int*>(smem + kXchgOff);
    if (tid < pieces) {
        const int planes = min(run.stages, (tid + 1) * q - plane0) - max(0, tid * q - plane0), cg = (group0 + tid) % groups;
        asm volatile("fence.acq_rel.gpu;" ::: "memory");         // after the barrier: the whole CTA's reductions before the count
        const unsigned have = atomicAdd(p.counters + cg, (unsigned)planes) + (unsigned)planes;
        if (have == (unsigned)(p.nslabs * q)) {
            asm volatile("fence.acq_rel.gpu;" ::: "memory");
            p.counters[cg] = 0u;                                 // ready for the next launch on this stream
            s_done[atomicAdd(s_count, 1)] = cg;
        }
    }
    __syncthreads();
    const int n = *s_count * (kStageCols / 4);
    for (int i = tid; i < n; i += kGemv2Threads) {
        const int c = s_done[i / (kStageCols / 4)] * kStageCols + 4 * (i % (kStageCols / 4));
        if (c >= N) continue;
        const float4 s = __ldcg(reinterpret_cast<const float4*>(p.partial + c));
        __stcg(reinterpret_cast<float4*>(p.partial + c), make_float4(0.f, 0.f, 0.f, 0.f));
        if (p.y32) *reinterpret_cast<float4*>(p.y32 + c) = s;
        if (p.y16) {
            __half2 lo = __floats2half2_rn(s.x, s.y), hi = __floats2half2_rn(s.z, s.w);
            *reinterpret_cast<uint2*>(p.y16 + c) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
        }
    }
}

}  // namespace lg
