// Batched BCQ matmul with the planes folded into one split operand, on the 5th-generation tensor cores, sm_100a.
//
// gemm_tc.cuh multiplies every bit plane by itself: q (or q + 1 with q_bias) tensor-core passes over the activations.
// Inside a scale group a weight takes only 2^q values, W = q_bias + sum_b +-alpha_b, so here each column's values are
// computed once per group in fp32, split as hi + lo (two fp16 numbers, lo = fp16(W - hi)) and the packed bits only
// choose between them: two passes whatever q is, and no rounding of the weight beyond 2^-22 of it.  So that hi never
// overflows a CTA scales every column by a power of two taken from the largest scale of that column in the CTA's k-range,
// and takes it out again in the epilogue.  Every W is a multiple of the last place of its group's smallest scale, at least
// 2^-24: scaled up, or left as it is (largest scale below 8192), lo's last place is no coarser than that and nothing is lost
// to fp16's subnormals.  Scaled down it may be, where a column has a scale of 8192 or more and one so small that its last
// place falls below 2^-24: the epilogue computes such a column anew, product by product.  It does the same for what is not
// finite in a row with an infinite activation: hi * inf + lo * inf has not the planes' signs.  (One plane without q_bias is exact
// as it is: one pass, no lo.)
//
//   CTA = 128 output columns x up to 256 activation rows x a k-range, walked in blocks of 64 k.
//   16 expansion warps: warp (quarter lq of the columns, sub) takes the blocks j with j mod 4 == sub.  Lane = column.  The
//   packed words and scales come straight from global memory, one block of this warp (four of the CTA) ahead.  The
//   lane writes the 2^q (hi, lo) pairs of its column to its own bank of a table in shared memory (no other lane reads
//   them: no synchronisation, no bank conflicts), turns the q words into one code per byte (a bit transpose of shifts
//   and LOP3s), looks 64 weights up (one PRMT makes a code byte and the lane's bank an address) and stores them with
//   tcgen05.st as the A operand in tensor memory.
//   Up to two planes the values (four at most) stay in registers and a PRMT picks two weights' halves at a time: no table, no
//   reads of shared memory.  Calls back to back on one weight, 8192 x 8192, q = 2, 128 rows 31.4 us (32.9 with the
//   table), q = 2 + q_bias, 64 rows 24.4 (27.4); on weights in turn that L2 does not hold 34.3.
//   One lane issues tcgen05.mma.kind::f16: M = 128 columns, N = rows, K = 16, A (hi, then lo) in tensor memory, the
//   activations [rows][64 k] (TMA, 128-byte swizzle) in shared memory, one fp32 accumulator.
//   Every accumulation of the tensor core cuts its fp32 sum off toward zero: measured, the error of a chain of n is 1.8e-8 n
//   of the result, whoever's chain it is.  SEG, for fp32 results and long k: chains no longer than gemm_tc's, which its
//   k-ranges cut.  Lo has an accumulator of its own up to 128 rows, and k is walked in segments: between two, the expansion
//   warps add the accumulators to sums of their own (fp32, rounded to nearest; in local memory, 64 a thread) while the next
//   blocks' operands wait.  Relative error of an fp32 result, gemm_tc / one chain / SEG: 28672 x 8192, q = 3, 100 rows 5.8e-6 /
//   1.8e-5 / 4.9e-6 (141 / 111 / 132 us); 8192 x 28672, q = 1, 300 rows 8.4e-6 / 3.4e-5 / 8.4e-6.  SEG's expansion loop issues some 10 %
//   more, which fp16 results, whose own rounding is 2.1e-4, do not pay.
//
// Tensor memory: 256 accumulator columns, then four operand stages of 64 columns (hi 32, lo 32), one per `sub`.
//
// At 256 rows a block of 64 k takes the tensor pipe 1024 cycles and shared memory about as long (the activations are read
// once for hi and once for lo: 64 KB, beside 32 KB arriving and 40 KB of table traffic, at 128 bytes a cycle); the expansion
// issues for about 700 cycles at q = 4 with q_bias and bounds the kernel below 200 rows.  Measured, us, 8192 x 8192, q = 4 +
// q_bias, 2048 rows: 424 (1296 as 16 launches of gemm_tc).  28672 x 8192, q = 4 + q_bias, 4 rows: 116 (160).
// All mbarrier waits are bounded, as in gemm_tc.cuh.
#pragma once
#include "gemm_tc.cuh"

namespace lg {

constexpr int kHlCols = 128;                  // output columns per CTA
constexpr int kHlStepK = 64;                  // k per block
constexpr int kHlRows = 256;                  // most activation rows per CTA
constexpr int kHlBoxRows = 128;               // rows per TMA box of the activations (fewer when the call has fewer)
constexpr int kHlExpWarps = 16, kHlMmaWarp = 0, kHlTmaWarp = 1, kHlFirstExpWarp = 2;
constexpr int kHlThreads = (kHlFirstExpWarp + kHlExpWarps) * 32;      // 576
constexpr int kHlStages = 4;                  // operand stages in tensor memory, one per `sub`
constexpr uint32_t kHlACol = 256;             // first operand column
constexpr int kHlMaxSlots = 8;                // activation ring
constexpr int kHlLoRows = 128;                // up to so many rows lo has accumulators of its own, at this column
constexpr int kHlTableBytes = kHlExpWarps * 16 * 128;                 // offset 0: [pair of warps][16 values][2 warps][32 lanes] x 4 B
constexpr int kHlScaleOff = kHlTableBytes;                            // [128] largest |scale| (fp16 bits) per column
constexpr int kHlBarOff = kHlScaleOff + kHlCols * 4;
constexpr int kHlXOff = kHlTableBytes + 1024;                         // multiple of 1024: swizzle atoms
constexpr int kHlXBudget = kSmemLimit - kHlXOff;                      // also the epilogue's transposes (16 x 16 x 33 floats)

struct HlParams {
    const uint32_t* bW;      // [K/32][q][N]
    const __half* alpha;     // [G][q][N]
    const __half* q_bias;    // [G][N] or nullptr
    const __half* x;         // [m][K], what tmX describes
    float* partial;          // [m][N] fp32, zero between launches (split-k only)
    unsigned* counters;      // one per output tile, zero between launches
    int* status;
    __half* y16;             // [m][N] or nullptr
    float* y32;              // [m][N] or nullptr
    int N, K, G, g, m;
    int col_tiles;           // tiles of 128 columns
    int full_items;          // items (column tile, 256 rows) that one CTA takes whole; the rest go as two halves of 128 rows
    int splits;              // k-ranges per item; a range is blocks_per_split blocks of 64 k
    int blocks_per_split;
    int segment_lo, segment; // most blocks between two drains, with lo in its own accumulator and without
    int box_rows;            // rows of a TMA box: 128, or m rounded up to 16 when that is less
    int x_slot_bytes, x_slots;
};

// One lane of a converged warp: 1 there, 0 elsewhere.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t e;
    asm volatile("{\n.reg .pred p;\nelect.sync _|p, 0xffffffff;\nselp.u32 %0, 1, 0, p;\n}\n" : "=r"(e));
    return e;
}
// umma_f16_ts / umma_commit under a predicate, for a warp that stays converged.
__device__ __forceinline__ void umma_f16_ts_if(uint32_t on, uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc,
                                               uint32_t accumulate) {
    asm volatile(
        "{\n.reg .pred p, q;\n"
        "setp.ne.b32 q, %5, 0;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "@q tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n}\n"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate), "r"(on) : "memory");
}
__device__ __forceinline__ void umma_commit_if(uint32_t on, uint32_t bar) {
    asm volatile(
        "{\n.reg .pred q;\n"
        "setp.ne.b32 q, %1, 0;\n"
        "@q tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}\n" ::"r"(bar), "r"(on) : "memory");
}

// (hi, lo) of two values, hi in the low half of an entry
__device__ __forceinline__ void hl_pack_pair(float v0, float v1, uint32_t& e0, uint32_t& e1) {
    const __half2 hi = __floats2half2_rn(v0, v1);
    const float2 f = __half22float2(hi);
    const __half2 lo = __floats2half2_rn(v0 - f.x, v1 - f.y);
    const uint32_t h = *reinterpret_cast<const uint32_t*>(&hi), l = *reinterpret_cast<const uint32_t*>(&lo);
    e0 = prmt_b32(h, l, 0x5410u);
    e1 = prmt_b32(h, l, 0x7632u);
}

// Groups that the k-range [k0, k1) touches in this column: is the last place of some scale, times 2^(12 - e) with e the
// exponent of the column's largest (`max_bits`, 8192 or more), below 2^-24?
template <int Q, bool BIAS>
__device__ __noinline__ bool hl_has_tiny_scale(const HlParams& p, int col, int k0, int k1, unsigned max_bits) {
    unsigned least = 0x7c00u;
    for (int grp = k0 / p.g; grp * p.g < k1; grp++)
        for (int b = 0; b < Q + (BIAS ? 1 : 0); b++) {
            const __half* src = b < Q ? p.alpha + ((size_t)grp * Q + b) * p.N : p.q_bias + (size_t)grp * p.N;
            const unsigned bits = __half_as_ushort(src[col]) & 0x7fffu;
            if (bits != 0u && bits < least) least = bits;
        }
    return (max_bits >> 10) - max(1u, least >> 10) > 26u;
}
// Whether this row's activations in [k0, k1) have an infinity, a NaN.  Called by a whole warp.
__device__ __noinline__ void hl_row_class(const HlParams& p, int row, int k0, int k1, int lane, bool* inf, bool* nan) {
    unsigned most = 0u;
    bool any_inf = false;
    for (int k = k0 + lane; k < k1; k += 32) {
        const unsigned bits = __half_as_ushort(p.x[(size_t)row * p.K + k]) & 0x7fffu;
        any_inf |= bits == 0x7c00u;
        most = max(most, bits);
    }
    *inf = __any_sync(0xffffffffu, any_inf);
    *nan = __any_sync(0xffffffffu, most > 0x7c00u);
}
// One output as the planes give it: products of +-alpha_b (and q_bias) with the activation, which are exact, summed in
// fp32, 32 k of a plane at a time.  Lane = column; every lane reads the same activations.
template <int Q, bool BIAS>
__device__ __noinline__ float hl_by_product(const HlParams& p, int row, int col, int k0, int k1) {
    const __half* x = p.x + (size_t)row * p.K;
    float sum = 0.f;
    for (int k = k0; k < k1; k += 32) {
        const size_t grp = k / p.g;
        for (int b = 0; b < Q + (BIAS ? 1 : 0); b++) {
            const uint32_t w = b < Q ? __ldg(p.bW + ((size_t)(k >> 5) * Q + b) * p.N + col) : 0xffffffffu;
            const float a = __half2float(b < Q ? p.alpha[(grp * Q + b) * p.N + col] : p.q_bias[grp * p.N + col]);
            float s = 0.f;
#pragma unroll 8
            for (int i = 0; i < 32; i++) s = fmaf((w >> i) & 1u ? a : -a, __half2float(x[k + i]), s);
            sum += s;
        }
    }
    return sum;
}

// Adds this warp's part of the accumulators (16 rows of every 64, lane = column) to `sums`, or puts it there.  lo_col: column
// of the accumulators of lo, 0 if there are none.
__device__ __noinline__ void hl_drain(float* sums, uint32_t t_acc, uint32_t lo_col, int sub, int rows, bool add) {
#pragma unroll 1
    for (int c = sub, at = 0; 16 * c < rows; c += 4, at += 16) {
        uint32_t r[16], l[16];
        tmem_ld_x16(t_acc + 16u * (uint32_t)c, r);
        if (lo_col) tmem_ld_x16(t_acc + lo_col + 16u * (uint32_t)c, l);
        tmem_ld_wait();
#pragma unroll
        for (int i = 0; i < 16; i++) {
            float v = __uint_as_float(r[i]);
            if (lo_col) v += __uint_as_float(l[i]);
            sums[at + i] = add ? sums[at + i] + v : v;
        }
    }
}

// Q: number of bit planes (1..4); BIAS: container has q_bias.  tmX: 2-D map {K, m} of fp16, box {64, box_rows}, 128-byte swizzle.
template <int Q, bool BIAS, bool SEG>
__global__ void __launch_bounds__(kHlThreads, 1)
gemm_hl_kernel(const __grid_constant__ CUtensorMap tmX, const __grid_constant__ HlParams p) {
    constexpr int NV = 1 << Q;
    constexpr int PASSES = (Q == 1 && !BIAS) ? 1 : 2;
    constexpr bool IN_REGS = Q <= 2;          // up to four values: a PRMT picks them out of two registers
    extern __shared__ __align__(1024) unsigned char smem[];
    const uint32_t smem_base = smem_u32(smem);
    const uint32_t bar_xfull = smem_base + kHlBarOff;             // kHlMaxSlots each
    const uint32_t bar_xempty = bar_xfull + 8 * kHlMaxSlots;
    const uint32_t bar_afull = bar_xempty + 8 * kHlMaxSlots;      // kHlStages each
    const uint32_t bar_aempty = bar_afull + 8 * kHlStages;
    const uint32_t bar_acc = bar_aempty + 8 * kHlStages;          // a segment's accumulators are complete
    const uint32_t bar_drained = bar_acc + 8;                     // ... and have been read
    uint32_t* s_tmem = reinterpret_cast<uint32_t*>(smem + kHlBarOff + 16 * kHlMaxSlots + 16 * kHlStages + 16);
    int* s_flag = reinterpret_cast<int*>(s_tmem + 1);
    unsigned* s_max = reinterpret_cast<unsigned*>(smem + kHlScaleOff);

    // the warp number through a shuffle: the compiler then knows it to be the same in every lane, and what depends on it
    // only (rows of words and scales, groups, block counts) is computed once per warp in uniform registers
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int N = p.N;
    // this CTA's item: 256 rows, or a half of one
    int item = blockIdx.x, half_row = 0, rows_cap = kHlRows;
    if (item >= p.full_items) {
        const int h = item - p.full_items;
        item = p.full_items + (h >> 1);
        half_row = (h & 1) * (kHlRows / 2);
        rows_cap = kHlRows / 2;
    }
    const int n0 = (item % p.col_tiles) * kHlCols;
    const int row0 = (item / p.col_tiles) * kHlRows + half_row;
    if (row0 >= p.m) return;                                      // the second half of a last, short item
    const int rows = min(rows_cap, p.m - row0);
    const int n_mma = (rows + 15) & ~15;
    const int blocks_total = (p.K + kHlStepK - 1) / kHlStepK;
    const int blk_begin = blockIdx.y * p.blocks_per_split;
    const int nblk = min(blocks_total, blk_begin + p.blocks_per_split) - blk_begin;      // >= 1 by the plan
    const uint32_t lo_col = SEG && PASSES == 2 && rows <= kHlLoRows ? (uint32_t)kHlLoRows : 0u;
    const int most = !SEG ? nblk : lo_col || PASSES == 1 ? p.segment_lo : p.segment;
    const int segments = SEG ? (nblk + most - 1) / most : 1, seg_blocks = SEG ? (nblk + segments - 1) / segments : nblk;

    if (tid == 0) {
        for (int s = 0; s < kHlMaxSlots; s++) {
            mbar_init(bar_xfull + 8 * s, 1);
            mbar_init(bar_xempty + 8 * s, 1);
        }
        for (int s = 0; s < kHlStages; s++) {
            mbar_init(bar_afull + 8 * s, 4);                      // the four column quarters
            mbar_init(bar_aempty + 8 * s, 1);
        }
        mbar_init(bar_acc, 1);
        mbar_init(bar_drained, kHlExpWarps);
        mbar_fence_init();
    }
    if (tid < kHlCols) s_max[tid] = 0u;
    if (warp == kHlMmaWarp) {
        tmem_alloc(smem_u32(s_tmem), kTcTmemCols);
        tmem_relinquish();
    }
    tc_fence_before_sync();
    __syncthreads();
    tc_fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *s_tmem, 0);
    bool timed_out = false;
    // the packed planes and scales are never written by a kernel: their stream starts while the previous kernel drains
    pdl_launch_dependents();

    const int lq = warp & 3;                                      // TMEM lane quarter this warp may access
    const int ew = warp - kHlFirstExpWarp, sub = ew >> 2;
    const int col_l = lq * 32 + lane, col = n0 + col_l;
    const uint32_t t_acc = tmem_base + ((uint32_t)(lq * 32) << 16);
    float unscale = 1.f;
    float sums[SEG ? kHlRows / 4 : 1];                            // of the segments that have been drained
    if (warp >= kHlFirstExpWarp) {
        // ---------------- expansion ----------------
        const size_t row_w = (size_t)Q * N;                       // words per k-word row, scales per group
        // one block ahead: with two or three a call of 16 to 128 rows took 1 to 2 us more (registers, moves)
        uint32_t w[2][Q];
        unsigned short av[2][Q], bv[2];
        // This warp's next block: its words, its group (advanced by 4 blocks = 256 k without a division).  Loads are not
        // predicated: a column beyond N reads column N - 1 (its accumulators are never stored), a word beyond K the block's
        // first word with that word's scales (the activations there are zero), a block beyond the range nothing at all.
        const unsigned col_c = (unsigned)min(col, N - 1);
        const uint32_t* wrow = p.bW + (size_t)(blk_begin + sub) * 2 * row_w;
        int knext = (blk_begin + sub) * kHlStepK;
        const int kend = min(p.K, (blk_begin + nblk) * kHlStepK);
        int grp = knext / p.g, grem = knext % p.g;
        const int ginc = (4 * kHlStepK) / p.g, grinc = (4 * kHlStepK) % p.g;
        auto fetch = [&]() {
            if (knext < kend) {                                   // warp-uniform
                const bool second = knext + 32 < kend;
                const uint32_t* wrow1 = second ? wrow + row_w : wrow;
                const unsigned short* arow = reinterpret_cast<const unsigned short*>(p.alpha) + (size_t)grp * row_w;
#pragma unroll
                for (int b = 0; b < Q; b++) {
                    w[0][b] = __ldg(wrow + (size_t)b * N + col_c);
                    w[1][b] = __ldg(wrow1 + (size_t)b * N + col_c);
                    av[0][b] = __ldg(arow + (size_t)b * N + col_c);
                }
                if (BIAS) bv[0] = __ldg(reinterpret_cast<const unsigned short*>(p.q_bias) + (size_t)grp * N + col_c);
                if (p.g < kHlStepK) {                             // g == 32: the second word has scales of its own
                    const int g1 = grp + (second ? 1 : 0);
                    const unsigned short* arow1 = reinterpret_cast<const unsigned short*>(p.alpha) + (size_t)g1 * row_w;
#pragma unroll
                    for (int b = 0; b < Q; b++) av[1][b] = __ldg(arow1 + (size_t)b * N + col_c);
                    if (BIAS) bv[1] = __ldg(reinterpret_cast<const unsigned short*>(p.q_bias) + (size_t)g1 * N + col_c);
                }
            }
            wrow += 8 * row_w;
            knext += 4 * kHlStepK;
            grp += ginc;
            grem += grinc;
            if (grem >= p.g) { grem -= p.g; grp++; }
        };
        fetch();
        // largest |scale| per column over this k-range: 16 threads x 8 columns per row of scales
        {
            const int grp0 = blk_begin * kHlStepK / p.g;
            const int grp1 = min(p.G, (kend + p.g - 1) / p.g);
            const int et = tid - kHlFirstExpWarp * 32, c8 = (et & 15) * 8;
            uint32_t mx[4] = {0u, 0u, 0u, 0u};
            if (n0 + c8 < N) {                                    // N % 8 == 0: whole chunks
                const int a_rows = (grp1 - grp0) * Q, all = a_rows + (BIAS ? grp1 - grp0 : 0);
#pragma unroll 4
                for (int r = et >> 4; r < all; r += kHlExpWarps * 2) {
                    const __half* src = r < a_rows ? p.alpha + ((size_t)grp0 * Q + r) * N : p.q_bias + (size_t)(grp0 + r - a_rows) * N;
                    const uint4 v = __ldg(reinterpret_cast<const uint4*>(src + n0 + c8));
                    const uint32_t vv[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
                    for (int i = 0; i < 4; i++) mx[i] = __vmaxu2(mx[i], vv[i] & 0x7fff7fffu);      // |fp16| orders like its bits
                }
            }
#pragma unroll
            for (int i = 0; i < 4; i++) mx[i] = __vmaxu2(mx[i], __shfl_xor_sync(0xffffffffu, mx[i], 16));
            if (lane < 16) {
#pragma unroll
                for (int i = 0; i < 4; i++) {
                    atomicMax(s_max + c8 + 2 * i, mx[i] & 0xffffu);
                    atomicMax(s_max + c8 + 2 * i + 1, mx[i] >> 16);
                }
            }
        }
        asm volatile("bar.sync 1, %0;" ::"n"(kHlExpWarps * 32) : "memory");
        // |W| <= (Q + 1) max < 5 * 2^(e + 1) with e = exponent of max: the scale 2^(12 - e) keeps |W| below 40960.  One
        // pass needs none (W = +-alpha).  All zero: 1.  Not finite: the column's result is not finite either, and the
        // scale for e = 15 keeps the finite weights beside it finite.
        float scale = 1.f;
        {
            const unsigned mbits = s_max[col_l];
            if (PASSES == 2 && mbits != 0u) {
                const int e = mbits >= 0x7c00u ? 15 : (int)(__float_as_uint(__half2float(__ushort_as_half((unsigned short)mbits))) >> 23) - 127;
                scale = __uint_as_float((uint32_t)(127 + 12 - e) << 23);
                unscale = __uint_as_float((uint32_t)(127 - 12 + e) << 23);
            }
        }
        // table entry of code c at (pair << 12) + (c << 8) + bank: the code byte carries the pair in its high nibble
        const uint32_t bank = (uint32_t)lane * 4u + (uint32_t)(ew & 1) * 128u;
        const uint32_t pair4 = (uint32_t)(ew >> 1) * 0x10101010u;
        unsigned char* tab = smem + (ew >> 1) * 4096 + bank;
        const uint32_t t_dst = tmem_base + ((uint32_t)(lq * 32) << 16) + kHlACol + (uint32_t)sub * 64u;
        int round = 0, j = sub;
        uint32_t t_hi[NV / 2] = {}, t_lo[NV / 2] = {};           // IN_REGS: the values' halves, two to a register
        // segment by segment: this warp's blocks up to and with its first one beyond the segment, then the drain, during which
        // those blocks wait for the tensor core (the stage of block j is free once block j - 4, of this segment, has been read)
#pragma unroll 1
        for (int seg = 0; seg < segments && !timed_out; seg++) {
        const int upto = seg + 1 < segments ? min(nblk, (seg + 1) * seg_blocks + kHlStages) : nblk;
        for (; j < upto; j += kHlStages, round++) {
            uint32_t cw[2][Q];
            float a[2][Q], qb[2] = {0.f, 0.f};
#pragma unroll
            for (int u = 0; u < 2; u++) {
#pragma unroll
                for (int b = 0; b < Q; b++) cw[u][b] = w[u][b];
                if (u == 0 || p.g < kHlStepK) {
#pragma unroll
                    for (int b = 0; b < Q; b++) a[u][b] = __half2float(__ushort_as_half(av[u][b])) * scale;
                    if (BIAS) qb[u] = __half2float(__ushort_as_half(bv[u])) * scale;
                }
            }
            fetch();
#pragma unroll
            for (int u = 0; u < 2; u++) {
                if (u == 0 || p.g < kHlStepK) {
                    // the column's 2^Q values: bit b of the code set = +alpha_b
                    float bound = fabsf(qb[u]);
#pragma unroll
                    for (int b = 0; b < Q; b++) bound += fabsf(a[u][b]);
                    // without q_bias the values of c and of its complement are each other's negatives
                    constexpr int NC = BIAS || Q == 1 ? NV : NV / 2;
                    float v[NC];
                    v[0] = BIAS || Q == 1 ? qb[u] : -a[u][Q - 1];
#pragma unroll
                    for (int b = (BIAS || Q == 1 ? Q : Q - 1) - 1; b >= 0; b--) {      // v[c] for c a multiple of 2^b, halving the stride
#pragma unroll
                        for (int c = 0; c < NC; c += 2 << b) {
                            const float s = v[c];
                            v[c] = s - a[u][b];
                            v[c + (1 << b)] = s + a[u][b];
                        }
                    }
                    if constexpr (IN_REGS) {
#pragma unroll
                        for (int c = 0; c < NV; c += 2) {
                            // without q_bias the upper half of four values are the lower's negatives, the other way round
                            const float v0 = c < NC ? v[c < NC ? c : 0] : -v[c < NC ? 0 : NV - 1 - c], v1 = c < NC ? v[c < NC ? c + 1 : 0] : -v[c < NC ? 0 : NV - 2 - c];
                            const __half2 h = __floats2half2_rn(v0, v1);
                            const float2 f = __half22float2(h);
                            const __half2 l = __floats2half2_rn(v0 - f.x, v1 - f.y);
                            t_hi[c / 2] = *reinterpret_cast<const uint32_t*>(&h);
                            t_lo[c / 2] = *reinterpret_cast<const uint32_t*>(&l);
                        }
                        if (!(bound <= 65504.f)) {                // an infinite or NaN scale: the value itself, lo = 0
#pragma unroll
                            for (int c = 0; c < NV / 2; c++) {
                                if ((t_hi[c] & 0x7c00u) == 0x7c00u) t_lo[c] &= 0xffff0000u;
                                if ((t_hi[c] & 0x7c000000u) == 0x7c000000u) t_lo[c] &= 0xffffu;
                            }
                        }
                    } else {
#pragma unroll
                        for (int c = 0; c < NC; c += 2) {
                            uint32_t e0, e1;
                            hl_pack_pair(v[c], v[c + 1], e0, e1);
                            *reinterpret_cast<uint32_t*>(tab + c * 256) = e0;
                            *reinterpret_cast<uint32_t*>(tab + (c + 1) * 256) = e1;
                            if (NC < NV) {
                                *reinterpret_cast<uint32_t*>(tab + (NV - 1 - c) * 256) = e0 ^ 0x80008000u;
                                *reinterpret_cast<uint32_t*>(tab + (NV - 2 - c) * 256) = e1 ^ 0x80008000u;
                            }
                        }
                        if (!(bound <= 65504.f)) {                    // an infinite or NaN scale: the value itself, lo = 0
#pragma unroll 1
                            for (int c = 0; c < NV; c++) {
                                uint32_t* e = reinterpret_cast<uint32_t*>(tab + c * 256);
                                if ((*e & 0x7c00u) == 0x7c00u) *e &= 0xffffu;
                            }
                        }
                    }
                }
                // q words of 32 bits -> nibble words (code of weight 4 i + r = nibble i of n[r]) -> one code per byte
                uint32_t lo4[4], hi4[4];
                {
                    const uint32_t w0 = cw[u][0], w1 = Q > 1 ? cw[u][Q > 1 ? 1 : 0] : 0u;
                    const uint32_t w2 = Q > 2 ? cw[u][Q > 2 ? 2 : 0] : 0u, w3 = Q > 3 ? cw[u][Q > 3 ? 3 : 0] : 0u;
                    const uint32_t e01 = (w0 & 0x55555555u) | ((w1 << 1) & 0xaaaaaaaau), o01 = ((w0 >> 1) & 0x55555555u) | (w1 & 0xaaaaaaaau);
                    const uint32_t e23 = (w2 & 0x55555555u) | ((w3 << 1) & 0xaaaaaaaau), o23 = ((w2 >> 1) & 0x55555555u) | (w3 & 0xaaaaaaaau);
                    uint32_t n[4];
                    n[0] = (e01 & 0x33333333u) | ((e23 << 2) & 0xccccccccu);
                    n[1] = (o01 & 0x33333333u) | ((o23 << 2) & 0xccccccccu);
                    n[2] = ((e01 >> 2) & 0x33333333u) | (e23 & 0xccccccccu);
                    n[3] = ((o01 >> 2) & 0x33333333u) | (o23 & 0xccccccccu);
#pragma unroll
                    for (int r = 0; r < 4; r++) {
                        lo4[r] = n[r] & 0x0f0f0f0fu;
                        hi4[r] = (n[r] >> 4) & 0x0f0f0f0fu;
                        // code c to the selectors of a value's two bytes, 2 c and 2 c + 1; or to its place in the table
                        lo4[r] = IN_REGS ? lo4[r] * 0x22u + 0x10101010u : lo4[r] | pair4;
                        hi4[r] = IN_REGS ? hi4[r] * 0x22u + 0x10101010u : hi4[r] | pair4;
                    }
                }
                uint32_t hi[16], lo[16];
#pragma unroll
                for (int i = 0; i < 8; i++) {
                    if constexpr (IN_REGS) {
#pragma unroll
                        for (int r = 0; r < 4; r += 2) {
                            // two weights at a time: a byte of selectors from each of two words
                            const uint32_t pick = (uint32_t)(i >> 1) | (uint32_t)(4 + (i >> 1)) << 4;
                            const uint32_t at = (i & 1) ? prmt_b32(hi4[r], hi4[r + 1], pick) : prmt_b32(lo4[r], lo4[r + 1], pick);
                            hi[2 * i + r / 2] = prmt_b32(t_hi[0], t_hi[NV / 2 - 1], at);
                            if (PASSES == 2) lo[2 * i + r / 2] = prmt_b32(t_lo[0], t_lo[NV / 2 - 1], at);
                        }
                    } else {
                        uint32_t e[4];
#pragma unroll
                        for (int r = 0; r < 4; r++)
                            e[r] = *reinterpret_cast<const uint32_t*>(smem + prmt_b32((i & 1) ? hi4[r] : lo4[r], bank, 0x6504u | (uint32_t)((i >> 1) << 4)));
                        hi[2 * i] = prmt_b32(e[0], e[1], 0x5410u);
                        hi[2 * i + 1] = prmt_b32(e[2], e[3], 0x5410u);
                        if (PASSES == 2) {
                            lo[2 * i] = prmt_b32(e[0], e[1], 0x7632u);
                            lo[2 * i + 1] = prmt_b32(e[2], e[3], 0x7632u);
                        }
                    }
                }
                if (u == 0 && round > 0) {                        // the stage is touched only here: the work above overlaps its last MMAs
                    if (!__all_sync(0xffffffffu, mbar_wait_bounded(bar_aempty + 8 * sub, (round - 1) & 1))) { timed_out = true; break; }
                    tc_fence_after_sync();
                }
                tmem_st_x16(t_dst + (uint32_t)u * 16u, hi);
                if (PASSES == 2) tmem_st_x16(t_dst + 32u + (uint32_t)u * 16u, lo);
            }
            if (timed_out) break;
            tmem_st_wait();
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_afull + 8 * sub);
        }
        if (SEG && seg + 1 < segments && !timed_out) {
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(bar_acc, seg & 1))) { timed_out = true; break; }
            tc_fence_after_sync();
            hl_drain(sums, t_acc, lo_col, sub, rows, seg > 0);
            tc_fence_before_sync();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_drained);
        }
        }
    } else if (warp == kHlTmaWarp) {
        // ---------------- TMA: activation blocks [rows][64 k] (the whole warp walks the loop, lane 0 issues) ----------------
        if (lane == 0) tma_prefetch_descriptor(&tmX);
        pdl_wait_prior_grids();                                   // the activations may come from the previous kernel
        const int boxes = (rows + p.box_rows - 1) / p.box_rows;
        const uint32_t box_bytes = (uint32_t)p.box_rows * 128u;
        int xs = 0, round = 0;
        for (int j = 0; j < nblk; j++) {
            if (round > 0) {
                if (!__all_sync(0xffffffffu, mbar_wait_bounded(bar_xempty + 8 * xs, (round - 1) & 1))) { timed_out = true; break; }
            }
            if (lane == 0) {
                const uint32_t dst = smem_base + kHlXOff + xs * p.x_slot_bytes;
                mbar_arrive_expect_tx(bar_xfull + 8 * xs, boxes * box_bytes);      // rows and k beyond the end are zero-filled and counted
                for (int i = 0; i < boxes; i++)
                    tma_load_2d(dst + i * box_bytes, &tmX, (blk_begin + j) * kHlStepK, row0 + i * p.box_rows, bar_xfull + 8 * xs);
            }
            __syncwarp();
            if (++xs == p.x_slots) { xs = 0; round++; }
        }
    } else {
        // ---------------- MMA issue ----------------
        // The whole warp walks straight through and one elected lane's predicate guards the instructions: their operands
        // stay in uniform registers.  Inside an `if (lane == 0)` every tcgen05.mma took ~120 cycles to issue, whatever
        // its N: more than it runs up to 240 rows (8192 x 8192, q = 2, 128 rows: 47.5 us against 37.6).
        const uint32_t idesc = umma_idesc_f16_f32(n_mma);
        const uint64_t dx0 = umma_desc_k_sw128(smem_base + kHlXOff);
        const uint32_t elected = elect_one();
        int xs = 0, xround = 0, seg = 0, left = 0;                // left: blocks of the segment that are to come
        for (int j = 0; j < nblk; j++) {
            const bool first = SEG ? left == 0 : j == 0;
            if (SEG && first) {
                if (seg > 0 && !__all_sync(0xffffffffu, mbar_wait_bounded(bar_drained, (seg - 1) & 1))) { timed_out = true; break; }
                left = seg_blocks;
                seg++;
            }
            if (SEG) left--;
            const int st = j & (kHlStages - 1);
            const uint32_t ap = (uint32_t)(j / kHlStages) & 1u;
            if (!__all_sync(0xffffffffu, mbar_wait_bounded(bar_xfull + 8 * xs, xround & 1) && mbar_wait_bounded(bar_afull + 8 * st, ap))) {
                timed_out = true;
                break;
            }
            tc_fence_after_sync();
            const uint32_t a_t = tmem_base + kHlACol + (uint32_t)st * 64u;
            const uint64_t dx = dx0 + (uint64_t)((xs * p.x_slot_bytes) >> 4);
#pragma unroll
            for (int ps = 0; ps < PASSES; ps++)
#pragma unroll
                for (int k16 = 0; k16 < 4; k16++)
                    umma_f16_ts_if(elected, tmem_base + (ps ? lo_col : 0u), a_t + (uint32_t)(ps * 32 + k16 * 8), dx + (uint64_t)(k16 * 2),
                                   idesc, k16 || !first || (ps && !lo_col) ? 1u : 0u);
            umma_commit_if(elected, bar_aempty + 8 * st);
            umma_commit_if(elected, bar_xempty + 8 * xs);
            if (SEG && left == 0 && j + 1 < nblk) umma_commit_if(elected, bar_acc);
            if (++xs == p.x_slots) { xs = 0; xround++; }
        }
        umma_commit_if(elected, bar_acc);
        __syncwarp();
    }
    pdl_wait_prior_grids();                  // before any store to global memory
    if (timed_out) atomicExch(p.status, kStatusTcTimeout);

    // ---------------- epilogue: TMEM lane = output column, TMEM column = activation row ----------------
    const bool split = p.splits > 1;
    if (warp >= kHlFirstExpWarp) {
        const bool ok = __all_sync(0xffffffffu, !timed_out && mbar_wait_bounded(bar_acc, (segments - 1) & 1));
        if (!ok) atomicExch(p.status, kStatusTcTimeout);
        tc_fence_after_sync();
        // the activation ring is idle: every load has been consumed when the accumulators are complete
        float* scratch = reinterpret_cast<float*>(smem + kHlXOff) + ew * (16 * 33);
        // columns that the split operand does not hold exactly (not finite: nothing to be exact about)
        const int k0 = blk_begin * kHlStepK, k1 = min(p.K, (blk_begin + nblk) * kHlStepK), col_c = min(col, N - 1);
        bool wide = false;
        if (PASSES == 2) {
            const unsigned max_bits = s_max[col_l];
            if (max_bits >= 0x7000u && max_bits < 0x7c00u) wide = hl_has_tiny_scale<Q, BIAS>(p, col_c, k0, k1, max_bits);
        }
        const bool any_wide = __any_sync(0xffffffffu, wide);
        for (int c = sub; 16 * c < rows && ok; c += 4) {          // 16 activation rows per tcgen05.ld; warp-uniform
            uint32_t r[16];
            tmem_ld_x16(t_acc + 16u * (uint32_t)c, r);
            if (SEG && lo_col) {
                uint32_t l[16];
                tmem_ld_x16(t_acc + lo_col + 16u * (uint32_t)c, l);
                tmem_ld_wait();
#pragma unroll
                for (int i = 0; i < 16; i++) r[i] = __float_as_uint(__uint_as_float(r[i]) + __uint_as_float(l[i]));
            }
            tmem_ld_wait();
            if (SEG && segments > 1) {
#pragma unroll
                for (int i = 0; i < 16; i++) r[i] = __float_as_uint(__uint_as_float(r[i]) + sums[4 * (c - sub) + i]);
            }
#pragma unroll
            for (int i = 0; i < 16; i++) r[i] = __float_as_uint(__uint_as_float(r[i]) * unscale);
            unsigned redo = wide ? 0xffffu : 0u;
#pragma unroll
            for (int i = 0; i < 16; i++) redo |= (r[i] & 0x7f800000u) == 0x7f800000u ? 1u << i : 0u;
            if (PASSES == 2 && __any_sync(0xffffffffu, redo != 0u)) {
#pragma unroll
                for (int i = 0; i < 16; i++) scratch[i * 33 + lane] = __uint_as_float(r[i]);
#pragma unroll 1
                for (int i = 0; i < 16 && 16 * c + i < rows; i++) {
                    if (!__any_sync(0xffffffffu, (redo >> i) & 1u)) continue;
                    bool inf, nan;
                    hl_row_class(p, row0 + 16 * c + i, k0, k1, lane, &inf, &nan);
                    if (nan || !(inf || any_wide)) continue;      // NaN: so is the row; finite: a scale is not, and that is right
                    const float v = hl_by_product<Q, BIAS>(p, row0 + 16 * c + i, col_c, k0, k1);
                    if (((redo >> i) & 1u) && (inf || wide)) scratch[i * 33 + lane] = v;
                }
#pragma unroll
                for (int i = 0; i < 16; i++) r[i] = __float_as_uint(scratch[i * 33 + lane]);
            }
            tc_store_block(scratch, r, lane, row0 + 16 * c, n0 + lq * 32, row0 + rows, N, split, p.partial, p.y16, p.y32);
        }
        tc_fence_before_sync();
    }
    __syncthreads();
    if (warp == kHlMmaWarp) {
        tc_fence_after_sync();
        tmem_dealloc(tmem_base, kTcTmemCols);
    }
    if (!split) return;

    // ---------------- split-k: the last CTA of the tile converts the reduced sums and zeroes the workspace ----------------
    if (tid == 0) *s_flag = arrive_acq_rel(p.counters + blockIdx.x) == (unsigned)p.splits - 1u;
    __syncthreads();
    if (!*s_flag) return;
    const int nvec = rows * (kHlCols / 4);
    for (int base = tid; base < nvec; base += 4 * kHlThreads) {
        float4 v[4];
        size_t off[4];
        bool live[4];
#pragma unroll
        for (int u = 0; u < 4; u++) {
            const int idx = base + u * kHlThreads;
            const int c = n0 + 4 * (idx % (kHlCols / 4));
            live[u] = idx < nvec && c < N;
            off[u] = (size_t)(row0 + idx / (kHlCols / 4)) * (size_t)N + c;
            if (live[u]) v[u] = __ldcg(reinterpret_cast<const float4*>(p.partial + off[u]));
        }
#pragma unroll
        for (int u = 0; u < 4; u++) {
            if (!live[u]) continue;
            __stcg(reinterpret_cast<float4*>(p.partial + off[u]), make_float4(0.f, 0.f, 0.f, 0.f));
            if (p.y32) *reinterpret_cast<float4*>(p.y32 + off[u]) = v[u];
            if (p.y16) {
                __half2 lo = __floats2half2_rn(v[u].x, v[u].y), hi = __floats2half2_rn(v[u].z, v[u].w);
                uint2 o;
                o.x = *reinterpret_cast<uint32_t*>(&lo);
                o.y = *reinterpret_cast<uint32_t*>(&hi);
                *reinterpret_cast<uint2*>(p.y16 + off[u]) = o;
            }
        }
    }
    if (tid == 0) p.counters[blockIdx.x] = 0u;
}

}  // namespace lg
