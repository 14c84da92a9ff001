// BCQ matmul for a handful of rows (up to 16) on the warp-level tensor instruction, sm_100a.
//
// With few rows the tcgen05 kernels are bound by what is not proportional to the rows: expanding every weight and passing
// it through tensor memory.  mma.sync takes its A operand from registers, so here a packed word becomes operand
// registers in the lane that loaded it and nothing of the expansion is ever stored:
//
//   A warp takes 32 output columns x 128 k, all planes, at a time (a "unit").  Lane (r = lane / 4, t = lane % 4) holds,
//   per plane, the packed words of columns 4 r .. 4 r + 3 at k-word t (one 128-bit load); columns 4 r, 4 r + 1 are rows
//   r, r + 8 of a first 16 x 16 operand tile, 4 r + 2, 4 r + 3 of a second.  The order of k inside a product is free as
//   long as both operands agree: bits (j, j + 16) of a word are the two halves of one operand register.  The activations of
//   the same k are the B operand, in registers for the whole kernel: a warp keeps its k-range and walks over the columns.
//   One LOP3 makes an operand register of a word whose bits lie at one of four places of the fp16 format: 15 (sign: -1 or
//   +1), 14 (exponent: 0 or 2), 10 (exponent: 2 or 4), 9 (mantissa: 4 or 6).  The two values differ by 2 each time, so the
//   sign's product is that of the operand less (1 + the lower value) times the activation: a sum over the group that does
//   not depend on the weights and is what the fp32 accumulator starts from.  16 bit positions then need 5 shifts, not 15.
//   (inf - inf: a row with an activation that is not finite is left out and computed product by product at the end.)
//   The accumulator of a plane and scale group is multiplied by alpha in fp32; q_bias takes the group's sum of activations.
//   Units come through a ring in shared memory that belongs to one warp (cp.async, no barriers).  The warps that
//   split k add up through shared memory once per 32 columns, k-ranges of different CTAs through fp32 reductions in L2.
//
// GW: packed words per scale group inside a unit: 4 (group size a multiple of 128), 2 (of 64), 1 (of 32).  With fewer
// than four, the four lanes t of a product share the words of one group (each takes NJ = 4 GW of the 16 bit positions).
// MT: tiles of 8 activation rows (1 or 2).  KS: units along k that a warp keeps activations for (2 for 8 rows, 1 for 16).
//
// Bound by the operands' making and the products together: per plane and 4096 weights 64 LOP3 on a pipe that takes half a warp a
// cycle (32 cycles per SM), 20 shifts as multiplications on the other, 16 MT mma.sync at 1024 multiply-adds a cycle (33 MT
// cycles): 52 cycles at MT = 1 and 88 at MT = 2 on registers alone.  What a unit costs beside its planes is then the rest,
// and is kept small: all planes' loops unrolled (Q), addresses as 32-bit offsets from the tensors' bases, pieces beyond an end
// fetched as zeros rather than branched around, words in shared memory at places that 16-byte reads find without conflicts
// (chunk XOR k-word), the accumulators' start as the first product's C operand (it was copied: 8 moves a plane).  156
// instructions a plane instead of 192.  Measured, us, with this / before, 28672 x 8192, q = 4 + q_bias, 4 rows: 64.8 / 80.0 = 2.1
// TB/s (160 with gemm_tc, 116 with gemm_hl); 49152 x 12288, q = 3, 4 rows: 126.7 / 149.6; 8192 x 8192, q = 2, 4 rows: 14.3 /
// 17.2; 2048 x 2048, q = 4, 4 rows: 4.37 / 4.43.  Activations in shared memory and runs of units per warp instead of a k-range
// per warp: 64.4, but 1 to 2 us more below 4096 x 4096.
#pragma once
#include "gemv_tma.cuh"

namespace lg {

constexpr int kFrWarps = 16;
constexpr int kFrThreads = kFrWarps * 32;
constexpr int kFrCols = 32;                   // columns per unit
constexpr int kFrMaxRows = 16;
constexpr int kFrRedStride = 12;              // floats between the rows of a reduction block: conflict-free stores
constexpr int kFrMaxDepth = 6;
constexpr int kFrSmemBytes = kSmemLimit;
constexpr int kFrTailBytes = 64;              // a flag, 16 bits of rows per warp
__host__ __device__ constexpr int fr_unit_bytes(int gw, int q, bool bias) { return q * 512 + (q + (bias ? 1 : 0)) * (4 / gw) * 64; }
__host__ __device__ constexpr int fr_red_floats(int mt) { return 4 * mt * 8 * kFrRedStride; }     // per warp
// units of a warp's ring (at least 2 are needed)
__host__ __device__ constexpr int fr_depth(int gw, int mt, int q, bool bias) {
    const int per_warp = (kFrSmemBytes - kFrTailBytes - 2 * kFrWarps * fr_red_floats(mt) * 4) / kFrWarps;
    const int d = per_warp / fr_unit_bytes(gw, q, bias);
    // a wait for each of these; 4 and 5 units are no faster than 3: 8196 x 8192, g = 64, q = 3, 8 rows 22.9 / 21.5 us, q = 2 + q_bias, 16 rows 29.9 / 29.0
    return d >= kFrMaxDepth ? kFrMaxDepth : d >= 3 ? 3 : d;
}

struct FrParams {
    const uint32_t* bW;      // [K/32][q][N]
    const __half* alpha;     // [G][q][N]
    const __half* q_bias;    // [G][N] or nullptr
    const __half* x;         // [m][K]
    float* partial;          // [m][N] fp32, zero between launches (more than one slab)
    unsigned* counters;      // [gridDim.x], zero between launches
    __half* y16;             // [m][N] or nullptr
    float* y32;              // [m][N] or nullptr
    int N, K, q, g, m;
    int kw;                  // warps that split a slab's k: 2, 4, 8 or 16; the other factor of 16 splits the columns
    int steps_per_slab;      // 128-k steps of a slab, at most kw * KS
    int tiles_per_cta;       // 32-column tiles per CTA
    int depth;               // units of a warp's ring
    // fp16 pairs of 1, 2 and 4: as arguments they stay in registers; as literals the compiler made them anew for every LOP3
    uint32_t ones, twos, fours;
    // k-word -> scale group: ceil(2^(32 + shift) / (g / 32)), 0 for g = 32.  shift: 0, or where WIDE the most that is less than g / 32,
    // which is exact for every k-word below 2^31
    uint32_t group_magic;
    int group_shift;
};

__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// D += A B, m16n8k16, fp16 in, fp32 accumulation
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2]) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
        : "+f"(d[0]), "+f"(d[1]), "+f"(d[2]), "+f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]));
}
// D = A B + C
__device__ __forceinline__ void mma_16816(float (&d)[4], const uint32_t (&a)[4], const uint32_t (&b)[2], const float4& c) {
    asm("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%10,%11,%12,%13};"
        : "=f"(d[0]), "=f"(d[1]), "=f"(d[2]), "=f"(d[3])
        : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b[0]), "r"(b[1]), "f"(c.x), "f"(c.y), "f"(c.z), "f"(c.w));
}
// Where bit position pos of a half goes (shift left by fr_shift) and what it becomes there: class 0 the sign, 1 to 3 as above.
__host__ __device__ constexpr int fr_shift(int pos) {
    return pos >= 14 || pos == 10 || pos == 9 ? 0 : pos >= 12 || pos == 8 || pos == 7 ? 2 : pos == 11 || pos == 6 || pos == 5 ? 4
           : pos >= 3 ? 6 : pos >= 1 ? 8 : 10;
}
__host__ __device__ constexpr int fr_class(int pos) {
    const int at = pos + fr_shift(pos);
    return at == 15 ? 0 : at == 14 ? 1 : at == 10 ? 2 : 3;
}
// minus (1 + the lower value) of the class, fp16 pair
__host__ __device__ constexpr uint32_t fr_offset(int pos) {
    return fr_class(pos) == 0 ? 0u : fr_class(pos) == 1 ? 0xbc00bc00u : fr_class(pos) == 2 ? 0xc200c200u : 0xc500c500u;
}
template <int LUT>
__device__ __forceinline__ uint32_t lop3(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, %4;" : "=r"(d) : "r"(a), "r"(b), "r"(c), "n"(LUT));
    return d;
}
// operand register of bit position POS (of both halves)
template <int POS>
__device__ __forceinline__ uint32_t fr_operand(uint32_t word, uint32_t ones, uint32_t twos, uint32_t fours) {
    const uint32_t w = word << fr_shift(POS);
    constexpr int cls = fr_class(POS);
    if constexpr (cls == 0) return lop3<0xae>(w, 0x80008000u, ones);              // (~w & mask) | 1: set -> +1, clear -> -1
    else if constexpr (cls == 1) return w & 0x40004000u;                            // 0 or 2
    else if constexpr (cls == 2) return lop3<0xea>(w, 0x04000400u, twos);         // (w & mask) | 2: 2 or 4
    else return lop3<0xea>(w, 0x02000200u, fours);                                 // (w & mask) | 4: 4 or 6
}
// One plane of one scale group: both operand tiles times MT x 8 rows.  Product S: positions FIRST + 2 S, FIRST + 2 S + 1.
template <int S, int COUNT, int FIRST, int MT>
__device__ __forceinline__ void fr_products(float (&d0)[MT][4], float (&d1)[MT][4], const uint32_t (&w)[4], const uint32_t (&bx)[COUNT][MT][2],
                                            const float4 (&start)[MT], uint32_t ones, uint32_t twos, uint32_t fours) {
    if constexpr (S < COUNT) {
        constexpr int P0 = FIRST + 2 * S, P1 = P0 + 1;
        const uint32_t a0[4] = {fr_operand<P0>(w[0], ones, twos, fours), fr_operand<P0>(w[1], ones, twos, fours),
                                fr_operand<P1>(w[0], ones, twos, fours), fr_operand<P1>(w[1], ones, twos, fours)};
        const uint32_t a1[4] = {fr_operand<P0>(w[2], ones, twos, fours), fr_operand<P0>(w[3], ones, twos, fours),
                                fr_operand<P1>(w[2], ones, twos, fours), fr_operand<P1>(w[3], ones, twos, fours)};
#pragma unroll
        for (int nt = 0; nt < MT; nt++) {
            if constexpr (S == 0) {
                mma_16816(d0[nt], a0, bx[S][nt], start[nt]);
                mma_16816(d1[nt], a1, bx[S][nt], start[nt]);
            } else {
                mma_16816(d0[nt], a0, bx[S][nt]);
                mma_16816(d1[nt], a1, bx[S][nt]);
            }
        }
        fr_products<S + 1, COUNT, FIRST, MT>(d0, d1, w, bx, start, ones, twos, fours);
    }
}
// What those accumulators start from: the offsets' products.
template <int S, int COUNT, int FIRST, int MT>
__device__ __forceinline__ void fr_start(float (&d)[MT][4], const uint32_t (&bx)[COUNT][MT][2]) {
    if constexpr (S < COUNT) {
        constexpr uint32_t o0 = fr_offset(FIRST + 2 * S), o1 = fr_offset(FIRST + 2 * S + 1);
        const uint32_t a[4] = {o0, o0, o1, o1};
#pragma unroll
        for (int nt = 0; nt < MT; nt++) mma_16816(d[nt], a, bx[S][nt]);
        fr_start<S + 1, COUNT, FIRST, MT>(d, bx);
    }
}

// A slab's sums of four columns: the output itself, or its share when k is cut into several slabs.
__device__ __forceinline__ void fr_store(const FrParams& p, size_t off, float4 f) {
    if (gridDim.y > 1) {
        red_add_v4(p.partial + off, f);
        return;
    }
    if (p.y32) *reinterpret_cast<float4*>(p.y32 + off) = f;
    if (p.y16) {
        __half2 lo = __floats2half2_rn(f.x, f.y), hi = __floats2half2_rn(f.z, f.w);
        *reinterpret_cast<uint2*>(p.y16 + off) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
    }
}

// Rows whose activations in this slab are not all finite (`rows`, a bit each): their sums over k-words [kw0, kw1) for columns
// [c0, c1), by all threads of the CTA, as the planes give them: products of +-alpha_b (and q_bias) with the activation,
// summed in fp32, 32 k of a plane at a time.
template <bool BIAS>
__device__ __noinline__ void fr_by_product(const FrParams& p, unsigned rows, int c0, int c1, int kw0, int kw1) {
    const int N = p.N, quads = (c1 - c0) / 4;
    for (int row = 0; row < p.m; row++) {
        if (!((rows >> row) & 1u)) continue;
        for (int at = threadIdx.x; at < quads; at += kFrThreads) {
            const int col = c0 + 4 * at;
            float sum[4] = {0.f, 0.f, 0.f, 0.f};
            for (int kw = kw0; kw < kw1; kw++) {
                const size_t grp = (size_t)(32 * kw / p.g);
                const __half* x = p.x + (size_t)row * p.K + 32 * kw;
                for (int b = 0; b < p.q + (BIAS ? 1 : 0); b++) {
                    const bool plane = !BIAS || b < p.q;
                    const uint4 w = plane ? __ldg(reinterpret_cast<const uint4*>(p.bW + ((size_t)kw * p.q + b) * N + col))
                                          : make_uint4(~0u, ~0u, ~0u, ~0u);
                    const uint2 av = __ldg(reinterpret_cast<const uint2*>((plane ? p.alpha + (grp * p.q + b) * N : p.q_bias + grp * N) + col));
                    const float2 a01 = half2_bits_to_float2(av.x), a23 = half2_bits_to_float2(av.y);
                    float s[4] = {0.f, 0.f, 0.f, 0.f};
                    for (int i = 0; i < 32; i++) {
                        const float v = __half2float(x[i]);
                        s[0] = fmaf((w.x >> i) & 1u ? a01.x : -a01.x, v, s[0]);
                        s[1] = fmaf((w.y >> i) & 1u ? a01.y : -a01.y, v, s[1]);
                        s[2] = fmaf((w.z >> i) & 1u ? a23.x : -a23.x, v, s[2]);
                        s[3] = fmaf((w.w >> i) & 1u ? a23.y : -a23.y, v, s[3]);
                    }
#pragma unroll
                    for (int c = 0; c < 4; c++) sum[c] += s[c];
                }
            }
            fr_store(p, (size_t)row * N + col, make_float4(sum[0], sum[1], sum[2], sum[3]));
        }
    }
}

// Q: planes, 0 for any number.  WIDE: byte offsets count from the slab's first k-word and group, not from the tensors' bases, so that
// those may be 4 GiB long or more (3 % slower).
template <int MT, int GW, bool BIAS, int Q, bool WIDE = false>
__global__ void __launch_bounds__(kFrThreads, 1)
gemm_frag_kernel(const __grid_constant__ FrParams p) {
    constexpr int KS = MT == 1 ? 2 : 1;
    constexpr int NG = 4 / GW;                // scale groups of a unit
    constexpr int NJ = 4 * GW;                // bit positions (of 16) that a lane takes of its word
    constexpr int FIRST = 16 - NJ;            // the lane's positions after its words are shifted up: FIRST .. 15
    extern __shared__ __align__(1024) unsigned char smem[];
    const int tid = threadIdx.x, lane = tid & 31, warp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const int r = lane >> 2, t = lane & 3;
    const int kw_log = 31 - __clz(p.kw), kw_mask = p.kw - 1;
    const int wk = warp & kw_mask, wc = warp >> kw_log, cw = kFrWarps >> kw_log;
    const int N = p.N, K = p.K, q = Q ? Q : p.q;
    const uint32_t ones = p.ones, twos = p.twos, fours = p.fours;
    const int P = q + (BIAS ? 1 : 0);
    const int a_off = q * 512, ub = a_off + P * NG * 64;          // a unit: words of the planes, then scales [plane][group][32 columns]
    unsigned char* ring = smem + warp * (p.depth * ub);
    const uint32_t ring_u = smem_u32(ring);
    float* red = reinterpret_cast<float*>(smem + kFrSmemBytes - kFrTailBytes - 2 * kFrWarps * fr_red_floats(MT) * 4);      // [parity][warp][fr_red_floats]
    int* s_flag = reinterpret_cast<int*>(smem + kFrSmemBytes - kFrTailBytes);
    unsigned short* s_open = reinterpret_cast<unsigned short*>(s_flag + 1);       // per warp: rows with an activation that is not finite

    const int words = K / 32;
    const int steps_total = (words + 3) / 4;
    const int slab0 = blockIdx.y * p.steps_per_slab, slab1 = min(steps_total, slab0 + p.steps_per_slab);
    int nsteps = 0;                           // this warp's steps: slab0 + wk + i kw
#pragma unroll
    for (int i = 0; i < KS; i++) nsteps += (slab0 + wk + i * p.kw < slab1) ? 1 : 0;
    const int tiles = (N + kFrCols - 1) / kFrCols;
    const int tile0 = blockIdx.x * p.tiles_per_cta, tile1 = min(tiles, tile0 + p.tiles_per_cta);

    // ---- the warp's stream of units: (tile, step) ----
    // Byte offsets are 32 bits wide; beyond the end of the stream, the columns or K zeros come instead.
    const uint32_t row_b = (uint32_t)q * (uint32_t)N * 4u;       // bytes of a k-word row of words
    const int f_kw = lane >> 3, f_chunk = lane & 7;
    int fi = 0, fslot = 0, fcol = (tile0 + wc) * kFrCols + 4 * f_chunk;
    const int fcol_end = nsteps ? min(N, tile1 * kFrCols) : 0;    // N % 4 == 0: whole quads
    // this lane's 16 bytes of every plane: chunks of a k-word's 128 bytes at their number XOR the k-word (conflict-free reads below)
    const uint32_t f_dst = ring_u + f_kw * 128 + (f_chunk ^ f_kw) * 16;
    // and its 8 bytes of scales: four (of NG groups: 4 / NG) planes at a time
    constexpr int PB = 4 / NG;
    const int f_plane = f_kw / NG, f_group = f_kw % NG;
    const uint32_t f_adst = ring_u + a_off + lane * 8;
    auto group_of = [&](int kw) {
        if (WIDE) return (p.group_magic ? __umulhi((unsigned)kw, p.group_magic) : (unsigned)kw) >> p.group_shift;
        return GW == 1 && !p.group_magic ? (unsigned)kw : __umulhi((unsigned)kw, p.group_magic);
    };
    const uint32_t grp0 = WIDE ? group_of(4 * slab0) : 0u;
    auto base = [&](const void* tensor, size_t offset) { return reinterpret_cast<const unsigned char*>(tensor) + (WIDE ? offset : 0); };
    auto fetch = [&]() {
        const int kw0 = 4 * (slab0 + wk + fi * p.kw), akw = kw0 + GW * f_group;
        const int end = fcol < fcol_end ? words : 0;
        const uint32_t size = kw0 + f_kw < end ? 16u : 0u, asize = akw < end ? 8u : 0u, at = fslot * ub;
        const uint32_t off = (uint32_t)(kw0 + f_kw - (WIDE ? 4 * slab0 : 0)) * row_b + (uint32_t)fcol * 4u;
        const int pu = Q ? Q : GW == 1 ? q : 8;      // GW = 1 copies scales as often as words: planes that are not there cost too much
#pragma unroll (Q ? Q : GW == 1 ? 4 : 8)
        for (int b = 0; b < pu; b++)
            if (Q || GW == 1 || b < q) cp_async16(f_dst + at + b * 512, base(p.bW, (size_t)(4 * slab0) * q * N * 4) + (off + b * ((uint32_t)N * 4u)), size);
        const uint32_t grp = WIDE ? group_of(akw) - grp0 : group_of(akw);
        const uint32_t aoff = ((grp * q + f_plane) * (uint32_t)N + fcol) * 2u;
#pragma unroll (Q ? Q : GW == 1 ? 2 : 8)
        for (int b = 0; b < pu; b += PB)
            if (b + f_plane < q) cp_async8(f_adst + at + b * (NG * 64), base(p.alpha, (size_t)grp0 * q * N * 2) + (aoff + b * ((uint32_t)N * 2u)), asize);
        if (BIAS && f_plane == 0) cp_async8(f_adst + at + q * (NG * 64), base(p.q_bias, (size_t)grp0 * N * 2) + (grp * (uint32_t)N + fcol) * 2u, asize);
        if (++fslot == p.depth) fslot = 0;
        if (++fi == nsteps) {
            fi = 0;
            fcol += cw * kFrCols;
        }
        cp_async_commit();                    // one group per unit: the wait below counts groups
    };
    auto wait_unit = [&]() {                  // all but the last depth - 2 groups
        if (p.depth == 2) cp_async_wait<0>();
        else if (p.depth == 3) cp_async_wait<1>();
        else cp_async_wait<kFrMaxDepth - 2>();
        __syncwarp();                         // every lane's copies of this unit have landed, every lane has read the previous one
    };
    // packed words and scales are never written by a kernel: the stream starts while the previous kernel drains
    pdl_launch_dependents();
#pragma unroll 1
    for (int i = 0; i < p.depth - 1; i++) fetch();
    pdl_wait_prior_grids();                   // the activations may come from the previous kernel

    // ---- activations of this warp's k-range, in operand order ----
    uint32_t bx[KS][NG][NJ / 2][MT][2];
    float4 start[KS][NG][MT];                 // what the accumulators start from: rows 8 nt + 2 t, + 1, the same of the tile's other half
    float sx[KS][NG][MT][2];                  // BIAS: sums of the group's activations for those rows
    unsigned open = 0u;                       // rows with an activation that is not finite: nor is, then, what they start from
#pragma unroll
    for (int i = 0; i < KS; i++)
#pragma unroll
        for (int gi = 0; gi < NG; gi++) {
            const int kw = 4 * (slab0 + wk + i * p.kw) + gi * GW + ((t * GW) >> 2);
            const int j0 = (t * GW % 4) * 4;  // this lane's first bit position
#pragma unroll
            for (int nt = 0; nt < MT; nt++) {
                uint32_t lo[NJ / 2] = {}, hi[NJ / 2] = {};        // activations j0 .. j0 + NJ - 1 of the word, and those + 16
                const int row = 8 * nt + r;
                if (i < nsteps && kw < words && row < p.m) {
                    const __half* src = p.x + (size_t)row * K + 32 * kw + j0;
                    if constexpr (NJ >= 8) {
#pragma unroll
                        for (int v = 0; v < NJ / 8; v++) {
                            const uint4 a = __ldcg(reinterpret_cast<const uint4*>(src) + v), b = __ldcg(reinterpret_cast<const uint4*>(src + 16) + v);
                            lo[4 * v] = a.x; lo[4 * v + 1] = a.y; lo[4 * v + 2] = a.z; lo[4 * v + 3] = a.w;
                            hi[4 * v] = b.x; hi[4 * v + 1] = b.y; hi[4 * v + 2] = b.z; hi[4 * v + 3] = b.w;
                        }
                    } else {
                        const uint2 a = __ldcg(reinterpret_cast<const uint2*>(src)), b = __ldcg(reinterpret_cast<const uint2*>(src + 16));
                        lo[0] = a.x; lo[1] = a.y;
                        hi[0] = b.x; hi[1] = b.y;
                    }
                }
#pragma unroll
                for (int s = 0; s < NJ / 2; s++) {
                    bx[i][gi][s][nt][0] = prmt_b32(lo[s], hi[s], 0x5410u);       // k of bits 2 s, 2 s + 16
                    bx[i][gi][s][nt][1] = prmt_b32(lo[s], hi[s], 0x7632u);       // k of bits 2 s + 1, 2 s + 17
                }
            }
            float d[MT][4];
#pragma unroll
            for (int nt = 0; nt < MT; nt++) d[nt][0] = d[nt][1] = d[nt][2] = d[nt][3] = 0.f;
            fr_start<0, NJ / 2, FIRST, MT>(d, bx[i][gi]);
#pragma unroll
            for (int nt = 0; nt < MT; nt++) {
                start[i][gi][nt] = make_float4(d[nt][0], d[nt][1], d[nt][0], d[nt][1]);
#pragma unroll
                for (int e = 0; e < 2; e++) open |= fabsf(d[nt][e]) <= 3.402823466e38f ? 0u : 1u << (8 * nt + 2 * t + e);
                if (BIAS) {
                    const uint32_t one[4] = {ones, ones, ones, ones};
                    float e[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
                    for (int s = 0; s < NJ / 2; s++) mma_16816(e, one, bx[i][gi][s][nt]);
                    sx[i][gi][nt][0] = e[0];
                    sx[i][gi][nt][1] = e[1];
                }
            }
        }

    open = __reduce_or_sync(0xffffffffu, open);
    if (lane == 0) s_open[warp] = (unsigned short)open;
    unsigned by_product = 0u;                 // rows left to fr_by_product

    // ---- columns ----
    const int my_tiles = (tile1 - tile0 + cw - 1) >> (4 - kw_log);      // every warp of the CTA walks as many: the barriers match
    const int quad = (r >> 1) + 4 * (r & 1);  // this lane's columns of a tile: two lanes r of a quarter warp are four chunks apart
    int slot = 0, parity = 0;
#pragma unroll 1
    for (int ti = 0; ti < my_tiles; ti++) {
        const int tile = tile0 + wc + ti * cw;
        float acc[4][MT][2];
#pragma unroll
        for (int c = 0; c < 4; c++)
#pragma unroll
            for (int nt = 0; nt < MT; nt++) acc[c][nt][0] = acc[c][nt][1] = 0.f;
        if (tile < tile1) {
#pragma unroll
            for (int i = 0; i < KS; i++) {
                if (i >= nsteps) continue;
                wait_unit();
                fetch();
                const unsigned char* u = ring + slot * ub;
                if (++slot == p.depth) slot = 0;
                auto plane = [&](int b) {
#pragma unroll
                    for (int gi = 0; gi < NG; gi++) {
                        const int kw = gi * GW + ((t * GW) >> 2);
                        const uint2 av = *reinterpret_cast<const uint2*>(u + a_off + (b * NG + gi) * 64 + quad * 8);
                        const uint4 wv = *reinterpret_cast<const uint4*>(u + b * 512 + kw * 128 + (quad ^ kw) * 16);
                        const float2 a01 = half2_bits_to_float2(av.x), a23 = half2_bits_to_float2(av.y);
                        uint32_t w[4] = {wv.x, wv.y, wv.z, wv.w};
                        if (GW < 4) {         // this lane's NJ positions to the top of each half
#pragma unroll
                            for (int c = 0; c < 4; c++) w[c] <<= FIRST - (t * GW % 4) * 4;
                        }
                        float d0[MT][4], d1[MT][4];
                        fr_products<0, NJ / 2, FIRST, MT>(d0, d1, w, bx[i][gi], start[i][gi], ones, twos, fours);
#pragma unroll
                        for (int nt = 0; nt < MT; nt++)
#pragma unroll
                            for (int e = 0; e < 2; e++) {
                                acc[0][nt][e] = fmaf(a01.x, d0[nt][e], acc[0][nt][e]);
                                acc[1][nt][e] = fmaf(a01.y, d0[nt][2 + e], acc[1][nt][e]);
                                acc[2][nt][e] = fmaf(a23.x, d1[nt][e], acc[2][nt][e]);
                                acc[3][nt][e] = fmaf(a23.y, d1[nt][2 + e], acc[3][nt][e]);
                            }
                    }
                };
                if constexpr (Q != 0) {
#pragma unroll
                    for (int b = 0; b < Q; b++) plane(b);
                } else {
#pragma unroll 1
                    for (int b = 0; b < q; b++) plane(b);
                }
                if (BIAS) {
#pragma unroll
                    for (int gi = 0; gi < NG; gi++) {
                        const uint2 av = *reinterpret_cast<const uint2*>(u + a_off + (q * NG + gi) * 64 + quad * 8);
                        const float2 a01 = half2_bits_to_float2(av.x), a23 = half2_bits_to_float2(av.y);
#pragma unroll
                        for (int nt = 0; nt < MT; nt++)
#pragma unroll
                            for (int e = 0; e < 2; e++) {
                                acc[0][nt][e] = fmaf(a01.x, sx[i][gi][nt][e], acc[0][nt][e]);
                                acc[1][nt][e] = fmaf(a01.y, sx[i][gi][nt][e], acc[1][nt][e]);
                                acc[2][nt][e] = fmaf(a23.x, sx[i][gi][nt][e], acc[2][nt][e]);
                                acc[3][nt][e] = fmaf(a23.y, sx[i][gi][nt][e], acc[3][nt][e]);
                            }
                    }
                }
            }
        }
        // ---- add the kw warps of this column group: block [column c of the quad][row][r] per warp ----
        {
            float* mine = red + (parity * kFrWarps + warp) * fr_red_floats(MT);
#pragma unroll
            for (int c = 0; c < 4; c++)
#pragma unroll
                for (int nt = 0; nt < MT; nt++)
#pragma unroll
                    for (int e = 0; e < 2; e++)
                        mine[((c * MT + nt) * 8 + 2 * t + e) * kFrRedStride + quad] = acc[c][nt][e];
            asm volatile("bar.sync %0, %1;" ::"r"(1 + wc), "r"(p.kw * 32) : "memory");
            // 64 MT (row, column quad) sums by two warps per 8 rows, other warps each time
            const int turn = (wk - ti * 2 * MT) & kw_mask;
            // the warps of this barrier hold all of the slab's activations: every column group finds the same rows
            if (ti == 0) by_product = __reduce_or_sync(0xffffffffu, s_open[wc * p.kw + (lane & kw_mask)]);
            for (int o = turn * 32 + lane; o < 64 * MT && tile < tile1; o += p.kw * 32) {
                const int row = o >> 3, rr = o & 7, nt = row >> 3, m8 = row & 7;
                const int col = tile * kFrCols + 4 * rr;
                if (row >= p.m || col >= N || ((by_product >> row) & 1u)) continue;
                const float* src = red + (parity * kFrWarps + wc * p.kw) * fr_red_floats(MT) + (nt * 8 + m8) * kFrRedStride + rr;
                float s[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll 4
                for (int v = 0; v < p.kw; v++)
#pragma unroll
                    for (int c = 0; c < 4; c++) s[c] += src[v * fr_red_floats(MT) + c * MT * 8 * kFrRedStride];
                fr_store(p, (size_t)row * N + col, make_float4(s[0], s[1], s[2], s[3]));
            }
            parity ^= 1;
        }
    }
    if (by_product) fr_by_product<BIAS>(p, by_product, tile0 * kFrCols, min(N, tile1 * kFrCols), 4 * slab0, min(words, 4 * slab1));
    if (gridDim.y == 1) return;

    // ---- slabs: the last CTA of the column range converts the reduced sums and zeroes the workspace ----
    __syncthreads();
    if (tid == 0) *s_flag = arrive_acq_rel(p.counters + blockIdx.x) == gridDim.y - 1u;
    __syncthreads();
    if (!*s_flag) return;
    const int c0 = tile0 * kFrCols, quads = (min(N, tile1 * kFrCols) - c0) / 4;
    for (int idx = tid; idx < quads * p.m; idx += kFrThreads) {
        const size_t off = (size_t)(idx / quads) * N + c0 + 4 * (idx % quads);
        const float4 v = __ldcg(reinterpret_cast<const float4*>(p.partial + off));
        __stcg(reinterpret_cast<float4*>(p.partial + off), make_float4(0.f, 0.f, 0.f, 0.f));
        if (p.y32) *reinterpret_cast<float4*>(p.y32 + off) = v;
        if (p.y16) {
            __half2 lo = __floats2half2_rn(v.x, v.y), hi = __floats2half2_rn(v.z, v.w);
            *reinterpret_cast<uint2*>(p.y16 + off) = make_uint2(*reinterpret_cast<uint32_t*>(&lo), *reinterpret_cast<uint32_t*>(&hi));
        }
    }
    if (tid == 0) p.counters[blockIdx.x] = 0u;
}

}  // namespace lg
