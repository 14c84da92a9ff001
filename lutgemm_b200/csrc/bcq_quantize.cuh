// BCQ quantiser on the device: greedy initialisation + alternating refinement, one warp per (row, group).
//
// Replaces quantize() of the reference's examples/bcq.py:23-98 (torch tensors on CUDA, a dozen library kernels per
// round over the whole layer) for its default, unweighted case (exponent 0, clipping 1, pruning 0):
//   greedy       examples/bcq.py:100-128   b_i = sign(r), alpha_i = mean |r|, r -= alpha_i b_i
//   refinement   examples/bcq.py:130-157   alpha from the normal equations (B^T B) alpha = B^T w by q steps of conjugate
//                                          gradient started at the current alpha (examples/bcq.py:190-206, 1e-6 added to
//                                          both denominators), |alpha| sorted descending, then every weight takes the
//                                          nearest of the 2^q levels sum_i +-alpha_i (examples/bcq.py:165-188: levels
//                                          sorted, q bisection steps on midpoints, `w < mid` goes left).
// Here a group up to 1024 wide never leaves its warp (wider ones take a CTA, see the end of this file): the weights stay in registers (lane l holds elements l, l + 32, ...), the
// q x q system is accumulated with warp reductions and solved redundantly by every lane, the 2^q levels are rank-sorted
// in shared memory.  Output in the quantiser's layout (alpha [N][G][q] fp32, binary int8 [N][G][g][q]) and/or directly
// in the matmul's container layout (bW uint32 [K/32][q][N] by warp ballots, alpha fp16 [G][q][N]).
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace lg {

constexpr int kBqMaxQ = 8;
constexpr int kBqWarps = 8;                   // warps (groups) per CTA

struct BqParams {
    const float* w;          // [N][K], groups of g consecutive k
    int N, K, g, q, rounds;
    float* alpha_py;         // [N][G][q] or nullptr
    signed char* binary_py;  // [N][G][g][q] or nullptr
    uint32_t* bW;            // [K/32][q][N] or nullptr (needs g % 32 == 0)
    __half* alpha_k;         // [G][q][N] or nullptr
};

__device__ __forceinline__ float warp_sum_f(float v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// code of one element: bits 0..7 = "+1" per plane, bits 8..15 = "non-zero" per plane
__device__ __forceinline__ float code_sign(uint32_t code, int i) {
    return ((code >> (8 + i)) & 1u) ? (((code >> i) & 1u) ? 1.f : -1.f) : 0.f;
}

template <int E>
__global__ void __launch_bounds__(kBqWarps * 32)
bcq_quantize_kernel(const BqParams p) {
    __shared__ float s_v[kBqWarps][1 << kBqMaxQ];
    __shared__ float s_vs[kBqWarps][1 << kBqMaxQ];
    __shared__ unsigned char s_ind[kBqWarps][1 << kBqMaxQ];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int G = p.K / p.g;
    const long long grp = (long long)blockIdx.x * kBqWarps + wib;
    if (grp >= (long long)p.N * G) return;                 // whole warps leave together
    const int n = (int)(grp / G), gi = (int)(grp % G);
    const int g = p.g, q = p.q;
    const float* wg = p.w + (size_t)n * p.K + (size_t)gi * g;

    float wv[E];
    uint32_t code[E];
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int idx = e * 32 + lane;
        wv[e] = idx < g ? wg[idx] : 0.f;
        code[e] = 0u;
    }
    float alpha[kBqMaxQ];
#pragma unroll
    for (int i = 0; i < kBqMaxQ; i++) alpha[i] = 0.f;

    // ---- greedy ----
    {
        float r[E];
#pragma unroll
        for (int e = 0; e < E; e++) r[e] = wv[e];
        for (int i = 0; i < q; i++) {
            float s = 0.f;
#pragma unroll
            for (int e = 0; e < E; e++) s += fabsf(r[e]);          // padding elements are 0
            float a = warp_sum_f(s) / (float)g;
            if (a != a) a = 0.f;
#pragma unroll
            for (int e = 0; e < E; e++) {
                const float b = r[e] > 0.f ? 1.f : (r[e] < 0.f ? -1.f : 0.f);
                if (b > 0.f) code[e] |= 1u << i;
                if (b != 0.f) code[e] |= 1u << (8 + i);
                r[e] -= b * a;
            }
#pragma unroll
            for (int j = 0; j < kBqMaxQ; j++) if (j == i) alpha[j] = a;
        }
    }

    // ---- alternating refinement ----
    if (q > 1) {
        const int nlev = 1 << q;
        for (int round = 0; round < p.rounds; round++) {
            // normal equations: integer Gram matrix and B^T w
            float A[kBqMaxQ][kBqMaxQ] = {}, btw[kBqMaxQ];
#pragma unroll
            for (int i = 0; i < kBqMaxQ; i++) {
                if (i >= q) { btw[i] = 0.f; continue; }
                float s = 0.f;
#pragma unroll
                for (int e = 0; e < E; e++) s += code_sign(code[e], i) * wv[e];
                btw[i] = warp_sum_f(s);
#pragma unroll
                for (int j = 0; j < kBqMaxQ; j++) {
                    if (j < i || j >= q) continue;
                    int c = 0;
#pragma unroll
                    for (int e = 0; e < E; e++) c += (int)(code_sign(code[e], i) * code_sign(code[e], j));
                    c = __reduce_add_sync(0xffffffffu, c);
                    A[i][j] = (float)c;
                    A[j][i] = (float)c;
                }
            }
            // q steps of conjugate gradient from the current alpha (every lane the same arithmetic)
            float x[kBqMaxQ], r[kBqMaxQ], pp[kBqMaxQ], Ap[kBqMaxQ];
            float rtr_new = 0.f;
#pragma unroll
            for (int i = 0; i < kBqMaxQ; i++) {
                x[i] = alpha[i];
                float s = 0.f;
#pragma unroll
                for (int j = 0; j < kBqMaxQ; j++) if (i < q && j < q) s += A[i][j] * alpha[j];
                r[i] = i < q ? btw[i] - s : 0.f;
                pp[i] = r[i];
                rtr_new += r[i] * r[i];
            }
            for (int it = 0; it < q; it++) {
                const float rtr = rtr_new;
                float pAp = 0.f;
#pragma unroll
                for (int i = 0; i < kBqMaxQ; i++) {
                    float s = 0.f;
#pragma unroll
                    for (int j = 0; j < kBqMaxQ; j++) if (i < q && j < q) s += A[i][j] * pp[j];
                    Ap[i] = i < q ? s : 0.f;
                    pAp += pp[i] * Ap[i];
                }
                const float a = rtr / (pAp + 1e-6f);
                rtr_new = 0.f;
#pragma unroll
                for (int i = 0; i < kBqMaxQ; i++) {
                    x[i] += a * pp[i];
                    r[i] -= a * Ap[i];
                    rtr_new += r[i] * r[i];
                }
                const float beta = rtr_new / (rtr + 1e-6f);
#pragma unroll
                for (int i = 0; i < kBqMaxQ; i++) pp[i] = r[i] + beta * pp[i];
            }
            // |alpha| descending (insertion sort over the q live entries)
#pragma unroll
            for (int i = 0; i < kBqMaxQ; i++) alpha[i] = i < q ? fabsf(x[i]) : -1.f;
#pragma unroll
            for (int i = 1; i < kBqMaxQ; i++) {
#pragma unroll
                for (int j = i; j > 0; j--) {
                    if (alpha[j] > alpha[j - 1]) { const float t = alpha[j]; alpha[j] = alpha[j - 1]; alpha[j - 1] = t; }
                }
            }
#pragma unroll
            for (int i = 0; i < kBqMaxQ; i++) if (i >= q) alpha[i] = 0.f;

            // the 2^q levels: level c has sign -1 on plane i iff bit q-1-i of c is set (examples/bcq.py:159-163)
            for (int c = lane; c < nlev; c += 32) {
                float v = 0.f;
#pragma unroll
                for (int i = 0; i < kBqMaxQ; i++) if (i < q) v += ((c >> (q - 1 - i)) & 1) ? -alpha[i] : alpha[i];
                s_v[wib][c] = v;
            }
            __syncwarp();
            for (int c = lane; c < nlev; c += 32) {          // rank sort, ties by index
                const float v = s_v[wib][c];
                int rank = 0;
                for (int d = 0; d < nlev; d++) {
                    const float u = s_v[wib][d];
                    rank += (u < v || (u == v && d < c)) ? 1 : 0;
                }
                s_vs[wib][rank] = v;
                s_ind[wib][rank] = (unsigned char)c;
            }
            __syncwarp();
            // nearest level by bisection on the midpoints
#pragma unroll
            for (int e = 0; e < E; e++) {
                int left = 0, right = nlev - 1;
                for (int it = 0; it < q; it++) {
                    const int ml = (left + right - 1) / 2, mr = ml + 1;
                    const float mid = (s_vs[wib][ml] + s_vs[wib][mr]) / 2.f;
                    if (wv[e] < mid) right = ml; else left = mr;
                }
                const uint32_t c = s_ind[wib][left];
                uint32_t pos = 0u;
                for (int i = 0; i < q; i++) pos |= (((c >> (q - 1 - i)) & 1u) ^ 1u) << i;
                if (e * 32 + lane < g) code[e] = pos | (((1u << q) - 1u) << 8);      // padding keeps code 0: it must not count in B^T B
            }
            __syncwarp();
        }
    }

    // ---- outputs ----
    if (p.alpha_py && lane < q) {
        float a = 0.f;
#pragma unroll
        for (int i = 0; i < kBqMaxQ; i++) if (i == lane) a = alpha[i];
        p.alpha_py[((size_t)n * G + gi) * q + lane] = a;
    }
    if (p.alpha_k && lane < q) {
        float a = 0.f;
#pragma unroll
        for (int i = 0; i < kBqMaxQ; i++) if (i == lane) a = alpha[i];
        p.alpha_k[((size_t)gi * q + lane) * p.N + n] = __float2half_rn(a);
    }
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int idx = e * 32 + lane;
        const bool valid = idx < g;
        if (p.binary_py && valid) {
            signed char* dst = p.binary_py + (((size_t)n * G + gi) * g + idx) * q;
            for (int i = 0; i < q; i++) dst[i] = (signed char)code_sign(code[e], i);
        }
        if (p.bW && e * 32 < g) {                          // g % 32 == 0: whole words; a zero code packs as -1
            for (int i = 0; i < q; i++) {
                const uint32_t word = __ballot_sync(0xffffffffu, valid && ((code[e] >> i) & 1u));
                if (lane == 0) p.bW[((size_t)((gi * g) / 32 + e) * q + i) * p.N + n] = word;
            }
        }
    }
}

// ---- groups up to 512 wide, up to four planes ----
// Same arithmetic, several groups to a warp.  LG lanes share one group and hold E weights each (LG * E >= g), so the
// conjugate gradient, whose arithmetic every lane of a group repeats, and the log2(LG) shuffles of a sum are paid once
// for 32 / LG groups.  Per round the group writes one table entry per level, in ascending order of the levels: the level's
// signs as floats and its Gram contributions (1 per pair of planes whose signs differ) packed in 10-bit fields, three
// pairs to a word.  A weight then costs its q comparisons, one table read, q multiply-adds (B^T w) and one integer add
// (B^T B) per word of pairs, and the sums of the next round are complete when the weights of this one are placed.
// Bound by instruction issue, not by memory: the weights are read once.  Measured, N = K = 4096, q = 3, g = 128, 15
// rounds: 406 us; bcq_quantize_kernel, which gives every group a whole warp, takes 3291 us.  Large layers of two to four planes take
// bcq_quantize_lane_kernel (below) instead.
// Sums are added in the order of bcq_quantize_kernel, whose lane L holds weights L, L + 32, ...: a lane here stands for
// NJ = 32 / LG of those lanes (lane, lane + LG, ...), keeps their partial sums apart and adds them first, which is that
// kernel's shuffle over distances 16 .. LG.  So both give the same bits, and which one a group takes does not show.
constexpr int kBqTileWarps = 4;               // 8: 423 us at q = 3, 270 at q = 2, g = 64; 4: 406 and 254
constexpr int kBqTileMaxG = 512;              // 32 lanes of 16 weights; a field of pair counts holds up to 1023
constexpr int kBqTileMaxQ = 4;                // the levels' signs are one 128-bit table entry

template <int LG>
__device__ __forceinline__ float group_sum_f(float v) {
#pragma unroll
    for (int o = LG / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}
template <int LG>
__device__ __forceinline__ uint32_t group_sum_u(uint32_t v) {
#pragma unroll
    for (int o = LG / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

// Partial sums of the NJ lanes that a lane stands for, then the shuffles.
template <int LG>
__device__ __forceinline__ float tile_sum_f(float (&v)[32 / LG]) {
#pragma unroll
    for (int d = 16 / LG; d > 0; d >>= 1)
#pragma unroll
        for (int j = 0; j < d; j++) v[j] += v[j + d];
    return group_sum_f<LG>(v[0]);
}

// The scales of a group from B^T B and B^T w: Q steps of conjugate gradient from the current ones, |alpha| in descending order.
template <int Q>
__device__ __forceinline__ void bq_solve(const float (&A)[Q][Q], const float (&btw)[Q], float (&alpha)[Q]) {
    float x[Q], r[Q], pp[Q], Ap[Q];
    float rtr_new = 0.f;
#pragma unroll
    for (int i = 0; i < Q; i++) {
        x[i] = alpha[i];
        float s = 0.f;
#pragma unroll
        for (int j = 0; j < Q; j++) s += A[i][j] * alpha[j];
        r[i] = btw[i] - s;
        pp[i] = r[i];
        rtr_new += r[i] * r[i];
    }
#pragma unroll
    for (int it = 0; it < Q; it++) {
        const float rtr = rtr_new;
        float pAp = 0.f;
#pragma unroll
        for (int i = 0; i < Q; i++) {
            float s = 0.f;
#pragma unroll
            for (int j = 0; j < Q; j++) s += A[i][j] * pp[j];
            Ap[i] = s;
            pAp += pp[i] * s;
        }
        const float a = rtr / (pAp + 1e-6f);
        rtr_new = 0.f;
#pragma unroll
        for (int i = 0; i < Q; i++) {
            x[i] += a * pp[i];
            r[i] -= a * Ap[i];
            rtr_new += r[i] * r[i];
        }
        const float beta = rtr_new / (rtr + 1e-6f);
#pragma unroll
        for (int i = 0; i < Q; i++) pp[i] = r[i] + beta * pp[i];
    }
    // insertion sort
#pragma unroll
    for (int i = 0; i < Q; i++) alpha[i] = fabsf(x[i]);
#pragma unroll
    for (int i = 1; i < Q; i++) {
#pragma unroll
        for (int j = i; j > 0; j--)
            if (alpha[j] > alpha[j - 1]) { const float t = alpha[j]; alpha[j] = alpha[j - 1]; alpha[j - 1] = t; }
    }
}

template <int LG, int Q>
__global__ void __launch_bounds__(kBqTileWarps * 32)
bcq_quantize_tile_kernel(const BqParams p) {
    constexpr int E = 16;                                  // weights per lane: register e is weight (e % EE) * 32 + LG * (e / EE) + l
    constexpr int NJ = 32 / LG, EE = E / NJ;
    constexpr int GPW = 32 / LG;                           // groups per warp
    constexpr int NLEV = 1 << Q;
    constexpr int PAIRS = Q * (Q - 1) / 2;
    constexpr int PW = (PAIRS + 2) / 3;                    // words of packed pair counts
    __shared__ float s_level[kBqTileWarps][GPW][NLEV];     // unsorted, then ascending
    __shared__ __align__(16) float s_sign[kBqTileWarps][GPW][NLEV][4];
    __shared__ uint32_t s_pair[kBqTileWarps][GPW][NLEV][PW > 0 ? PW : 1];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int l = lane % LG, sub = lane / LG;
    const int G = p.K / p.g, g = p.g;
    const long long groups = (long long)p.N * G;
    const long long first = ((long long)blockIdx.x * kBqTileWarps + wib) * GPW;
    if (first >= groups) return;                           // whole warps leave together
    // groups of consecutive rows share a warp: their packed words are neighbours
    const bool live = first + sub < groups;                // a group beyond the end repeats the warp's first one
    const long long grp = live ? first + sub : first;
    const int gi = (int)(grp / p.N), n = (int)(grp % p.N);
    const float* wg = p.w + (size_t)n * p.K + (size_t)gi * g;

    float wv[E];
    uint32_t valid = 0u;                                   // bit e: register e holds a weight
#pragma unroll
    for (int e = 0; e < E; e++) {
        const int at = (e % EE) * 32 + LG * (e / EE) + l;
        wv[e] = at < g ? __ldg(wg + at) : 0.f;
        valid |= (at < g ? 1u : 0u) << e;
    }

    float alpha[Q], btw[Q];
    uint32_t pos[Q], nz[Q];                                // per plane: sign is +1 / sign is not 0, bit e for register e
    float A[Q][Q];                                         // B^T B
    // ---- greedy ----
    {
        float r[E];
#pragma unroll
        for (int e = 0; e < E; e++) r[e] = wv[e];
#pragma unroll
        for (int i = 0; i < Q; i++) {
            float s[NJ] = {}, t[NJ] = {};
#pragma unroll
            for (int e = 0; e < E; e++) s[e / EE] += fabsf(r[e]);            // padding elements are 0
            float a = tile_sum_f<LG>(s) / (float)g;
            if (a != a) a = 0.f;
            alpha[i] = a;
            pos[i] = nz[i] = 0u;
#pragma unroll
            for (int e = 0; e < E; e++) {
                const float b = r[e] > 0.f ? 1.f : (r[e] < 0.f ? -1.f : 0.f);
                if (b > 0.f) pos[i] |= 1u << e;
                if (b != 0.f) nz[i] |= 1u << e;
                t[e / EE] += b * wv[e];
                r[e] -= b * a;
            }
            // padding never counts: its weight is 0, and its code is masked out
            pos[i] &= valid;
            nz[i] &= valid;
            btw[i] = tile_sum_f<LG>(t);
        }
#pragma unroll
        for (int i = 0; i < Q; i++)
#pragma unroll
            for (int j = i; j < Q; j++) {
                const uint32_t both = nz[i] & nz[j];
                const int c = __popc(both) - 2 * __popc((pos[i] ^ pos[j]) & both);
                A[i][j] = A[j][i] = (float)(int)group_sum_u<LG>((uint32_t)c);
            }
    }

    // ---- alternating refinement ----
    const uint32_t pad = (uint32_t)(E - __popc(valid));
    for (int round = 0; Q > 1 && round < p.rounds; round++) {
        bq_solve<Q>(A, btw, alpha);
        // the levels, in ascending order, ties by index: level c has sign -1 on plane i iff bit Q-1-i of c is set
        constexpr int LPL = (NLEV + LG - 1) / LG;          // levels per lane
        float lv[LPL];
        __syncwarp();                                      // the previous round's tables have been read
#pragma unroll
        for (int u = 0; u < LPL; u++) {
            const int c = l + u * LG;
            float v = 0.f;
#pragma unroll
            for (int i = 0; i < Q; i++) v += ((c >> (Q - 1 - i)) & 1) ? -alpha[i] : alpha[i];
            lv[u] = v;
            if (c < NLEV) s_level[wib][sub][c] = v;
        }
        __syncwarp();
        int rank[LPL];
#pragma unroll
        for (int u = 0; u < LPL; u++) rank[u] = 0;
#pragma unroll
        for (int d = 0; d < NLEV; d++) {
            const float o = s_level[wib][sub][d];
#pragma unroll
            for (int u = 0; u < LPL; u++) rank[u] += (o < lv[u] || (o == lv[u] && d < l + u * LG)) ? 1 : 0;
        }
        __syncwarp();
#pragma unroll
        for (int u = 0; u < LPL; u++) {
            const int c = l + u * LG;
            if (c >= NLEV) continue;
            s_level[wib][sub][rank[u]] = lv[u];
            float sg[4];
#pragma unroll
            for (int i = 0; i < 4; i++) sg[i] = i < Q ? (((c >> (Q - 1 - i)) & 1) ? -1.f : 1.f) : 0.f;
            *reinterpret_cast<float4*>(s_sign[wib][sub][rank[u]]) = make_float4(sg[0], sg[1], sg[2], sg[3]);
            uint32_t pk[PW > 0 ? PW : 1] = {};
            int t = 0;
#pragma unroll
            for (int i = 0; i < Q; i++)
#pragma unroll
                for (int j = i + 1; j < Q; j++, t++) pk[t / 3] |= (uint32_t)(((c >> (Q - 1 - i)) ^ (c >> (Q - 1 - j))) & 1) << (10 * (t % 3));
#pragma unroll
            for (int i = 0; i < PW; i++) s_pair[wib][sub][rank[u]][i] = pk[i];
        }
        __syncwarp();
        // every weight to its nearest level: bisection on the midpoints, `w < mid` goes left
        float mid[NLEV - 1];
#pragma unroll
        for (int c = 0; c + 1 < NLEV; c++) mid[c] = (s_level[wib][sub][c] + s_level[wib][sub][c + 1]) / 2.f;
        const bool last = round + 1 == p.rounds;
        auto place = [&](float w) {
            int at = 0;
            float m = mid[NLEV / 2 - 1];
#pragma unroll
            for (int s = NLEV / 2; s > 0; s >>= 1) {
                at = w < m ? at : at + s;
                if (s > 1) {
                    // the midpoint of the half that is left: at + s / 2 - 1, out of registers
                    float next = mid[s / 2 - 1];
#pragma unroll
                    for (int c = s; c < NLEV; c += s) next = at == c ? mid[c + s / 2 - 1] : next;
                    m = next;
                }
            }
            return at;
        };
        if (!last) {
            uint32_t pk[PW > 0 ? PW : 1] = {};
            float part[Q][NJ] = {};
#pragma unroll
            for (int e = 0; e < E; e++) {
                const int at = place(wv[e]);
                const float4 sg = *reinterpret_cast<const float4*>(s_sign[wib][sub][at]);
                const float sv[4] = {sg.x, sg.y, sg.z, sg.w};
#pragma unroll
                for (int i = 0; i < Q; i++) part[i][e / EE] = fmaf(sv[i], wv[e], part[i][e / EE]);
#pragma unroll
                for (int i = 0; i < PW; i++) pk[i] += s_pair[wib][sub][at][i];
            }
            // padding registers hold 0 and were placed with it: their pairs come off again
            if (pad) {
                const int at = place(0.f);
#pragma unroll
                for (int i = 0; i < PW; i++) pk[i] -= pad * s_pair[wib][sub][at][i];
            }
#pragma unroll
            for (int i = 0; i < Q; i++) {
                btw[i] = tile_sum_f<LG>(part[i]);
                A[i][i] = (float)g;
            }
#pragma unroll
            for (int i = 0; i < PW; i++) pk[i] = group_sum_u<LG>(pk[i]);
            int t = 0;
#pragma unroll
            for (int i = 0; i < Q; i++)
#pragma unroll
                for (int j = i + 1; j < Q; j++, t++)
                    A[i][j] = A[j][i] = (float)(g - 2 * (int)((pk[t / 3] >> (10 * (t % 3))) & 1023u));
        } else {
#pragma unroll
            for (int i = 0; i < Q; i++) { pos[i] = 0u; nz[i] = valid; }
#pragma unroll
            for (int e = 0; e < E; e++) {
                const float4 sg = *reinterpret_cast<const float4*>(s_sign[wib][sub][place(wv[e])]);
                const float sv[4] = {sg.x, sg.y, sg.z, sg.w};
#pragma unroll
                for (int i = 0; i < Q; i++) pos[i] |= (sv[i] > 0.f ? 1u : 0u) << e;
            }
#pragma unroll
            for (int i = 0; i < Q; i++) pos[i] &= valid;
        }
    }

    // ---- outputs ----
    if (live && l == 0) {
#pragma unroll
        for (int i = 0; i < Q; i++) {
            if (p.alpha_py) p.alpha_py[((size_t)n * G + gi) * Q + i] = alpha[i];
            if (p.alpha_k) p.alpha_k[((size_t)gi * Q + i) * p.N + n] = __float2half_rn(alpha[i]);
        }
    }
    if (live && p.binary_py) {
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int at = (e % EE) * 32 + LG * (e / EE) + l;
            if (at < g) {
                signed char* dst = p.binary_py + (((size_t)n * G + gi) * g + at) * Q;
#pragma unroll
                for (int i = 0; i < Q; i++) dst[i] = (signed char)(((nz[i] >> e) & 1u) ? (((pos[i] >> e) & 1u) ? 1 : -1) : 0);
            }
        }
    }
    if (p.bW) {                                            // g % 32 == 0: whole words; a zero code packs as -1
#pragma unroll
        for (int kw = 0; kw < EE; kw++)                    // word of the group: registers kw, kw + EE, ... of all its lanes
#pragma unroll
            for (int b = 0; b < Q; b++) {
                uint32_t word = 0u;
#pragma unroll
                for (int j = 0; j < NJ; j++) word |= ((pos[b] >> (j * EE + kw)) & 1u) << (LG * j + l);
#pragma unroll
                for (int o = LG / 2; o > 0; o >>= 1) word |= __shfl_xor_sync(0xffffffffu, word, o);
                if (live && l == kw % LG && kw * 32 < g) p.bW[((size_t)(gi * (g / 32) + kw) * Q + b) * p.N + n] = word;
            }
    }
}

// ---- the same, a group to a lane: two to four planes, refined at least once ----
// The levels come in pairs +-v, so the midpoints do too and the middle one is 0: a weight's level is decided by |w| among the
// 2^(Q-1) levels of the upper half and by its sign, and sign times weight by the level's signs and |w|.  A plane's sign is a step
// function of |w|: one multiply-add per midpoint with the comparison's 1 or 0 and the step's height (0 or +-2, of this group's
// levels).  Nothing is searched or looked up: at Q = 3 a weight and round is 3 comparisons, 6 multiply-adds for the signs, 3
// for B^T w and 3 for B^T B.  A lane does that for a group of its own, so there is nothing to reduce, and the solve costs the
// warp once for 32 groups instead of once for 32 / LG.  The weights lie in shared memory, four of a group to 16 bytes, at
// places that reading (a lane per group) and filling (a row of the matrix at a time) both find without bank conflicts.
// `w < mid goes left` is strict on both sides: a negative weight leaves the inner level only if |w| > midpoint.  Those compare with
// the float below |w|: w plus the smallest float, cut off toward zero, which leaves the others as they are from 2^-125 on; a group with a
// midpoint no larger than that compares everything times 2^60.
// Sums are added in the order of the other kernels: per residue of 32 the weights in turn, then residues 16, 8, 4, 2 and 1 apart.  So
// all give the same bits.
//
// Bound by issue and its latencies on 14 warps to an SM: an ALU instruction (a comparison) keeps a scheduler for two cycles, an
// fp32 one for one, some 20 cycles a weight and round at Q = 3.  Measured, us, this / tiled kernel, 15 rounds, 4096 x 4096: q = 3, g = 128,
// 256 / 409, g = 256 276 / 422, g = 512 421 / 462; q = 2, g = 64, 184 / 257, g = 128 123 / 231; q = 4, g = 128, 616 / 842.  A round takes
// 14 us of the 256; reading, greedy start and packing 50.
// Sums of |w| per midpoint, two packed instructions for two weights, are a third faster (171 us) but round otherwise: then a
// weight in a million takes another level.
constexpr int kBqLaneWarps = 7;               // 16 KB a warp at g = 128: two CTAs of 7 warps to an SM
constexpr int kBqLaneMaxG = 512;
__host__ __device__ constexpr int bq_lane_warp_bytes(int g) { return (g + 31) / 32 * 4096; }
__host__ __device__ constexpr int bq_lane_warps(int g) {
    return 232448 / bq_lane_warp_bytes(g) < kBqLaneWarps ? 232448 / bq_lane_warp_bytes(g) : kBqLaneWarps;
}

// What a weight is compared with: |w|, or for a negative one the float below (the sum with the smallest float, cut off toward zero); times unit.
__device__ __forceinline__ float bq_key(float w, float unit) { return fabsf(__fmaf_rz(w, unit, 1.401298464324817e-45f)); }
// 1 where key >= mid, else 0
__device__ __forceinline__ float bq_from(float key, float mid) {
    float f;
    asm("set.ge.f32.f32 %0, %1, %2;" : "=f"(f) : "f"(key), "f"(mid));
    return f;
}
__device__ __forceinline__ float4 bq_add4(float4 a, float4 b) { return make_float4(a.x + b.x, a.y + b.y, a.z + b.z, a.w + b.w); }

template <int Q>
__global__ void __launch_bounds__(kBqLaneWarps * 32, 2)
bcq_quantize_lane_kernel(const BqParams p) {
    constexpr int NH = 1 << (Q - 1);                       // levels of the upper half
    extern __shared__ __align__(1024) unsigned char smem[];
    const int lane = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int G = p.K / p.g, g = p.g, words = (g + 31) / 32;
    const long long groups = (long long)p.N * G;
    const long long first = ((long long)blockIdx.x * (blockDim.x >> 5) + wib) * 32;
    if (first >= groups) return;                           // whole warps leave together
    // groups of consecutive rows share a warp: their packed words are neighbours
    const bool live = first + lane < groups;               // a group beyond the end repeats the warp's first one
    const long long grp = live ? first + lane : first;
    const int gi = (int)(grp / p.N), n = (int)(grp % p.N);
    const float* wg = p.w + (size_t)n * p.K + (size_t)gi * g;
    unsigned char* mine = smem + (size_t)wib * bq_lane_warp_bytes(g);
    // quad j + 8 e of row r: weights 32 e + 4 j .. + 3
    auto place = [&](int j, int e, int row) { return mine + e * 4096 + (j * 32 + (row ^ j)) * 16; };

    // ---- the weights, zeros up to whole words of 32: the whole warp takes one group after the other ----
    const bool wide = g % 4 == 0 && ((uintptr_t)p.w & 15) == 0;      // then every group begins on 16 bytes
#pragma unroll 16
    for (int r = 0; r < 32; r++) {
        const float* src = reinterpret_cast<const float*>(__shfl_sync(0xffffffffu, (unsigned long long)wg, r));
        if (wide) {
            for (int k4 = lane; k4 < words * 8; k4 += 32)
                *reinterpret_cast<float4*>(place(k4 & 7, k4 >> 3, r)) = 4 * k4 < g ? __ldg(reinterpret_cast<const float4*>(src) + k4) : make_float4(0.f, 0.f, 0.f, 0.f);
        } else {
            for (int k = lane; k < words * 32; k += 32)
                reinterpret_cast<float*>(place((k >> 2) & 7, k >> 5, r))[k & 3] = k < g ? __ldg(src + k) : 0.f;
        }
    }
    __syncwarp();

    // Sums over the group's weights, COUNT at a time: f(w, part) adds what a weight contributes to part[0 .. COUNT-1].
    auto sums = [&](auto& out, auto&& f) {
        constexpr int COUNT = sizeof(out) / sizeof(float), UNROLL = Q == 4 ? 1 : 2;       // twice as much: 261 and, Q = 4, 671 us
        float4 even[COUNT], acc[COUNT];                    // residues 4 j .. 4 j + 3 for j = 0, 4, 2, 6, and then 1, 5, 3, 7
#pragma unroll 1
        for (int jj = 0; jj < 4; jj++) {
            const int j = (jj & 1) << 1 | jj >> 1;
            const unsigned char *at0 = place(j, 0, lane), *at1 = place(j + 4, 0, lane);
            float part[2][4][COUNT] = {};
#pragma unroll UNROLL
            for (int e = 0; e < words; e++) {
                const float4 v = *reinterpret_cast<const float4*>(at0 + e * 4096), u = *reinterpret_cast<const float4*>(at1 + e * 4096);
                f(v.x, part[0][0]); f(v.y, part[0][1]); f(v.z, part[0][2]); f(v.w, part[0][3]);
                f(u.x, part[1][0]); f(u.y, part[1][1]); f(u.z, part[1][2]); f(u.w, part[1][3]);
            }
#pragma unroll
            for (int i = 0; i < COUNT; i++) {
                const float4 both = make_float4(part[0][0][i] + part[1][0][i], part[0][1][i] + part[1][1][i],
                                                part[0][2][i] + part[1][2][i], part[0][3][i] + part[1][3][i]);
                acc[i] = jj & 1 ? bq_add4(acc[i], both) : both;
                if (jj == 1) even[i] = acc[i];
            }
        }
#pragma unroll
        for (int i = 0; i < COUNT; i++) {
            const float4 all = bq_add4(even[i], acc[i]);
            out[i] = (all.x + all.z) + (all.y + all.w);
        }
    };

    // ---- greedy ----
    float alpha[Q], btw[Q];
    float A[Q][Q];                                         // B^T B
    auto scale = [&](float sum) {
        const float a = sum / (float)g;
        return a != a ? 0.f : a;
    };
    // By signs relative to the weight's own: plane 0 is +, r = |w| - alpha_0 decides plane 1, and so on.  A residual that is 0 (a
    // weight that is 0, to begin with) has no sign: a warp that meets one does it over below.
    auto toward0 = [](float r, float a) { return r - copysignf(a, r); };
    float whole;                                           // sum of |w|
    float least = __int_as_float(0x7f800000);              // of the |residuals| whose signs were used
    {
        float s[1];
        sums(s, [&](float w, float (&part)[1]) {
            least = fminf(least, fabsf(w));
            part[0] += fabsf(w);
        });
        whole = btw[0] = s[0];
        alpha[0] = scale(s[0]);
    }
#pragma unroll
    for (int i = 1; i < Q; i++) {
        float s[1];
        sums(s, [&](float w, float (&part)[1]) {
            float r = fabsf(w) - alpha[0];
#pragma unroll
            for (int j = 1; j < i; j++) r = toward0(r, alpha[j]);
            least = fminf(least, fabsf(r));
            part[0] += fabsf(r);
        });
        alpha[i] = scale(s[0]);
    }
    {
        float t[Q - 1];
        float both[Q][Q] = {};                             // [j][i], j < i: sum of the products of the signs
        sums(t, [&](float w, float (&part)[Q - 1]) {
            float r[Q];
            r[1] = fabsf(w) - alpha[0];
#pragma unroll
            for (int i = 2; i < Q; i++) r[i] = toward0(r[i - 1], alpha[i - 1]);
#pragma unroll
            for (int i = 1; i < Q; i++) {
                part[i - 1] += copysignf(w, r[i]);
                both[0][i] += copysignf(1.f, r[i]);
#pragma unroll
                for (int j = 1; j < i; j++) both[j][i] += copysignf(1.f, __uint_as_float(__float_as_uint(r[i]) ^ __float_as_uint(r[j])));
            }
        });
#pragma unroll
        for (int i = 0; i < Q; i++) {
            if (i) btw[i] = t[i ? i - 1 : 0];
            A[i][i] = (float)g;
#pragma unroll
            for (int j = 0; j < i; j++) A[j][i] = A[i][j] = both[j][i];
        }
    }
    if (__any_sync(0xffffffffu, !(least > 0.f))) {         // (so do the zeros behind a group's end)
        auto take = [&](float r, float a) { return r != 0.f ? toward0(r, a) : r; };
#pragma unroll
        for (int i = 1; i < Q; i++) {
            float s[1];
            sums(s, [&](float w, float (&part)[1]) {
                float r = w;
#pragma unroll
                for (int j = 0; j < i; j++) r = take(r, alpha[j]);
                part[0] += fabsf(r);
            });
            alpha[i] = scale(s[0]);
        }
        float both[Q][Q] = {};
        sums(btw, [&](float w, float (&part)[Q]) {
            float r = w, b[Q];
#pragma unroll
            for (int i = 0; i < Q; i++) {
                b[i] = r > 0.f ? 1.f : (r < 0.f ? -1.f : 0.f);
                r = take(r, alpha[i]);
                part[i] = fmaf(b[i], w, part[i]);
#pragma unroll
                for (int j = 0; j <= i; j++) both[j][i] = fmaf(b[j], b[i], both[j][i]);
            }
        });
#pragma unroll
        for (int i = 0; i < Q; i++)
#pragma unroll
            for (int j = 0; j <= i; j++) A[j][i] = A[i][j] = both[j][i];
    }

    // ---- alternating refinement ----
    float mid[NH];                                         // [1 ..]: between the upper half's levels, times unit
    float unit;                                            // 1, or 2^60 where a midpoint is so low that bq_key would move positive weights
    uint32_t code[NH];                                     // bit Q - 1 - i set: plane i is -1 in this level
    const float pad = (float)(words * 32 - g);
#pragma unroll 1
    for (int round = 0;; round++) {
        bq_solve<Q>(A, btw, alpha);
        // the upper half's levels in ascending order, ties by index: of c and its complement the one above 0, the larger one at 0
        float v[NH];
#pragma unroll
        for (int c = 0; c < NH; c++) {
            float x = 0.f;
#pragma unroll
            for (int i = 0; i < Q; i++) x += ((c >> (Q - 1 - i)) & 1) ? -alpha[i] : alpha[i];
            v[c] = fabsf(x);
            code[c] = x > 0.f ? c : 2 * NH - 1 - c;
        }
#pragma unroll
        for (int c = 1; c < NH; c++)
#pragma unroll
            for (int d = c; d > 0; d--)
                if (v[d] < v[d - 1] || (v[d] == v[d - 1] && code[d] < code[d - 1])) {
                    const float t = v[d]; v[d] = v[d - 1]; v[d - 1] = t;
                    const uint32_t u = code[d]; code[d] = code[d - 1]; code[d - 1] = u;
                }
#pragma unroll
        for (int c = 1; c < NH; c++) mid[c] = (v[c - 1] + v[c]) / 2.f;
        unit = 1.f;
#pragma unroll
        for (int c = 1; c < NH; c++) unit = mid[c] > 0.f && mid[c] <= 2.350988701644575e-38f ? 1.152921504606846976e18f : unit;
#pragma unroll
        for (int c = 1; c < NH; c++) mid[c] *= unit;
        if (round + 1 == p.rounds) break;
        // a plane's sign: in the lowest level, and the steps at the midpoints
        float step[Q][NH];
#pragma unroll
        for (int i = 0; i < Q; i++) {
            float last = 0.f;
#pragma unroll
            for (int c = 0; c < NH; c++) {
                const float sign = ((code[c] >> (Q - 1 - i)) & 1u) ? -1.f : 1.f;
                step[i][c] = sign - last;
                last = sign;
            }
        }
        float both[Q][Q] = {};
        // KIND 1, Q = 3: above the lowest level the codes are 1, 2, ... from the top, as they are without ties, and steps are known.
        // 2, Q = 2: the codes are 0 and 1, and plane 0 is + throughout.
        auto refine = [&](auto kind) {
            constexpr int KIND = decltype(kind)::value;
            auto signs = [&](float key, float (&sg)[Q]) {
                float from[NH];
#pragma unroll
                for (int c = 1; c < NH; c++) from[c] = bq_from(key, mid[c]);
#pragma unroll
                for (int i = 0; i < Q; i++) {
                    if (KIND == 2) {
                        sg[i] = i ? fmaf(2.f, from[1], -1.f) : 1.f;
                    } else {
                        sg[i] = step[i][0];
#pragma unroll
                        for (int c = 1; c < NH; c++) {
                            if (KIND == 1 && c >= 2) {
                                if (i == 1 && c == 2 || i == 2 && c == 3) sg[i] = fmaf(2.f, from[c], sg[i]);
                                if (i == 2 && c == 2) sg[i] = fmaf(-2.f, from[c], sg[i]);
                            } else {
                                sg[i] = fmaf(step[i][c], from[c], sg[i]);
                            }
                        }
                    }
                }
            };
            constexpr int FROM = KIND == 2 ? 1 : 0;       // first plane whose sum changes
            float t[Q - FROM];
            sums(t, [&](float w, float (&part)[Q - FROM]) {
                float sg[Q];
                signs(bq_key(w, unit), sg);
#pragma unroll
                for (int i = 0; i < Q; i++) {
                    if (i >= FROM) part[i >= FROM ? i - FROM : 0] = fmaf(sg[i], fabsf(w), part[i >= FROM ? i - FROM : 0]);
#pragma unroll
                    for (int j = 0; j < i; j++) both[j][i] = fmaf(sg[j], sg[i], both[j][i]);
                }
            });
            if (FROM) btw[0] = whole;
#pragma unroll
            for (int i = FROM; i < Q; i++) btw[i] = t[i - FROM];
            if (pad != 0.f) {                              // the zeros behind the group's end were counted
                float sg[Q];
                signs(bq_key(0.f, unit), sg);
#pragma unroll
                for (int i = 0; i < Q; i++)
#pragma unroll
                    for (int j = 0; j < i; j++) both[j][i] -= pad * (sg[i] * sg[j]);
            }
        };
        if constexpr (Q == 3) {
            if (__all_sync(0xffffffffu, code[3] == 0u && code[2] == 1u && code[1] == 2u)) refine(std::integral_constant<int, 1>{});
            else refine(std::integral_constant<int, 0>{});
        } else if constexpr (Q == 2) {
            if (__all_sync(0xffffffffu, code[1] == 0u && code[0] == 1u)) refine(std::integral_constant<int, 2>{});
            else refine(std::integral_constant<int, 0>{});
        } else {
            refine(std::integral_constant<int, 0>{});
        }
#pragma unroll
        for (int i = 0; i < Q; i++) {
            A[i][i] = (float)g;
#pragma unroll
            for (int j = 0; j < i; j++) A[j][i] = A[i][j] = both[j][i];
        }
    }

    // ---- outputs ----
    if (live) {
#pragma unroll
        for (int i = 0; i < Q; i++) {
            if (p.alpha_py) p.alpha_py[((size_t)n * G + gi) * Q + i] = alpha[i];
            if (p.alpha_k) p.alpha_k[((size_t)gi * Q + i) * p.N + n] = __float2half_rn(alpha[i]);
        }
    }
    if (!p.bW && !p.binary_py) return;
    // 32 weights at a time: a bit per weight of every plane, 1 for +1
    for (int kw = 0; kw < words; kw++) {
        uint32_t from[NH] = {}, neg = 0u;                  // [1 ..]: from mid on
        auto mark = [&](float w, int e) {
            const float key = bq_key(w, unit);
            neg |= w < 0.f ? 1u << e : 0u;
#pragma unroll
            for (int c = 1; c < NH; c++) from[c] |= key >= mid[c] ? 1u << e : 0u;
        };
#pragma unroll
        for (int j = 0; j < 8; j++) {
            const float4 v = *reinterpret_cast<const float4*>(place(j, kw, lane));
            mark(v.x, 4 * j); mark(v.y, 4 * j + 1); mark(v.z, 4 * j + 2); mark(v.w, 4 * j + 3);
        }
        from[0] = 0xffffffffu;
        uint32_t plus[Q] = {};
#pragma unroll
        for (int c = 0; c < NH; c++) {
            const uint32_t here = c + 1 < NH ? from[c] & ~from[c + 1] : from[c];
#pragma unroll
            for (int i = 0; i < Q; i++) plus[i] |= ((code[c] >> (Q - 1 - i)) & 1u) ? 0u : here;
        }
#pragma unroll
        for (int i = 0; i < Q; i++) {
            plus[i] ^= neg;
            if (p.bW && live) p.bW[((size_t)(gi * (g / 32) + kw) * Q + i) * p.N + n] = plus[i];      // g % 32 == 0: whole words
        }
        if (p.binary_py) {
            // a row after the other, by the whole warp: consecutive bytes of it
            const int count = min(32, g - 32 * kw);
            for (int r = 0; r < 32; r++) {
                const bool there = __shfl_sync(0xffffffffu, live ? 1 : 0, r);
                signed char* dst = p.binary_py + ((size_t)__shfl_sync(0xffffffffu, n, r) * G + __shfl_sync(0xffffffffu, gi, r)) * g * Q + (size_t)32 * kw * Q;
                uint32_t row[Q];
#pragma unroll
                for (int i = 0; i < Q; i++) row[i] = __shfl_sync(0xffffffffu, plus[i], r);
                for (int at = lane; there && at < count * Q; at += 32) {
                    const int e = at / Q, i = at % Q;
                    uint32_t bits = row[0];
#pragma unroll
                    for (int j = 1; j < Q; j++) bits = i == j ? row[j] : bits;
                    dst[at] = (bits >> e) & 1u ? 1 : -1;
                }
            }
        }
    }
}

// ---- groups wider than 1024 (the reference's default is one group per row): one CTA per (row, group) ----
// Same arithmetic; the codes live in shared memory (2 bytes per weight), the weights are re-read from global memory
// (L2) twice per round, sums go through warp shuffles and a shared-memory stage, and warp 0 solves for alpha and
// sorts the levels.
constexpr int kBqBlockThreads = 256;

__device__ __forceinline__ float block_sum_f(float v, float* s_stage, int tid) {
    v = warp_sum_f(v);
    __syncthreads();                                   // s_stage free
    if ((tid & 31) == 0) s_stage[tid >> 5] = v;
    __syncthreads();
    float t = 0.f;
#pragma unroll
    for (int w = 0; w < kBqBlockThreads / 32; w++) t += s_stage[w];
    return t;
}

__global__ void __launch_bounds__(kBqBlockThreads)
bcq_quantize_block_kernel(const BqParams p) {
    extern __shared__ unsigned short s_code[];         // [g]: bits 0..7 "+1" per plane, 8..15 "non-zero" per plane
    __shared__ float s_stage[kBqBlockThreads / 32];
    __shared__ float s_acc[kBqMaxQ + kBqMaxQ * kBqMaxQ];
    __shared__ float s_alpha[kBqMaxQ];
    __shared__ float s_v[1 << kBqMaxQ];
    __shared__ float s_vs[1 << kBqMaxQ];
    __shared__ unsigned char s_ind[1 << kBqMaxQ];
    const int tid = threadIdx.x, lane = tid & 31;
    const int G = p.K / p.g, g = p.g, q = p.q;
    const int n = blockIdx.x / G, gi = blockIdx.x % G;
    const float* wg = p.w + (size_t)n * p.K + (size_t)gi * g;
    if (tid < kBqMaxQ) s_alpha[tid] = 0.f;
    for (int idx = tid; idx < g; idx += kBqBlockThreads) s_code[idx] = 0;
    __syncthreads();

    auto residual = [&](int idx, int upto) {           // w - sum_{j < upto} alpha_j b_j
        float r = wg[idx];
        const uint32_t c = s_code[idx];
        for (int j = 0; j < upto; j++) r -= s_alpha[j] * code_sign(c, j);
        return r;
    };
    // ---- greedy ----
    for (int i = 0; i < q; i++) {
        float s = 0.f;
        for (int idx = tid; idx < g; idx += kBqBlockThreads) s += fabsf(residual(idx, i));
        float a = block_sum_f(s, s_stage, tid) / (float)g;
        if (a != a) a = 0.f;
        for (int idx = tid; idx < g; idx += kBqBlockThreads) {
            const float r = residual(idx, i);
            unsigned short c = s_code[idx];
            if (r > 0.f) c |= (unsigned short)(1u << i);
            if (r != 0.f) c |= (unsigned short)(1u << (8 + i));
            s_code[idx] = c;
        }
        __syncthreads();
        if (tid == 0) s_alpha[i] = a;
        __syncthreads();
    }
    // ---- alternating refinement ----
    if (q > 1) {
        const int nlev = 1 << q;
        for (int round = 0; round < p.rounds; round++) {
            // B^T w and the Gram matrix, reduced over the block
            float btw[kBqMaxQ];
            int cov[kBqMaxQ * (kBqMaxQ + 1) / 2];
#pragma unroll
            for (int i = 0; i < kBqMaxQ; i++) btw[i] = 0.f;
#pragma unroll
            for (int i = 0; i < kBqMaxQ * (kBqMaxQ + 1) / 2; i++) cov[i] = 0;
            for (int idx = tid; idx < g; idx += kBqBlockThreads) {
                const float wv = wg[idx];
                const uint32_t c = s_code[idx];
                int t = 0;
#pragma unroll
                for (int i = 0; i < kBqMaxQ; i++) {
                    const float bi = i < q ? code_sign(c, i) : 0.f;
                    btw[i] += bi * wv;
#pragma unroll
                    for (int j = i; j < kBqMaxQ; j++, t++) cov[t] += (int)(bi * (j < q ? code_sign(c, j) : 0.f));
                }
            }
            {
                int t = 0;
                for (int i = 0; i < kBqMaxQ; i++) {
                    const float sb = block_sum_f(i < q ? btw[i] : 0.f, s_stage, tid);
                    if (tid == 0) s_acc[i] = sb;
                    for (int j = i; j < kBqMaxQ; j++, t++) {
                        if (i < q && j < q) {
                            const float sc = block_sum_f((float)cov[t], s_stage, tid);      // integer counts below 2^24: exact
                            if (tid == 0) { s_acc[kBqMaxQ + i * kBqMaxQ + j] = sc; s_acc[kBqMaxQ + j * kBqMaxQ + i] = sc; }
                        }
                    }
                }
            }
            __syncthreads();
            if (tid < 32) {
                // warp 0: q steps of conjugate gradient from the current alpha, |alpha| descending, levels rank-sorted
                float x[kBqMaxQ], r[kBqMaxQ], pp[kBqMaxQ], Ap[kBqMaxQ], al[kBqMaxQ];
                float rtr_new = 0.f;
#pragma unroll
                for (int i = 0; i < kBqMaxQ; i++) al[i] = s_alpha[i];
#pragma unroll
                for (int i = 0; i < kBqMaxQ; i++) {
                    x[i] = al[i];
                    float sdot = 0.f;
#pragma unroll
                    for (int j = 0; j < kBqMaxQ; j++) if (i < q && j < q) sdot += s_acc[kBqMaxQ + i * kBqMaxQ + j] * al[j];
                    r[i] = i < q ? s_acc[i] - sdot : 0.f;
                    pp[i] = r[i];
                    rtr_new += r[i] * r[i];
                }
                for (int it = 0; it < q; it++) {
                    const float rtr = rtr_new;
                    float pAp = 0.f;
#pragma unroll
                    for (int i = 0; i < kBqMaxQ; i++) {
                        float sdot = 0.f;
#pragma unroll
                        for (int j = 0; j < kBqMaxQ; j++) if (i < q && j < q) sdot += s_acc[kBqMaxQ + i * kBqMaxQ + j] * pp[j];
                        Ap[i] = i < q ? sdot : 0.f;
                        pAp += pp[i] * Ap[i];
                    }
                    const float a = rtr / (pAp + 1e-6f);
                    rtr_new = 0.f;
#pragma unroll
                    for (int i = 0; i < kBqMaxQ; i++) {
                        x[i] += a * pp[i];
                        r[i] -= a * Ap[i];
                        rtr_new += r[i] * r[i];
                    }
                    const float beta = rtr_new / (rtr + 1e-6f);
#pragma unroll
                    for (int i = 0; i < kBqMaxQ; i++) pp[i] = r[i] + beta * pp[i];
                }
#pragma unroll
                for (int i = 0; i < kBqMaxQ; i++) al[i] = i < q ? fabsf(x[i]) : -1.f;
#pragma unroll
                for (int i = 1; i < kBqMaxQ; i++) {
#pragma unroll
                    for (int j = i; j > 0; j--) {
                        if (al[j] > al[j - 1]) { const float t2 = al[j]; al[j] = al[j - 1]; al[j - 1] = t2; }
                    }
                }
#pragma unroll
                for (int i = 0; i < kBqMaxQ; i++) if (i >= q) al[i] = 0.f;
                __syncwarp();
                if (lane < kBqMaxQ) {
                    float a = 0.f;
#pragma unroll
                    for (int i = 0; i < kBqMaxQ; i++) if (i == lane) a = al[i];
                    s_alpha[lane] = a;
                }
                for (int c = lane; c < nlev; c += 32) {
                    float v = 0.f;
#pragma unroll
                    for (int i = 0; i < kBqMaxQ; i++) if (i < q) v += ((c >> (q - 1 - i)) & 1) ? -al[i] : al[i];
                    s_v[c] = v;
                }
                __syncwarp();
                for (int c = lane; c < nlev; c += 32) {
                    const float v = s_v[c];
                    int rank = 0;
                    for (int d = 0; d < nlev; d++) {
                        const float u = s_v[d];
                        rank += (u < v || (u == v && d < c)) ? 1 : 0;
                    }
                    s_vs[rank] = v;
                    s_ind[rank] = (unsigned char)c;
                }
            }
            __syncthreads();
            for (int idx = tid; idx < g; idx += kBqBlockThreads) {
                const float wv = wg[idx];
                int left = 0, right = nlev - 1;
                for (int it = 0; it < q; it++) {
                    const int ml = (left + right - 1) / 2, mr = ml + 1;
                    const float mid = (s_vs[ml] + s_vs[mr]) / 2.f;
                    if (wv < mid) right = ml; else left = mr;
                }
                const uint32_t c = s_ind[left];
                uint32_t pos = 0u;
                for (int i = 0; i < q; i++) pos |= (((c >> (q - 1 - i)) & 1u) ^ 1u) << i;
                s_code[idx] = (unsigned short)(pos | (((1u << q) - 1u) << 8));
            }
            __syncthreads();
        }
    }
    // ---- outputs ----
    if (tid < q) {
        if (p.alpha_py) p.alpha_py[((size_t)n * G + gi) * q + tid] = s_alpha[tid];
        if (p.alpha_k) p.alpha_k[((size_t)gi * q + tid) * p.N + n] = __float2half_rn(s_alpha[tid]);
    }
    const int g_pad = (g + 31) / 32 * 32;
    for (int idx = tid; idx < g_pad; idx += kBqBlockThreads) {        // whole warps walk whole 32-element words
        const bool valid = idx < g;
        const uint32_t c = valid ? s_code[idx] : 0u;
        if (p.binary_py && valid) {
            signed char* dst = p.binary_py + (((size_t)n * G + gi) * g + idx) * q;
            for (int i = 0; i < q; i++) dst[i] = (signed char)code_sign(c, i);
        }
        if (p.bW) {                                         // g % 32 == 0 here; a zero code packs as -1
            for (int i = 0; i < q; i++) {
                const uint32_t word = __ballot_sync(0xffffffffu, valid && ((c >> i) & 1u));
                if (lane == 0) p.bW[((size_t)((gi * g + idx) / 32) * q + i) * p.N + n] = word;
            }
        }
    }
}

}  // namespace lg
