// Small device kernels beside the matmul: dense dequantisation, the bit-plane packer and the
// uniform -> BCQ converter.  All are plain HBM-streaming kernels.
#pragma once
#include <cuda_fp16.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace lg {

// W = sum_b +-alpha (fp32 sum in plane order, one fp16 rounding), no q_bias: bit-identical to
// lutGEMM::dequantize_cpu (lutGEMM/src/nQWeight_fp16.cu:38-59).  One thread per (k-word, n):
// the q packed words are read once and expanded to 32 outputs.
// Column-wise output W[k][N]; row-wise output W[n][K].
__global__ void __launch_bounds__(256)
dequantize_kernel(const uint32_t* __restrict__ bW, const __half* __restrict__ alpha, __half* __restrict__ W,
                  int N, int K, int q, int g, int row_wise) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const int kw = blockIdx.y;
    if (n >= N) return;
    const int grp = (kw * 32) / g;
    uint32_t word[8];
    float av[8];
#pragma unroll
    for (int b = 0; b < 8; b++) {
        if (b < q) {
            word[b] = bW[((size_t)kw * q + b) * N + n];
            av[b] = __half2float(alpha[((size_t)grp * q + b) * N + n]);
        } else {
            word[b] = 0u;
            av[b] = 0.f;
        }
    }
    if (!row_wise) {
        for (int t = 0; t < 32; t++) {
            float s = 0.f;
#pragma unroll
            for (int b = 0; b < 8; b++)
                if (b < q) s = ((word[b] >> t) & 1u) ? s + av[b] : s - av[b];
            W[(size_t)(kw * 32 + t) * N + n] = __float2half_rn(s);
        }
    } else {
        __half out[32];
#pragma unroll
        for (int t = 0; t < 32; t++) {
            float s = 0.f;
#pragma unroll
            for (int b = 0; b < 8; b++)
                if (b < q) s = ((word[b] >> t) & 1u) ? s + av[b] : s - av[b];
            out[t] = __float2half_rn(s);
        }
        uint4* dst = reinterpret_cast<uint4*>(W + (size_t)n * K + kw * 32);   // 64 B, 64-B aligned
        const uint4* src = reinterpret_cast<const uint4*>(out);
#pragma unroll
        for (int i = 0; i < 4; i++) dst[i] = src[i];
    }
}

// planes int8 [K][q][N] of +-1 -> bW [K/32][q][N]; bit t of word kw <=> planes[32 kw + t] > 0
// (packing rule of tests/opt/fp16/int3_col_wise_matmul_fp16.cu:200-215).
__global__ void __launch_bounds__(256)
pack_planes_kernel(const int8_t* __restrict__ planes, uint32_t* __restrict__ bW, int K, int q, int N) {
    const size_t col = (size_t)blockIdx.x * blockDim.x + threadIdx.x;   // over q*N
    const int kw = blockIdx.y;
    if (col >= (size_t)q * N) return;
    uint32_t s = 0;
#pragma unroll 8
    for (int t = 0; t < 32; t++)
        if (planes[(size_t)(kw * 32 + t) * q * N + col] > 0) s |= 1u << t;
    bW[(size_t)kw * q * N + col] = s;
}

// Four planes, from b on, of eight rows x 32 codes that eight lanes hold (lane l8 codes 4 l8 .. + 3 of every row, the low bytes
// of code u in byte u of t): lane l8 gets row l8's four words.
__device__ __forceinline__ void u2b_words(const uint32_t (&t)[8], int b, int l8, uint32_t (&w)[4]) {
    // per row 16 bits, the four codes' bits of a plane side by side (a 4 x 4 transpose); two rows to a register
    uint32_t r[4];
#pragma unroll
    for (int i = 0; i < 4; i++) {
        const uint32_t u0 = (t[2 * i] >> b) & 0x0f0f0f0fu, u1 = (t[2 * i + 1] >> b) & 0x0f0f0f0fu;
        uint32_t x = __byte_perm(u0 | (u0 >> 4), u1 | (u1 >> 4), 0x6420), y;
        y = (x ^ (x >> 3)) & 0x0a0a0a0au;
        x ^= y ^ (y << 3);
        y = (x ^ (x >> 6)) & 0x00cc00ccu;
        r[i] = x ^ y ^ (y << 6);
    }
    // rows 4 .. 7 for the same of the lane four on, then rows 2, 3 of each four with the lane two on: sources in the order of lanes
    const bool up4 = l8 & 4, up2 = l8 & 2, up1 = l8 & 1;
    uint32_t s[4];
    {
        const uint32_t v0 = __shfl_xor_sync(0xffffffffu, up4 ? r[0] : r[2], 4), v1 = __shfl_xor_sync(0xffffffffu, up4 ? r[1] : r[3], 4);
        const uint32_t a0 = up4 ? v0 : r[0], a1 = up4 ? v1 : r[1], c0 = up4 ? r[2] : v0, c1 = up4 ? r[3] : v1;
        const uint32_t x0 = __shfl_xor_sync(0xffffffffu, up2 ? a0 : a1, 2), x1 = __shfl_xor_sync(0xffffffffu, up2 ? c0 : c1, 2);
        s[0] = up2 ? x0 : a0;
        s[1] = up2 ? a1 : x0;
        s[2] = up2 ? x1 : c0;
        s[3] = up2 ? c1 : x1;
    }
    // a row of the pair for the other of the neighbour
    const uint32_t mine = up1 ? 0x7632u : 0x5410u, other = up1 ? 0x5410u : 0x7632u;
    const uint32_t x0 = __shfl_xor_sync(0xffffffffu, __byte_perm(s[0], s[1], other), 1), x1 = __shfl_xor_sync(0xffffffffu, __byte_perm(s[2], s[3], other), 1);
    const uint32_t o0 = __byte_perm(s[0], s[1], mine), o1 = __byte_perm(s[2], s[3], mine);
    const uint32_t even0 = up1 ? x0 : o0, odd0 = up1 ? o0 : x0, even1 = up1 ? x1 : o1, odd1 = up1 ? o1 : x1;
    // nibbles of lanes 2 i and 2 i + 1 to byte i of their plane's word
    const uint32_t p0 = (even0 & 0x0f0f0f0fu) | ((odd0 << 4) & 0xf0f0f0f0u), p1 = (even1 & 0x0f0f0f0fu) | ((odd1 << 4) & 0xf0f0f0f0u);
    const uint32_t q0 = ((even0 >> 4) & 0x0f0f0f0fu) | (odd0 & 0xf0f0f0f0u), q1 = ((even1 >> 4) & 0x0f0f0f0fu) | (odd1 & 0xf0f0f0f0u);
    w[0] = __byte_perm(p0, p1, 0x6420);
    w[2] = __byte_perm(p0, p1, 0x7531);
    w[1] = __byte_perm(q0, q1, 0x6420);
    w[3] = __byte_perm(q0, q1, 0x7531);
}

// Uniform (scale, zero, code) -> kernel-layout BCQ with offset, following
// RTNParameter.convert_bcq_format (examples/rtn_parameter.py:77-96):
//   alpha_b = scale/2 * 2^b, plane b = bit b of the code, q_bias = sum_b alpha_b - scale*zero (fp32),
// then rounded to the container's fp16.  A warp takes 32 rows x 128 k (four k-words), eight rows at a time: a lane reads four
// codes of each (128 bits, the warp 512 contiguous bytes), lays its codes' bits of a plane side by side, and eight lanes exchange
// their eight rows (u2b_words) until each has one row's words: the stores are whole 32-byte sectors.  Bound by HBM (4 bytes read
// per code).  Measured, N = K = 8192, q = 4, g = 128: 53.4 us (5.8 TB/s); 61.5 with three shuffles per row and plane; now memory
// holds it (issue slots 41 % taken); one thread per word and row takes 250 us (every lane on another row's line).
constexpr int kU2bWarps = 8;
template <int Q>
__global__ void __launch_bounds__(kU2bWarps * 32)
uniform_to_bcq_kernel(const float* __restrict__ scale, const float* __restrict__ zero,
                      const int32_t* __restrict__ code, int N, int G, int g,
                      uint32_t* __restrict__ bW, __half* __restrict__ alpha, __half* __restrict__ q_bias) {
    const int lane = threadIdx.x & 31, l8 = lane & 7, n0 = blockIdx.x * 32;
    const size_t K = (size_t)G * g;
    const size_t k0 = ((size_t)blockIdx.y * kU2bWarps + (threadIdx.x >> 5)) * 128;
    if (k0 >= K) return;                                     // whole warps leave together
    const size_t k = k0 + 4 * lane;                          // this lane's four codes; K % 32 == 0: whole octets of lanes
    const bool k_ok = k < K;
    const bool vec = (reinterpret_cast<uintptr_t>(code) & 15) == 0;
    // beyond the last row or K the last row's or first codes are read: their words are not stored
    const int32_t* c = code + (size_t)n0 * K + (k_ok ? k : 0);
    const int last = min(32, N - n0) - 1;
    uint32_t words[4][Q];                                    // rows l8, l8 + 8, ... of k-word k0 / 32 + lane / 8
#pragma unroll
    for (int rb = 0; rb < 4; rb++) {
        int4 v[8];
        if (vec) {
#pragma unroll
            for (int i = 0; i < 8; i++) v[i] = __ldcs(reinterpret_cast<const int4*>(c + (size_t)min(8 * rb + i, last) * K));
        } else {
#pragma unroll
            for (int i = 0; i < 8; i++) {
                const int32_t* src = c + (size_t)min(8 * rb + i, last) * K;
                v[i] = make_int4(src[0], src[1], src[2], src[3]);
            }
        }
        // the low byte of each code (planes 0..7), code t in byte t
        uint32_t t[8];
#pragma unroll
        for (int i = 0; i < 8; i++) t[i] = __byte_perm(__byte_perm(v[i].x, v[i].y, 0x0040), __byte_perm(v[i].z, v[i].w, 0x0040), 0x5410);
#pragma unroll
        for (int b = 0; b < Q; b += 4) {
            uint32_t w[4];
            u2b_words(t, b, l8, w);
#pragma unroll
            for (int i = 0; i < 4; i++)
                if (b + i < Q) words[rb][b + i] = w[i];
        }
    }
#pragma unroll
    for (int rb = 0; rb < 4; rb++) {
        const int n = n0 + 8 * rb + l8;
        if (k_ok && n < N) {
#pragma unroll
            for (int b = 0; b < Q; b++) bW[((k0 / 32 + lane / 8) * Q + b) * N + n] = words[rb][b];
        }
    }
    // the first k-word of a group writes the group's scales; lane = row
    const int n = n0 + lane;
    for (size_t kw = k0; kw < k0 + 128 && kw < K; kw += 32) {
        if (kw % g != 0 || n >= N) continue;
        const size_t grp = kw / g;
        const float sc = scale[(size_t)n * G + grp];
        const float z = sc * zero[(size_t)n * G + grp];
        const float half_s = sc / 2.0f;
        float sum = 0.f;
        for (int b = 0; b < Q; b++) {
            const float a = half_s * (float)(1u << b);
            alpha[(grp * Q + b) * N + n] = __float2half_rn(a);
            sum += a;
        }
        q_bias[grp * N + n] = __float2half_rn(sum - z);
    }
}

// The Python examples' uint8 interchange format (Packer.pack / Packer.unpack, examples/utils.py:162-181):
// L values of +-1, byte j of the L/8 packed bytes = sum_i 2^i [flat[i L/8 + j] > 0].  One thread per byte:
// eight strided reads (or writes), each coalesced across the warp.
__global__ void __launch_bounds__(256)
packer_pack_kernel(const int8_t* __restrict__ flat, size_t cols, uint8_t* __restrict__ packed) {
    const size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cols) return;
    unsigned v = 0;
#pragma unroll
    for (int i = 0; i < 8; i++) v |= (flat[(size_t)i * cols + j] > 0 ? 1u : 0u) << i;
    packed[j] = (uint8_t)v;
}
__global__ void __launch_bounds__(256)
packer_unpack_kernel(const uint8_t* __restrict__ packed, size_t cols, int8_t* __restrict__ flat) {
    const size_t j = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= cols) return;
    const unsigned v = packed[j];
#pragma unroll
    for (int i = 0; i < 8; i++) flat[(size_t)i * cols + j] = ((v >> i) & 1u) ? 1 : -1;
}

// The quantisers' tensors (alpha float [N][G][q], binary [N][G][g][q] of +-1, offset float [N][G] or null;
// examples/bcq_parameter.py:41-48, examples/rtn_parameter.py:77-96) -> the container layout on the device:
// bW [K/32][q][N], alpha fp16 [G][q][N], q_bias fp16 [G][N].  PACKED: the binary tensor arrives as Packer bytes
// (element e of the flattened tensor is bit e / (L/8) of byte e % (L/8)) and is never expanded in memory.
// One thread per (k-word, n): its 32 q signs are consecutive elements of the flattened tensor.
template <bool PACKED>
__global__ void __launch_bounds__(128)
python_layout_kernel(const float* __restrict__ alpha_py, const void* __restrict__ binary, const float* __restrict__ offset_py,
                     int N, int K, int g, int q, uint32_t* __restrict__ bW, __half* __restrict__ alpha,
                     __half* __restrict__ q_bias) {
    const int n = blockIdx.x * blockDim.x + threadIdx.x;
    const int kw = blockIdx.y;
    if (n >= N) return;
    const int k = kw * 32, G = K / g, grp = k / g;
    const size_t e0 = ((size_t)n * K + k) * q;                 // first element of this thread in the flattened tensor
    const size_t cols = (size_t)N * K * q / 8;                 // PACKED: bytes in the stream
    uint32_t words[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    for (int t = 0; t < 32; t++) {
#pragma unroll
        for (int b = 0; b < 8; b++) {
            if (b < q) {
                const size_t e = e0 + (size_t)t * q + b;
                bool plus;
                if (PACKED) {
                    const size_t i = e / cols, j = e - i * cols;
                    plus = (reinterpret_cast<const uint8_t*>(binary)[j] >> i) & 1u;
                } else {
                    plus = reinterpret_cast<const int8_t*>(binary)[e] > 0;
                }
                words[b] |= (plus ? 1u : 0u) << t;
            }
        }
    }
    for (int b = 0; b < q; b++) bW[((size_t)kw * q + b) * N + n] = words[b];
    if (k == grp * g) {   // first word of the group moves the group's scales
        const size_t ng = (size_t)n * G + grp;
        for (int b = 0; b < q; b++) alpha[((size_t)grp * q + b) * N + n] = __float2half_rn(alpha_py[ng * q + b]);
        if (offset_py) q_bias[(size_t)grp * N + n] = __float2half_rn(offset_py[ng]);
    }
}

}  // namespace lg
