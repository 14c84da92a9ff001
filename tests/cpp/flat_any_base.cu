// gemv_flat_kernel where the start of dynamic shared memory is not the address that its lookups expect: the same result as with
// that address, out of the same kernel instantiated for another one.
#include <cuda.h>

#include <cstdio>
#include <cstdlib>
#include <vector>

#include "../../lutgemm_b200/csrc/gemv_flat.cuh"

#define OK(x)                                                    \
    do {                                                         \
        const int e = (int)(x);                                  \
        if (e) { std::printf("%s: %d\n", #x, e); std::exit(1); } \
    } while (0)

template <class T>
T* to_device(const std::vector<T>& v) {
    T* d = nullptr;
    OK(cudaMalloc(&d, v.size() * sizeof(T)));
    OK(cudaMemcpy(d, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice));
    return d;
}

int main() {
    const int N = 520, K = 2560, q = 3, g = 128, G = K / g, slabs = K / 512, groups = (N + 255) / 256, ctas = 7;
    std::vector<uint32_t> bW((size_t)K / 32 * q * N);
    std::vector<__half> alpha((size_t)G * q * N), q_bias((size_t)G * N), x(K);
    srand(1);
    auto real = [](float scale) { return __float2half(scale * ((float)rand() / (float)RAND_MAX - 0.3f)); };
    for (auto& v : bW) v = (uint32_t)rand() * 65539u + (uint32_t)rand();
    for (auto& v : alpha) v = real(0.02f);
    for (auto& v : q_bias) v = real(0.02f);
    for (auto& v : x) v = real(1.f);
    void* fn = nullptr;
    cudaDriverEntryPointQueryResult found;
    OK(cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &fn, cudaEnableDefault, &found));
    auto map = [&](CUtensorMapDataType type, void* base, int rows, int bytes, int box_rows) {
        CUtensorMap m;
        const cuuint64_t dims[3] = {(cuuint64_t)N, (cuuint64_t)q, (cuuint64_t)rows}, strides[2] = {(cuuint64_t)N * bytes, (cuuint64_t)q * N * bytes};
        const cuuint32_t box[3] = {(cuuint32_t)lg::kStageCols, 1, (cuuint32_t)box_rows}, es[3] = {1, 1, 1};
        OK(reinterpret_cast<decltype(&cuTensorMapEncodeTiled)>(fn)(&m, type, 3, base, dims, strides, box, es, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE));
        return m;
    };
    lg::Gemv2Params p = {};
    p.bW = to_device(bW); p.alpha = to_device(alpha); p.q_bias = to_device(q_bias); p.x = to_device(x);
    p.partial = to_device(std::vector<float>(N)); p.counters = to_device(std::vector<unsigned>(groups)); p.status = to_device(std::vector<int>(1));
    p.N = N; p.K = K; p.q = q; p.g = g; p.nslabs = slabs; p.n_tile = lg::kStageCols; p.a_rows = 512 / g;
    const CUtensorMap tmW = map(CU_TENSOR_MAP_DATA_TYPE_UINT32, (void*)p.bW, K / 32, 4, lg::kSlabWords);
    const CUtensorMap tmA = map(CU_TENSOR_MAP_DATA_TYPE_UINT16, (void*)p.alpha, G, 2, p.a_rows);
    lg::FlatRuns runs = {};
    lg::flat_plan(runs, slabs, groups, q, ctas);
    std::vector<double> ref(N), size(N);
    for (int n = 0; n < N; n++)
        for (int k = 0; k < K; k++) {
            const double xv = __half2float(x[k]);
            for (int b = 0; b < q; b++) {
                const double a = __half2float(alpha[((size_t)(k / g) * q + b) * N + n]);
                ref[n] += ((bW[((size_t)(k / 32) * q + b) * N + n] >> (k % 32)) & 1u ? a : -a) * xv;
                size[n] += std::abs(a * xv);
            }
            const double z = __half2float(q_bias[(size_t)(k / g) * N + n]);
            ref[n] += z * xv;
            size[n] += std::abs(z * xv);
        }
    auto run = [&](auto kernel) {
        std::vector<float> y(N, 1e30f);
        p.y32 = to_device(y);
        OK(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, lg::kSmemLimit));
        kernel<<<ctas, lg::kGemv2Threads, lg::gemv2_smem_bytes(p.a_rows)>>>(tmW, tmA, p, runs);
        OK(cudaGetLastError());
        OK(cudaDeviceSynchronize());
        OK(cudaMemcpy(y.data(), p.y32, N * sizeof(float), cudaMemcpyDeviceToHost));
        for (int n = 0; n < N; n++)      // fp32 sums of the 64 chunks of every slab, plane and offset
            if (!(std::abs(y[n] - ref[n]) <= (K / 8 * (q + 1)) * 6e-8 * size[n])) { std::printf("column %d: %g, not %g\n", n, y[n], ref[n]); std::exit(1); }
    };
    run(lg::gemv_flat_kernel<2, true>);
    run(lg::gemv_flat_kernel<2, true, 0x800>);
    std::printf("flat ok\n");
    return 0;
}
