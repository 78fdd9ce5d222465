// Stand-alone activation quantiser (one CTA per token row).
#include "quant.cuh"
#include "leanstage.cuh"
#include "model.cuh"

namespace rb {

__global__ void __launch_bounds__(1024) quantize_rows_kernel(const float* __restrict__ x, int k, int kpad,
                                                             int terms, int8_t* __restrict__ xq,
                                                             float* __restrict__ sx, int32_t* __restrict__ xsum,
                                                             int32_t* __restrict__ zero, size_t zero_n, int early) {
    if (early) pdl_trigger();  // launched as an ordinary kernel: everything before it is complete
    for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < zero_n; i += (size_t)gridDim.x * blockDim.x) zero[i] = 0;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float* scratch = reinterpret_cast<float*>(smem_raw);
    float* row = scratch + 64;
    const size_t m = blockIdx.x;
    for (int i = threadIdx.x; i < k; i += blockDim.x) row[i] = x[m * k + i];
    __syncthreads();
    quantize_row_from_smem(row, k, kpad, terms, xq + m * terms * (size_t)kpad, sx + m * terms,
                           xsum + m * terms, scratch);
    if (!early) pdl_trigger();
}

// The same with the row in registers (rows of up to 4 V TH elements): a thread owns groups of four consecutive elements, all
// requested together, and the quantised bytes leave as words.  13 rows of 1923, three terms: 6.7 -> 4.3 us.
template <int V, int TH>
__global__ void __launch_bounds__(TH) quantize_rows_lean_kernel(const float* __restrict__ x, int k, int kpad, int terms, int8_t* __restrict__ xq,
                                                                float* __restrict__ sx, int32_t* __restrict__ xsum, int32_t* __restrict__ zero,
                                                                size_t zero_n, int early) {
    if (early) pdl_trigger();  // (as above)
    const float* row = x + (size_t)blockIdx.x * k;
    float4 v[V];
    if (((uintptr_t)x & 15) == 0 && (k & 3) == 0) {
#pragma unroll
        for (int j = 0; j < V; ++j) {
            const int i = 4 * (threadIdx.x + j * TH);
            v[j] = i < k ? __ldg(reinterpret_cast<const float4*>(row + i)) : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    } else {
#pragma unroll
        for (int j = 0; j < V; ++j) {
            const int i = 4 * (threadIdx.x + j * TH);
            v[j] = make_float4(i < k ? __ldg(row + i) : 0.f, i + 1 < k ? __ldg(row + i + 1) : 0.f, i + 2 < k ? __ldg(row + i + 2) : 0.f,
                               i + 3 < k ? __ldg(row + i + 3) : 0.f);
        }
    }
    for (size_t i = (size_t)blockIdx.x * TH + threadIdx.x; i < zero_n; i += (size_t)gridDim.x * TH) zero[i] = 0;
    __shared__ float scratch[64];
    LeanStage q = {};
    q.n = (k + 3) & ~3;
    q.norm_n = k;
    q.kpad = kpad;
    q.terms = terms;
    int rk = 0;
    const size_t m = blockIdx.x;
    lean_quantize<V, false, true, true>(q, v, scratch, xq + m * terms * (size_t)kpad, (size_t)kpad, sx + m * terms, xsum + m * terms, rk);
    if (!early) pdl_trigger();
}

int launch_quantize_rows(const float* x, size_t m, size_t k, int terms, int8_t* xq, float* sx, int32_t* xsum, int32_t* zero,
                         size_t zero_n, bool early, cudaStream_t st) {
    RB_REQUIRE(x && xq && sx && xsum && m > 0 && k > 0 && terms >= 1 && terms <= 4);
    RB_REQUIRE(k <= 49152 && m < (1u << 31));
    RB_REQUIRE(((uintptr_t)xq & 3) == 0);
    const size_t smem = 64 * 4 + k * 4;
    if (smem > 48 * 1024) {
        static PerDevice<bool> once;
        bool& configured = once.here();
        if (!configured) {
            RB_CUDA(cudaFuncSetAttribute(quantize_rows_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                         64 * 4 + 49152 * 4));
            configured = true;
        }
    }
    const size_t kpad = kpad_of(k);
    if (kpad <= 8 * 1024) {
        const unsigned rows = (unsigned)m;
        const int ki = (int)k, kp = (int)kpad;
        if (kpad <= 4 * 128)
            quantize_rows_lean_kernel<1, 128><<<rows, 128, 0, st>>>(x, ki, kp, terms, xq, sx, xsum, zero, zero_n, early);
        else if (kpad <= 4 * 512)
            quantize_rows_lean_kernel<1, 512><<<rows, 512, 0, st>>>(x, ki, kp, terms, xq, sx, xsum, zero, zero_n, early);
        else if (kpad <= 8 * 512)
            quantize_rows_lean_kernel<2, 512><<<rows, 512, 0, st>>>(x, ki, kp, terms, xq, sx, xsum, zero, zero_n, early);
        else
            quantize_rows_lean_kernel<2, 1024><<<rows, 1024, 0, st>>>(x, ki, kp, terms, xq, sx, xsum, zero, zero_n, early);
        return launch_status();
    }
    const int threads = k >= 4096 ? 1024 : (k >= 1024 ? 512 : 128);
    quantize_rows_kernel<<<(unsigned)m, threads, smem, st>>>(x, (int)k, (int)kpad_of(k), terms, xq, sx, xsum, zero, zero_n, early);
    return launch_status();
}

}  // namespace rb

using namespace rb;

extern "C" int rotor_b200_quantize_rows(const float* x, size_t m, size_t k, int terms, int8_t* xq, float* sx,
                                        int32_t* xsum, void* stream) {
    return launch_quantize_rows(x, m, k, terms, xq, sx, xsum, nullptr, 0, true, as_stream(stream));
}
