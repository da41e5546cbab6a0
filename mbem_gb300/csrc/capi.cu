// Library identity, error reporting, and the not-yet-specialised paths.
#include <stdarg.h>
#include <stdio.h>

#include <atomic>

#include "common.cuh"
#include "dp_math.cuh"

namespace mbem {

static thread_local char g_last_error[512] = "";

int set_error(int code, const char* fmt, ...) {
    va_list ap;
    va_start(ap, fmt);
    vsnprintf(g_last_error, sizeof(g_last_error), fmt, ap);
    va_end(ap);
    return code;
}

static std::atomic<unsigned long long> g_launches{0};

void count_launches(int n) { g_launches.fetch_add((unsigned long long)n, std::memory_order_relaxed); }

int launch_status(const char* what, int n_launched) {
    count_launches(n_launched);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return set_error(MBEM_ERR_CUDA, "%s: %s", what, cudaGetErrorString(e));
    return MBEM_OK;
}

}  // namespace mbem

namespace mbem {

// Independent DFMA chains (8 per thread) for the FP64 pipe's throughput.
__global__ void fp64_fma_probe_kernel(double* out, int64_t iters) {
    double a[8];
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = 1.0 + 1e-9 * (threadIdx.x + k);
    const double m = 0.999999999, c = 1e-12;
    for (int64_t i = 0; i < iters; i++) {
#pragma unroll
        for (int k = 0; k < 8; k++) a[k] = fma(a[k], m, c);
    }
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 8; k++) s += a[k];
    if (s == 12345.678) out[0] = s;   // keeps the chains live; never true
}

// The pair kernels' FP64 functions, one value a thread.
__global__ void dp_math_probe_kernel(int fn, const double* __restrict__ x, const double* __restrict__ y, int64_t n,
                                     double* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double v = x[i];
    out[i] = fn == 0   ? rcp64(v)
             : fn == 1 ? log64(v)
             : fn == 2 ? angle64(y[i], v)
             : fn == 3 ? inv_pow64<3>(v)
                       : inv_pow64<5>(v);
}

// Independent FP32 FMA chains for the FP32 pipe's throughput: 16 scalar
// chains (FFMA) or 8 float2 chains (packed FFMA2), the same FLOPs per thread.
template <bool PACKED>
__global__ void fp32_fma_probe_kernel(float* out, int64_t iters) {
    float s = 0.0f;
    if (PACKED) {
        float2 a[8];
#pragma unroll
        for (int k = 0; k < 8; k++) a[k] = make_float2(1.0f + 1e-6f * (threadIdx.x + k), 1.0f - 1e-6f * k);
        const float2 m = make_float2(0.9999999f, 0.9999998f), c = make_float2(1e-7f, 2e-7f);
        for (int64_t i = 0; i < iters; i++) {
#pragma unroll
            for (int k = 0; k < 8; k++) a[k] = __ffma2_rn(a[k], m, c);
        }
#pragma unroll
        for (int k = 0; k < 8; k++) s += a[k].x + a[k].y;
    } else {
        float a[16];
#pragma unroll
        for (int k = 0; k < 16; k++) a[k] = 1.0f + 1e-6f * (threadIdx.x + k);
        const float m = 0.9999999f, c = 1e-7f;
        for (int64_t i = 0; i < iters; i++) {
#pragma unroll
            for (int k = 0; k < 16; k++) a[k] = fmaf(a[k], m, c);
        }
#pragma unroll
        for (int k = 0; k < 16; k++) s += a[k];
    }
    if (s == 12345.678f) out[0] = s;   // keeps the chains live; never true
}

}  // namespace mbem

extern "C" {

int mbem_fp32_fma_probe(float* out, int64_t iters, int blocks, int threads, int packed, void* stream) {
    MBEM_REQUIRE(out && iters > 0 && blocks > 0 && threads > 0 && threads <= 1024, MBEM_ERR_ARG,
                 "bad probe launch");
    if (packed)
        mbem::fp32_fma_probe_kernel<true><<<blocks, threads, 0, (cudaStream_t)stream>>>(out, iters);
    else
        mbem::fp32_fma_probe_kernel<false><<<blocks, threads, 0, (cudaStream_t)stream>>>(out, iters);
    return mbem::launch_status("fp32_fma_probe_kernel");
}

unsigned long long mbem_launch_count(void) { return mbem::g_launches.load(); }

int mbem_dp_math_probe(int fn, const double* x, const double* y, int64_t n, double* out, void* stream) {
    MBEM_REQUIRE(fn >= 0 && fn <= 4 && n >= 0 && (n == 0 || (x && out && (fn != 2 || y))), MBEM_ERR_ARG,
                 "bad FP64 function probe");
    MBEM_REQUIRE(mbem::ceil_div(n, 256) < INT32_MAX, MBEM_ERR_SIZE, "too many values");
    if (n == 0) return MBEM_OK;
    mbem::dp_math_probe_kernel<<<(unsigned)mbem::ceil_div(n, 256), 256, 0, (cudaStream_t)stream>>>(fn, x, y, n, out);
    return mbem::launch_status("dp_math_probe_kernel");
}

int mbem_fp64_fma_probe(double* out, int64_t iters, int blocks, int threads, void* stream) {
    MBEM_REQUIRE(out && iters > 0 && blocks > 0 && threads > 0 && threads <= 1024, MBEM_ERR_ARG,
                 "bad probe launch");
    mbem::fp64_fma_probe_kernel<<<blocks, threads, 0, (cudaStream_t)stream>>>(out, iters);
    return mbem::launch_status("fp64_fma_probe_kernel");
}

int mbem_version(void) { return 1; }

const char* mbem_last_error(void) { return mbem::g_last_error; }

}  // extern "C"
