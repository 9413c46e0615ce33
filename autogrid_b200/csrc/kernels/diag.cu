// Microbenchmarks for the roofline denominators (MUFU rsqrt rate and FP32 FMA
// rate), and checks of the arithmetic that the kernels rest on.
#include <algorithm>
#include <cstring>
#include <cuda_runtime.h>

#include "agb_device.cuh"
#include "autogrid_b200_diag.h"

namespace agb {

__global__ void __launch_bounds__(256) k_peak_rsqrt(float *out, int iters)
{
    float a[8];
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = 1.0f + 1e-3f * (threadIdx.x + k);
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int k = 0; k < 8; k++) a[k] = rsqrt_approx(a[k]);
    }
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) s += a[k];
    if (s == 12345.f) out[threadIdx.x] = s;
}

__global__ void __launch_bounds__(256) k_peak_ffma(float *out, int iters)
{
    float2 a[8];
    const float2 m = make_float2(0.9999f, 0.9999f), c = make_float2(1e-4f, 1e-4f);
#pragma unroll
    for (int k = 0; k < 8; k++) a[k] = make_float2(1.0f + k, 2.0f + k);
    for (int i = 0; i < iters; i++) {
#pragma unroll
        for (int k = 0; k < 8; k++) a[k] = __ffma2_rn(a[k], m, c);
    }
    float s = 0.f;
#pragma unroll
    for (int k = 0; k < 8; k++) s += a[k].x + a[k].y;
    if (s == 12345.f) out[threadIdx.x] = s;
}

// Relative error of rsqrt.approx.f32 at every float of [2^lo_exp, 2^hi_exp):
// the largest |rsqrt(x)*sqrt(x) - 1| (FP64) as order-preserving bits of a
// non-negative double.
__global__ void __launch_bounds__(256) k_rsqrt_error(uint32_t bits0, uint32_t n, unsigned long long *max_bits)
{
    double worst = 0.0;
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < n; i += gridDim.x * 256u) {
        const float x = __uint_as_float(bits0 + i);
        const double e = fabs((double)rsqrt_approx(x) * sqrt((double)x) - 1.0);
        worst = fmax(worst, e);
    }
    for (int o = 16; o; o >>= 1) worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, o));
    if ((threadIdx.x & 31) == 0) atomicMax(max_bits, (unsigned long long)__double_as_longlong(worst));
}

// The far kernel's units of 2^24 bins against bins, for the squared distances
// x = every float of [2^lo_exp, ..): the distance, both guard bins and whether
// they differ.  bad[0..2]: how many floats disagree in each.
__global__ void __launch_bounds__(256) k_far_units(uint32_t bits0, uint32_t n, float edge_lo, float edge_hi,
                                                   unsigned long long *bad)
{
    const float2 nlom = make_float2(-edge_lo * FAR_EDGE_DOWN, -edge_lo * FAR_EDGE_DOWN);
    const float2 himd = make_float2(edge_hi * FAR_EDGE_DOWN, edge_hi * FAR_EDGE_DOWN);
    const float2 lom = make_float2(edge_lo, edge_lo), him = make_float2(edge_hi, edge_hi);
    unsigned b[3] = {0, 0, 0};
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < n; i += gridDim.x * 256u) {
        const float x = __uint_as_float(bits0 + i);
        const float t = __fmul_rn(x, rsqrt_approx(x));
        const float xd = x * FAR_DOWN * FAR_DOWN, td = __fmul_rn(xd, rsqrt_approx(xd));
        b[0] += __float_as_uint(td) != __float_as_uint(t * FAR_DOWN);
        const float2 t2 = make_float2(t, t), td2 = make_float2(td, td);
        float2 lo, hi;
        far_guard_bins(t2, lom, him, lo, hi);
        const float2 nlo = far_units_lo(td2, nlom), E = far_units_hi(td2, himd, nlo);
        // the kernel's table offset: the sign bit leaves with the shift
        b[1] += (__float_as_uint(nlo.x) << 2) != (__float_as_uint(lo.x) - MAGIC_BITS) << 2;
        b[2] += __float_as_uint(E.x) != __float_as_uint(hi.x) - __float_as_uint(lo.x);
    }
    for (int k = 0; k < 3; k++) {
        const unsigned s = __reduce_add_sync(0xffffffffu, b[k]);
        if ((threadIdx.x & 31) == 0 && s) atomicAdd(bad + k, (unsigned long long)s);
    }
}

// sqrt_markstein against sqrt.rn at every float of [bits0, bits0 + n): out[0]
// counts the differences.
__global__ void __launch_bounds__(256) k_root_differences(uint32_t bits0, uint32_t n, unsigned long long *out)
{
    unsigned bad = 0;
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < n; i += gridDim.x * 256u) {
        const float x = __uint_as_float(bits0 + i);
        float inv;
        bad += __float_as_uint(sqrt_markstein(x, inv)) != __float_as_uint(__fsqrt_rn(x));
    }
    bad = __reduce_add_sync(0xffffffffu, bad);
    if ((threadIdx.x & 31) == 0 && bad) atomicAdd(out, (unsigned long long)bad);
}

// Largest relative error of rsqrt_f64 over samples of each binade [2^e, 2^(e+1)),
// e = lo_exp + blockIdx.y: mantissas spread over the binade, its ends among
// them.  The error is (1 - x y^2) / 2 with y^2 in two doubles.
__global__ void __launch_bounds__(256) k_rsqrt64_error(int lo_exp, uint32_t n, unsigned long long *max_bits)
{
    double worst = 0.0;
    const unsigned long long exp = (unsigned long long)(lo_exp + (int)blockIdx.y + 1023) << 52;
    for (uint32_t i = blockIdx.x * 256u + threadIdx.x; i < n; i += gridDim.x * 256u) {
        // an odd multiplier visits the mantissas without pattern; the first and the
        // last 256 samples are the binade's ends
        unsigned long long m = (i * 0x9E3779B97F4A7C15ull) >> 12;
        if (i < 256) m = i;
        else if (i >= n - 256) m = (1ull << 52) - (n - i);
        const double x = __longlong_as_double((long long)(exp | m));
        const double y = rsqrt_f64(x);
        const double h = __dmul_rn(y, y), l = __fma_rn(y, y, -h);
        worst = fmax(worst, 0.5 * fabs(__fma_rn(-x, l, __fma_rn(-x, h, 1.0))));
    }
    for (int o = 16; o; o >>= 1) worst = fmax(worst, __shfl_xor_sync(0xffffffffu, worst, o));
    if ((threadIdx.x & 31) == 0) atomicMax(max_bits, (unsigned long long)__double_as_longlong(worst));
}

// Run `launch` on zeroed counters in device memory and read them.
template <class Launch>
static int with_counters(int32_t device, unsigned long long *h, int n, Launch launch)
{
    if (cudaSetDevice(device) != cudaSuccess) return 1;
    unsigned long long *d = nullptr;
    if (cudaMalloc(&d, n * sizeof *d) != cudaSuccess) return 1;
    cudaMemset(d, 0, n * sizeof *d);
    launch(d);
    const cudaError_t e = cudaMemcpy(h, d, n * sizeof *d, cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess && cudaGetLastError() == cudaSuccess ? 0 : 1;
}

}  // namespace agb

extern "C" int ag_diag_far_units(int32_t device, int32_t lo_exp, int32_t hi_exp, float edge_lo, float edge_hi,
                                 int64_t differences[3])
{
    // t * edge stays below 2^23, and x * 2^-48 normal
    if (!differences || lo_exp < 0 || hi_exp > 44 || lo_exp >= hi_exp || !(edge_lo > 0.5f && edge_lo <= edge_hi && edge_hi < 2.f))
        return 1;
    unsigned long long h[3];
    const uint32_t b0 = (uint32_t)(lo_exp + 127) << 23, b1 = (uint32_t)(hi_exp + 127) << 23;
    if (agb::with_counters(device, h, 3, [&](unsigned long long *d) {
            agb::k_far_units<<<4096, 256>>>(b0, b1 - b0, edge_lo, edge_hi, d);
        }))
        return 1;
    for (int k = 0; k < 3; k++) differences[k] = (int64_t)h[k];
    return 0;
}

extern "C" int ag_diag_root_errors(int32_t device, int64_t *sqrt_differences, int32_t lo_exp, int32_t hi_exp,
                                   double *rsqrt64_max_ulps)
{
    if (!sqrt_differences || !rsqrt64_max_ulps || lo_exp < -1000 || hi_exp > 1000 || lo_exp >= hi_exp) return 1;
    unsigned long long h[2];
    const float lo = 1.0e-12f, hi = 64.0f;
    uint32_t b0, b1;
    std::memcpy(&b0, &lo, 4);
    std::memcpy(&b1, &hi, 4);
    if (agb::with_counters(device, h, 2, [&](unsigned long long *d) {
            agb::k_root_differences<<<4096, 256>>>(b0, b1 - b0 + 1, d);
            agb::k_rsqrt64_error<<<dim3(64, (unsigned)(hi_exp - lo_exp)), 256>>>(lo_exp, 1u << 22, d + 1);
        }))
        return 1;
    *sqrt_differences = (int64_t)h[0];
    double v;
    std::memcpy(&v, &h[1], sizeof v);
    *rsqrt64_max_ulps = v * 9007199254740992.0;
    return 0;
}

extern "C" int ag_diag_rsqrt_error(int32_t device, int32_t lo_exp, int32_t hi_exp, double *max_rel_ulps)
{
    if (!max_rel_ulps || lo_exp < -126 || hi_exp > 127 || lo_exp >= hi_exp) return 1;
    if (cudaSetDevice(device) != cudaSuccess) return 1;
    unsigned long long *d = nullptr;
    if (cudaMalloc(&d, sizeof *d) != cudaSuccess) return 1;
    cudaMemset(d, 0, sizeof *d);
    const uint32_t b0 = (uint32_t)(lo_exp + 127) << 23, b1 = (uint32_t)(hi_exp + 127) << 23;
    agb::k_rsqrt_error<<<4096, 256>>>(b0, b1 - b0, d);
    unsigned long long h = 0;
    const cudaError_t e = cudaMemcpy(&h, d, sizeof h, cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e != cudaSuccess || cudaGetLastError() != cudaSuccess) return 1;
    double v;
    std::memcpy(&v, &h, sizeof v);
    *max_rel_ulps = v * 16777216.0;
    return 0;
}

extern "C" int ag_diag_peak_rates(int32_t device, double *rsqrt_per_s, double *fp32_flops_per_s,
                                  double *sm_clock_mhz)
{
    if (cudaSetDevice(device) != cudaSuccess) return 1;
    cudaDeviceProp prop;
    if (cudaGetDeviceProperties(&prop, device) != cudaSuccess) return 1;
    float *out = nullptr;
    if (cudaMalloc(&out, 1024 * sizeof(float)) != cudaSuccess) return 1;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    const int blocks = prop.multiProcessorCount * 8, threads = 256, iters = 4096;
    double best_r = 0, best_f = 0;
    for (int rep = 0; rep < 3; rep++) {
        float ms = 0;
        cudaEventRecord(e0);
        agb::k_peak_rsqrt<<<blocks, threads>>>(out, iters);
        cudaEventRecord(e1);
        cudaEventSynchronize(e1);
        cudaEventElapsedTime(&ms, e0, e1);
        if (ms > 0) best_r = std::max(best_r, (double)blocks * threads * iters * 8 / (ms * 1e-3));
        cudaEventRecord(e0);
        agb::k_peak_ffma<<<blocks, threads>>>(out, iters);
        cudaEventRecord(e1);
        cudaEventSynchronize(e1);
        cudaEventElapsedTime(&ms, e0, e1);
        if (ms > 0) best_f = std::max(best_f, (double)blocks * threads * iters * 8 * 2 * 2 / (ms * 1e-3));
    }
    int clk_khz = 0;
    cudaDeviceGetAttribute(&clk_khz, cudaDevAttrClockRate, device);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(out);
    if (rsqrt_per_s) *rsqrt_per_s = best_r;
    if (fp32_flops_per_s) *fp32_flops_per_s = best_f;
    if (sm_clock_mhz) *sm_clock_mhz = clk_khz / 1000.0;
    return cudaGetLastError() == cudaSuccess ? 0 : 1;
}
