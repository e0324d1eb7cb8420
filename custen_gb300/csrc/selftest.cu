// Self-test of the bounded mbarrier wait of the TMA-staged stencil kernels (stencil_tma.cuh).
//
// One CTA initialises an mbarrier that nothing will ever arrive on and waits on it with the same
// mbar_wait as the stencil kernels, with a short round limit. The wait must give up, the kernel must
// record kErrMbarrierTimeout in the device error flags and return, and the context must stay usable.
// No copy is in flight and no thread traps: this exercises the failure path the stencil kernels take
// when a tensor copy never completes, without making one fail.
//
// And a self-test of fp64_offload.cuh: its conversions and divisions against the compiler's own operators.
#include <cuda_runtime.h>

#include "../../include/custen_gb300.h"
#include "fp64_offload.cuh"
#include "stencil_tma.cuh"

namespace custen {
namespace {

__global__ void wait_expiry_kernel(long long limit) {
    __shared__ __align__(8) uint64_t bar;
    if (threadIdx.x == 0) mbar_init(&bar, 1);
    __syncthreads();
    const bool ok = threadIdx.x == 0 ? mbar_wait(&bar, 0, limit) : true;
    if (__syncthreads_or(!ok) && threadIdx.x == 0) atomicOr(&g_custen_device_error, kErrMbarrierTimeout);
}

__device__ __forceinline__ unsigned long long mix64(unsigned long long z) {   // splitmix64
    z += 0x9e3779b97f4a7c15ull;
    z = (z ^ (z >> 30)) * 0xbf58476d1ce4e5b9ull;
    z = (z ^ (z >> 27)) * 0x94d049bb133111ebull;
    return z ^ (z >> 31);
}

// A test operand: random bits; a random significand within 2^-60 .. 2^60; one with few bits set (exact and
// halfway quotients, ties of the conversion); a significand next to all ones or all zeros; or a special value.
__device__ double fp64_operand(unsigned long long r) {
    const unsigned long long sign = r & 0x8000000000000000ull;
    const unsigned long long frac = mix64(r) & 0xfffffffffffffull;
    const unsigned long long ex = (1023ull - 60 + mix64(r + 1) % 121) << 52;
    switch (mix64(r + 2) % 6) {
    case 0: return __longlong_as_double((long long)mix64(r + 3));
    case 1: return __longlong_as_double((long long)(sign | ex | (frac & ~0xfffffffffull)));
    case 2: return __longlong_as_double((long long)(sign | ex | (frac & 0xfffffffe0000000ull) | 0x10000000ull));   // a float tie
    case 3: return __longlong_as_double((long long)(sign | ex | ((r & 1) ? 0xfffffffffffffull - (frac & 3) : (frac & 3))));
    case 4: {
        const double sp[12] = {0.0, 4.9e-324, 2.2250738585072014e-308, 1.1754943508222875e-38, 1.401298464324817e-45,
                               3.4028234663852886e38, 3.4028235677973366e38, 1.7976931348623157e308,
                               __longlong_as_double(0x7ff0000000000000ll), __longlong_as_double(0x7ff8000000000000ll),
                               1.0, 7.006492321624085e-46};
        const double v = sp[mix64(r + 4) % 12];
        return sign ? -v : v;
    }
    default: return __longlong_as_double((long long)(sign | ex | frac));
    }
}

__device__ __forceinline__ bool same_bits(double a, double b) {
    return __double_as_longlong(a) == __double_as_longlong(b) || (isnan(a) && isnan(b));
}

// out[0 .. 5]: mismatches of to_float, to_double_pos (plain and quartered), div_by_float, reciprocal, Divider, and
// of the sums, differences and products as multiply-adds
__global__ void fp64_offload_kernel(unsigned long long seed, long long samples, unsigned long long* out) {
    const double cs[3] = {0.1, 0.6, 0.3};
    const f64::F64 f64c;
    for (long long i = blockIdx.x * (long long)blockDim.x + threadIdx.x; i < samples;
         i += (long long)gridDim.x * blockDim.x) {
        const unsigned long long r = mix64(seed + 8ull * (unsigned long long)i);
        const double a = fp64_operand(r), b = fp64_operand(r + 77);
        const float f = f64::to_float(a);
        const float fr = (float)a;
        if (__float_as_uint(f) != __float_as_uint(fr) && !(isnan(f) && isnan(fr))) atomicAdd(&out[0], 1ull);
        const float p = fabsf(fr);
        if (!same_bits(f64::to_double_pos(p), (double)p) || !same_bits(f64::to_double_pos<-2>(p), 0.25 * (double)p))
            atomicAdd(&out[1], 1ull);
        for (int k = 0; k < 3; ++k)
            if (!same_bits(f64::div_by_float(f64c, cs[k], p), cs[k] / (double)p)) atomicAdd(&out[2], 1ull);
        if (!same_bits(f64::reciprocal(f64c, b), 1.0 / b)) atomicAdd(&out[3], 1ull);
        if (!same_bits(f64::Divider(f64c, b)(a), a / b)) atomicAdd(&out[4], 1ull);
        if (!same_bits(f64c.add(a, b), __dadd_rn(a, b)) || !same_bits(f64c.sub(a, b), __dsub_rn(a, b)) ||
            !same_bits(f64c.mul(a, b), __dmul_rn(a, b)))
            atomicAdd(&out[5], 1ull);
    }
}

}  // namespace
}  // namespace custen

// Runs the wait with `rounds` try_wait rounds (1 .. 2^22) and returns the device error flags seen
// afterwards in *flags (bit 0 expected); the flags are left set for the caller to read and clear with
// custen_device_error. Returns 0 when the kernel ran and returned.
extern "C" int custen_selftest_wait_expiry(long long rounds, unsigned int* flags) {
    if (rounds < 1 || rounds > custen::kWaitLimit || !flags) return 2;
    custen::wait_expiry_kernel<<<1, 32>>>(rounds);
    cudaError_t e = cudaGetLastError();
    if (e == cudaSuccess) e = cudaDeviceSynchronize();
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(flags, custen::g_custen_device_error, sizeof(unsigned int));
    return e == cudaSuccess ? 0 : 1;
}

// Compares fp64_offload.cuh with the compiler's operators on `samples` operands; mismatches[0 .. 5] receive
// the counts for the conversions to float and to double, c / float, 1 / x, a / b, and a + b, a - b, a b (all
// expected zero).
extern "C" int custen_selftest_fp64(unsigned long long seed, long long samples, unsigned long long* mismatches) {
    if (samples < 1 || samples > (1ll << 34) || !mismatches) return 2;
    unsigned long long* d = nullptr;
    cudaError_t e = cudaMalloc(&d, 6 * sizeof(unsigned long long));
    if (e == cudaSuccess) e = cudaMemset(d, 0, 6 * sizeof(unsigned long long));
    if (e == cudaSuccess) {
        custen::fp64_offload_kernel<<<1216, 256>>>(seed, samples, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(mismatches, d, 6 * sizeof(unsigned long long), cudaMemcpyDeviceToHost);
    cudaFree(d);
    return e == cudaSuccess ? 0 : 1;
}
