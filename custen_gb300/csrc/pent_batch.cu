// Batched pentadiagonal factorisation and solve over the interleaved layout of cuPentBatch
// (cuPentCahnADI/src/cuPentBatch.cu): element (row i, system s) of every diagonal and of the
// right-hand side lives at [i * batch + s]; ds / dl are the diagonals two and one below the main one
// (ds[0], ds[1], dl[0] zero), du / dw one and two above (du[m-1], dw[m-2], dw[m-1] zero).
//
// pent_factor: in place, the reference's pentFactorBatch (:35-113) -- the same expressions in the same
// order, so every factor is bit-identical to the reference kernel's on the same GPU.
// pent_solve: the reference's pentSolveBatch (:119-198), bit-identical as well.
// pent_invert_pivots / pent_solve_rcp: the fast variant this library's ADI solver uses -- pivots
// inverted once, the solve multiplies instead of dividing (rounding differs from the reference by about
// one unit in the last place per row).
//
// GB300 shape: one thread per system, coalesced across systems (the layout's purpose), one warp per CTA so that a
// batch spreads evenly over the SMs. The per-row recurrence is a dependent chain; the rows ahead of it are copied
// into a shared-memory ring while it runs, and the rows it refers back to stay in registers. The divisions of the
// exact variants are the correctly rounded ones of fp64_offload.cuh (5 FP64 operations, 8 for the two that
// share a pivot, against 9.4 each for the operator). The exact variants are bound by the FP64 pipe (12 and 9
// operations a row), the reciprocal variant by HBM.
// Measured, 262144 systems of 256 rows, G rows/s (before: operator divisions, loads staged in registers):
// factorisation 27.9 -> 48.6, exact solve 44.2 -> 62.7, inverted-pivot solve 80.8 -> 93.9 (6.8 TB/s); 4096 systems of
// 512 rows: 4.6 -> 6.0, 3.6 -> 7.7, 4.6 -> 13.8.
#include <cuda_runtime.h>

#include <atomic>

#include <algorithm>
#include <cstdio>
#include <string>

#include "../../include/custen_gb300.h"
#include "fp64_offload.cuh"

namespace custen {
namespace pent {
namespace {

constexpr int kThreads = 128;    // pivot inversion
constexpr int kLine = 32;        // systems per CTA of the factorisation and the solves: one warp

// Rows in flight: every thread copies the values of the next D rows of its own system into its own slots of a
// shared-memory ring (cp.async, one group per row), so the loads take no registers and no barrier. A row beyond
// the end leaves an empty group, which keeps the group count per row fixed.
__device__ __forceinline__ void copy8(double* dst, const double* src) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src) : "memory");
}
__device__ __forceinline__ void commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void wait_group() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

// Expressions and order of the reference's pentFactorBatch (cuPentBatch.cu:35-113): rows 0 and 1 lack the terms
// of the rows before them, row m-2 has no dw, row m-1 neither du nor dw.
template <int D>
__global__ void __launch_bounds__(kLine) factor_kernel(const double* __restrict__ ds, double* dl, double* d, double* du,
                                                       double* dw, int m, int batch) {
    __shared__ double ring[D][5][kLine];
    const int t = threadIdx.x;
    const int s = blockIdx.x * kLine + t;
    if (s >= batch) return;
    const size_t B = (size_t)batch;
    const f64::F64 f;
    auto issue = [&](int i) {
        if (i < m) {
            const size_t q = (size_t)i * B + s;
            double(*r)[kLine] = ring[i % D];
            if (i >= 2) copy8(&r[0][t], ds + q);
            if (i >= 1) copy8(&r[1][t], dl + q);
            copy8(&r[2][t], d + q);
            if (i < m - 1) copy8(&r[3][t], du + q);
            if (i < m - 2) copy8(&r[4][t], dw + q);
        }
        commit();
    };
#pragma unroll
    for (int i = 0; i < D; ++i) issue(i);
    // (du, dw) of the two previous rows: P2 = row i-2, P1 = row i-1
    double duP2 = 0.0, dwP2 = 0.0, duP1 = 0.0, dwP1 = 0.0;
#pragma unroll 1
    for (int i = 0; i < m; ++i) {
        wait_group<D - 1>();
        const size_t q = (size_t)i * B + s;
        const double(*r)[kLine] = ring[i % D];
        double dd = r[2][t], l = 0.0;
        if (i >= 2) {   // interior rows (:75-80)
            const double vs = r[0][t];
            l = r[1][t] - vs * duP2;
            dd = dd - vs * dwP2 - l * duP1;
            dl[q] = l;
            d[q] = dd;
        } else if (i == 1) {
            l = r[1][t];
            dd = dd - l * duP1;
            d[q] = dd;
        }
        const f64::Divider by(f, dd);
        duP2 = duP1;
        const double dwL = dwP1;
        dwP2 = dwP1;
        if (i < m - 2) {
            dwP1 = by(r[4][t]);
            dw[q] = dwP1;
        }
        if (i < m - 1) {
            const double vu = r[3][t];
            duP1 = by(i >= 1 ? vu - l * dwL : vu);
            du[q] = duP1;
        }
        issue(i + D);
    }
}

// pentSolveBatch (cuPentBatch.cu:119-198): forward substitution (:153-171), then backward (:178-196). RCP: d holds
// the inverted pivots. Each thread re-reads in the backward pass what it stored itself in the forward pass.
template <int D, bool RCP>
__global__ void __launch_bounds__(kLine) solve_kernel(const double* __restrict__ ds, const double* __restrict__ dl,
                                                      const double* __restrict__ d, const double* __restrict__ du,
                                                      const double* __restrict__ dw, double* b, int m, int batch) {
    __shared__ double ring[D][4][kLine];
    const int t = threadIdx.x;
    const int s = blockIdx.x * kLine + t;
    if (s >= batch) return;
    const size_t B = (size_t)batch;
    const f64::F64 f;
    auto issue = [&](int i) {
        if (i < m) {
            const size_t q = (size_t)i * B + s;
            double(*r)[kLine] = ring[i % D];
            if (i >= 2) copy8(&r[0][t], ds + q);
            if (i >= 1) copy8(&r[1][t], dl + q);
            copy8(&r[2][t], d + q);
            copy8(&r[3][t], b + q);
        }
        commit();
    };
#pragma unroll
    for (int i = 0; i < D; ++i) issue(i);
    double p2 = 0.0, p1 = 0.0;
#pragma unroll 1
    for (int i = 0; i < m; ++i) {
        wait_group<D - 1>();
        const double(*r)[kLine] = ring[i % D];
        double v = r[3][t];
        if (i >= 2) v = v - r[0][t] * p2 - r[1][t] * p1;
        else if (i == 1) v = v - r[1][t] * p1;
        v = RCP ? f.mul(v, r[2][t]) : f64::Divider(f, r[2][t])(v);
        b[(size_t)i * B + s] = v;
        p2 = p1;
        p1 = v;
        issue(i + D);
    }
    wait_group<0>();
    // row m-1 is done; p1, p2: rows i+1, i+2
    auto issue_back = [&](int k) {   // k rows above row m-2
        const int i = m - 2 - k;
        if (i >= 0) {
            const size_t q = (size_t)i * B + s;
            double(*r)[kLine] = ring[k % D];
            copy8(&r[0][t], du + q);
            if (k > 0) copy8(&r[1][t], dw + q);
            copy8(&r[2][t], b + q);
        }
        commit();
    };
#pragma unroll
    for (int k = 0; k < D; ++k) issue_back(k);
    p2 = 0.0;
#pragma unroll 1
    for (int k = 0; k < m - 1; ++k) {
        wait_group<D - 1>();
        const double(*r)[kLine] = ring[k % D];
        double v = r[2][t] - r[0][t] * p1;
        if (k > 0) v = v - r[1][t] * p2;
        b[(size_t)(m - 2 - k) * B + s] = v;
        p2 = p1;
        p1 = v;
        issue_back(k + D);
    }
}

__global__ void __launch_bounds__(kThreads) invert_kernel(double* __restrict__ d, size_t count) {
    const size_t step = (size_t)gridDim.x * blockDim.x;
    size_t q = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (q >= count) return;
    double x = d[q];   // on its way while the constants are read
    const f64::F64 f;
    for (;;) {
        d[q] = f64::reciprocal(f, x);
        if ((q += step) >= count) return;
        x = d[q];
    }
}

thread_local std::string g_err;
std::atomic<int> g_kr[3] = {0, 0, 0};   // rows in flight of factor, exact solve, inverted-pivot solve; 0: by the rule

// Rows in flight: 8 while at most two warps share an FP64 sub-partition (4 per SM) and the copies' latency shows,
// else 4, since a deep ring limits the resident warps. Measured (us, 4 / 8 rows): inverted-pivot solve 179 / 152 with
// 4096 systems of 512 rows, 41 / 38 with 20000 of 100, 369 / 451 with 131072 of 256; exact solve 287 / 271, 65 / 64,
// 561 / 629; factorisation 352 / 352, 78 / 79, 709 / 760.
int rows_in_flight(int which, int blocks) {
    const int set = g_kr[which].load();
    if (set) return set;
    static std::atomic<int> sms[64] = {};   // threads that race store the same value
    int dev = 0, n = 0;
    if (cudaGetDevice(&dev) == cudaSuccess && dev >= 0 && dev < 64) {
        n = sms[dev].load(std::memory_order_relaxed);
        if (n == 0 && cudaDeviceGetAttribute(&n, cudaDevAttrMultiProcessorCount, dev) == cudaSuccess)
            sms[dev].store(n, std::memory_order_relaxed);
    }
    return blocks <= 8 * n ? 8 : 4;
}

template <typename F2, typename F4, typename F8>
void by_depth(int kr, F2 f2, F4 f4, F8 f8) {
    if (kr <= 2) f2();
    else if (kr <= 4) f4();
    else f8();
}

int check(cudaError_t e, const char* what) {
    if (e == cudaSuccess) return 0;
    g_err = std::string("Error while '") + what + "': " + cudaGetErrorString(e);
    cudaGetLastError();
    return 1;
}

int check_args(const void* a, const void* b, const void* c, const void* dd, const void* e, int m, int batch) {
    if (!a || !b || !c || !dd || !e) {
        g_err = "diagonal pointers must not be NULL";
        return 2;
    }
    if (m < 4 || batch < 1) {
        g_err = "need m >= 4 unknowns and batch >= 1 systems";
        return 2;
    }
    return 0;
}

}  // namespace
}  // namespace pent
}  // namespace custen

using namespace custen::pent;

extern "C" {

const char* custen_pent_last_error(void) { return g_err.c_str(); }

// Rows in flight ahead of the chain (2, 4 or 8; 0: by the batch size) of the factorisation (which = 0),
// the exact solve (1) and the inverted-pivot solve (2). Results do not depend on it.
int custen_pent_set_depth(int which, int rows) {
    if (which < 0 || which > 2 || (rows != 0 && rows != 2 && rows != 4 && rows != 8)) {
        g_err = "invalid prefetch depth";
        return 2;
    }
    g_kr[which] = rows;
    return 0;
}

// Rows in flight that a call for `batch` systems on the current device takes; 0 for invalid arguments.
int custen_pent_depth(int which, int batch) {
    return which < 0 || which > 2 || batch < 1 ? 0 : rows_in_flight(which, (batch - 1) / kLine + 1);
}

int custen_pent_factor_batch(double* ds, double* dl, double* d, double* du, double* dw, int m, int batch,
                             void* stream) {
    if (int st = check_args(ds, dl, d, du, dw, m, batch)) return st;
    const int blocks = (batch + kLine - 1) / kLine;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    by_depth(
        rows_in_flight(0, blocks), [&] { factor_kernel<2><<<blocks, kLine, 0, st>>>(ds, dl, d, du, dw, m, batch); },
        [&] { factor_kernel<4><<<blocks, kLine, 0, st>>>(ds, dl, d, du, dw, m, batch); },
        [&] { factor_kernel<8><<<blocks, kLine, 0, st>>>(ds, dl, d, du, dw, m, batch); });
    return check(cudaGetLastError(), "Launching the batched factorisation");
}

int custen_pent_solve_batch(const double* ds, const double* dl, const double* d, const double* du, const double* dw,
                            double* b, int m, int batch, void* stream) {
    if (int st = check_args(ds, dl, d, du, dw, m, batch)) return st;
    if (!b) {
        g_err = "right-hand side pointer must not be NULL";
        return 2;
    }
    const int blocks = (batch + kLine - 1) / kLine;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    by_depth(
        rows_in_flight(1, blocks), [&] { solve_kernel<2, false><<<blocks, kLine, 0, st>>>(ds, dl, d, du, dw, b, m, batch); },
        [&] { solve_kernel<4, false><<<blocks, kLine, 0, st>>>(ds, dl, d, du, dw, b, m, batch); },
        [&] { solve_kernel<8, false><<<blocks, kLine, 0, st>>>(ds, dl, d, du, dw, b, m, batch); });
    return check(cudaGetLastError(), "Launching the batched solve");
}

int custen_pent_invert_pivots(double* d, int m, int batch, void* stream) {
    if (!d || m < 4 || batch < 1) {
        g_err = "invalid arguments";
        return 2;
    }
    int sms = 0, dev = 0;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    invert_kernel<<<sms * 8, kThreads, 0, static_cast<cudaStream_t>(stream)>>>(d, (size_t)m * batch);
    return check(cudaGetLastError(), "Inverting the pivots");
}

int custen_pent_solve_batch_rcp(const double* ds, const double* dl, const double* rd, const double* du,
                                const double* dw, double* b, int m, int batch, void* stream) {
    if (int st = check_args(ds, dl, rd, du, dw, m, batch)) return st;
    if (!b) {
        g_err = "right-hand side pointer must not be NULL";
        return 2;
    }
    const int blocks = (batch + kLine - 1) / kLine;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    by_depth(
        rows_in_flight(2, blocks), [&] { solve_kernel<2, true><<<blocks, kLine, 0, st>>>(ds, dl, rd, du, dw, b, m, batch); },
        [&] { solve_kernel<4, true><<<blocks, kLine, 0, st>>>(ds, dl, rd, du, dw, b, m, batch); },
        [&] { solve_kernel<8, true><<<blocks, kLine, 0, st>>>(ds, dl, rd, du, dw, b, m, batch); });
    return check(cudaGetLastError(), "Launching the batched solve");
}

}  // extern "C"
