// Cahn-Hilliard ADI solver on sm_103a: one time step of many periodic grids of different sizes.
//
// Scheme of the reference solver (cuPentCahnADI/src/cuPentCahnADI.cu:528-596, and its CPU twin
// cuPentSpeedUp/serialCahnADITiming/serialCahnADI.c:1010-1047), per grid of n x n points:
//   cBar = 2 cCurr - cOld
//   rhs  = Lin5x5(cBar) + Nl3x3(cCurr^3 - cCurr) - (2/3)(cCurr - cOld)
//   (1 + s Dx4)(1 + s Dy4) delta = rhs   -- two cyclic pentadiagonal sweeps, x then y
//   cNew = cBar + delta;  cOld <- cCurr;  cCurr <- cNew
//
// GB300 shape: FP64 FMAs (about 2 per clock per SM) bound this solver, not HBM, so the kernels
// minimise FP64 operations (about 26 per point and step, against about 100 in the reference: the two
// explicit stencils as two 5-point Laplacians, cBar and c^3 - c computed once per point, the line operators
// factored with constant coefficients) and keep every SM sub-partition busy:
//   K1 ch_rhs_kernel / ch_h_kernel + ch_rhs2_kernel -- right-hand side, 32 x 32 blocks, lane = column, all points
//                           in parallel.
//   K2 ch_xsweep_kernel  -- x sweep, two chains (warps) per 32 rows, lane = row.
//   K3 ch_ysweep_kernel  -- y sweep, two chains per 32 columns, lane = column.
//   K4 ch_update_kernel  -- cNew = cBar + delta, written over cOld (the two field buffers swap roles every step).
// Each launch covers all grids of a work list (largest first), so grids of different sizes share it; pairs of steps
// are captured in a CUDA graph.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <complex>
#include <cstdio>
#include <cstring>
#include <string>
#include <type_traits>
#include <vector>

#include "../../include/custen_gb300.h"
#include "ch_internal.cuh"
#include "checked.cuh"
#include "fp64_offload.cuh"
#include "stencil_launch.cuh"   // mbarrier and TMA helpers, the tensor map encoder

namespace custen {
namespace ch {

// ------------------------------------------------------------------------------------------------
// K1: right-hand side
// ------------------------------------------------------------------------------------------------
// T = double: FP64 arithmetic; T = float: the FP32 precision variant (cBar, c^3 - c, the inner Laplacian
// and h in FP32 from inputs and coefficients rounded to float; the outer Laplacian of the FP32 h values
// and the time-derivative term summed in FP64, which keeps the mass conserved to FP64 rounding).
//
// The reference's two explicit stencils are the 13-point biharmonic sigma_lin * [-1; -2 8 -2; -1 8 -20
// 8 -1; ...] on cBar and the 5-point Laplacian sigma_nl * [1; 1 -4 1; 1] on c^3 - c
// (cuPentCahnADI.cu:463-467, 509-513). The biharmonic is the 5-point Laplacian applied twice, so
//   Lin(cBar) + Nl(g) = Lap(h),   h = sigma_nl * g - sigma_lin * Lap(cBar),
// with Lap the unit-weight 5-point Laplacian (N + S + W + E - 4 C). The kernel evaluates that form:
// about 14 FP64 operations per point instead of 24 for the two stencils taken separately. The sums are
// the same mathematically; their rounding differs from the reference's weight-by-weight chain at the
// level of one rounding per term, far inside the solver's 1e-10 parity bar.
// NW warps per CTA share one 32 x 32 work item: shared memory limits residency to a few CTAs per SM, so
// more warps per CTA give the FP64 pipe more warps to issue from (the tuned choice, ChConfig).
//
// The constant factors 2, -4 and -2/3 are read from device memory into registers once per thread: an
// FP64 FMA that takes a literal or a kernel parameter as an operand issues about 19% slower on GB300
// (507 against 602-628 G FMA/s measured) than one whose operands are all registers. The values, and
// so the results, are the same as with literals.
__device__ double g_rhs_factors[3] = {2.0, -4.0, -2.0 / 3.0};

// Sums and products: FP64 ones as multiply-adds (fp64_offload.cuh; at first use h kernel 459 -> 425 us and pass 2 320 ->
// 296 us at 24 grids of 1024^2), FP32 ones as they are.
template <typename T>
struct Arith {
    __device__ __forceinline__ T add(T a, T b) const { return a + b; }
    __device__ __forceinline__ T sub(T a, T b) const { return a - b; }
    __device__ __forceinline__ T mul(T a, T b) const { return a * b; }
};
template <>
struct Arith<double> : f64::F64 {};

// The five-point Laplacian N + S + W + E - 4 C. The FP64 one adds N + E and W + S first: with d(r, c) = v(r, c) +
// v(r + 1, c + 1) these are d of the point above and d of the point to the left, so the kernels of the two-pass form
// add d once per point (diagonal_sums) and take two additions where the points apart take three.
template <typename T>
__device__ __forceinline__ T laplacian(const Arith<T>& ar, T m_four, T c, T n, T s, T w, T e) {
    if constexpr (std::is_same<T, double>::value) return fma(m_four, c, ar.add(ar.add(n, e), ar.add(w, s)));
    else return fma(m_four, c, ar.add(ar.add(n, s), ar.add(w, e)));
}
// d over a 32 x 32 block with its halo: 1089 sums for 1024 points. The caller synchronises before and after.
template <int NT>
__device__ __forceinline__ void diagonal_sums(const Arith<double>& ar, const double* v, double (&d)[33][33], int tid) {
#pragma unroll
    for (int e = tid; e < 33 * 33; e += NT) {
        const int r = e / 33, c = e - r * 33;
        d[r][c] = ar.add(v[r * 35 + c], v[(r + 1) * 35 + c + 1]);
    }
}

// h from c and Lap(cBar), in units of sigma_nl in FP64 (one operation less): c (c^2 - 1) - ratio Lap(cBar), ratio =
// sigma_lin / sigma_nl, with a = ratio; in FP32 sigma_nl (c^3 - c) - sigma_lin Lap(cBar), with a, b = sigma_lin,
// sigma_nl.
template <typename T>
struct HValue {
    T a, b;
    __device__ __forceinline__ explicit HValue(const double* tab) {
        constexpr bool d = std::is_same<T, double>::value;
        a = (T)tab[d ? TAB_RATIO : TAB_SLIN];
        b = (T)tab[TAB_SNL];
    }
    __device__ __forceinline__ T operator()(const Arith<T>& ar, T c, T lap) const {
        if constexpr (std::is_same<T, double>::value) return fma(c, fma(c, c, -ar.one), ar.mul(-a, lap));
        else return fma(-a, lap, ar.mul(b, fma(ar.mul(c, c), c, -c)));
    }
};

// The right-hand side (findRHS, cuPentCahnADI.cu:72-86) from Lap(h) and cCurr - cOld: over FP64 h in units of 2/3,
// (3/2) sigma_nl Lap(h) - (cCurr - cOld), which the update takes back (TAB_KAPPA, TAB_OUT); over FP32 h as it stands.
template <typename T>
struct RhsValue {
    double k;
    __device__ __forceinline__ explicit RhsValue(const double* tab) {
        k = std::is_same<T, double>::value ? tab[TAB_LAP] : ((const volatile double*)g_rhs_factors)[2];
    }
    __device__ __forceinline__ double operator()(double lap, double dco) const {
        return std::is_same<T, double>::value ? fma(k, lap, -dco) : fma(k, dco, lap);
    }
};

template <typename T, int NW>
__global__ void __launch_bounds__(NW * BLK) ch_rhs_kernel(const GridDev* __restrict__ grids,
                                                          const Item* __restrict__ items, int n_items, int parity) {
    __shared__ T cb[36][37];        // cBar over the block and a 2-point halo
    __shared__ T hh[34][35];        // c, then h, over the block and a 1-point halo
    __shared__ double dco[32][33];  // cCurr - cOld at the block's points (FP64 in both variants)
    constexpr int NT = NW * BLK;
    const int tid = threadIdx.x;
    const int lane = tid & (BLK - 1), warp = tid / BLK;
    const volatile double* factors = g_rhs_factors;
    const T two = (T)factors[0], m_four = (T)factors[1];
    const double m_four_d = factors[1];
    const Arith<T> ar;
    const Arith<double> ar_d;
    launch_wait();
    for (int it = blockIdx.x; it < n_items; it += gridDim.x) {
        const Item item = items[it];
        const GridDev gd = grids[item.grid];
        const int n = gd.n;
        // selects rather than gd.buf[parity]: a run-time index would put the descriptor in local memory
        const double* cur = parity ? gd.buf[1] : gd.buf[0];
        const double* old = parity ? gd.buf[0] : gd.buf[1];
        const double* tab = gd.tab;
        const int bpr = n / BLK;
        const int y0 = (item.block / bpr) * BLK, x0 = (item.block % bpr) * BLK;
        const HValue<T> h(tab);
        // stage the 36 x 36 window (periodic wrap)
#pragma unroll 4
        for (int e = tid; e < 36 * 36; e += NT) {
            const int r = e / 36, c = e - r * 36;
            int gy = y0 - 2 + r, gx = x0 - 2 + c;
            gy = gy < 0 ? gy + n : (gy >= n ? gy - n : gy);
            gx = gx < 0 ? gx + n : (gx >= n ? gx - n : gx);
            const double cv = cur[(size_t)gy * n + gx];
            const double ov = old[(size_t)gy * n + gx];
            const T c32 = (T)cv, o32 = (T)ov;
            cb[r][c] = fma(two, c32, -o32);
            if (r >= 1 && r < 35 && c >= 1 && c < 35) hh[r - 1][c - 1] = c32;
            if (r >= 2 && r < 34 && c >= 2 && c < 34) dco[r - 2][c - 2] = ar_d.sub(cv, ov);
        }
        __syncthreads();
        // h over the 34 x 34 block + halo
#pragma unroll 4
        for (int e = tid; e < 34 * 34; e += NT) {
            const int r = e / 34, c = e - r * 34;
            const T lap = laplacian(ar, m_four, cb[r + 1][c + 1], cb[r][c + 1], cb[r + 2][c + 1], cb[r + 1][c], cb[r + 1][c + 2]);
            hh[r][c] = h(ar, hh[r][c], lap);
        }
        __syncthreads();
        // rhs = Lap(h) - (2/3)(cCurr - cOld)  (findRHS, cuPentCahnADI.cu:72-86); lane = column. Summed in
        // FP64 in both variants: over FP32 values of h (the precision variant) the FP64 sums are exact, so
        // the discrete Laplacian sums to zero over the periodic grid and the mass is conserved to FP64
        // rounding, as in the FP64 variant.
        const RhsValue<T> rhs(tab);
        const int j = lane;
        double* out = gd.tmp + (size_t)y0 * n + x0 + j;
#pragma unroll 4
        for (int rr = warp; rr < BLK; rr += NW) {
            const double lap = laplacian(ar_d, m_four_d, (double)hh[rr + 1][j + 1], (double)hh[rr][j + 1],
                                         (double)hh[rr + 2][j + 1], (double)hh[rr + 1][j], (double)hh[rr + 1][j + 2]);
            if (!in_bounds((long long)(y0 + rr) * n + x0 + j, 0, (long long)n * n)) continue;
            out[(size_t)rr * n] = rhs(lap, dco[rr][j]);
        }
        __syncthreads();
    }
}

// ------------------------------------------------------------------------------------------------
// K1 in two passes (configurations with warps2): h is formed once per point and kept in the grid's h buffer, so that no
// block recomputes its neighbours' halo values of h (K1 above forms cBar on a 2-point halo and h on a 1-point halo of
// every block, 15.1 FP64 operations per point), and the Laplacians' diagonal sums are added once per point: 7.3
// operations in pass 1 and 5.1 in pass 2. The values are those of K1 bit for bit.
// One CTA per block, its descriptor read before the wait for the previous kernel: 7 to 9 CTAs of 8 warps share an SM and
// hide one another's loads and barriers. At 24 grids of 1024^2, us (share of the FP64 pipe): pass 1 312 (94%), pass 2
// 221 (94%); before, persistent CTAs without shared sums and with h and the sum in plain units 428 (89%) and 296 (84%,
// with a cp.async double buffer); persistent CTAs with them 363 (85%) and 248 (87%). 96 grids of 64^2 .. 1024^2 in all:
// 1231, 1423 and 1317 us a step; over FP32 values 1294, 1379 and 1330.
// ------------------------------------------------------------------------------------------------
// Pass 1: h = sigma_nl * (c^3 - c) - sigma_lin * Lap(cBar), cBar over the block and a 1-point halo.
template <typename T, int NW>
__global__ void __launch_bounds__(NW * BLK) ch_h_kernel(const GridDev* __restrict__ grids, const Item* __restrict__ items,
                                                        int parity) {
    constexpr bool kFp64 = std::is_same<T, double>::value;
    __shared__ T cb[34][35];
    __shared__ T cc[32][33];
    __shared__ double diag[kFp64 ? 33 : 1][33];
    constexpr int NT = NW * BLK;
    const int tid = threadIdx.x;
    const volatile double* factors = g_rhs_factors;
    const T two = (T)factors[0], m_four = (T)factors[1];
    const Arith<T> ar;
    const Item item = items[blockIdx.x];
    const GridDev gd = grids[item.grid];
    const HValue<T> h(gd.tab);
    launch_wait();
    const int n = gd.n;
    const double* cur = parity ? gd.buf[1] : gd.buf[0];
    const double* old = parity ? gd.buf[0] : gd.buf[1];
    const int bpr = n / BLK;
    const int y0 = (item.block / bpr) * BLK, x0 = (item.block % bpr) * BLK;
#pragma unroll 4
    for (int e = tid; e < 34 * 34; e += NT) {
        const int r = e / 34, c = e - r * 34;
        int gy = y0 - 1 + r, gx = x0 - 1 + c;
        gy = gy < 0 ? gy + n : (gy >= n ? gy - n : gy);
        gx = gx < 0 ? gx + n : (gx >= n ? gx - n : gx);
        const double cv = cur[(size_t)gy * n + gx];
        const double ov = old[(size_t)gy * n + gx];
        const T c32 = (T)cv, o32 = (T)ov;
        cb[r][c] = fma(two, c32, -o32);
        if (r >= 1 && r < 33 && c >= 1 && c < 33) cc[r - 1][c - 1] = c32;
    }
    __syncthreads();
    if constexpr (kFp64) {
        diagonal_sums<NT>(ar, &cb[0][0], diag, tid);
        __syncthreads();
    }
#pragma unroll 4
    for (int e = tid; e < 32 * 32; e += NT) {
        const int r = e / 32, c = e - r * 32;
        T lap;
        if constexpr (kFp64) lap = fma(m_four, cb[r + 1][c + 1], ar.add(diag[r][c + 1], diag[r + 1][c]));
        else lap = laplacian(ar, m_four, cb[r + 1][c + 1], cb[r][c + 1], cb[r + 2][c + 1], cb[r + 1][c], cb[r + 1][c + 2]);
        const long long q = (long long)(y0 + r) * n + x0 + c;
        if (in_bounds(q, 0, (long long)n * n)) gd.hbuf[q] = (double)h(ar, cc[r][c], lap);
    }
}

// Pass 2: rhs = Lap(h) - (2/3)(cCurr - cOld) (findRHS, cuPentCahnADI.cu:72-86), h over the block and a
// 1-point halo from the h buffer.
// cp.async helpers (8-byte copies into shared memory, grouped, waited on by group count)
__device__ __forceinline__ void cp_async8(void* smem, const void* gmem) {
    const unsigned s = (unsigned)__cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(s), "l"(gmem) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N) : "memory"); }

template <typename T, int NW>
__global__ void __launch_bounds__(NW * BLK) ch_rhs2_kernel(const GridDev* __restrict__ grids,
                                                           const Item* __restrict__ items, int parity) {
    __shared__ double hh[34 * 35];
    __shared__ double diag[33][33];
    constexpr int NT = NW * BLK, R = BLK / NW;   // rows per warp
    const int tid = threadIdx.x;
    const int j = tid & (BLK - 1), warp = tid / BLK;
    const volatile double* factors = g_rhs_factors;
    const double m_four = factors[1];
    const Arith<double> ar;
    const Item item = items[blockIdx.x];
    const GridDev gd = grids[item.grid];
    launch_wait();
    const int n = gd.n;
    const double* cur = parity ? gd.buf[1] : gd.buf[0];
    const double* old = parity ? gd.buf[0] : gd.buf[1];
    const int bpr = n / BLK;
    const int y0 = (item.block / bpr) * BLK, x0 = (item.block % bpr) * BLK;
    for (int e = tid; e < 34 * 34; e += NT) {
        const int r = e / 34, c = e - r * 34;
        int gy = y0 - 1 + r, gx = x0 - 1 + c;
        gy = gy < 0 ? gy + n : (gy >= n ? gy - n : gy);
        gx = gx < 0 ? gx + n : (gx >= n ? gx - n : gx);
        cp_async8(hh + r * 35 + c, gd.hbuf + (size_t)gy * n + gx);
    }
    cp_async_commit();
    const size_t at = (size_t)(y0 + warp) * n + x0 + j;
    double cv[R], ov[R];
#pragma unroll
    for (int r = 0; r < R; ++r) {
        cv[r] = cur[at + (size_t)(r * NW) * n];
        ov[r] = old[at + (size_t)(r * NW) * n];
    }
    const RhsValue<T> rhs(gd.tab);
    cp_async_wait<0>();
    __syncthreads();
    diagonal_sums<NT>(ar, hh, diag, tid);
    __syncthreads();
#pragma unroll
    for (int r = 0; r < R; ++r) {
        const int rr = warp + r * NW;
        const double lap = fma(m_four, hh[(rr + 1) * 35 + j + 1], ar.add(diag[rr][j + 1], diag[rr + 1][j]));
        const size_t q = at + (size_t)(r * NW) * n;
        if (in_bounds((long long)q, 0, (long long)n * n)) gd.tmp[q] = rhs(lap, ar.sub(cv[r], ov[r]));
    }
}

// ------------------------------------------------------------------------------------------------
// K2 / K3: the line solves
// ------------------------------------------------------------------------------------------------
// Each line is a circulant pentadiagonal system A x = r, A = 1 + sigma_lin D^4 (the two unknowns that the reference
// splits off, BatchHyper.cu:195-259, are its way of closing the same circulant). Its symbol is positive, so it
// factors as A = G P(z) P(1/z) with P(z) = 1 + p1 / z + p2 / z^2 causal and minimum phase (line_factor, below):
// constant coefficients, two multiply-adds per element and direction, no pivots and no tables, against five and
// a table row for the banded factors. The constant G is applied once, in the update.
//
// A line is solved by two chains that meet in its middle (one warp each, a lane per line):
//   - cut the ring between its last and first element and let the right-hand side be zero beyond both ends: on that
//     infinite line chain A runs u = r / P(z) from the left end to the middle, chain B the mirrored w = r / P(1/z)
//     from the right end. v = A^-1 r satisfies P(1/z) v = u left of the middle and P(z) v = w right of it, which
//     makes the four values of v around the middle a constant 4 x 4 system in the chains' last two values each
//     (TAB_MID); from there each chain runs back to its end;
//   - close the ring: the periodic solution is v summed over all its translates by n. To the right of the line v
//     decays as the homogeneous solutions of P, so the translates from the left add alpha1 f1(i) + alpha2 f2(i) with
//     (alpha1, alpha2) = (1 - M^n)^-1 (v[n-1], v[n-2]) (TAB_CLOSE; M the one-step matrix), and the mirrored sum at
//     the other end adds beta1 f1(n-1-i) + beta2 f2(n-1-i). f1 and f2 fall off; beyond TAB_REACH entries (2^-56 of
//     their peak) they are left out.
// The x sweep's closure is applied where the y sweep reads, the y sweep's in the update. Per point that is 8
// multiply-adds for the recurrences and 2 for each end within reach, against 10 and 4, and a line's dependent chain
// is half as long. The arithmetic is a function of n, lx, gamma and dt alone, so a grid's result does not depend
// on its batch.
//
// Short and very long lines are cut into two segments, four chains (line_cuts): each segment is
// solved as above, zero beyond its ends, and the closure of a segment's end sums the other segment's tail and, once
// around the ring, its own: (1 - M^n)^-1 applied to the neighbour's end values (TAB_CLOSE) and to its own carried
// through the neighbour, M to its length (TAB_CLOSE2). A segment is a CTA; the one that finishes last forms the amplitudes of both. The closure then reaches
// every point of most lines, up to two multiply-adds a sweep more, for chains of half the length.
//
// A warp's FP64 instruction holds its sub-partition's FP64 pipe for 64 cycles however few lanes it has, so with
// fewer chains than FP64 sub-partitions (4 per SM) a step takes the chain's instruction count: n / 2 elements
// of 4 instructions per sweep. Measured, us per step (before: banded factors, one warp per 32 lines, and the former
// right-hand side): one grid of 256^2 45 (159), 512^2 73 (298), 1024^2 231 (601), 2048^2 353 (1331); 96 grids of 64^2 ..
// 1024^2 1231 (1973).

// Chunks of kChunk elements of a warp's 32 lines move between the work field and a shared-memory ring of kStages
// stages by the tensor memory accelerator, one copy per chunk each way, issued by a copy warp per chain (two chain
// warps and two copy warps make a CTA): the recurrence has the issue slots to itself, and a chain alone on its
// sub-partition keeps the FP64 pipe busy. Measured, x sweep of one 512^2 grid (32 us of FP64 instructions): 44 us;
// the copies issued by the chain warp itself 48 us; its lanes copying with 8-byte cp.async and stores 63 us; with bulk
// copies of 128 bytes per lane 106 us (each occupies the copy engine for about 50 cycles). A
// chunk is solved in place in its stage and copied back from there. At the middle the last kStages chunks are
// still in the ring; the backward pass starts from them and they never make the round trip through the work field.
constexpr int kChunk = 16, kStages = 4;
using Forward = std::true_type;
using Backward = std::false_type;

__device__ __forceinline__ void pair_barrier() { asm volatile("bar.sync 1, 64;" ::: "memory"); }

__device__ __forceinline__ void bulk_load(void* smem, const void* gmem, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(smem)),
                 "l"(gmem), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}
__device__ __forceinline__ void tma_store_2d(const CUtensorMap* map, int x, int y, const void* smem) {
    asm volatile("cp.async.bulk.tensor.2d.global.shared::cta.bulk_group [%0, {%1, %2}], [%3];" ::"l"(
                     reinterpret_cast<uint64_t>(map)),
                 "r"(x), "r"(y), "r"(smem_u32(smem))
                 : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// this thread's copies out of shared memory have read their source / have completed
__device__ __forceinline__ void bulk_wait_read_all() { asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory"); }
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }

// The map lies in device memory that the host writes between launches: made visible to the copy engine.
__device__ __forceinline__ void acquire_map(const CUtensorMap* map) {
    asm volatile("fence.proxy.tensormap::generic.acquire.sys [%0], 128;" ::"l"(reinterpret_cast<uint64_t>(map))
                 : "memory");
}

// The value next to the chain's end and the one behind it, from the chains' ends (TAB_MID row 0 and 1).
__device__ __forceinline__ double mid_value(const double* q, double own1, double own2, double oth1, double oth2) {
    return fma(q[0], own1, fma(q[1], own2, fma(q[2], oth1, q[3] * oth2)));
}

// The ring of one chain: full[s] completes when a chunk has arrived in stage s, done[s] when it has been solved
// there and may be copied out. failed: a wait for a chunk has expired.
struct ChainBars {
    uint64_t full[kStages], done[kStages];
    unsigned failed;
};

__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.release.cta.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Waits on the stages' barriers in turn; after one has expired (stencil_tma.cuh) none waits any more, so the
// warps of a CTA run to their end and meet at its barriers whatever happened; the results are void then. The copy
// warp then starts no further copy and stays until those in flight have landed (bounded as well).
struct RingWait {
    long long limit;
    unsigned* failed;      // set at an expiry, or null
    unsigned parity = 0;   // per stage: the phase its next completion ends
    bool ok = true;
    __device__ __forceinline__ explicit RingWait(long long limit_, unsigned* failed_ = nullptr) : limit(limit_), failed(failed_) {}
    __device__ __forceinline__ void operator()(uint64_t* bars, int st) {
        if (ok && !mbar_wait(&bars[st], (parity >> st) & 1u, limit)) {
            ok = false;
            if (failed) *(volatile unsigned*)failed = 1u;
        }
        parity ^= 1u << st;
    }
    __device__ __forceinline__ void report() const {
        if (!ok) atomicOr(&g_custen_device_error, kErrMbarrierTimeout);
    }
};

// The chain is done with a chunk in stage st (by every lane).
__device__ __forceinline__ void chunk_solved(ChainBars& bars, int st, int lane) {
    __syncwarp();   // every lane's writes
    if (lane == 0) mbar_arrive(&bars.done[st]);
}

// The copy warp of a chain (one lane): load(c, stage, pass) starts the copy of chunk c on the stage's full
// barrier, store(c, stage) the copy back. A stage is refilled once its store has read it.
template <class Load, class Store>
__device__ __forceinline__ void run_copies(int nchunk, ChainBars& bars, Load load, Store store, long long limit = kWaitLimit) {
    RingWait done(limit);
    auto solved = [&](int st) {
        done(bars.done, st);
        return done.ok && *(const volatile unsigned*)&bars.failed == 0u;
    };
    for (int c = 0; c < kStages && c < nchunk; ++c) load(c, c, Forward{});
    unsigned last = 0;   // per stage: the phase that its last copy ends
    bool ok = true;
    for (int c = 0; c < nchunk - kStages; ++c) {
        const int st = c % kStages;
        if (!(ok = solved(st))) break;
        fence_proxy_async_smem();
        store(c, st);
        bulk_wait_read_all();
        load(c + kStages, st, Forward{});
        last ^= 1u << st;
    }
    bulk_wait_all();   // the backward pass reads the forward pass's chunks again
    for (int c = nchunk - 1; ok && c >= 0; --c) {
        const int st = c % kStages;
        if (!(ok = solved(st))) break;
        fence_proxy_async_smem();
        store(c, st);
        if (c >= kStages) {
            bulk_wait_read_all();
            load(c - kStages, st, Backward{});
            last ^= 1u << st;
        }
    }
    bulk_wait_all();
    if (!ok)
        for (int st = 0; st < kStages && st < nchunk; ++st) mbar_wait(&bars.full[st], (last >> st) & 1u, limit);
    done.report();
}

// The chain itself (a lane per line): solve(stage, a1, a2, pass) runs the recurrence over a chunk in place, from
// the last two values; v1, v2: the values at the chain's outer end.
template <class Solve>
__device__ __forceinline__ void run_chain(int nchunk, ChainBars& bars, double (*own)[BLK], double (*other)[BLK], int lane,
                                          const double* mid, double& v1, double& v2, Solve solve,
                                          long long limit = kWaitLimit) {
    RingWait full(limit, &bars.failed);
    auto solved = [&](int st) { chunk_solved(bars, st, lane); };
    double u1 = 0.0, u2 = 0.0;
    for (int c = 0; c < nchunk; ++c) {
        const int st = c % kStages;
        full(bars.full, st);
        solve(st, u1, u2, Forward{});
        if (c < nchunk - kStages) solved(st);
    }
    __syncwarp();   // the y sweep's exchange lies where other lanes may still read the first stage's amplitudes
    own[0][lane] = u1;
    own[1][lane] = u2;
    pair_barrier();
    const double o1 = other[0][lane], o2 = other[1][lane];
    v1 = mid_value(mid, u1, u2, o1, o2);
    v2 = mid_value(mid + 4, u1, u2, o1, o2);
    for (int c = nchunk - 1; c >= 0; --c) {
        const int st = c % kStages;
        if (c < nchunk - kStages) full(bars.full, st);
        solve(st, v1, v2, Backward{});
        solved(st);
    }
    full.report();
}

// The recurrence over kChunk values in registers, w[0] first: v = w + np1 v1 + np2 v2.
__device__ __forceinline__ void recur(double (&w)[kChunk], double np1, double np2, double& v1, double& v2) {
#pragma unroll
    for (int k = 0; k < kChunk; ++k) {
        w[k] = fma(np1, v1, fma(np2, v2, w[k]));
        v2 = v1;
        v1 = w[k];
    }
}

// x sweep: DIR = 1 is chain A (columns upwards), -1 chain B. A stage holds 32 rows of 128 bytes in the 128-byte
// swizzle (the 16-byte unit u of row r lies at u ^ (r & 7)), in which a lane per row reads and writes 16 bytes at a
// time without bank conflicts.
struct Segment {
    int block, seg, lo, len;   // line block, segment of the line, its first element and length
    __device__ __forceinline__ Segment(const GridDev& gd, const Item& item)
        : block(gd.cuts == 2 ? item.block >> 1 : item.block), seg(gd.cuts == 2 ? item.block & 1 : 0),
          lo(seg ? first_segment(gd.n, gd.cuts) : 0),
          len(seg ? gd.n - first_segment(gd.n, gd.cuts) : first_segment(gd.n, gd.cuts)) {}
    __device__ __forceinline__ int chunks() const { return len / 2 / kChunk; }
};
template <int DIR>
__device__ __forceinline__ int chunk_origin(const Segment& sg, int c) {
    return DIR > 0 ? sg.lo + c * kChunk : sg.lo + sg.len - (c + 1) * kChunk;
}

// The closure amplitudes of a chain's end for its 32 lines: four per line at ends[4 (seg n + line)], alpha1, alpha2
// (from the left) by chain B, beta1, beta2 (from the right) by chain A. With one segment they follow from the
// chain's own end values; with two, the values themselves are left there and the CTA that arrives last replaces
// those of both segments.
template <int DIR>
__device__ __forceinline__ void close_segment(const GridDev& gd, const Segment& sg, double* ends, int line, int lane, double v1,
                                              double v2, unsigned int* arrived, int* flag) {
    const double* cl = gd.tab + TAB_CLOSE;
    const int n = gd.n;
    double2* mine = reinterpret_cast<double2*>(ends + 4 * (sg.seg * n + line) + (DIR > 0 ? 2 : 0));
    if (!in_bounds(4 * (sg.seg * n + line) + 3, 0, 4 * n * gd.cuts)) return;
    if (gd.cuts == 1) {
        *mine = make_double2(fma(cl[0], v1, cl[1] * v2), fma(cl[2], v1, cl[3] * v2));
        return;
    }
    *mine = make_double2(v1, v2);
    __threadfence();
    pair_barrier();
    if (DIR > 0 && lane == 0) *flag = (int)atomicAdd(arrived, 1u);
    pair_barrier();
    if (*flag == 0) return;   // the other segment's CTA has yet to arrive
    if (DIR > 0 && lane == 0) *arrived = 0;   // for the next sweep
    __threadfence();
    double2* theirs = reinterpret_cast<double2*>(ends + 4 * ((sg.seg ^ 1) * n + line) + (DIR > 0 ? 2 : 0));
    const double2 o = __ldcg(theirs);
    auto amplitude = [&](int seg, double a1, double a2, double b1, double b2) {   // neighbour a, itself b
        const double* c2 = gd.tab + TAB_CLOSE2 + 4 * seg;
        return make_double2(fma(cl[0], a1, fma(cl[1], a2, fma(c2[0], b1, c2[1] * b2))),
                            fma(cl[2], a1, fma(cl[3], a2, fma(c2[2], b1, c2[3] * b2))));
    };
    *mine = amplitude(sg.seg, o.x, o.y, v1, v2);
    *theirs = amplitude(sg.seg ^ 1, v1, v2, o.x, o.y);
}

template <int DIR>
__device__ __forceinline__ void xsweep_copies(const GridDev& gd, const CUtensorMap* map, const Segment& sg,
                                              double (*stage)[BLK][kChunk], ChainBars& bars) {
    const int n = gd.n, block = sg.block;
    auto load = [&](int c, int st, auto) {
        mbar_arrive_expect_tx(&bars.full[st], BLK * kChunk * sizeof(double));
        tma_load_2d(&stage[st][0][0], map, chunk_origin<DIR>(sg, c), block * BLK, &bars.full[st]);
    };
    auto store = [&](int c, int st) {
        const int x = chunk_origin<DIR>(sg, c);
        if (!in_bounds(x, 0, n - kChunk + 1) || !in_bounds(block * BLK, 0, n - BLK + 1)) return;
        tma_store_2d(map, x, block * BLK, &stage[st][0][0]);
        bulk_commit();
    };
    run_copies(sg.chunks(), bars, load, store);
}

template <int DIR>
__device__ __forceinline__ void xsweep_chain(const GridDev& gd, const Segment& sg, int lane, double (*stage)[BLK][kChunk],
                                             ChainBars& bars, double (*own)[BLK], double (*other)[BLK],
                                             unsigned int* arrived, int* flag) {
    const double np1 = gd.tab[TAB_NP1], np2 = gd.tab[TAB_NP2];
    const int swz = lane & 7;
    auto solve = [&](int st, double& a1, double& a2, auto forward) {
        double2* p = reinterpret_cast<double2*>(&stage[st][lane][0]);
        constexpr bool up = (DIR > 0) == decltype(forward)::value;
        double w[kChunk];
#pragma unroll
        for (int k = 0; k < kChunk / 2; ++k) {
            const double2 q = p[(up ? k : kChunk / 2 - 1 - k) ^ swz];
            w[2 * k] = up ? q.x : q.y;
            w[2 * k + 1] = up ? q.y : q.x;
        }
        recur(w, np1, np2, a1, a2);
#pragma unroll
        for (int k = 0; k < kChunk / 2; ++k)
            p[(up ? k : kChunk / 2 - 1 - k) ^ swz] =
                up ? make_double2(w[2 * k], w[2 * k + 1]) : make_double2(w[2 * k + 1], w[2 * k]);
    };
    double v1, v2;
    run_chain(sg.chunks(), bars, own, other, lane, gd.tab + TAB_MID, v1, v2, solve);
    close_segment<DIR>(gd, sg, gd.ends, sg.block * BLK + lane, lane, v1, v2, arrived, flag);
}

__device__ __forceinline__ void init_ring(ChainBars (&bars)[2]) {
    if (threadIdx.x == 0) {
        for (int k = 0; k < 2; ++k)
            for (int st = 0; st < kStages; ++st) {
                mbar_init(&bars[k].full[st], 1);
                mbar_init(&bars[k].done[st], 1);
                bars[k].failed = 0u;
            }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}

// The ring's base, aligned inside its slack (x: 1 KB for the 128-byte swizzle; y: 128 bytes; as in stencil_tma.cuh, through an opaque
// value, since the compiler may not assume more than the declared alignment).
template <uint32_t kRingAlign>
__device__ __forceinline__ double* ring_base(unsigned char* raw) {
    uint32_t addr = smem_u32(raw);
    asm volatile("" : "+r"(addr));
    return reinterpret_cast<double*>(raw + ((kRingAlign - (addr & (kRingAlign - 1))) & (kRingAlign - 1)));
}

constexpr int kStageWords = BLK * kChunk;
constexpr size_t kRingBytes = 2 * kStages * kStageWords * sizeof(double);
constexpr size_t kXSweepBytes = kRingBytes + 1024, kYSweepBytes = kRingBytes + 128;   // dynamic shared memory

constexpr int kSweepThreads = 4 * BLK;   // warps: chain A, chain B, the copies of A, the copies of B

__global__ void __launch_bounds__(kSweepThreads) ch_xsweep_kernel(const GridDev* __restrict__ grids,
                                                                  const Item* __restrict__ items,
                                                                  const CUtensorMap* maps, unsigned int* arrived) {
    extern __shared__ __align__(16) unsigned char sweep_smem[];
    __shared__ double ex[2][2][BLK];
    __shared__ int flag;
    __shared__ __align__(8) ChainBars bars[2];
    init_ring(bars);
    const int lane = threadIdx.x & (BLK - 1), warp = threadIdx.x / BLK;
    const Item item = items[blockIdx.x];
    const GridDev gd = grids[item.grid];
    const CUtensorMap* map = maps + 2 * item.grid;
    auto* stage = reinterpret_cast<double(*)[BLK][kChunk]>(ring_base<1024>(sweep_smem));
    launch_wait();
    const Segment sg(gd, item);
    arrived += blockIdx.x - sg.seg;   // of the line block
    if (warp == 0) xsweep_chain<1>(gd, sg, lane, stage, bars[0], ex[0], ex[1], arrived, &flag);
    else if (warp == 1) xsweep_chain<-1>(gd, sg, lane, stage + kStages, bars[1], ex[1], ex[0], arrived, &flag);
    else if (lane == 0) {
        acquire_map(map);
        if (warp == 2) xsweep_copies<1>(gd, map, sg, stage, bars[0]);
        else xsweep_copies<-1>(gd, map, sg, stage + kStages, bars[1]);
    }
}

// y sweep: DIR = 1 is chain A (rows upwards). CLOSE: the x sweep's closure is added to the right-hand side as a
// chunk is read, in the columns within reach of either end, by the rows' amplitudes (copied with the chunk).
// Without it ch_xclose_kernel has added it, with the same operations.
__device__ __forceinline__ int tab_int(const GridDev& gd, int k) { return (int)__double_as_longlong(gd.tab[k]); }
__device__ __forceinline__ int reach_of(const GridDev& gd) { return tab_int(gd, TAB_REACH); }

// The closure of one end over N values, or of none: branches around whole loops, since the compiler turns a
// condition at each value into both ends' multiply-adds and selections.
template <int N, class Amp>
__device__ __forceinline__ void close_end(bool within, double (&v)[N], double f1, double f2, Amp amp) {
    if (within) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const double2 a = amp(k);
            v[k] = fma(f1, a.x, fma(f2, a.y, v[k]));
        }
    }
}

// Where the 32 elements from i0 lie in their segment of a line, and whether within reach of either end.
struct CloseEnds {
    int seg, at, len;   // segment, position in it, its length
    bool left, right;
    __device__ __forceinline__ CloseEnds(const GridDev& gd, int i0) {
        const int reach = reach_of(gd);
        const int first = first_segment(gd.n, gd.cuts);
        seg = i0 >= first;
        at = seg ? i0 - first : i0;
        len = seg ? gd.n - first : first;
        left = at < reach;
        right = at + BLK > len - reach;
    }
};

template <int DIR, bool CLOSE>
__device__ __forceinline__ void ysweep_copies(const GridDev& gd, const CUtensorMap* map, const Segment& sg,
                                              double (*stage)[kChunk][BLK], double (*amp)[kChunk][4], ChainBars& bars) {
    const int n = gd.n, block = sg.block;
    const CloseEnds ends(gd, block * BLK);
    auto load = [&](int c, int st, auto forward) {
        const int y = chunk_origin<DIR>(sg, c);
        const bool amps = CLOSE && decltype(forward)::value && (ends.left || ends.right);
        mbar_arrive_expect_tx(&bars.full[st], kChunk * BLK * sizeof(double) + (amps ? kChunk * 4 * sizeof(double) : 0));
        tma_load_2d(&stage[st][0][0], map, block * BLK, y, &bars.full[st]);
        if (amps) bulk_load(&amp[st][0][0], gd.ends + 4 * (ends.seg * n + y), kChunk * 4 * sizeof(double), &bars.full[st]);
    };
    auto store = [&](int c, int st) {
        const int y = chunk_origin<DIR>(sg, c);
        if (!in_bounds(y, 0, n - kChunk + 1) || !in_bounds(block * BLK, 0, n - BLK + 1)) return;
        tma_store_2d(map, block * BLK, y, &stage[st][0][0]);
        bulk_commit();
    };
    run_copies(sg.chunks(), bars, load, store);
}

template <int DIR, bool CLOSE>
__device__ __forceinline__ void ysweep_chain(const GridDev& gd, const Segment& sg, int lane, double (*stage)[kChunk][BLK],
                                             double (*amp)[kChunk][4], ChainBars& bars, double (*own)[BLK],
                                             double (*other)[BLK], unsigned int* arrived, int* flag) {
    const int n = gd.n, block = sg.block;
    const double np1 = gd.tab[TAB_NP1], np2 = gd.tab[TAB_NP2];
    const int x = block * BLK + lane;
    double l1 = 0.0, l2 = 0.0, r1 = 0.0, r2 = 0.0;
    const CloseEnds in(gd, block * BLK);
    const bool left = in.left, right = in.right;   // uniform over the warp
    if (CLOSE) {
        const double *f1 = gd.tab + kTabParams, *f2 = f1 + n;
        const int i = in.at + lane, j = in.len - 1 - i;
        l1 = f1[i]; l2 = f2[i]; r1 = f1[j]; r2 = f2[j];
    }
    auto solve = [&](int st, double& a1, double& a2, auto forward) {
        constexpr bool up = (DIR > 0) == decltype(forward)::value;
        double w[kChunk];
#pragma unroll
        for (int k = 0; k < kChunk; ++k) w[k] = stage[st][up ? k : kChunk - 1 - k][lane];
        if (CLOSE && decltype(forward)::value) {
            auto e = [&](int k) { return reinterpret_cast<const double2*>(amp[st][up ? k : kChunk - 1 - k]); };
            close_end(left, w, l1, l2, [&](int k) { return e(k)[0]; });
            close_end(right, w, r1, r2, [&](int k) { return e(k)[1]; });
        }
        recur(w, np1, np2, a1, a2);
#pragma unroll
        for (int k = 0; k < kChunk; ++k) stage[st][up ? k : kChunk - 1 - k][lane] = w[k];
    };
    double v1, v2;
    run_chain(sg.chunks(), bars, own, other, lane, gd.tab + TAB_MID, v1, v2, solve);
    close_segment<DIR>(gd, sg, gd.ends + 4 * n * gd.cuts, x, lane, v1, v2, arrived, flag);
}

template <bool CLOSE>
__global__ void __launch_bounds__(kSweepThreads) ch_ysweep_kernel(const GridDev* __restrict__ grids,
                                                                  const Item* __restrict__ items,
                                                                  const CUtensorMap* maps, unsigned int* arrived) {
    extern __shared__ __align__(16) unsigned char sweep_smem[];
    __shared__ int flag;
    // A chain leaves its end values for the other in its own amplitude area, which the backward pass does not use:
    // 37 KB per CTA, so six fit an SM.
    __shared__ __align__(16) double amp[CLOSE ? 2 * kStages : 4][kChunk][4];
    __shared__ __align__(8) ChainBars bars[2];
    init_ring(bars);
    const int lane = threadIdx.x & (BLK - 1), warp = threadIdx.x / BLK;
    const Item item = items[blockIdx.x];
    const GridDev gd = grids[item.grid];
    const CUtensorMap* map = maps + 2 * item.grid + 1;
    auto* stage = reinterpret_cast<double(*)[kChunk][BLK]>(ring_base<128>(sweep_smem));
    launch_wait();
    auto* amp_b = amp + (CLOSE ? kStages : 2);
    auto *ex_a = reinterpret_cast<double(*)[BLK]>(amp), *ex_b = reinterpret_cast<double(*)[BLK]>(amp_b);
    const Segment sg(gd, item);
    arrived += blockIdx.x - sg.seg;
    if (warp == 0) ysweep_chain<1, CLOSE>(gd, sg, lane, stage, amp, bars[0], ex_a, ex_b, arrived, &flag);
    else if (warp == 1)
        ysweep_chain<-1, CLOSE>(gd, sg, lane, stage + kStages, amp_b, bars[1], ex_b, ex_a, arrived, &flag);
    else if (lane == 0) {
        acquire_map(map);
        if (warp == 2) ysweep_copies<1, CLOSE>(gd, map, sg, stage, amp, bars[0]);
        else ysweep_copies<-1, CLOSE>(gd, map, sg, stage + kStages, amp_b, bars[1]);
    }
}

// The x sweep's closure as an element-wise kernel over the 32 x 32 blocks, for batches with few chains (it spreads
// over every SM, where in the y sweep it would lengthen the chains).
__global__ void __launch_bounds__(256, 6) ch_xclose_kernel(const GridDev* __restrict__ grids,
                                                        const Item* __restrict__ items) {
    const Item item = items[blockIdx.x];
    const GridDev gd = grids[item.grid];
    launch_wait();
    if (gd.general) return;
    const int n = gd.n;
    const int bpr = n / BLK;
    const int y0 = (item.block / bpr) * BLK, x0 = (item.block % bpr) * BLK;
    const CloseEnds in(gd, x0);
    const bool left = in.left, right = in.right;
    if (!left && !right) return;
    const int lane = threadIdx.x & (BLK - 1), x = x0 + lane, i = in.at + lane, j = in.len - 1 - i;
    const double *f1 = gd.tab + kTabParams, *f2 = f1 + n;
    const double l1 = f1[i], l2 = f2[i], r1 = f1[j], r2 = f2[j];
    const int r0 = threadIdx.x / BLK;
    double v[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) v[k] = gd.tmp[(size_t)(y0 + r0 + 8 * k) * n + x];
    auto e = [&](int k) { return reinterpret_cast<const double2*>(gd.ends + 4 * (in.seg * n + y0 + r0 + 8 * k)); };
    close_end(left, v, l1, l2, [&](int k) { return e(k)[0]; });
    close_end(right, v, r1, r2, [&](int k) { return e(k)[1]; });
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const long long q = (long long)(y0 + r0 + 8 * k) * n + x;
        if (in_bounds(q, 0, (long long)n * n)) gd.tmp[q] = v[k];
    }
}

// K4: cNew = cBar + delta written over cOld (cuPentCahnADI.cu:58-69, 89-100), one 32 x 32 block per CTA: delta is
// kappa times the y solution with its closure, for the rows within reach of either end.
__global__ void __launch_bounds__(256, 4) ch_update_kernel(const GridDev* __restrict__ grids,
                                                        const Item* __restrict__ items, int parity) {
    const Item item = items[blockIdx.x];
    const GridDev gd = grids[item.grid];
    launch_wait();
    if (gd.general) return;   // ch_update_general_kernel does it
    const int n = gd.n;
    const int bpr = n / BLK;
    const int y0 = (item.block / bpr) * BLK, x0 = (item.block % bpr) * BLK;
    const int x = x0 + (threadIdx.x & (BLK - 1));
    const CloseEnds in(gd, y0);
    const double *f1 = gd.tab + kTabParams, *f2 = f1 + n;
    const double two = ((const volatile double*)g_rhs_factors)[0];
    const double kappa = gd.tab[TAB_KAPPA];
    const double* cur = parity ? gd.buf[1] : gd.buf[0];
    double* old = parity ? gd.buf[0] : gd.buf[1];
    const int r0 = threadIdx.x / BLK;
    double v[4], cv[4], ov[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const size_t q = (size_t)(y0 + r0 + 8 * k) * n + x;
        v[k] = gd.tmp[q];
        cv[k] = cur[q];
        ov[k] = old[q];
    }
    const double2* e = reinterpret_cast<const double2*>(gd.ends + 4 * n * gd.cuts + 4 * (in.seg * n + x));
    if (in.left) {
        __syncwarp();   // keeps the branch: predicated-off multiply-adds take the FP64 pipe (4.9 -> 3.9 per point and 219 -> 169 us at
        // 24 grids of 1024^2)
        const double2 a = e[0];
#pragma unroll
        for (int k = 0; k < 4; ++k) v[k] = fma(f1[in.at + r0 + 8 * k], a.x, fma(f2[in.at + r0 + 8 * k], a.y, v[k]));
    }
    if (in.right) {
        __syncwarp();
        const double2 a = e[1];
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            const int i = in.len - 1 - (in.at + r0 + 8 * k);
            v[k] = fma(f1[i], a.x, fma(f2[i], a.y, v[k]));
        }
    }
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const long long q = (long long)(y0 + r0 + 8 * k) * n + x;
        if (in_bounds(q, 0, (long long)n * n)) old[q] = fma(kappa, v[k], fma(two, cv[k], -ov[k]));
    }
}

// ------------------------------------------------------------------------------------------------
// General sweeps: the line solved as the (n-2) x (n-2) banded block with its pre-computed factors plus the 2 x 2
// Schur complement on the last two unknowns (cuPentBatch.cu:35-198, BatchHyper.cu:195-259, 421-514). For
//   - a negative sigma_lin (a negative gamma or time step): the symbol may vanish and has no real causal factor;
//   - the precision variant: it rounds the fields to FP32 every step, which turns any other last bit of a solve into
//     a difference of FP32 rounding size (2e-7 after 40 steps), so its results are tied to these operations.
// One chain per 32 lines (the whole line), with the ring and the copy warp of the factored sweeps; the table entries
// of a chunk arrive with it, and in the part of the line where the factors have converged to the last bit they stay
// in registers. 24 grids of 96^2 .. 384^2, FP32 stencils: 204 us per step (263 with cp.async double buffers and the
// table entries read per chunk into registers); 96 grids of 64^2 .. 1024^2: 1294 (1571; 1378 with the
// sweeps alone).
// ------------------------------------------------------------------------------------------------
struct BandChunk {
    double ds[kChunk], dl[kChunk], rd[kChunk], du[kChunk], dw[kChunk];
};
constexpr uint32_t kBandBytes = sizeof(BandChunk);

// The table's arrays (ch_internal.cuh) and the chunks in which they are constant.
struct BandTable {
    const double* t;
    int m, const_lo, const_hi;
    __device__ __forceinline__ explicit BandTable(const GridDev& gd)
        : t(gd.tab + kTabParams), m(gd.n - 2), const_lo(tab_int(gd, TAB_BAND_LO)), const_hi(tab_int(gd, TAB_BAND_HI)) {}
    __device__ __forceinline__ void load(BandChunk& to, int c, uint64_t* bar) const {
        bulk_load(to.ds, t + c * kChunk, kChunk * sizeof(double), bar);
        bulk_load(to.dl, t + m + c * kChunk, kChunk * sizeof(double), bar);
        bulk_load(to.rd, t + 2 * m + c * kChunk, kChunk * sizeof(double), bar);
        bulk_load(to.du, t + 3 * m + c * kChunk, kChunk * sizeof(double), bar);
        bulk_load(to.dw, t + 4 * m + c * kChunk, kChunk * sizeof(double), bar);
    }
};

// The chain of 32 lines of n elements: get(stage, w, pass) and put(stage, w) move a chunk between its stage and
// registers, ascending. x2, x1: the last two unknowns.
template <class Get, class Put>
__device__ __forceinline__ void run_band(const GridDev& gd, const BandTable& bt, ChainBars& bars, const BandChunk* band,
                                         int lane, double& x2, double& x1, Get get, Put put) {
    const int nchunk = gd.n / kChunk;
    RingWait full(kWaitLimit, &bars.failed);
    auto solved = [&](int st) { chunk_solved(bars, st, lane); };
    const double* tc = bt.t + min(bt.const_lo, nchunk - 1) * kChunk;
    const double cs = tc[0], cl = tc[bt.m], cr = tc[2 * bt.m], cu = tc[3 * bt.m], cw = tc[4 * bt.m];
    double b1 = 0.0, b2 = 0.0, r2 = 0.0, r1 = 0.0;
    for (int c = 0; c < nchunk; ++c) {   // forward elimination
        const int st = c % kStages;
        full(bars.full, st);
        double w[kChunk];
        get(st, w, Forward{});
        if (c >= bt.const_lo && c < bt.const_hi) {
#pragma unroll
            for (int k = 0; k < kChunk; ++k) {
                double t = fma(-cs, b2, w[k]);
                t = fma(-cl, b1, t);
                t *= cr;
                b2 = b1;
                b1 = t;
                w[k] = t;
            }
        } else {
            const BandChunk& q = band[st];
            const bool last = c == nchunk - 1;
#pragma unroll
            for (int k = 0; k < kChunk; ++k) {
                if (k >= kChunk - 2 && last) break;   // the two unknowns outside the band
                double t = fma(-q.ds[k], b2, w[k]);
                t = fma(-q.dl[k], b1, t);
                t *= q.rd[k];
                b2 = b1;
                b1 = t;
                w[k] = t;
            }
            if (last) {
                r2 = w[kChunk - 2];
                r1 = w[kChunk - 1];
            }
        }
        put(st, w);
        if (c < nchunk - kStages) solved(st);
    }
    double f1 = 0.0, f2 = 0.0, y0v = 0.0, y1v = 0.0, ym2 = 0.0, ym1 = 0.0;
    for (int c = nchunk - 1; c >= 0; --c) {   // backward substitution
        const int st = c % kStages;
        if (c < nchunk - kStages) full(bars.full, st);
        double w[kChunk];
        get(st, w, Backward{});
        if (c >= bt.const_lo && c < bt.const_hi) {
#pragma unroll
            for (int k = kChunk - 1; k >= 0; --k) {
                double y = fma(-cu, f1, w[k]);
                y = fma(-cw, f2, y);
                f2 = f1;
                f1 = y;
                w[k] = y;
            }
        } else {
            const BandChunk& q = band[st];
            const bool last = c == nchunk - 1;
#pragma unroll
            for (int k = kChunk - 1; k >= 0; --k) {
                if (k >= kChunk - 2 && last) continue;
                double y = fma(-q.du[k], f1, w[k]);
                y = fma(-q.dw[k], f2, y);
                f2 = f1;
                f1 = y;
                w[k] = y;
            }
            if (last) {
                ym2 = w[kChunk - 4];
                ym1 = w[kChunk - 3];
            }
        }
        if (c == 0) {
            y0v = w[0];
            y1v = w[1];
        }
        put(st, w);
        solved(st);
    }
    // the last two unknowns through the 2 x 2 Schur complement (BatchHyper.cu:195-227)
    const double* om = bt.t + 7 * bt.m;
    const double a = om[4], b = om[5], d = om[6], e = om[7];
    const double nx2 = r2 - (e * y0v + a * ym2 + b * ym1);
    const double nx1 = r1 - (d * y0v + e * y1v + a * ym1);
    x2 = om[0] * nx2 + om[1] * nx1;
    x1 = om[2] * nx2 + om[3] * nx1;
    full.report();
}

constexpr int kBandThreads = 2 * BLK;   // warps: the chain, its copies
constexpr size_t kBandRingBytes = kStages * kStageWords * sizeof(double);
constexpr size_t kXBandBytes = kBandRingBytes + 1024, kYBandBytes = kBandRingBytes + 128;   // dynamic shared memory

__device__ __forceinline__ void init_bars(ChainBars& bars) {
    if (threadIdx.x == 0) {
        for (int st = 0; st < kStages; ++st) {
            mbar_init(&bars.full[st], 1);
            mbar_init(&bars.done[st], 1);
            bars.failed = 0u;
        }
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
}

// x sweep (lane = row); leaves the banded solution and the two border values of every row, which the ends buffer
// keeps as well.
__global__ void __launch_bounds__(kBandThreads) ch_xband_kernel(const GridDev* __restrict__ grids,
                                                                const Item* __restrict__ items, const CUtensorMap* maps) {
    extern __shared__ __align__(16) unsigned char sweep_smem[];
    __shared__ __align__(16) BandChunk band[kStages];
    __shared__ __align__(8) ChainBars bars;
    init_bars(bars);
    const int lane = threadIdx.x & (BLK - 1);
    const Item item = items[blockIdx.x];
    const GridDev gd = grids[item.grid];
    const CUtensorMap* map = maps + 2 * item.grid;
    const BandTable bt(gd);
    const int n = gd.n, y0 = item.block * BLK;
    auto* stage = reinterpret_cast<double(*)[BLK][kChunk]>(ring_base<1024>(sweep_smem));
    launch_wait();
    if (threadIdx.x >= BLK) {
        if (lane == 0) {
            acquire_map(map);
            auto load = [&](int c, int st, auto) {
                mbar_arrive_expect_tx(&bars.full[st], BLK * kChunk * sizeof(double) + kBandBytes);
                tma_load_2d(&stage[st][0][0], map, c * kChunk, y0, &bars.full[st]);
                bt.load(band[st], c, &bars.full[st]);
            };
            auto store = [&](int c, int st) {
                if (!in_bounds(c * kChunk, 0, n - kChunk + 1) || !in_bounds(y0, 0, n - BLK + 1)) return;
                tma_store_2d(map, c * kChunk, y0, &stage[st][0][0]);
                bulk_commit();
            };
            run_copies(n / kChunk, bars, load, store);
            asm volatile("fence.proxy.async;" ::: "memory");   // the chain's stores below follow the copies'
        }
        __syncwarp();
        pair_barrier();
        return;
    }
    const int swz = lane & 7;
    auto get = [&](int st, double (&w)[kChunk], auto) {
        const double2* p = reinterpret_cast<const double2*>(&stage[st][lane][0]);
#pragma unroll
        for (int k = 0; k < kChunk / 2; ++k) {
            const double2 q = p[k ^ swz];
            w[2 * k] = q.x;
            w[2 * k + 1] = q.y;
        }
    };
    auto put = [&](int st, const double (&w)[kChunk]) {
        double2* p = reinterpret_cast<double2*>(&stage[st][lane][0]);
#pragma unroll
        for (int k = 0; k < kChunk / 2; ++k) p[k ^ swz] = make_double2(w[2 * k], w[2 * k + 1]);
    };
    double x2, x1;
    run_band(gd, bt, bars, band, lane, x2, x1, get, put);
    pair_barrier();   // the last chunk has been copied out with the border values' right-hand sides
    const int y = y0 + lane;
    double* row = gd.tmp + (size_t)y * n;
    if (in_bounds(2 * y + 1, 0, 2 * n)) {
        row[n - 2] = x2;
        row[n - 1] = x1;
        gd.ends[2 * y] = x2;
        gd.ends[2 * y + 1] = x1;
    }
}

// y sweep (lane = column); leaves the banded solution and, at ends + 2 n, the two border values of every column.
// CLOSE: with the x sweep's rank-2 correction of the columns x < n - 2 as rows are read (BatchHyper.cu:233-259), by
// the rows' border values, copied with the chunk; without it ch_xcorr_general_kernel has applied it.
template <bool CLOSE>
__global__ void __launch_bounds__(kBandThreads) ch_yband_kernel(const GridDev* __restrict__ grids,
                                                                const Item* __restrict__ items, const CUtensorMap* maps) {
    extern __shared__ __align__(16) unsigned char sweep_smem[];
    __shared__ __align__(16) BandChunk band[kStages];
    __shared__ __align__(16) double amp[CLOSE ? kStages : 1][kChunk][2];
    __shared__ __align__(8) ChainBars bars;
    init_bars(bars);
    const int lane = threadIdx.x & (BLK - 1);
    const Item item = items[blockIdx.x];
    const GridDev gd = grids[item.grid];
    const CUtensorMap* map = maps + 2 * item.grid + 1;
    const BandTable bt(gd);
    const int n = gd.n, x0 = item.block * BLK, x = x0 + lane;
    auto* stage = reinterpret_cast<double(*)[kChunk][BLK]>(ring_base<128>(sweep_smem));
    launch_wait();
    if (threadIdx.x >= BLK) {
        if (lane == 0) {
            acquire_map(map);
            auto load = [&](int c, int st, auto forward) {
                const uint32_t amps = CLOSE && decltype(forward)::value ? 2 * kChunk * sizeof(double) : 0;
                mbar_arrive_expect_tx(&bars.full[st], BLK * kChunk * sizeof(double) + kBandBytes + amps);
                tma_load_2d(&stage[st][0][0], map, x0, c * kChunk, &bars.full[st]);
                bt.load(band[st], c, &bars.full[st]);
                if (amps) bulk_load(&amp[st][0][0], gd.ends + 2 * c * kChunk, amps, &bars.full[st]);
            };
            auto store = [&](int c, int st) {
                if (!in_bounds(c * kChunk, 0, n - kChunk + 1) || !in_bounds(x0, 0, n - BLK + 1)) return;
                tma_store_2d(map, x0, c * kChunk, &stage[st][0][0]);
                bulk_commit();
            };
            run_copies(n / kChunk, bars, load, store);
        }
        return;
    }
    const bool corr = CLOSE && x < bt.m;
    const double cx1 = corr ? bt.t[5 * bt.m + x] : 0.0, cx2 = corr ? bt.t[6 * bt.m + x] : 0.0;
    auto get = [&](int st, double (&w)[kChunk], auto forward) {
#pragma unroll
        for (int k = 0; k < kChunk; ++k) w[k] = stage[st][k][lane];
        if (CLOSE && decltype(forward)::value) {
#pragma unroll
            for (int k = 0; k < kChunk; ++k) {
                const double2 e = *reinterpret_cast<const double2*>(amp[st][k]);
                const double v = fma(-cx1, e.x, fma(-cx2, e.y, w[k]));
                w[k] = corr ? v : w[k];
            }
        }
    };
    auto put = [&](int st, const double (&w)[kChunk]) {
#pragma unroll
        for (int k = 0; k < kChunk; ++k) stage[st][k][lane] = w[k];
    };
    double x2, x1;
    run_band(gd, bt, bars, band, lane, x2, x1, get, put);
    if (in_bounds(2 * n + 2 * x + 1, 0, 4 * n)) {
        gd.ends[2 * n + 2 * x] = x2;
        gd.ends[2 * n + 2 * x + 1] = x1;
    }
}

// One 32 x 32 block of a grid per CTA (the right-hand side's work list): t[y][x] -= inv1[x] x2(y) +
// inv2[x] x1(y) for the columns x < n - 2 of the block's rows, as fma(-inv1, x2, fma(-inv2, x1, t)).
__global__ void __launch_bounds__(256) ch_xcorr_general_kernel(const GridDev* __restrict__ grids,
                                                       const Item* __restrict__ items) {
    const Item item = items[blockIdx.x];
    const GridDev gd = grids[item.grid];
    launch_wait();
    if (!gd.general) return;
    const int n = gd.n, m = n - 2;
    const int bpr = n / BLK;
    const int y0 = (item.block / bpr) * BLK, x0 = (item.block % bpr) * BLK;
    const int x = x0 + (threadIdx.x & (BLK - 1));
    if (x >= m) return;
    const double cx1 = gd.tab[kTabParams + 5 * m + x], cx2 = gd.tab[kTabParams + 6 * m + x];
    for (int r = threadIdx.x / BLK; r < BLK; r += blockDim.x / BLK) {
        const int y = y0 + r;
        const long long q = (long long)y * n + x;
        if (!in_bounds(q, 0, (long long)n * n)) continue;
        gd.tmp[q] = fma(-cx1, gd.ends[2 * y], fma(-cx2, gd.ends[2 * y + 1], gd.tmp[q]));
    }
}

// One 32 x 32 block per CTA: cNew = cBar + delta written over cOld (cuPentCahnADI.cu:58-69, 89-100), delta
// from the banded y solution in the work field and the column's cyclic unknowns in GridDev::ends.
__global__ void __launch_bounds__(256) ch_update_general_kernel(const GridDev* __restrict__ grids,
                                                        const Item* __restrict__ items, int parity) {
    const Item item = items[blockIdx.x];
    const GridDev gd = grids[item.grid];
    launch_wait();
    if (!gd.general) return;
    const int n = gd.n, m = n - 2;
    const int bpr = n / BLK;
    const int y0 = (item.block / bpr) * BLK, x0 = (item.block % bpr) * BLK;
    const int x = x0 + (threadIdx.x & (BLK - 1));
    const double two = ((const volatile double*)g_rhs_factors)[0], unit = gd.tab[TAB_OUT];
    const double x2 = gd.ends[2 * n + 2 * x], x1 = gd.ends[2 * n + 2 * x + 1];
    const double* cur = parity ? gd.buf[1] : gd.buf[0];
    double* old = parity ? gd.buf[0] : gd.buf[1];
    for (int r = threadIdx.x / BLK; r < BLK; r += blockDim.x / BLK) {
        const int y = y0 + r;
        const long long q = (long long)y * n + x;
        double dlt;
        if (y < m) dlt = fma(-gd.tab[kTabParams + 5 * m + y], x2, fma(-gd.tab[kTabParams + 6 * m + y], x1, gd.tmp[q]));
        else dlt = (y == m) ? x2 : x1;
        const double cbar = fma(two, cur[q], -old[q]);
        if (in_bounds(q, 0, (long long)n * n)) old[q] = fma(unit, dlt, cbar);
    }
}

// Whether the element-wise parts of a sweep run as kernels of their own. With fewer chains than FP64 sub-partitions (4
// per SM) a sweep takes as long as one chain, so they are taken out of it; for lines in two segments, which the
// closure reaches everywhere, that is no slower with many chains either. Measured (us per step, x closure in the y
// sweep / apart): 24 grids of 96^2 .. 384^2 (672 chains) 123 / 116, of 512^2 (1536) 372 / 367; 8 grids of 1024^2 (512
// chains) 474 / 485, 24 (1536) 1201 / 1252; one of 1024^2 (64) 262 / 231.
static bool few_chains(int chains, int sms) { return chains < 4 * sms; }
static bool close_apart(const ChConfig& c, const ChWork& w, int sms) {
    return c.close == 2 || (c.close == 0 && (w.n_whole == 0 || 2 * (w.n_lines - w.n_general) < 3 * sms));
}

int ch_launches_per_step(const ChConfig& c, const ChWork& w, int sms) {
    return (c.warps2 ? 2 : 1) + (w.n_lines > w.n_general ? 3 + close_apart(c, w, sms) : 0) +
           (w.n_general > 0 ? 3 + few_chains(w.n_general, sms) : 0);
}

ChConfig ch_config(int index) {
    // {warps per right-hand-side CTA, of pass 2 (0: one pass), x closure}
    static const ChConfig tab[kChConfigs] = {
        {1, 0, 1}, {2, 0, 1}, {4, 0, 1}, {8, 0, 1}, {1, 1, 1}, {2, 2, 1}, {4, 4, 1}, {8, 8, 1}, {4, 2, 1}, {8, 4, 1}, {4, 8, 1},
        {1, 0, 2}, {4, 0, 0}, {2, 0, 2}, {4, 0, 2}, {8, 0, 2}, {2, 2, 2}, {4, 4, 2}, {8, 8, 2}, {8, 4, 2}, {8, 8, 0}, {4, 4, 0}};
    return tab[(index >= 0 && index < kChConfigs) ? index : 0];
}

void config_name(const ChConfig& c, char* name, size_t len) {
    char second[16] = "";
    if (c.warps2) snprintf(second, sizeof(second), "_2pass%d", c.warps2);
    snprintf(name, len, "rhs_warps%d%s%s", c.rhs_warps, second, c.close == 2 ? "_close_apart" : (c.close ? "_close_fused" : ""));
}

// The two passes of the right-hand side run one CTA per block. Pass 2 runs in FP64 in both variants: the precision
// variant's h buffer holds FP32 values, whose FP64 Laplacian is exact, so its mass is conserved to FP64 rounding (the
// one-pass kernel does the same).
template <typename F>
static cudaError_t with_warps(int warps, F f) {
    switch (warps) {
    case 1: return f(std::integral_constant<int, 1>{});
    case 2: return f(std::integral_constant<int, 2>{});
    case 4: return f(std::integral_constant<int, 4>{});
    default: return f(std::integral_constant<int, 8>{});
    }
}

template <typename T>
static cudaError_t launch_rhs(const ChConfig& c, const ChWork& w, int parity, int sms, cudaStream_t s) {
    if (!c.warps2)
        return with_warps(c.rhs_warps, [&](auto nw) {
            constexpr int NW = decltype(nw)::value;   // persistent over the work list
            return launch_overlapped(ch_rhs_kernel<T, NW>, std::max(1, std::min(w.n_blocks, sms * 32 / NW)), dim3(NW * BLK), 0, s,
                                     w.grids, w.blocks, w.n_blocks, parity);
        });
    const cudaError_t e = with_warps(c.rhs_warps, [&](auto nw) {
        constexpr int NW = decltype(nw)::value;
        return launch_overlapped(ch_h_kernel<T, NW>, w.n_blocks, dim3(NW * BLK), 0, s, w.grids, w.blocks, parity);
    });
    if (e != cudaSuccess) return e;
    return with_warps(c.warps2, [&](auto nw) {
        constexpr int NW = decltype(nw)::value;
        return launch_overlapped(ch_rhs2_kernel<T, NW>, w.n_blocks, dim3(NW * BLK), 0, s, w.grids, w.blocks, parity);
    });
}

cudaError_t launch_ch_step(const ChConfig& c, bool rhs_fp32, const ChWork& w, int parity, int sms, cudaStream_t s) {
    cudaError_t e = rhs_fp32 ? launch_rhs<float>(c, w, parity, sms, s) : launch_rhs<double>(c, w, parity, sms, s);
    if (e != cudaSuccess) return e;
    const int n = w.n_lines - w.n_general;
    const dim3 sweep(kSweepThreads), line(kBandThreads), block(256);
    auto then = [&](auto kern, int grid, dim3 threads, size_t smem, auto... args) {
        if (e == cudaSuccess) e = launch_overlapped(kern, grid, threads, smem, s, args...);
    };
    if (n > 0) {   // one CTA (two chains) per 32 lines, largest grids first
        then(ch_xsweep_kernel, n, sweep, kXSweepBytes, w.grids, w.lines, w.maps, w.arrived);
        if (close_apart(c, w, sms)) {
            then(ch_xclose_kernel, w.n_blocks, block, 0, w.grids, w.blocks);
            then(ch_ysweep_kernel<false>, n, sweep, kYSweepBytes, w.grids, w.lines, w.maps, w.arrived);
        } else {
            then(ch_ysweep_kernel<true>, n, sweep, kYSweepBytes, w.grids, w.lines, w.maps, w.arrived);
        }
        then(ch_update_kernel, w.n_blocks, block, 0, w.grids, w.blocks, parity);
    }
    if (w.n_general > 0) {
        const Item* lines = w.lines + n;
        then(ch_xband_kernel, w.n_general, line, kXBandBytes, w.grids, lines, w.maps);
        if (few_chains(w.n_general, sms)) {
            then(ch_xcorr_general_kernel, w.n_blocks, block, 0, w.grids, w.blocks);
            then(ch_yband_kernel<false>, w.n_general, line, kYBandBytes, w.grids, lines, w.maps);
        } else {
            then(ch_yband_kernel<true>, w.n_general, line, kYBandBytes, w.grids, lines, w.maps);
        }
        then(ch_update_general_kernel, w.n_blocks, block, 0, w.grids, w.blocks, parity);
    }
    return e;
}

// Self-test of the rings' failure path (custen_selftest_ring_expiry): two chains of `nchunk` chunks whose copies are plain
// arrivals, but the copy of chunk `lost` of chain A never arrives (a byte count that nothing delivers; no copy is in flight).
// counts: copies started and stored back by chain A, then by chain B.
__global__ void __launch_bounds__(kSweepThreads) ch_ring_expiry_kernel(long long limit, int nchunk, int lost, int* counts) {
    __shared__ double ex[2][2][BLK], mid[8];
    __shared__ __align__(8) ChainBars bars[2];
    if (threadIdx.x < 8) mid[threadIdx.x] = 0.0;
    init_ring(bars);
    const int lane = threadIdx.x & (BLK - 1), warp = threadIdx.x / BLK, chain = warp & 1;
    if (warp < 2) {
        double v1, v2;
        run_chain(nchunk, bars[chain], ex[chain], ex[chain ^ 1], lane, mid, v1, v2, [](int, double&, double&, auto) {}, limit);
    } else if (lane == 0) {
        auto load = [&](int c, int st, auto) {
            ++counts[2 * chain];
            mbar_arrive_expect_tx(&bars[chain].full[st], chain == 0 && c == lost ? 16 : 0);
        };
        auto store = [&](int, int) { ++counts[2 * chain + 1]; };
        run_copies(nchunk, bars[chain], load, store, limit);
    }
}

// Compensated (Neumaier) sum of one grid: every thread, then every CTA, then the CTA that finishes last over the
// CTAs' partial sums, combines with two-sums and carries the rounding errors apart. One CTA over the whole grid took
// 0.5 ms at 512^2, bound by its own six FP64 operations per value; a CTA per kMassSpan values, at most kMassBlocks, takes 28 us with its
// launch and read-back (547 before; 2048^2: 90 against 8449).
__device__ __forceinline__ void two_sum(double a, double b, double& s, double& err) {
    s = a + b;
    const double bb = s - a;
    err = (a - (s - bb)) + (b - bb);
}

__device__ __forceinline__ void mass_reduce(double (&ss)[256], double (&sc)[256]) {
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) {
            double t, e;
            two_sum(ss[threadIdx.x], ss[threadIdx.x + w], t, e);
            ss[threadIdx.x] = t;
            sc[threadIdx.x] += sc[threadIdx.x + w] + e;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256) ch_mass_kernel(const double* __restrict__ f, long long count, MassScratch* out) {
    __shared__ double ss[256], sc[256];
    __shared__ bool last;
    const int t = threadIdx.x;
    double s = 0.0, c = 0.0;
    for (long long k = blockIdx.x * 256ll + t; k < count; k += gridDim.x * 256ll) {
        double v, e;
        two_sum(s, f[k], v, e);
        s = v;
        c += e;
    }
    ss[t] = s;
    sc[t] = c;
    mass_reduce(ss, sc);
    if (t == 0) {
        out->part[blockIdx.x][0] = ss[0];
        out->part[blockIdx.x][1] = sc[0];
        __threadfence();
        last = atomicAdd(&out->arrived, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    ss[t] = t < gridDim.x ? __ldcg(&out->part[t][0]) : 0.0;
    sc[t] = t < gridDim.x ? __ldcg(&out->part[t][1]) : 0.0;
    mass_reduce(ss, sc);
    if (t == 0) {
        out->sum = ss[0] + sc[0];
        out->arrived = 0;   // for the next sum on this stream
    }
}

cudaError_t launch_ch_mass(const double* f, long long count, MassScratch* out, cudaStream_t s) {
    const long long want = (count + kMassSpan - 1) / kMassSpan;
    ch_mass_kernel<<<(int)std::min<long long>(want, kMassBlocks), 256, 0, s>>>(f, count, out);
    return cudaGetLastError();
}

// ------------------------------------------------------------------------------------------------
// Host side
// ------------------------------------------------------------------------------------------------

// sigma_lin of an n x n grid of side lx with D = 1, gamma, dt = dt_factor * dx (the reference defaults are gamma =
// 0.01, dt = 0.1 dx: cuPentCahnADI.cu:204-221).
static double sigma_lin(int n, double lx, double gamma, double dt_factor) {
    const double D = 1.0, dx = lx / n, dt = dt_factor * dx;
    return 2.0 * dt * D * gamma / (3.0 * (dx * dx * dx * dx));
}

// Two segments halve a chain, which is the time of a sweep when fewer chains than FP64 sub-partitions are resident,
// and add up to two multiply-adds per point and sweep (of 26 in a step) where the closure's reach is long against
// half a line, which is the time when more are. A grid's segments may depend on n alone, or its bits would depend on
// its batch, so each size takes the side that loses less: up to 512 points at most 1.5% in a full chip against up to
// 1.55x alone; 544 to 1024 one segment, since a full chip would lose 5.5%, at the price of 1.5x for a grid alone;
// above, where chains are longest and eight grids are needed to fill the chip, two (1.4x alone, 8% lost with eight).
// Measured with the persistent right-hand side (us per step, one / two segments): one grid of 256^2 64 / 46, 512^2
// 116 / 75, 24 grids of 96^2 .. 384^2 152 / 123, 96 grids of 64^2 .. 1024^2 with those up to 512^2 cut 1466 / 1488;
// one grid of 1024^2 242 / 161, but the 96 grids 1488 / 1570 with the 1024^2 ones cut as well; 2048^2: one grid 547 /
// 388, four 1092 / 1039, eight 1909 / 2054.
constexpr int kCutUpTo = 512, kCutAbove = 1024;
int line_cuts(int n, bool general) {
    return !general && (n <= kCutUpTo || n > kCutAbove) ? 2 : 1;
}

bool line_is_general(int n, double lx, double gamma, double dt_factor, bool rhs_fp32) {
    return rhs_fp32 || !(sigma_lin(n, lx, gamma, dt_factor) >= 0.0);
}

// Causal factor of the circulant line operator 1 + s D^4, s >= 0: its symbol 1 + s w^2, w = 2 - z - 1/z, vanishes at
// w = +-i / sqrt(s); P(z) = (1 - z1 / z)(1 - conj(z1) / z) with z1 the root inside the unit circle of z + 1/z = 2 - w.
static void line_factor(double s, double* p1, double* p2) {
    *p1 = *p2 = 0.0;
    if (s < 1e-36) return;   // P = 1 to double precision
    const long double a = 0.5L / sqrtl((long double)s);
    const std::complex<long double> t(1.0L, -a), r = std::sqrt(std::complex<long double>(-a * a, -2.0L * a));
    const std::complex<long double> big = std::norm(t + r) > std::norm(t - r) ? t + r : t - r;
    const std::complex<long double> z = 1.0L / big;
    *p1 = (double)(-2.0L * z.real());
    *p2 = (double)std::norm(z);
}

// -(p1 a + p2 b) of pairs of doubles a, b (their low parts to first order): the homogeneous solutions' recurrence, whose
// n steps in long double are software on the host of a GB300 (0.25 us each).
struct Pair {
    double hi, lo;
};
static Pair next_term(double p1, Pair a, double p2, Pair b) {
    const double u = -p1 * a.hi, eu = std::fma(-p1, a.hi, -u) - p1 * a.lo;
    const double v = -p2 * b.hi, ev = std::fma(-p2, b.hi, -v) - p2 * b.lo;
    const double s = u + v, bb = s - u, es = (u - (s - bb)) + (v - bb);   // two-sum
    const double lo = es + (eu + ev), hi = s + lo;
    return {hi, lo - (hi - s)};
}

// The factored sweeps' part of the table: parameters and homogeneous solutions (see K2 / K3).
static void fill_line_table(double* t, int n, double s) {
    const int cuts = line_cuts(n, false), len = first_segment(n, cuts), other = n - len;   // len >= other
    double p1d, p2d;
    line_factor(s, &p1d, &p2d);
    const long double p1 = p1d, p2 = p2d;
    t[TAB_NP1] = -p1d;
    t[TAB_NP2] = -p2d;
    const long double at1 = 1.0L + p1 + p2;   // P(1): G P(1)^2 = 1, the operator on constants
    t[TAB_KAPPA] = (double)(at1 * at1 * at1 * at1 * 2.0L / 3.0L);
    // the four values around the middle (X1, X2 | Y1, Y2) from the chains' ends (a1, a2 | b1, b2)
    long double m[4][8] = {{1, 0, p1, p2, 1, 0, 0, 0},
                           {p1, 1, p2, 0, 0, 1, 0, 0},
                           {p1, p2, 1, 0, 0, 0, 1, 0},
                           {p2, 0, p1, 1, 0, 0, 0, 1}};
    for (int c = 0; c < 4; ++c) {
        int piv = c;
        for (int r = c + 1; r < 4; ++r)
            if (fabsl(m[r][c]) > fabsl(m[piv][c])) piv = r;
        for (int k = 0; k < 8; ++k) std::swap(m[c][k], m[piv][k]);
        const long double inv = 1.0L / m[c][c];
        for (int k = 0; k < 8; ++k) m[c][k] *= inv;
        for (int r = 0; r < 4; ++r) {
            if (r == c) continue;
            const long double f = m[r][c];
            for (int k = 0; k < 8; ++k) m[r][k] -= f * m[c][k];
        }
    }
    for (int k = 0; k < 4; ++k) {
        t[TAB_MID + k] = (double)m[2][4 + k];
        t[TAB_MID + 4 + k] = (double)m[3][4 + k];
    }
    // f1, f2: P f = 0 from (f[-1], f[-2]) = (1, 0) and (0, 1)
    double *f1 = t + kTabParams, *f2 = f1 + n;
    Pair a1{1.0, 0.0}, a2{0.0, 0.0}, b1{0.0, 0.0}, b2{1.0, 0.0};
    double peak = 1.0;
    long double step[2][4] = {};   // per segment
    auto power = [&](long double* to) {   // M^i from the last two terms
        const Pair from[4] = {a1, b1, a2, b2};
        for (int k = 0; k < 4; ++k) to[k] = (long double)from[k].hi + from[k].lo;
    };
    for (int i = 0; i < n; ++i) {
        const Pair a = next_term(p1d, a1, p2d, a2), b = next_term(p1d, b1, p2d, b2);
        a2 = a1;
        a1 = a;
        b2 = b1;
        b1 = b;
        if (i >= len) continue;
        f1[i] = a.hi;
        f2[i] = b.hi;
        peak = std::max(peak, std::max(std::fabs(a.hi), std::fabs(b.hi)));
        for (int k = 0; k < 2; ++k)
            if (i == (k ? len : other) - 1) power(step[k]);   // M^len, M^other: the way through the other segment
    }
    int reach = len;
    while (reach > 0 && std::max(fabs(f1[reach - 1]), fabs(f2[reach - 1])) <= ldexp(peak, -56)) --reach;
    const long long reach_bits = reach;   // as bits: a conversion on the device would take the FP64 pipe
    memcpy(&t[TAB_REACH], &reach_bits, sizeof(reach_bits));
    // (1 - M^n)^-1, M^n = [f1[n-1] f2[n-1]; f1[n-2] f2[n-2]]
    long double mn[4];
    power(mn);
    const long double c00 = 1.0L - mn[0], c01 = -mn[1], c10 = -mn[2], c11 = 1.0L - mn[3], det = c00 * c11 - c01 * c10;
    const long double inv[4] = {c11 / det, -c01 / det, -c10 / det, c00 / det};
    for (int r = 0; r < 2; ++r)
        for (int c = 0; c < 2; ++c) {
            t[TAB_CLOSE + 2 * r + c] = (double)inv[2 * r + c];
            for (int k = 0; k < 2; ++k)
                t[TAB_CLOSE2 + 4 * k + 2 * r + c] = (double)(inv[2 * r] * step[k][c] + inv[2 * r + 1] * step[k][2 + c]);
        }
}

// Solver table for an n x n grid (layout in ch_internal.cuh), written into t (tab_size(n) doubles) with `work`
// (7 * (n - 2) doubles) as scratch.
static void fill_table(double* t, double* work, int n, double lx, double gamma, double dt_factor, bool general, bool rhs_fp32) {
    const int m = n - 2;
    const double D = 1.0, dx = lx / n, dt = dt_factor * dx;
    const double sl = sigma_lin(n, lx, gamma, dt_factor);
    for (int k = 0; k < tab_size(n); ++k) t[k] = 0.0;
    t[TAB_SLIN] = sl;
    t[TAB_SNL] = (dt / 3.0) * D * (2.0 / (dx * dx));
    t[TAB_RATIO] = t[TAB_SNL] != 0.0 ? sl / t[TAB_SNL] : 0.0;
    t[TAB_LAP] = 1.5 * t[TAB_SNL];
    t[TAB_OUT] = rhs_fp32 ? 1.0 : 2.0 / 3.0;
    if (!general) {
        fill_line_table(t, n, sl);
        return;
    }
    double* params = t;
    t += kTabParams;
    const double a = sl, b = -4 * sl, c = 1 + 6 * sl, d = -4 * sl, e = sl;
    double *ds = work, *dl = work + m, *dg = work + 2 * m, *du = work + 3 * m, *dw = work + 4 * m;
    double *inv1 = work + 5 * m, *inv2 = work + 6 * m;
    for (int i = 0; i < m; ++i) {
        ds[i] = (i > 1) ? a : 0.0;
        dl[i] = (i > 0) ? b : 0.0;
        dg[i] = c;
        du[i] = (i < m - 1) ? d : 0.0;
        dw[i] = (i < m - 2) ? e : 0.0;
    }
    // in-place factorisation of the banded block (cuPentBatch.cu:35-113)
    du[0] = du[0] / dg[0];
    dw[0] = dw[0] / dg[0];
    dg[1] = dg[1] - dl[1] * du[0];
    du[1] = (du[1] - dl[1] * dw[0]) / dg[1];
    dw[1] = dw[1] / dg[1];
    for (int i = 2; i < m; ++i) {
        dl[i] = dl[i] - ds[i] * du[i - 2];
        dg[i] = dg[i] - ds[i] * dw[i - 2] - dl[i] * du[i - 1];
        if (i < m - 2) dw[i] = dw[i] / dg[i];
        if (i < m - 1) du[i] = (du[i] - dl[i] * dw[i - 1]) / dg[i];
    }
    auto solve = [&](double* x) {
        x[0] = x[0] / dg[0];
        x[1] = (x[1] - dl[1] * x[0]) / dg[1];
        for (int i = 2; i < m; ++i) x[i] = (x[i] - ds[i] * x[i - 2] - dl[i] * x[i - 1]) / dg[i];
        x[m - 2] = x[m - 2] - du[m - 2] * x[m - 1];
        for (int i = m - 3; i >= 0; --i) x[i] = x[i] - du[i] * x[i + 1] - dw[i] * x[i + 2];
    };
    // border columns and omega (BatchHyper.cu:421-514)
    for (int i = 0; i < m; ++i) inv1[i] = inv2[i] = 0.0;
    inv1[0] = a; inv1[m - 2] = e; inv1[m - 1] = d;
    inv2[0] = b; inv2[1] = a; inv2[m - 1] = e;
    solve(inv1);
    solve(inv2);
    const double z11 = e * inv1[0] + a * inv1[m - 2] + b * inv1[m - 1];
    const double z12 = e * inv2[0] + a * inv2[m - 2] + b * inv2[m - 1];
    const double z21 = d * inv1[0] + e * inv1[1] + a * inv1[m - 1];
    const double z22 = d * inv2[0] + e * inv2[1] + a * inv2[m - 1];
    const double y11 = c - z11, y12 = d - z12, y21 = b - z21, y22 = c - z22;
    const double det = 1.0 / (y11 * y22 - y21 * y12);
    for (int i = 0; i < m; ++i) {
        t[i] = (i > 1) ? ds[i] : 0.0;
        t[m + i] = (i > 0) ? dl[i] : 0.0;
        t[2 * m + i] = 1.0 / dg[i];
        t[3 * m + i] = (i < m - 1) ? du[i] : 0.0;
        t[4 * m + i] = (i < m - 2) ? dw[i] : 0.0;
        t[5 * m + i] = inv1[i];
        t[6 * m + i] = inv2[i];
    }
    // the chunks, short of the last, whose entries are all those of their neighbours to the last bit
    const int nchunk = n / kChunk;
    int lo = nchunk - 1;
    auto same = [&](int i, int j) {
        for (int k = 0; k < 5; ++k)
            if (memcmp(&t[k * m + i], &t[k * m + j], sizeof(double)) != 0) return false;
        return true;
    };
    for (int i = (nchunk - 1) * kChunk - 1; i >= 0 && same(i, (nchunk - 1) * kChunk - 1); --i)
        if (i % kChunk == 0) lo = i / kChunk;
    const long long band[2] = {lo, nchunk - 1};
    memcpy(params + TAB_BAND_LO, &band[0], sizeof(double));
    memcpy(params + TAB_BAND_HI, &band[1], sizeof(double));
    double* om = &t[7 * m];
    om[0] = y22 * det;
    om[1] = -y12 * det;
    om[2] = -y21 * det;
    om[3] = y11 * det;
    om[4] = a; om[5] = b; om[6] = d; om[7] = e;
}

std::vector<double> build_table(int n, double lx, double gamma, double dt_factor, bool general, bool rhs_fp32) {
    std::vector<double> t(tab_size(n)), work(7 * (n - 2));
    fill_table(t.data(), work.data(), n, lx, gamma, dt_factor, general, rhs_fp32);
    return t;
}

// Tensor maps of a grid's work field for the sweeps: [0] 16 columns by 32 rows in the 128-byte swizzle (x), [1] 32
// columns by 16 rows (y). False when the driver cannot encode them.
bool sweep_maps(CUtensorMap maps[2], double* tmp, int n) {
    auto enc = tensor_map_encoder();
    if (!enc) return false;
    cuuint64_t dims[2] = {(cuuint64_t)n, (cuuint64_t)n};
    cuuint64_t strides[1] = {(cuuint64_t)n * sizeof(double)};
    cuuint32_t estr[2] = {1, 1};
    for (int k = 0; k < 2; ++k) {
        cuuint32_t box[2] = {(cuuint32_t)(k ? BLK : kChunk), (cuuint32_t)(k ? kChunk : BLK)};
        if (enc(&maps[k], CU_TENSOR_MAP_DATA_TYPE_FLOAT64, 2, tmp, dims, strides, box, estr,
                CU_TENSOR_MAP_INTERLEAVE_NONE, k ? CU_TENSOR_MAP_SWIZZLE_NONE : CU_TENSOR_MAP_SWIZZLE_128B,
                CU_TENSOR_MAP_L2_PROMOTION_NONE, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE) != CUDA_SUCCESS)
            return false;
    }
    return true;
}

struct Batch {
    int device = 0;
    int rhs_fp32 = 0;
    int parity = 0;   // cCurr = buf[parity]
    long long steps_done = 0;
    std::vector<int> n;
    std::vector<double> lx;
    std::vector<GridDev> grids_h;
    std::vector<double*> allocs;
    std::vector<std::pair<std::string, double*>> tables;   // key "n/lx/gamma/dtf" -> device table
    GridDev* grids_d = nullptr;
    CUtensorMap* maps_d = nullptr;   // two per grid (sweep_maps)
    Item* items_rhs = nullptr;
    Item* items_rows = nullptr;   // K2 and K3 share the per-grid block lists (row / column blocks)
    int n_items_rhs = 0, n_items_rows = 0, n_general = 0, n_whole = 0;   // as in ChWork; those of general grids are the last
    unsigned int* arrived = nullptr;   // of the sweeps, one per line entry
    MassScratch* mass_d = nullptr;
    cudaStream_t stream = nullptr;
    bool own_stream = false;
    cudaGraphExec_t graph_exec[2] = {nullptr, nullptr};   // pair of steps starting at parity 0 / 1
    int sms = 0;
    int cfg = -1;   // ch_config index; -1: kChBatchDefault
    unsigned long long launches = 0;
};

static ChConfig batch_config(const Batch* b) { return ch_config(b->cfg >= 0 ? b->cfg : kChBatchDefault); }

static ChWork batch_work(const Batch* b) {
    return ChWork{b->grids_d, b->items_rhs, b->items_rows, b->maps_d, b->arrived, b->n_items_rhs, b->n_items_rows, b->n_general, b->n_whole};
}

static thread_local std::string g_ch_err;
static int ch_fail(cudaError_t e, const char* what) {
    g_ch_err = std::string("Error while '") + what + "': " + cudaGetErrorString(e);
    cudaGetLastError();
    return 1;
}
static int ch_fail_arg(const std::string& msg) {
    g_ch_err = msg;
    return 2;
}
#define CH_TRY(x, what)                             \
    do {                                            \
        cudaError_t _e = (x);                       \
        if (_e != cudaSuccess) return ch_fail(_e, what); \
    } while (0)

static int enqueue_step(Batch* b, int parity) {
    CH_TRY(launch_ch_step(batch_config(b), b->rhs_fp32 != 0, batch_work(b), parity, b->sms, b->stream),
           "Launching a step");
    return 0;
}

static int capture_pairs(Batch* b) {
    for (int p = 0; p < 2; ++p) {
        if (b->graph_exec[p]) continue;
        cudaGraph_t g;
        CH_TRY(cudaStreamBeginCapture(b->stream, cudaStreamCaptureModeThreadLocal), "Beginning graph capture");
        int st = enqueue_step(b, p);
        if (st == 0) st = enqueue_step(b, p ^ 1);
        cudaError_t e = cudaStreamEndCapture(b->stream, &g);
        if (st != 0) return st;
        CH_TRY(e, "Ending graph capture");
        e = cudaGraphInstantiate(&b->graph_exec[p], g, 0);
        cudaGraphDestroy(g);
        CH_TRY(e, "Instantiating graph");
    }
    return 0;
}

// ------------------------------------------------------------------------------------------------
// Allocation-free single-grid step (custen_ch_step_noalloc)
// ------------------------------------------------------------------------------------------------
// Some callers cannot allocate device memory at all: a plug-in running inside a host application
// that owns every device allocation through its own budgeted pool, or a latency-critical loop that
// must never enter cudaMalloc / cudaFree (they synchronise the device). For them one step of one
// grid runs with all of its work buffers in this file-scope array: the right-hand side / x-sweep
// field, the closure amplitudes, the solver table, the descriptor, the work lists,
// the tensor maps and the sweeps' arrival counts.
// Maximum grid: kNoAllocMaxN x kNoAllocMaxN. Every GPU that loads the library holds the array
// (about 560 KiB) until the process exits.
constexpr int kNoAllocMaxN = 256;
constexpr size_t align256(size_t v) { return (v + 255) / 256 * 256; }
constexpr size_t kNoAllocTmpOff = 0;
constexpr size_t kNoAllocEndsOff = align256(kNoAllocTmpOff + sizeof(double) * kNoAllocMaxN * kNoAllocMaxN);
constexpr size_t kNoAllocTabOff = align256(kNoAllocEndsOff + sizeof(double) * 16 * kNoAllocMaxN);
constexpr int kNoAllocTabLen = kTabParams + 7 * (kNoAllocMaxN - 2) + 8;
constexpr size_t kNoAllocGridOff = align256(kNoAllocTabOff + sizeof(double) * kNoAllocTabLen);
constexpr int kNoAllocBlocks = (kNoAllocMaxN / BLK) * (kNoAllocMaxN / BLK);
constexpr int kNoAllocRows = 2 * kNoAllocMaxN / BLK;   // two segments per line block
constexpr size_t kNoAllocRhsOff = align256(kNoAllocGridOff + sizeof(GridDev));
constexpr size_t kNoAllocRowsOff = align256(kNoAllocRhsOff + sizeof(Item) * kNoAllocBlocks);
constexpr size_t kNoAllocMapsOff = align256(kNoAllocRowsOff + sizeof(Item) * kNoAllocRows);
constexpr size_t kNoAllocArrivedOff = align256(kNoAllocMapsOff + 2 * sizeof(CUtensorMap));   // zero between calls
constexpr size_t kNoAllocBytes = align256(kNoAllocArrivedOff + kNoAllocRows * sizeof(unsigned int));

static __device__ __align__(256) unsigned char g_ch_noalloc_scratch[kNoAllocBytes];

// Device address of the array for each device, taken once with that device current. In host code the
// array's name is only a host-side stand-in, never a device address.
static std::atomic<unsigned char*> g_noalloc_base[64] = {};

}  // namespace ch
}  // namespace custen

using namespace custen::ch;

extern "C" {

const char* custen_ch_last_error(void) { return g_ch_err.c_str(); }

int custen_selftest_ring_expiry(long long rounds, int nchunk, int lost, unsigned int* flags, int* counts) {
    if (rounds < 1 || rounds > custen::kWaitLimit || nchunk < 1 || nchunk > 4096 || !flags || !counts)
        return ch_fail_arg("invalid arguments");
    int* d = nullptr;
    CH_TRY(cudaMalloc(&d, 4 * sizeof(int)), "Allocating the self-test's counts");
    cudaError_t e = cudaMemset(d, 0, 4 * sizeof(int));
    if (e == cudaSuccess) {
        ch_ring_expiry_kernel<<<1, kSweepThreads>>>(rounds, nchunk, lost, d);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(counts, d, 4 * sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(d);
    if (e == cudaSuccess) e = cudaMemcpyFromSymbol(flags, custen::g_custen_device_error, sizeof(unsigned int));
    return e == cudaSuccess ? 0 : ch_fail(e, "Running the ring's self-test");
}

int custen_ch_batch_create(void** out, int nsims, const int* n, const double* lx, double gamma, double dt_factor,
                           int rhs_dtype, void* stream) {
    if (!out || nsims < 1 || !n) return ch_fail_arg("invalid arguments");
    for (int s = 0; s < nsims; ++s)
        if (n[s] < 64 || n[s] % BLK != 0) return ch_fail_arg("grid sizes must be multiples of 32, at least 64");
    Batch* b = new Batch();
    cudaGetDevice(&b->device);
    b->rhs_fp32 = rhs_dtype == CUSTEN_F32;
    if (stream) {
        b->stream = static_cast<cudaStream_t>(stream);
    } else {
        cudaError_t e = cudaStreamCreateWithFlags(&b->stream, cudaStreamNonBlocking);
        if (e != cudaSuccess) { delete b; return ch_fail(e, "Creating stream"); }
        b->own_stream = true;
    }
    auto cleanup_fail = [&](int st) {
        for (double* p : b->allocs) cudaFree(p);
        for (auto& t : b->tables) cudaFree(t.second);
        if (b->own_stream) cudaStreamDestroy(b->stream);
        delete b;
        return st;
    };
    b->n.assign(n, n + nsims);
    b->lx.resize(nsims);
    for (int s = 0; s < nsims; ++s) b->lx[s] = lx ? lx[s] : 2.0 * M_PI;
    b->grids_h.resize(nsims);
    for (int s = 0; s < nsims; ++s) {
        const int ns = n[s];
        const bool general = line_is_general(ns, b->lx[s], gamma, dt_factor, b->rhs_fp32 != 0);
        char key[128];
        snprintf(key, sizeof(key), "%d/%.17g/%.17g/%.17g", ns, b->lx[s], gamma, dt_factor);
        double* tab = nullptr;
        for (auto& t : b->tables)
            if (t.first == key) tab = t.second;
        if (!tab) {
            std::vector<double> h = build_table(ns, b->lx[s], gamma, dt_factor, general, b->rhs_fp32 != 0);
            cudaError_t e = cudaMalloc(&tab, h.size() * sizeof(double));
            if (e != cudaSuccess) return cleanup_fail(ch_fail(e, "Allocating solver table"));
            e = cudaMemcpy(tab, h.data(), h.size() * sizeof(double), cudaMemcpyHostToDevice);
            if (e != cudaSuccess) return cleanup_fail(ch_fail(e, "Uploading solver table"));
            b->tables.push_back({key, tab});
        }
        GridDev g{};
        const size_t bytes = (size_t)ns * ns * sizeof(double);
        for (int k = 0; k < 4; ++k) {   // cCurr / cOld, tmp, h of the two-pass right-hand side
            double* p = nullptr;
            cudaError_t e = cudaMalloc(&p, bytes);
            if (e != cudaSuccess) return cleanup_fail(ch_fail(e, "Allocating grid fields"));
            b->allocs.push_back(p);
            if (k < 2) g.buf[k] = p; else if (k == 2) g.tmp = p; else g.hbuf = g.ends = p;
        }
        g.tab = tab;
        g.n = ns;
        g.general = general;
        g.cuts = line_cuts(ns, general);
        b->grids_h[s] = g;
    }
    // work lists, largest grids first
    std::vector<int> order(nsims);
    for (int s = 0; s < nsims; ++s) order[s] = s;
    std::stable_sort(order.begin(), order.end(), [&](int x, int y) { return n[x] > n[y]; });
    std::vector<Item> rhs, rows;
    for (int s : order) {
        const int bpr = n[s] / BLK;
        for (int k = 0; k < bpr * bpr; ++k) rhs.push_back({s, k});
        if (!b->grids_h[s].general)
            for (int k = 0; k < bpr * b->grids_h[s].cuts; ++k) {
                rows.push_back({s, k});
                b->n_whole += b->grids_h[s].cuts == 1;
            }
    }
    for (int s : order)
        if (b->grids_h[s].general)
            for (int k = 0; k < n[s] / BLK; ++k, ++b->n_general) rows.push_back({s, k});
    b->n_items_rhs = (int)rhs.size();
    b->n_items_rows = (int)rows.size();
    cudaError_t e = cudaMalloc(&b->grids_d, nsims * sizeof(GridDev));
    if (e == cudaSuccess) e = cudaMemcpy(b->grids_d, b->grids_h.data(), nsims * sizeof(GridDev), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMalloc(&b->items_rhs, rhs.size() * sizeof(Item));
    if (e == cudaSuccess) e = cudaMemcpy(b->items_rhs, rhs.data(), rhs.size() * sizeof(Item), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMalloc(&b->items_rows, rows.size() * sizeof(Item));
    if (e == cudaSuccess)
        e = cudaMemcpy(b->items_rows, rows.data(), rows.size() * sizeof(Item), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMalloc(&b->arrived, rows.size() * sizeof(unsigned int));
    if (e == cudaSuccess) e = cudaMemset(b->arrived, 0, rows.size() * sizeof(unsigned int));
    if (e == cudaSuccess) e = cudaMalloc(&b->mass_d, sizeof(MassScratch));
    if (e == cudaSuccess) e = cudaMemset(b->mass_d, 0, sizeof(MassScratch));
    std::vector<CUtensorMap> maps(2 * (size_t)nsims);
    for (int s = 0; s < nsims && e == cudaSuccess; ++s)
        if (!sweep_maps(&maps[2 * s], b->grids_h[s].tmp, n[s])) e = cudaErrorNotSupported;
    if (e == cudaSuccess) e = cudaMalloc(&b->maps_d, maps.size() * sizeof(CUtensorMap));
    if (e == cudaSuccess)
        e = cudaMemcpy(b->maps_d, maps.data(), maps.size() * sizeof(CUtensorMap), cudaMemcpyHostToDevice);
    if (e != cudaSuccess) return cleanup_fail(ch_fail(e, "Allocating work lists"));
    cudaDeviceGetAttribute(&b->sms, cudaDevAttrMultiProcessorCount, b->device);
    *out = b;
    return 0;
}

int custen_ch_batch_set_state(void* h, int sim, const double* c_cur, const double* c_old) {
    Batch* b = static_cast<Batch*>(h);
    if (!b || sim < 0 || sim >= (int)b->n.size() || !c_cur) return ch_fail_arg("invalid arguments");
    const size_t bytes = (size_t)b->n[sim] * b->n[sim] * sizeof(double);
    GridDev& g = b->grids_h[sim];
    CH_TRY(cudaMemcpyAsync(g.buf[b->parity], c_cur, bytes, cudaMemcpyDefault, b->stream), "Uploading cCurr");
    CH_TRY(cudaMemcpyAsync(g.buf[b->parity ^ 1], c_old ? c_old : c_cur, bytes, cudaMemcpyDefault, b->stream),
           "Uploading cOld");
    CH_TRY(cudaStreamSynchronize(b->stream), "Synchronising upload");
    return 0;
}

int custen_ch_batch_get_state(void* h, int sim, double* c_cur, double* c_old) {
    Batch* b = static_cast<Batch*>(h);
    if (!b || sim < 0 || sim >= (int)b->n.size()) return ch_fail_arg("invalid arguments");
    const size_t bytes = (size_t)b->n[sim] * b->n[sim] * sizeof(double);
    GridDev& g = b->grids_h[sim];
    if (c_cur) CH_TRY(cudaMemcpyAsync(c_cur, g.buf[b->parity], bytes, cudaMemcpyDefault, b->stream), "Reading cCurr");
    if (c_old)
        CH_TRY(cudaMemcpyAsync(c_old, g.buf[b->parity ^ 1], bytes, cudaMemcpyDefault, b->stream), "Reading cOld");
    CH_TRY(cudaStreamSynchronize(b->stream), "Synchronising read");
    return 0;
}

// Snapshot of one grid in the reference's HDF5 format (Print_Out, cuPentCahnADI.cu:103-140): dataset
// "c" = cCurr (n x n doubles), plus "c_old" = cOld and "t" = the time (1 x 1), which a resume needs
// and a reader of the reference's files ignores.
int custen_ch_batch_save(void* h, int sim, const char* path, double time) {
    Batch* b = static_cast<Batch*>(h);
    if (!b || sim < 0 || sim >= (int)b->n.size() || !path) return ch_fail_arg("invalid arguments");
    const long long n = b->n[sim];
    std::vector<double> cur((size_t)(n * n)), old((size_t)(n * n));
    const int rc = custen_ch_batch_get_state(h, sim, cur.data(), old.data());
    if (rc) return rc;
    const char* names[3] = {"c", "c_old", "t"};
    const double* data[3] = {cur.data(), old.data(), &time};
    const long long dims[6] = {n, n, n, n, 1, 1};
    if (custen_h5_write(path, 3, names, data, dims)) return ch_fail_arg(std::string("Writing the snapshot: ") + custen_h5_last_error());
    return 0;
}

// Resume one grid from a snapshot: "c" (required, n x n) becomes cCurr; cOld is "c_old" when present,
// else cCurr too, as the reference starts from its initial condition (cuPentCahnADI.cu:295-305).
// *time receives "t", or NaN when the file has none (the reference's own snapshots).
int custen_ch_batch_load(void* h, int sim, const char* path, double* time) {
    Batch* b = static_cast<Batch*>(h);
    if (!b || sim < 0 || sim >= (int)b->n.size() || !path) return ch_fail_arg("invalid arguments");
    const long long n = b->n[sim];
    long long dims[2] = {0, 0};
    if (custen_h5_read(path, "c", nullptr, 0, dims)) return ch_fail_arg(std::string("Reading the snapshot: ") + custen_h5_last_error());
    if (dims[0] != n || dims[1] != n)
        return ch_fail_arg("snapshot grid is " + std::to_string(dims[0]) + " x " + std::to_string(dims[1]) +
                           ", grid " + std::to_string(sim) + " is " + std::to_string(n) + " x " + std::to_string(n));
    std::vector<double> cur((size_t)(n * n)), old;
    if (custen_h5_read(path, "c", cur.data(), n * n, dims)) return ch_fail_arg(std::string("Reading the snapshot: ") + custen_h5_last_error());
    long long od[2] = {0, 0};
    if (custen_h5_read(path, "c_old", nullptr, 0, od) == 0) {
        if (od[0] != n || od[1] != n) return ch_fail_arg("snapshot c_old does not match c");
        old.resize((size_t)(n * n));
        if (custen_h5_read(path, "c_old", old.data(), n * n, od))
            return ch_fail_arg(std::string("Reading the snapshot: ") + custen_h5_last_error());
    }
    double t = std::nan("");
    long long td[2];
    if (custen_h5_read(path, "t", nullptr, 0, td) == 0 && td[0] * td[1] == 1) custen_h5_read(path, "t", &t, 1, td);
    if (time) *time = t;
    return custen_ch_batch_set_state(h, sim, cur.data(), old.empty() ? nullptr : old.data());
}

// Advance every grid by `steps` steps; asynchronous on the batch's stream (graph replays for pairs of
// steps, plain launches for an odd remainder) unless use_graph == 0.
int custen_ch_batch_step(void* h, int steps, int use_graph) {
    Batch* b = static_cast<Batch*>(h);
    if (!b || steps < 0) return ch_fail_arg("invalid arguments");
    cudaSetDevice(b->device);
    int left = steps;
    const int per_step = ch_launches_per_step(batch_config(b), batch_work(b), b->sms);   // kernel launches in one step
    if (use_graph && left >= 2) {
        int st = capture_pairs(b);
        if (st) return st;
        while (left >= 2) {
            CH_TRY(cudaGraphLaunch(b->graph_exec[b->parity], b->stream), "Launching step graph");
            b->launches += 2 * per_step;
            left -= 2;
            b->steps_done += 2;
        }
    }
    while (left > 0) {
        int st = enqueue_step(b, b->parity);
        if (st) return st;
        b->launches += per_step;
        b->parity ^= 1;
        --left;
        ++b->steps_done;
    }
    return 0;
}

int custen_ch_batch_synchronize(void* h) {
    Batch* b = static_cast<Batch*>(h);
    CH_TRY(cudaStreamSynchronize(b->stream), "Synchronising batch");
    return 0;
}

// Mean of a grid's cCurr with a compensated FP64 sum (device side).
int custen_ch_batch_mean(void* h, int sim, double* mean) {
    Batch* b = static_cast<Batch*>(h);
    if (!b || sim < 0 || sim >= (int)b->n.size() || !mean) return ch_fail_arg("invalid arguments");
    const long long count = (long long)b->n[sim] * b->n[sim];
    CH_TRY(launch_ch_mass(b->grids_h[sim].buf[b->parity], count, b->mass_d, b->stream), "Launching mass sum");
    double s = 0.0;
    CH_TRY(cudaMemcpyAsync(&s, &b->mass_d->sum, sizeof(double), cudaMemcpyDeviceToHost, b->stream), "Reading mass");
    CH_TRY(cudaStreamSynchronize(b->stream), "Synchronising mass");
    *mean = s / (double)count;
    return 0;
}

unsigned long long custen_ch_batch_launches(void* h) { return static_cast<Batch*>(h)->launches; }

// One step of one n x n grid (n a multiple of 32, 64 <= n <= 256) without any device allocation.
// c_old, c_cur: the two previous fields; c_new receives the next one (it may be the c_old buffer,
// not the c_cur buffer). All three are device-accessible n*n double arrays. The first call on a
// device looks up the scratch array's device address (make it before any stream capture). Calls
// share the array: two calls that overlap on the GPU (different streams, no ordering) race.
int custen_ch_step_noalloc(const double* c_old, const double* c_cur, double* c_new, int n, double lx, double gamma,
                           double dt_factor, void* stream) {
    if (!c_old || !c_cur || !c_new) return ch_fail_arg("custen_ch_step_noalloc: NULL field pointer");
    if (n < 64 || n % BLK != 0) return ch_fail_arg("custen_ch_step_noalloc: n must be a multiple of 32, at least 64");
    if (n > kNoAllocMaxN) {
        char msg[160];
        snprintf(msg, sizeof(msg), "custen_ch_step_noalloc: n = %d exceeds the allocation-free maximum of %d", n,
                 kNoAllocMaxN);
        return ch_fail_arg(msg);
    }
    if (c_new == c_cur) return ch_fail_arg("custen_ch_step_noalloc: c_new must not be the c_cur buffer");
    int dev = 0;
    CH_TRY(cudaGetDevice(&dev), "Querying the current device");
    if (dev < 0 || dev >= 64) return ch_fail_arg("custen_ch_step_noalloc: device index out of range");
    unsigned char* base = g_noalloc_base[dev].load(std::memory_order_acquire);
    if (base == nullptr) {   // the same address whichever thread looks it up first
        void* p = nullptr;
        CH_TRY(cudaGetSymbolAddress(&p, g_ch_noalloc_scratch), "Looking up the scratch array's device address");
        base = static_cast<unsigned char*>(p);
        g_noalloc_base[dev].store(base, std::memory_order_release);
    }
    cudaStream_t s = static_cast<cudaStream_t>(stream);

    // host-side inputs in stack buffers (no heap either)
    double tab[kNoAllocTabLen];
    double work[7 * (kNoAllocMaxN - 2)];
    GridDev g{};
    g.general = line_is_general(n, lx, gamma, dt_factor, false);
    fill_table(tab, work, n, lx, gamma, dt_factor, g.general != 0, false);
    g.buf[0] = const_cast<double*>(c_cur);
    g.buf[1] = c_new;
    g.tmp = reinterpret_cast<double*>(base + kNoAllocTmpOff);
    g.ends = reinterpret_cast<double*>(base + kNoAllocEndsOff);
    g.tab = reinterpret_cast<const double*>(base + kNoAllocTabOff);
    g.n = n;
    const int bpr = n / BLK;
    Item rhs[kNoAllocBlocks], rows[kNoAllocRows];
    for (int k = 0; k < bpr * bpr; ++k) rhs[k] = Item{0, k};
    g.cuts = line_cuts(n, g.general != 0);
    const int n_lines = bpr * g.cuts;
    for (int k = 0; k < n_lines; ++k) rows[k] = Item{0, k};

    const size_t bytes = (size_t)n * n * sizeof(double);
    // the update is written over the "old" buffer: start it from c_old
    if (c_new != c_old) CH_TRY(cudaMemcpyAsync(c_new, c_old, bytes, cudaMemcpyDefault, s), "Copying c_old");
    CH_TRY(cudaMemcpyAsync(base + kNoAllocTabOff, tab, sizeof(double) * tab_size(n), cudaMemcpyHostToDevice, s),
           "Uploading the solver table");
    CH_TRY(cudaMemcpyAsync(base + kNoAllocGridOff, &g, sizeof(g), cudaMemcpyHostToDevice, s),
           "Uploading the grid descriptor");
    CH_TRY(cudaMemcpyAsync(base + kNoAllocRhsOff, rhs, sizeof(Item) * bpr * bpr, cudaMemcpyHostToDevice, s),
           "Uploading the work list");
    CH_TRY(cudaMemcpyAsync(base + kNoAllocRowsOff, rows, sizeof(Item) * n_lines, cudaMemcpyHostToDevice, s),
           "Uploading the work list");
    const GridDev* gd = reinterpret_cast<const GridDev*>(base + kNoAllocGridOff);
    const Item* it_rhs = reinterpret_cast<const Item*>(base + kNoAllocRhsOff);
    const Item* it_rows = reinterpret_cast<const Item*>(base + kNoAllocRowsOff);
    int sms = 0;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    CUtensorMap maps[2];
    if (!sweep_maps(maps, g.tmp, n)) return ch_fail(cudaErrorNotSupported, "Encoding the tensor maps");
    CH_TRY(cudaMemcpyAsync(base + kNoAllocMapsOff, maps, sizeof(maps), cudaMemcpyHostToDevice, s),
           "Uploading the tensor maps");
    const ChWork w{gd, it_rhs, it_rows, reinterpret_cast<const CUtensorMap*>(base + kNoAllocMapsOff),
                   reinterpret_cast<unsigned int*>(base + kNoAllocArrivedOff), bpr * bpr, n_lines,
                   g.general ? n_lines : 0, g.cuts == 1 ? n_lines : 0};
    CH_TRY(launch_ch_step(ch_config(kChOneGrid), false, w, 0, sms, s), "Launching the step");
    return 0;
}

// Kernel configuration of a batch: time every configuration (ch_config) over `steps` steps of the
// batch itself, then restore the fields it started from, so tuning changes no result. Writes the
// chosen configuration's name to `name`. No reference counterpart.
int custen_ch_batch_autotune(void* h, int steps, char* name, size_t len) {
    Batch* b = static_cast<Batch*>(h);
    if (!b || steps < 1) return ch_fail_arg("invalid arguments");
    CH_TRY(cudaSetDevice(b->device), "Setting device");
    size_t total = 0;
    for (const auto& g : b->grids_h) total += (size_t)g.n * g.n;
    double* save = nullptr;
    CH_TRY(cudaMalloc(&save, 2 * total * sizeof(double)), "Allocating the saved state");
    auto copy_state = [&](bool to_save) -> cudaError_t {
        size_t off = 0;
        for (const auto& g : b->grids_h) {
            const size_t bytes = (size_t)g.n * g.n * sizeof(double);
            for (int k = 0; k < 2; ++k) {
                double* dev = g.buf[k];
                double* sv = save + off;
                cudaError_t e = cudaMemcpyAsync(to_save ? sv : dev, to_save ? dev : sv, bytes,
                                                cudaMemcpyDeviceToDevice, b->stream);
                if (e != cudaSuccess) return e;
                off += (size_t)g.n * g.n;
            }
        }
        return cudaSuccess;
    };
    const int parity0 = b->parity;
    const long long done0 = b->steps_done;
    const unsigned long long launches0 = b->launches;
    cudaEvent_t e0 = nullptr, e1 = nullptr;
    cudaError_t err = copy_state(true);
    if (err == cudaSuccess) err = cudaEventCreate(&e0);
    if (err == cudaSuccess) err = cudaEventCreate(&e1);
    int best = -1;
    float best_ms = 0.f;
    for (int c = 0; c < kChConfigs && err == cudaSuccess; ++c) {
        b->cfg = c;
        for (int p = 0; p < 2; ++p)
            if (b->graph_exec[p]) {
                cudaGraphExecDestroy(b->graph_exec[p]);
                b->graph_exec[p] = nullptr;
            }
        if (custen_ch_batch_step(h, 2, 1) != 0) break;   // warm-up, graph capture
        cudaEventRecord(e0, b->stream);
        if (custen_ch_batch_step(h, steps, 1) != 0) break;
        cudaEventRecord(e1, b->stream);
        if ((err = cudaEventSynchronize(e1)) != cudaSuccess) break;
        float ms = 0.f;
        cudaEventElapsedTime(&ms, e0, e1);
        if (best < 0 || ms < best_ms) {
            best = c;
            best_ms = ms;
        }
        if ((err = copy_state(false)) != cudaSuccess) break;
        b->parity = parity0;
        b->steps_done = done0;
    }
    if (e0) cudaEventDestroy(e0);
    if (e1) cudaEventDestroy(e1);
    if (err == cudaSuccess) err = cudaStreamSynchronize(b->stream);
    cudaFree(save);
    b->parity = parity0;
    b->steps_done = done0;
    b->launches = launches0;
    for (int p = 0; p < 2; ++p)
        if (b->graph_exec[p]) {
            cudaGraphExecDestroy(b->graph_exec[p]);
            b->graph_exec[p] = nullptr;
        }
    if (err != cudaSuccess) return ch_fail(err, "Tuning the batch");
    if (best < 0) return 1;
    b->cfg = best;
    if (name && len) {
        const ChConfig c = ch_config(best);
        config_name(c, name, len);
    }
    return 0;
}

int custen_ch_batch_set_config(void* h, int index) {
    Batch* b = static_cast<Batch*>(h);
    if (!b || index < -1 || index >= kChConfigs) return ch_fail_arg("invalid arguments");
    CH_TRY(cudaStreamSynchronize(b->stream), "Synchronising the batch");
    b->cfg = index;
    for (int p = 0; p < 2; ++p)
        if (b->graph_exec[p]) {
            cudaGraphExecDestroy(b->graph_exec[p]);
            b->graph_exec[p] = nullptr;
        }
    return 0;
}

int custen_ch_batch_config(void* h, char* name, size_t len) {
    Batch* b = static_cast<Batch*>(h);
    if (!b || !name || !len) return ch_fail_arg("invalid arguments");
    const ChConfig c = batch_config(b);
    config_name(c, name, len);
    return 0;
}

int custen_ch_batch_destroy(void* h) {
    Batch* b = static_cast<Batch*>(h);
    if (!b) return 0;
    cudaStreamSynchronize(b->stream);
    for (int p = 0; p < 2; ++p)
        if (b->graph_exec[p]) cudaGraphExecDestroy(b->graph_exec[p]);
    for (double* p : b->allocs) cudaFree(p);
    for (auto& t : b->tables) cudaFree(t.second);
    cudaFree(b->grids_d);
    cudaFree(b->maps_d);
    cudaFree(b->items_rhs);
    cudaFree(b->items_rows);
    cudaFree(b->mass_d);
    cudaFree(b->arrived);
    if (b->own_stream) cudaStreamDestroy(b->stream);
    delete b;
    return 0;
}

}  // extern "C"


