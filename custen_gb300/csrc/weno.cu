// WENO5 advection stencil, periodic in x and y (the thirteenth cuSten operator,
// cuSten/src/kernels/2d_xyADVWENO_p_kernel.cu), for sm_103a.
//
// out[y][x] = u[y][x] * Fx + v[y][x] * Fy, where Fx (Fy) is the fifth-order WENO reconstruction of the
// upwind one-sided differences D[i] = (in[i] - in[i-1]) * coeDx along x (along y with coeDy): for u > 0
// the differences at x-2 .. x+2, otherwise those at x+3 .. x-1 in reverse order (the reference's
// upwind selection, 2d_xyADVWENO_p_kernel.cu:286-348 and :352-414).
//
// GB300 shape: about 100 FP64 operations per point against 32 bytes of compulsory traffic, so the FP64 pipe
// bounds this operator by a wide margin (issue slots 30%). The kernel therefore spends no
// FP64 work twice or where another pipe can do it:
//   - a 64 x TH tile with its 3-point periodic halo is staged once, and the x and y differences and the squared
//     second differences are formed once per tile into shared memory (the reference forms five differences and
//     three second differences per point and direction);
//   - the 36 conversions per point between double and the float smoothness terms, and all but 3 operations of
//     each division (4 of the reciprocal's), run on the integer and FP32 pipes (fp64_offload.cuh).
// The reconstruction keeps the reference's operation order, including its single-precision powf on the
// smoothness terms, so that results are bit-identical to the reference's kernel on the same GPU.
// Measured (2048^2): 1418 us with hardware conversions and divisions (about 200 FP64 instructions per point),
// 913 us with those moved off the FP64 pipe (112), 817 us with the shared second differences and the shorter
// divisions (103; 5.1 Gpts/s; 4096^2: 5.3, about 94% of the rate of multiply-adds).
#include <cuda_runtime.h>

#include <atomic>

#include "checked.cuh"
#include "custen_internal.h"
#include "fp64_offload.cuh"

namespace custen {
namespace {

constexpr int kWenoTW = 64;                 // tile columns (one per thread column)
constexpr int kWenoHalo = 3;                // i-3 .. i+3
constexpr int kWenoThreads = 256;           // 64 columns x 4 thread rows
constexpr int kWenoSW = kWenoTW + 2 * kWenoHalo;   // 70 staged columns
constexpr int kWenoDXW = kWenoTW + 5;       // x differences at columns x0-2 .. x0+TW+2
constexpr int kWenoSXW = kWenoTW + 3;       // x second differences at columns x0-1 .. x0+TW+1

// Shared memory of a tile of TH rows: the staged field, the differences (y differences at rows y0-2 ..
// y0+TH+2), and the squared second differences of either orientation (floats; y: rows y0-1 .. y0+TH+1).
template <int TH>
struct WenoTile {
    static constexpr int SH = TH + 2 * kWenoHalo, DYH = TH + 5, SYH = TH + 3;
    static constexpr size_t bytes = sizeof(double) * ((size_t)SH * kWenoSW + (size_t)TH * kWenoDXW + (size_t)DYH * kWenoTW) +
                                    2 * sizeof(float) * ((size_t)TH * kWenoSXW + (size_t)SYH * kWenoTW);
};

// Coefficients of the reconstruction. They are read from device memory into registers once per
// thread (WenoCoeffs::load): an FP64 FMA or add with a literal or kernel-parameter operand issues about
// 19% slower on GB300 than one whose operands are all registers (507 against 602-628 G FMA/s
// measured). The values are the literals of the reference's expressions, so every result is the same.
__device__ double g_weno_coeffs[14] = {1.0 / 3.0, 7.0 / 6.0, 11.0 / 6.0, 1.0 / 6.0, 5.0 / 6.0,
                                       2.0,       4.0,       3.0,        13.0 / 12.0, 0.25,
                                       1e-06,     0.1,       0.6,        0.3};

struct WenoCoeffs {
    double third, seven_sixths, eleven_sixths, sixth, five_sixths, two, four, three, thirteen_twelfths,
        eps, g1, g2, g3;
    f64::F64 f;
    __device__ __forceinline__ void load() {
        const volatile double* k = g_weno_coeffs;
        third = k[0]; seven_sixths = k[1]; eleven_sixths = k[2]; sixth = k[3]; five_sixths = k[4];
        two = k[5]; four = k[6]; three = k[7]; thirteen_twelfths = k[8];
        eps = k[10]; g1 = k[11]; g2 = k[12]; g3 = k[13];
    }
};

// t^2 by single-precision powf.
__device__ __forceinline__ float square(double t) { return powf(f64::to_float(t), 2.0f); }
// A quarter of it, as a double (exact: an exponent shift).
__device__ __forceinline__ double quarter_square(double t) { return f64::to_double_pos<-2>(square(t)); }

// Fifth-order WENO reconstruction (Jiang & Shu 1996, in the notation of Osher & Fedkiw, "Level Set
// Methods and Dynamic Implicit Surfaces", 3.4) from five consecutive differences a..e, given the squared second
// differences s1 = (a - 2b + c)^2, s2 = (b - 2c + d)^2, s3 = (c - 2d + e)^2 (floats; each belongs to one cell
// and is shared by the three points whose windows hold it). The three candidate stencils, the smoothness
// indicators and the nonlinear weights are evaluated in the order of the reference's wenoSten
// (2d_xyADVWENO_p_kernel.cu:52-88): same expressions, same contraction, and the smoothness squares and the
// squared (indicator + 1e-6) taken by powf in single precision.
__device__ __forceinline__ double weno5(const WenoCoeffs& k, double a, double b, double c, double d, double e, float s1,
                                        float s2, float s3) {
    // each sum of products is the contraction fma(x, y, z w) the compiler gives the reference's expression
    const f64::F64& f = k.f;
    const double q1 = fma(k.eleven_sixths, c, fma(k.third, a, -f.mul(k.seven_sixths, b)));
    const double q2 = fma(k.third, d, fma(k.five_sixths, c, -f.mul(k.sixth, b)));
    const double q3 = fma(-k.sixth, e, fma(k.third, c, f.mul(k.five_sixths, d)));

    const double is1 = fma(k.thirteen_twelfths, f64::to_double_pos(s1), quarter_square(fma(k.three, c, fma(-k.four, b, a))));
    const double is2 = fma(k.thirteen_twelfths, f64::to_double_pos(s2), quarter_square(f.sub(b, d)));
    const double is3 =
        fma(k.thirteen_twelfths, f64::to_double_pos(s3), quarter_square(f.add(fma(k.three, c, -f64::times4(d)), e)));

    const double g1 = f64::div_by_float(f, k.g1, square(f.add(is1, k.eps)));
    const double g2 = f64::div_by_float(f, k.g2, square(f.add(is2, k.eps)));
    const double g3 = f64::div_by_float(f, k.g3, square(f.add(is3, k.eps)));
    const double norm = f64::reciprocal(f, f.add(f.add(g1, g2), g3));
    const double w1 = f.mul(g1, norm), w2 = f.mul(g2, norm), w3 = f.mul(g3, norm);
    return fma(q3, w3, fma(q1, w1, f.mul(q2, w2)));
}

__device__ __forceinline__ int wrap_col(int c, int nx) {
    if (c < 0) c += nx;
    else if (c >= nx) c -= nx;
    if (c < 0 || c >= nx) {   // a field narrower than the staged window
        c %= nx;
        if (c < 0) c += nx;
    }
    return c;
}

// One CTA per 64 x TH tile of the launch's rows. Rows above / below the launch come from the T = 3
// halo rows at `top` / `bot` (the handle's boundaryTop/boundaryBottom of the tile, periodic); columns
// wrap around the field.
template <int TH>
__global__ void __launch_bounds__(kWenoThreads, 2) weno_adv_kernel(double* __restrict__ out,
                                                                   const double* __restrict__ in,
                                                                   const double* __restrict__ uvel,
                                                                   const double* __restrict__ vvel,
                                                                   const double* __restrict__ top,
                                                                   const double* __restrict__ bot, double cdx,
                                                                   double cdy, int nx, int rows) {
    extern __shared__ __align__(16) double wsm[];
    using G = WenoTile<TH>;
    double* tile = wsm;                                   // [SH][SW]
    double* dxs = tile + G::SH * kWenoSW;                 // [TH][DXW]
    double* dys = dxs + TH * kWenoDXW;                    // [DYH][TW]
    float* sxf = reinterpret_cast<float*>(dys + G::DYH * kWenoTW);   // [TH][SXW], upwind from the left
    float* sxb = sxf + TH * kWenoSXW;                     // from the right
    float* syf = sxb + TH * kWenoSXW;                     // [SYH][TW]
    float* syb = syf + G::SYH * kWenoTW;
    const int x0 = blockIdx.x * kWenoTW, y0 = blockIdx.y * TH;
    const int tid = threadIdx.x;
    WenoCoeffs k;
    k.load();
    const double dx = k.f.add(cdx, k.f.nzero), dy = k.f.add(cdy, k.f.nzero);   // the parameters in registers

    // stage the tile and its halo: staged (r, c) is field row y0-3+r, column x0-3+c (wrapped)
    for (int e = tid; e < G::SH * kWenoSW; e += kWenoThreads) {
        const int r = e / kWenoSW, c = e - r * kWenoSW;
        const int gy = y0 - kWenoHalo + r;
        const int gx = wrap_col(x0 - kWenoHalo + c, nx);
        double val = 0.0;
        if (gy < 0) val = top[(size_t)(gy + kWenoHalo) * nx + gx];
        else if (gy < rows) val = in[(size_t)gy * nx + gx];
        else if (gy < rows + kWenoHalo) val = bot[(size_t)(gy - rows) * nx + gx];
        tile[e] = val;
    }
    __syncthreads();
    // differences, each formed once: D(i) = (f[i] - f[i-1]) * coe (2d_xyADVWENO_p_kernel.cu:290-309)
    for (int e = tid; e < TH * kWenoDXW; e += kWenoThreads) {
        const int r = e / kWenoDXW, c = e - r * kWenoDXW;
        const double* row = tile + (r + kWenoHalo) * kWenoSW;
        dxs[e] = k.f.mul(k.f.sub(row[c + 1], row[c]), dx);
    }
    for (int e = tid; e < G::DYH * kWenoTW; e += kWenoThreads) {
        const int r = e / kWenoTW, c = e - r * kWenoTW;
        dys[e] = k.f.mul(k.f.sub(tile[(r + 1) * kWenoSW + c + kWenoHalo], tile[r * kWenoSW + c + kWenoHalo]), dy);
    }
    __syncthreads();

    // squared second differences of every cell, once in each orientation (the order of the sum differs): the
    // three smoothness indicators of a point take them from its window's three middle cells
    for (int e = tid; e < TH * kWenoSXW; e += kWenoThreads) {
        const int r = e / kWenoSXW, c = e - r * kWenoSXW;   // cell: column x0 - 1 + c
        const double* d = dxs + r * kWenoDXW + c;
        sxf[e] = square(k.f.add(fma(-k.two, d[1], d[0]), d[2]));
        sxb[e] = square(k.f.add(fma(-k.two, d[1], d[2]), d[0]));
    }
    for (int e = tid; e < G::SYH * kWenoTW; e += kWenoThreads) {   // cell: row y0 - 1 + e / TW
        const double* d = dys + e;
        syf[e] = square(k.f.add(fma(-k.two, d[kWenoTW], d[0]), d[2 * kWenoTW]));
        syb[e] = square(k.f.add(fma(-k.two, d[kWenoTW], d[2 * kWenoTW]), d[0]));
    }
    __syncthreads();

    const int tx = tid % kWenoTW;
    const int x = x0 + tx;
    if (x >= nx) return;
#pragma unroll(TH == 16 ? 2 : 1)
    for (int ty = tid / kWenoTW; ty < TH; ty += kWenoThreads / kWenoTW) {
        const int y = y0 + ty;
        if (y >= rows) break;
        const size_t q = (size_t)y * nx + x;
        const double uu = uvel[q], vv = vvel[q];
        // Upwind side: the five differences are selected first and reconstructed once (two calls in a
        // conditional expression would let the compiler evaluate both and double the FP64 work).
        if (!span_ok((long long)ty * kWenoDXW + tx, 6, (long long)TH * kWenoDXW) ||
            !span_ok((long long)ty * kWenoTW + tx, 5 * kWenoTW + 1, (long long)G::DYH * kWenoTW) ||
            !in_bounds((long long)q, 0, (long long)rows * nx))
            continue;
        const double* dr = dxs + ty * kWenoDXW + tx;      // dr[k] = D at column x - 2 + k
        const float* sf = sxf + ty * kWenoSXW + tx;       // sf[k] = cell at column x - 1 + k
        const float* sb = sxb + ty * kWenoSXW + tx;
        const bool ux = uu > 0.0;
        const double fx = weno5(k, ux ? dr[0] : dr[5], ux ? dr[1] : dr[4], dr[2 + !ux], ux ? dr[3] : dr[2],
                                ux ? dr[4] : dr[1], ux ? sf[0] : sb[3], ux ? sf[1] : sb[2], ux ? sf[2] : sb[1]);
        const double* dc = dys + ty * kWenoTW + tx;       // dc[k * TW] = D at row y - 2 + k
        const float* tf = syf + ty * kWenoTW + tx;        // tf[k * TW] = cell at row y - 1 + k
        const float* tb = syb + ty * kWenoTW + tx;
        const bool vy = vv > 0.0;
        const double fy = weno5(k, vy ? dc[0] : dc[5 * kWenoTW], vy ? dc[kWenoTW] : dc[4 * kWenoTW],
                                dc[(2 + !vy) * kWenoTW], vy ? dc[3 * kWenoTW] : dc[2 * kWenoTW],
                                vy ? dc[4 * kWenoTW] : dc[kWenoTW], vy ? tf[0] : tb[3 * kWenoTW],
                                vy ? tf[kWenoTW] : tb[2 * kWenoTW], vy ? tf[2 * kWenoTW] : tb[kWenoTW]);
        // (2d_xyADVWENO_p_kernel.cu:424)
        out[q] = fma(uu, fx, k.f.mul(vv, fy));
    }
}

template <int TH>
cudaError_t launch_tile(const StencilArgs& a, cudaStream_t s, int dev) {
    // setting the attribute is idempotent: threads that race here both set it
    static std::atomic<bool> attr_set[64] = {};
    if (dev >= 0 && dev < 64 && !attr_set[dev].load(std::memory_order_acquire)) {
        cudaError_t e = cudaFuncSetAttribute(weno_adv_kernel<TH>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             (int)WenoTile<TH>::bytes);
        if (e != cudaSuccess) return e;
        attr_set[dev].store(true, std::memory_order_release);
    }
    dim3 grid((a.nx + kWenoTW - 1) / kWenoTW, (a.rows + TH - 1) / TH);
    weno_adv_kernel<TH><<<grid, kWenoThreads, WenoTile<TH>::bytes, s>>>(
        static_cast<double*>(a.out), static_cast<const double*>(a.in), static_cast<const double*>(a.u),
        static_cast<const double*>(a.v), static_cast<const double*>(a.top), static_cast<const double*>(a.bot),
        a.cdx, a.cdy, a.nx, a.rows);
    return cudaGetLastError();
}

}  // namespace

// Two CTAs are resident per SM (304 on GB300) and each tile is a long stretch of FP64 work, so
// few tiles leave SMs idle and few waves end in an uneven one; a lower tile forms more differences of its halo
// twice. Measured (us, 8 / 16 / 32 rows): 300^2 40 / 44 / 77, 600^2 101 / 122 / 123, 1000 x 777 187 / 189 / 201
// (400 tiles of 32 rows), 1500 x 1400 453 / 431 / 454 (1056), 2048^2 - / 817 / 838 (2048), 4096^2 - / 3199 / 3141.
int weno_tile_rows(int nx, int rows) {
    const long long tiles = (long long)((nx + kWenoTW - 1) / kWenoTW) * ((rows + 31) / 32);
    return tiles < 512 ? 8 : (tiles < 4096 ? 16 : 32);
}

cudaError_t launch_weno_adv(const StencilArgs& a, cudaStream_t s) {
    int dev = 0;
    cudaError_t e = cudaGetDevice(&dev);
    if (e != cudaSuccess) return e;
    if (a.rows <= 0 || a.nx <= 0) return cudaSuccess;
    switch (weno_tile_rows(a.nx, a.rows)) {
    case 8: return launch_tile<8>(a, s, dev);
    case 16: return launch_tile<16>(a, s, dev);
    default: return launch_tile<32>(a, s, dev);
    }
}

}  // namespace custen
