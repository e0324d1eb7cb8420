// Kernel entry and launcher template for the shared-memory tiled stencil (see stencil_kernel.cuh).
#pragma once

#include <cudaTypedefs.h>

#include <algorithm>
#include <atomic>
#include <cstring>

#include "stencil_async.cuh"
#include "stencil_configs.h"
#include "stencil_kernel.cuh"
#include "stencil_tma.cuh"

namespace custen {

// Largest dynamic shared memory a block may opt in to on the current device.
inline int smem_optin_limit() {
    static std::atomic<int> cached[64] = {};   // threads that race store the same value
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64) {
        const int c = cached[dev].load(std::memory_order_relaxed);
        if (c) return c;
    }
    int v = 0;
    if (cudaDeviceGetAttribute(&v, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev) != cudaSuccess) v = 48 * 1024;
    if (dev >= 0 && dev < 64) cached[dev].store(v, std::memory_order_relaxed);
    return v;
}

template <typename Kernel>
inline cudaError_t ensure_smem(Kernel k, size_t smem) {
    if (smem <= 48 * 1024) return cudaSuccess;
    if (smem > (size_t)smem_optin_limit()) return cudaErrorInvalidConfiguration;
    return cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
}

// cuTensorMapEncodeTiled through the runtime's driver entry point (no link-time libcuda dependency).
// Looked up once (a function-local static: initialised once even when host threads race).
inline PFN_cuTensorMapEncodeTiled_v12000 tensor_map_encoder() {
    static const PFN_cuTensorMapEncodeTiled_v12000 fn = []() -> PFN_cuTensorMapEncodeTiled_v12000 {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &q) ==
                cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            return reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(p);
        cudaGetLastError();
        return nullptr;
    }();
    return fn;
}

template <typename T>
inline bool encode_rows_map(CUtensorMap* m, const void* base, int nx, int rows, int box_w, int box_h) {
    auto enc = tensor_map_encoder();
    if (!enc || base == nullptr || rows < 1 || box_h < 1) return false;
    cuuint64_t dims[2] = {(cuuint64_t)nx, (cuuint64_t)rows};
    cuuint64_t strides[1] = {(cuuint64_t)nx * sizeof(T)};
    cuuint32_t box[2] = {(cuuint32_t)box_w, (cuuint32_t)box_h};
    cuuint32_t estr[2] = {1, 1};
    CUresult r = enc(m, sizeof(T) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2,
                     const_cast<void*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                     CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                     CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    return r == CUDA_SUCCESS;
}

inline int sm_count() {
    static std::atomic<int> cached[64] = {};   // threads that race store the same value
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < 64) {
        const int c = cached[dev].load(std::memory_order_relaxed);
        if (c) return c;
    }
    int v = 0;
    cudaDeviceGetAttribute(&v, cudaDevAttrMultiProcessorCount, dev);
    if (dev >= 0 && dev < 64) cached[dev].store(v, std::memory_order_relaxed);
    return v;
}

// Resident threads per SM of the persistent FP32 grid. These launches are bound by HBM or L2. Beyond about 2e7 points
// (input and output exceed L2) more resident CTAs, each keeping S windows in flight, make them slower: over the twelve
// operators at 16384^2, 650 Gpts/s with every CTA that fits, 730 capped at 768 threads per SM, 624 at 512. Below, a
// few more keep the SMs busier (768 / 1024 / 1536 threads, us): 1024^2 58 / 50 / 50, 2048^2 121 / 113 / 115, 4096^2
// 317 / 310 / 313.
inline int f32_threads_per_sm(const StencilArgs& a) { return (double)a.nx * a.rows < 2e7 ? 1024 : 768; }

// CTAs of a persistent launch: those that fit, at most one per tile, under the test cap.
inline int persistent_grid(int tiles_total, int per_sm) {
    const int grid = std::min(tiles_total, per_sm * sm_count());
    const int cap = persistent_grid_cap();
    return cap > 0 ? std::min(grid, cap) : grid;
}

// Launch with programmatic stream serialization: the kernel may start before the previous kernel of the stream has
// ended and waits for it itself (launch_wait). Each CTA allows that when its first warp has computed its last tile:
// 256^2, twelve FP64 operators in stream order, 99 us when allowed from the kernel's start, 56 us from the last tile's
// start, 49 us so (116 us without, and with the former set-up and tiles); 4096^2 FP32 in four tiles: 352, 322, 316 and
// 343 us. Any earlier, the next launch's CTAs take the room beside the running ones, several on one SM and none on
// another: a 33-point Y window at 512^2 28.3 us against 19.7.
template <typename... P, typename... A>
cudaError_t launch_overlapped(void (*kern)(P...), int grid, dim3 block, size_t smem, cudaStream_t s, const A&... args) {
    cudaLaunchAttribute attr;
    attr.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    attr.val.programmaticStreamSerializationAllowed = 1;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = s;
    cfg.attrs = &attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kern, args...);
}

// cp.async path, for every geometry whose window fits shared memory: as many ring stages as leave two CTAs per SM,
// at least one.
template <typename T, int TW, int TH, int RPT, int VEC, int MODE>
cudaError_t launch_async_mode(const StencilArgs& a, cudaStream_t s) {
    TileGeom<T, TW, TH> g(a);
    auto kern = stencil_async_kernel<T, TW, TH, RPT, VEC, MODE>;
    const size_t stage = async_stage_bytes<T>(g.SR, g.SW);
    const size_t limit = smem_optin_limit();
    int stages = kAsyncStages;
    while (stages > 1 && 2 * (stages * stage + g.coef_bytes(a)) > limit) --stages;
    const size_t smem = stages * stage + g.coef_bytes(a) + 16;
    cudaError_t e = ensure_smem(kern, smem);
    if (e != cudaSuccess) return e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, (TW / VEC) * (TH / RPT), smem);
    if (e != cudaSuccess) return e;
    if (per_sm < 1) return cudaErrorInvalidConfiguration;
    const int tiles_x = (a.nx + TW - 1) / TW;
    const int tiles_total = tiles_x * ((a.rows + TH - 1) / TH);
    return launch_overlapped(kern, persistent_grid(tiles_total, per_sm), dim3(TW / VEC, TH / RPT), smem, s, a, tiles_x,
                             tiles_total, stages);
}

// TMA path: returns cudaErrorNotSupported (without launching) when the geometry does not allow it.
template <typename T, int TW, int TH, int RPT, int VEC, int S, int MODE, bool WRAP, bool KEEP>
cudaError_t launch_tma_mode(const StencilArgs& a, cudaStream_t s) {
    TileGeom<T, TW, TH> g(a);
    // One box per window: at most 256 columns and 256 rows; rows 16-byte aligned (global address and stride
    // rules of cuTensorMapEncodeTiled).
    if (!a.vec_ok || g.SW > 256 || g.SR > 256) return cudaErrorNotSupported;
    TmaMaps maps;
    memset(&maps, 0, sizeof(maps));
    if (!encode_rows_map<T>(&maps.win, a.in, a.nx, a.rows, g.SW, g.SR)) return cudaErrorNotSupported;
    // periodic in x: wrap-around boxes of the LP / RP edge columns (x = nx - LP and x = 0 are 16-byte
    // aligned: rows are, and LP, RP are whole 16-byte units)
    const int wl_bytes = WRAP ? g.wrap_l_bytes(a) : 0, wr_bytes = WRAP ? g.wrap_r_bytes(a) : 0;
    if (wl_bytes && !encode_rows_map<T>(&maps.wrap_l, a.in, a.nx, a.rows, g.LP, g.SR)) return cudaErrorNotSupported;
    if (wr_bytes && !encode_rows_map<T>(&maps.wrap_r, a.in, a.nx, a.rows, g.RP, g.SR)) return cudaErrorNotSupported;
    const size_t stage_bytes = round_up_int((int)((size_t)g.SR * g.SW * sizeof(T)), 128);
    const size_t smem = S * (stage_bytes + wl_bytes + wr_bytes) + g.coef_bytes(a) +
                        256;   // 128 bytes of alignment slack for the ring base + tail padding
    auto kern = stencil_tma_kernel<T, TW, TH, RPT, VEC, S, MODE, WRAP, KEEP>;
    cudaError_t e = ensure_smem(kern, smem);
    if (e != cudaSuccess) return e == cudaErrorInvalidConfiguration ? cudaErrorNotSupported : e;
    int per_sm = 0;
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, (TW / VEC) * (TH / RPT), smem);
    if (e != cudaSuccess || per_sm < 1) return cudaErrorNotSupported;
    // The FP64 launches, bound by the FP64 pipe, keep every CTA that fits (a 768 cap cost them 0.3%).
    if (sizeof(T) == 4) per_sm = std::min(per_sm, std::max(1, f32_threads_per_sm(a) / ((TW / VEC) * (TH / RPT))));
    const int tiles_x = (a.nx + TW - 1) / TW;
    const int tiles_total = tiles_x * ((a.rows + TH - 1) / TH);
    return launch_overlapped(kern, persistent_grid(tiles_total, per_sm), dim3(TW / VEC, TH / RPT), smem, s, maps, a,
                             tiles_x, tiles_total);
}

// The instantiation that keeps or skips zero weights: FP32 shapes only.
template <typename T, int TW, int TH, int RPT, int VEC, int S, int MODE, bool WRAP>
cudaError_t launch_tma_zeros(const StencilArgs& a, cudaStream_t s) {
    if constexpr (sizeof(T) == 4 && MODE >= MODE_FIRST_SHAPE)
        if (a.keep_zeros) return launch_tma_mode<T, TW, TH, RPT, VEC, S, MODE, WRAP, true>(a, s);
    return launch_tma_mode<T, TW, TH, RPT, VEC, S, MODE, WRAP, false>(a, s);
}

// The instantiation with or without the wrap-around boxes; the Y shapes have no columns to wrap.
template <typename T, int TW, int TH, int RPT, int VEC, int S, int MODE>
cudaError_t launch_tma_wrap(const StencilArgs& a, cudaStream_t s, bool wrap) {
    if constexpr (MODE >= 5 && MODE <= 7) {
        return launch_tma_zeros<T, TW, TH, RPT, VEC, S, MODE, false>(a, s);
    } else {
        return wrap ? launch_tma_zeros<T, TW, TH, RPT, VEC, S, MODE, true>(a, s)
                    : launch_tma_zeros<T, TW, TH, RPT, VEC, S, MODE, false>(a, s);
    }
}

// The kernel mode of a launch.
inline int launch_mode(const StencilArgs& a) {
    return (variant_is_fun(a.variant) && !a.pre) ? (int)MODE_FUN : shape_mode(a.H, a.L, a.V, a.T);
}

template <typename T, int TW, int TH, int RPT, int VEC, int S>
cudaError_t launch_tma(const StencilArgs& a, cudaStream_t s) {
    const bool wrap = a.wrap_x && (a.L > 0 || a.R > 0);
    switch (launch_mode(a)) {
    case MODE_FUN: return launch_tma_wrap<T, TW, TH, RPT, VEC, S, MODE_FUN>(a, s, wrap);
    case 2: return launch_tma_wrap<T, TW, TH, RPT, VEC, S, 2>(a, s, wrap);
    case 3: return launch_tma_wrap<T, TW, TH, RPT, VEC, S, 3>(a, s, wrap);
    case 4: return launch_tma_wrap<T, TW, TH, RPT, VEC, S, 4>(a, s, wrap);
    case 5: return launch_tma_wrap<T, TW, TH, RPT, VEC, S, 5>(a, s, wrap);
    case 6: return launch_tma_wrap<T, TW, TH, RPT, VEC, S, 6>(a, s, wrap);
    case 7: return launch_tma_wrap<T, TW, TH, RPT, VEC, S, 7>(a, s, wrap);
    case 8: return launch_tma_wrap<T, TW, TH, RPT, VEC, S, 8>(a, s, wrap);
    case 9: return launch_tma_wrap<T, TW, TH, RPT, VEC, S, 9>(a, s, wrap);
    default: return launch_tma_wrap<T, TW, TH, RPT, VEC, S, MODE_LIST>(a, s, wrap);
    }
}

template <typename T, int TW, int TH, int RPT, int VEC>
cudaError_t launch_async(const StencilArgs& a, cudaStream_t s) {
    switch (launch_mode(a)) {
    case MODE_FUN: return launch_async_mode<T, TW, TH, RPT, VEC, MODE_FUN>(a, s);
    case 2: return launch_async_mode<T, TW, TH, RPT, VEC, 2>(a, s);
    case 3: return launch_async_mode<T, TW, TH, RPT, VEC, 3>(a, s);
    case 4: return launch_async_mode<T, TW, TH, RPT, VEC, 4>(a, s);
    case 5: return launch_async_mode<T, TW, TH, RPT, VEC, 5>(a, s);
    case 6: return launch_async_mode<T, TW, TH, RPT, VEC, 6>(a, s);
    case 7: return launch_async_mode<T, TW, TH, RPT, VEC, 7>(a, s);
    case 8: return launch_async_mode<T, TW, TH, RPT, VEC, 8>(a, s);
    case 9: return launch_async_mode<T, TW, TH, RPT, VEC, 9>(a, s);
    default: return launch_async_mode<T, TW, TH, RPT, VEC, MODE_LIST>(a, s);
    }
}

}  // namespace custen
