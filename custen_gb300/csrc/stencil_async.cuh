// cp.async-staged, persistent stencil kernel (sm_103a) for the geometries TMA cannot take: rows that are not 16-byte
// aligned (an odd number of doubles, a number of floats that is not a multiple of four, an unaligned base) and windows
// of more than 256 columns or rows.
//
// Like the TMA kernel (stencil_tma.cuh) each CTA walks the tiles tile = blockIdx.x + k * gridDim.x with the next
// windows in flight in a shared-memory ring and runs the same compute stage on them; the elements are copied one by
// one (8 or 4 bytes, the alignment such rows have), a warp per window row, from the launch's rows or its halo rows,
// wrapped (periodic) or zero-filled where a variant has no value. Windows of nine weights or more are
// bound by the FP64 pipe (77 to 85%), shorter ones by issue slots and the copies themselves (47%). Measured, 1999 x 1501, FP64 (FP32): 9-point X 57 (12) us, 5 x 5 with zeros 81 (14), dense
// 3 x 3 58 (12); the kernel before it, one tile per CTA staged with plain loads and every window through the generic
// weight list, took 70 (25), 96 (32) and 70 (25). On aligned rows (2000 x 1500) the TMA kernel takes 50, 70 and 50.
#pragma once

#include "stencil_kernel.cuh"

namespace custen {

constexpr int kAsyncStages = 3;

template <typename T>
__host__ __device__ inline size_t async_stage_bytes(int SR, int SW) {
    return ((size_t)SR * SW * sizeof(T) + 15) / 16 * 16;
}

// One element into shared memory: copied, or zero when src_bytes is 0.
template <typename T>
__device__ __forceinline__ void copy_element(T* dst, const T* src, int src_bytes) {
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2, %3;\n" ::"r"(d), "l"(src), "n"((int)sizeof(T)), "r"(src_bytes)
                 : "memory");
}

// Start the copies of one tile window and commit them as one group.
template <typename T, int TW, int TH, int NT>
__device__ __forceinline__ void issue_elements(const StencilArgs& a, T* tile, const TileGeom<T, TW, TH>& g, int x0, int y0,
                                               int tid) {
    const int lane = tid & 31;
    for (int r = tid >> 5; r < g.SR; r += NT / 32) {
        const T* row = launch_row<T>(a, y0 - a.T + r);
        T* dst = tile + r * g.SW;
        for (int c = lane; c < g.SW; c += 32) {
            int x = x0 - g.LP + c;
            if (a.wrap_x) x = x < 0 ? x + a.nx : (x >= a.nx ? x - a.nx : x);
            const bool has = row != nullptr && x >= 0 && x < a.nx;
            if (!in_bounds((long long)r * g.SW + c, 0, (long long)g.SR * g.SW)) continue;
            copy_element(dst + c, has ? row + x : reinterpret_cast<const T*>(a.in), has ? (int)sizeof(T) : 0);
        }
    }
    asm volatile("cp.async.commit_group;\n" ::: "memory");
}

template <typename T, int TW, int TH, int RPT, int VEC, int MODE>
__global__ void __launch_bounds__((TW / VEC) * (TH / RPT), min_blocks_for((TW / VEC) * (TH / RPT), MODE == MODE_FUN))
stencil_async_kernel(const __grid_constant__ StencilArgs a, int tiles_x, int tiles_total, int stages) {
    constexpr int NTX = TW / VEC;
    constexpr int NT = NTX * (TH / RPT);
    static_assert(NT % 32 == 0, "whole warps");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    TileGeom<T, TW, TH> g(a);
    const size_t stage = async_stage_bytes<T>(g.SR, g.SW);
    unsigned char* after = smem_raw + stages * stage;
    T* coef_s = reinterpret_cast<T*>(after);
    int* list_off = reinterpret_cast<int*>(after + g.list_off(a));
    T* list_w = reinterpret_cast<T*>(after + g.listw_off(a));
    const int tid = threadIdx.x + threadIdx.y * NTX;
    const Zeros<T> zeros;
    launch_wait();
    auto window = [&](int k) { return reinterpret_cast<T*>(smem_raw + (size_t)k * stage); };
    // Group k of the thread holds the copies of the CTA's k-th tile (empty past the last), so the group to await is
    // always the one `stages - 2` groups back.
    auto issue = [&](int it, int k) {
        const int t = blockIdx.x + it * gridDim.x;
        if (t < tiles_total) issue_elements<T, TW, TH, NT>(a, window(k), g, (t % tiles_x) * TW, (t / tiles_x) * TH, tid);
        else asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    for (int k = 0; k + 1 < stages; ++k) issue(k, k);
    const int nlist = stage_coefficients<T, NT>(a, coef_s, list_off, list_w, g.SW, tid, MODE == MODE_FUN,
                                                MODE >= MODE_FIRST_SHAPE);  // syncs
    int cur = 0, next = stages - 1;   // stages of this tile and of the one to fetch (stages - 1 tiles ahead)
    for (int it = 0;; ++it) {
        const int t = blockIdx.x + it * gridDim.x;
        if (t >= tiles_total) break;
        if (stages == 1) {
            __syncthreads();   // every thread is done with the stage
            issue(it, 0);
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            __syncthreads();
        } else {
            if (stages == 2) asm volatile("cp.async.wait_group 0;\n" ::: "memory");
            else asm volatile("cp.async.wait_group 1;\n" ::: "memory");
            __syncthreads();   // the window is complete, and every thread is done with the previous tile's stage
            issue(it + stages - 1, next);
        }
        T* tile = window(cur);
        const int x0 = (t % tiles_x) * TW, y0 = (t / tiles_x) * TH;
        if (a.pre) {
            apply_cube<T, NT>(tile, g.SR * g.SW, tid, zeros);
            __syncthreads();
        }
        const bool all_write = tile_all_write(a, x0, x0 + TW, a.row0 + y0, a.row0 + y0 + TH);
        compute_tile<T, TW, TH, RPT, VEC, MODE, false>(a, tile, coef_s, list_off, list_w, nlist, g, x0, y0, all_write, zeros);
        if (t + gridDim.x >= tiles_total) launch_dependents();   // a warp is done with the CTA's last tile
        cur = cur + 1 == stages ? 0 : cur + 1;
        next = next + 1 == stages ? 0 : next + 1;
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

}  // namespace custen
