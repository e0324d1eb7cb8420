// Shared declarations of the Cahn-Hilliard ADI kernels (ch_solver.cu) for the batch and server hosts.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <string>
#include <vector>

namespace custen {
namespace ch {

constexpr int BLK = 32;   // rows / columns per work item; n must be a multiple of 32

// Per-grid descriptor (device).
struct GridDev {
    double* buf[2];       // the two field buffers: cCurr = buf[parity], cOld = buf[parity ^ 1]
    double* tmp;          // n x n work field (rhs, then the line solutions)
    double* ends;         // 8 n cuts values: closure amplitudes of the rows (four per row, segment by segment), then
                          // of the columns; may lie in hbuf, which the sweeps do not read
    double* hbuf;         // n x n h of the two-pass right-hand side (null in the allocation-free step)
    const double* tab;    // solver table for n (layout below)
    int n;
    int general;          // 1: general sweeps (banded factors) instead of the factored ones
    int cuts;             // segments per line, 1 or 2 (line_cuts)
    int pad;
};

// Table layout for one n, all double. First kTabParams parameters:
enum : int {
    TAB_SLIN = 0,    // sigma_lin, weight of the explicit biharmonic
    TAB_SNL = 1,     // sigma_nl, weight of the explicit Laplacian of c^3 - c
    TAB_NP1 = 2,     // -p1, -p2 of the causal factor P(z) = 1 + p1 / z + p2 / z^2 of the line operator
    TAB_NP2 = 3,
    TAB_KAPPA = 4,   // (2/3) / G^2: the two line operators are G P(z) P(1/z), the right-hand side is in units of 2/3
    TAB_REACH = 5,   // entries of f1, f2 that are not negligible (the bits of an integer)
    TAB_MID = 6,     // 2 x 4: the other chain's two values next to the middle from (own, own, other, other) ends
    TAB_CLOSE = 14,  // 2 x 2: closure amplitudes from the two values at the outer end of the neighbouring segment
    TAB_CLOSE2 = 18, // 2 x 2 for each of two segments: from those of the segment itself, once around the ring
    TAB_BAND_LO = 26,   // general grids: first and end chunk of 16 entries in which the factors are constant (the bits of
    TAB_BAND_HI = 27,   // integers)
    TAB_RATIO = 28,  // sigma_lin / sigma_nl and 3/2 sigma_nl: the FP64 right-hand side's units (h in sigma_nl, the sum in 2/3)
    TAB_LAP = 29,
    TAB_OUT = 30,    // general grids: the unit of the right-hand side, 2/3 in FP64 and 1 over FP32 stencils
    kTabParams = 32
};
// then f1[n], f2[n] (homogeneous solutions, as many entries used as the first segment has), or for a general grid (m = n - 2) the banded factors
//   [0, m) ds  [m, 2m) dl  [2m, 3m) rd = 1/diag  [3m, 4m) du  [4m, 5m) dw   (zero-padded: ds[0] = ds[1] = dl[0]
//   = 0, du[m-1] = 0, dw[m-2] = dw[m-1] = 0)  [5m, 6m) inv1  [6m, 7m) inv2   border columns of the cyclic
//   correction  [7m, 7m+4) omega  [7m+4, 7m+8) a, b, d, e
__host__ __device__ inline int tab_size(int n) { return kTabParams + 7 * (n - 2) + 8; }

struct Item {
    int grid;
    int block;   // right-hand side and update: 32 x 32 block index (row-major over the grid); sweeps: row / column block
                 // times cuts, plus the segment (segments of a block are neighbours in the list)
};

// Sum of `count` values into out->sum (zeroed before the first call; one sum at a time on a scratch).
constexpr int kMassBlocks = 256, kMassSpan = 2048;
struct MassScratch {
    double sum;
    unsigned int arrived;
    double part[kMassBlocks][2];
};
cudaError_t launch_ch_mass(const double* f, long long count, MassScratch* out, cudaStream_t s);

// Kernel configuration of a step: warps per right-hand-side CTA (of pass 1), one or two passes, and where the x sweep's
// closure is applied. Every configuration computes the same values; the batch tuner times them.
struct ChConfig {
    int rhs_warps;   // 1, 2, 4 or 8
    int warps2;      // of the right-hand side in two passes, warps per CTA of pass 2; 0: one pass (no h buffer)
    int close;       // x closure: 1 as the y sweep reads, 2 in a kernel of its own, 0 by the number of chains
};
constexpr int kChOneGrid = 12;        // needs no h buffer (the allocation-free step)
constexpr int kChBatchDefault = 20;   // batches and the server (they allocate the h buffer)
constexpr int kChConfigs = 22;
ChConfig ch_config(int index);   // 0 .. kChConfigs-1
void config_name(const ChConfig& c, char* name, size_t len);

// The work lists of a set of grids, on the device: 32 x 32 blocks, and line blocks with those of general grids last.
struct ChWork {
    const GridDev* grids;
    const Item* blocks;
    const Item* lines;
    const CUtensorMap* maps;   // two per grid (sweep_maps)
    unsigned int* arrived;     // one per line block entry, zero between sweeps
    int n_blocks, n_lines, n_general;   // n_lines counts the line entries of all grids, n_general the general ones'
    int n_whole;                        // entries that are whole lines (one segment)
};
int ch_launches_per_step(const ChConfig& c, const ChWork& w, int sms);

// One step of every grid of the work lists: right-hand side (one or two passes), x sweep, y sweep, update.
cudaError_t launch_ch_step(const ChConfig& c, bool rhs_fp32, const ChWork& w, int parity, int sms, cudaStream_t s);

// Whether an n x n grid takes the general sweeps (GridDev::general).
bool line_is_general(int n, double lx, double gamma, double dt_factor, bool rhs_fp32);

// Segments per line of a grid, and the length of the first: whole blocks, at least half of the line.
int line_cuts(int n, bool general);
__host__ __device__ inline int first_segment(int n, int cuts) { return cuts == 2 ? (n / BLK + 1) / 2 * BLK : n; }

// Tensor maps of an n x n work field for the sweeps (two); false when they cannot be encoded.
bool sweep_maps(CUtensorMap maps[2], double* tmp, int n);

// Solver table of an n x n grid (tab_size(n) doubles) built on the host.
std::vector<double> build_table(int n, double lx, double gamma, double dt_factor, bool general, bool rhs_fp32);

}  // namespace ch
}  // namespace custen
