// Batched tridiagonal line solves (definitions in tri.cu).
#pragma once

#include <cuda_runtime.h>

#include "device.cuh"

namespace fb {

constexpr int kYLines = 2;  // contiguous lines per block
constexpr int kYWarps = 2;  // warps per contiguous line
constexpr int kYPoissonWarps = 4;  // warps per line of the Poisson mode solves
constexpr int kZLines = 4;  // strided lines per block (one warp each)

constexpr int kWinMax = 24;  // longest truncation window of the windowed helsolve

// Rows of the windowed helsolve's tiles (32 columns wide, two fields): 64, or 32
// where 64 would leave SMs without a tile.  Measured with 64 / 32 rows: 48 x 32
// 6.3 / 5.4 us, 384 x 256 (96 tiles of 64 rows) 6.7 / 5.8 us; with 192 tiles (512 x
// 384) 64 rows are the faster ones.
inline int win_tile_rows(int n2m, int n3m, int sms = 148) {
    return 2 * ((n2m + 31) / 32) * ((n3m + 63) / 64) < sms ? 32 : 64;
}

cudaError_t scan_configure();
// blocks: forward recurrences in blocks (the split-precision Poisson form)
void launch_win_helsolve(const Dev &d, const SubDev &s, cudaStream_t st, bool blocks);
void launch_scan_helsolve(const Dev &d, const SubDev &s, cudaStream_t st);
// rmax (may be null): n2m row maxima of |hmn| (over the modes) accumulated for
// the INT8 digit cut; one_warp: one warp per mode at any size (the
// split-precision form)
void launch_scan_poisson(const Dev &d, cudaStream_t st, double *rmax = nullptr, bool one_warp = false);
void glaunch_win_helsolve(const Group &g, int n, cudaStream_t st, bool blocks);  // substep n (0-based)
void glaunch_scan_poisson(const Group &g, cudaStream_t st, bool one_warp = false);

}  // namespace fb
