// pair_hist.cuh -- the per-thread FP32 pair histogram shared by the planar
// and spherical pair kernels: layout [bin][quantity][thread] in shared
// memory (a warp's read-modify-writes hit 32 distinct banks), folded into FP64
// every ~4096 sources.
#pragma once
#include <cuda_runtime.h>

#include "tpcf_internal.cuh"

namespace tpcf {

template <int QA, int NC>
__device__ __forceinline__ void hist_add(float* hcol, int bin, const float* v) {
  float* h = hcol + bin * (QA * NC);
#pragma unroll
  for (int q = 0; q < QA; ++q) h[q * NC] += v[q];
}

// Fold this warp's 32 histogram columns into its FP64 sums (times the lens
// factors val*w or w) and, when lens_col is set, each lane's per-lens FP64
// column (zeroed before the launch; a lens's pairs between two folds fall in
// few bins, so only its non-zero cells are added, as fire-and-forget FP64
// reductions: each column has one writer, so the adds land in program order
// and the result is deterministic, and no load latency is waited for); then
// clear the columns.  Called by all lanes of the warp.
template <int QA, int BT>
__device__ __forceinline__ void warp_fold(const float* hist, float* hcol, double* wsum, const double* fvw,
                                          const double* fw, int nb, double* lens_col, size_t lens_stride, int warp,
                                          int lane) {
  __syncwarp();
  if (lens_col) {
    for (int q = 0; q < kQ; ++q) {
      const int qa = (q == QK && QA == 5) ? QW : q;
      for (int b = 0; b < nb; ++b) {
        const float v = hcol[(b * QA + qa) * BT];
        if (v != 0.f) atomicAdd(lens_col + (size_t)(q * nb + b) * lens_stride, (double)v);
      }
    }
  }
  const int cb = warp * 32;
  for (int e = lane; e < kQ * nb; e += 32) {
    const int q = e / nb, b = e - q * nb;
    if (q == QK && QA == 5) continue;  // K == w: copied from the w row at item end
    const float* row = hist + (b * QA + q) * BT + cb;
    double s = 0.0;
    if (q == QN) {
      for (int l = 0; l < 32; ++l) s += (double)row[(l + lane) & 31];
    } else {
      const double* f = ((q == QGT || q == QGX) ? fvw : fw) + cb;
      for (int l = 0; l < 32; ++l) {
        const int c = (l + lane) & 31;
        s = fma((double)row[c], f[c], s);
      }
    }
    wsum[e] += s;
  }
  __syncwarp();
  for (int e = 0; e < nb * QA; ++e) hcol[e * BT] = 0.f;
}

}  // namespace tpcf
