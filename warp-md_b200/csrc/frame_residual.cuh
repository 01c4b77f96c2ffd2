// frame_residual.cuh -- a frame's RMSD from explicit residuals, and the gradient's
// rotation record, shared by the streaming and the one-CTA-per-frame kernels.
#pragma once

#include <cstdint>

#include "qcp.cuh"
#include "wmd_internal.h"

namespace wmd {

// The RMSD of a queued frame (near zero) from explicit residuals
// sum |R (x_k - x_bar) - (y_k - y_bar)|^2 in FP64, as the reference's
// rmsd_aligned_selected computes every frame (plan.rs:1223-1247), with R from
// the QCP eigenvector.  rec: finish_totals' record; red: 8 doubles of shared
// memory.  Called by a whole CTA of 256 threads.
template <int STRIDE>
__device__ __forceinline__ void residual_rmsd(const FrameLaunch& L, const double* rec, double* red) {
  __shared__ double sh_r[12];
  const int64_t n_sel = L.ref.n_sel;
  const double inv_n = 1.0 / (double)n_sel;
  if (threadIdx.x == 0) {
    double h[9], r[9];
    for (int e = 0; e < 9; ++e) h[e] = rec[4 + e];
    rotation_from_qcp(h, rec[13], r);
    for (int e = 0; e < 9; ++e) sh_r[e] = r[e];
    sh_r[9] = rec[1]; sh_r[10] = rec[2]; sh_r[11] = rec[3];
  }
  __syncthreads();
  const int64_t f = (int64_t)rec[0];
  double R[9], c[3];
  for (int e = 0; e < 9; ++e) R[e] = sh_r[e];
  c[0] = sh_r[9]; c[1] = sh_r[10]; c[2] = sh_r[11];
  const double my0 = ref_sum_c(L.ref, 0) * inv_n, my1 = ref_sum_c(L.ref, 1) * inv_n,
               my2 = ref_sum_c(L.ref, 2) * inv_n;
  const float* frame = L.coords + (size_t)f * L.n_atoms * STRIDE;
  double acc = 0.0;
  for (int64_t k = threadIdx.x; k < n_sel; k += blockDim.x) {
    int64_t atom = L.sel ? (int64_t)L.sel[k] : k;
    if (atom >= L.n_atoms) atom = 0;  // reported by the forward kernel
    const float* p = frame + atom * STRIDE;
    const double d0 = (double)p[0] - c[0], d1 = (double)p[1] - c[1], d2 = (double)p[2] - c[2];
    const double* y = L.ref.yc + k * 3;
    const double r0 = R[0] * d0 + R[1] * d1 + R[2] * d2 - (y[0] - my0);
    const double r1 = R[3] * d0 + R[4] * d1 + R[5] * d2 - (y[1] - my1);
    const double r2 = R[6] * d0 + R[7] * d1 + R[8] * d2 - (y[2] - my2);
    acc += r0 * r0 + r1 * r1 + r2 * r2;
  }
  for (int o = 16; o; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double t = 0.0;
    for (int w = 0; w < 8; ++w) t += red[w];
    const double rmsd = sqrt(t * inv_n);
    if (L.out.rmsd) L.out.rmsd[f] = rmsd;
    if (L.out.stats) L.out.stats[f * kStatDoubles + 13] = rmsd;
  }
}

// Frame f's rotation record for the gradient: R from the QCP eigenvector of the
// stored H, the centroid and the scale dL/drmsd / (n rmsd).
__device__ __forceinline__ void frame_rotation(const double* stats, const float* grad_rmsd, const double* grad_f64,
                                               int64_t grad_stride, int64_t f, double* o) {
  const double* st = stats + f * kStatDoubles;
  double h[9], r[9];
  for (int e = 0; e < 9; ++e) h[e] = st[3 + e];
  rotation_from_qcp(h, st[12], r);
  const double rmsd = st[13], n = st[14];
  const double g = grad_f64 ? grad_f64[f * grad_stride] : grad_rmsd ? (double)grad_rmsd[f] : 1.0;
  const double scale = (rmsd > 0.0 && n > 0.0) ? g / (n * rmsd) : 0.0;
  for (int e = 0; e < 9; ++e) o[e] = r[e];
  o[9] = st[0]; o[10] = st[1]; o[11] = st[2];
  o[12] = scale; o[13] = 0; o[14] = 0; o[15] = 0;
}

}  // namespace wmd
