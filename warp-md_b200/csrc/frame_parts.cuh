// frame_parts.cuh -- pieces shared by the per-frame forward kernels: the sums of
// a tile of gathered atoms by one warp, and a frame's outputs from its sums.
#pragma once

#include <cstdint>

#include "device_util.cuh"
#include "qcp.cuh"
#include "wmd_internal.h"

namespace wmd {

enum Mode : int { kFwdFit = 0, kFwdRaw = 1, kBwd = 2, kFwdW = 3 };

// Frame f's outputs from its 15 sums (raw: tot[0] alone); one thread.
__device__ __forceinline__ void finish_totals(const FrameLaunch& L, int64_t f, const double (&tot)[16], int mode) {
  const double n = (double)L.ref.n_sel;
  if (mode == kFwdRaw) {
    // tot[0] = sum |x - y|^2 accumulated directly
    const double msd = n > 0 ? tot[0] / n : 0.0;
    if (L.out.rmsd) L.out.rmsd[f] = sqrt(msd);
    return;
  }
  const double inv_n = 1.0 / n;
  const double sx[3] = {tot[0], tot[1], tot[2]};
  const double sxx = tot[3] + tot[4] + tot[5];
  double h[9];
#pragma unroll
  for (int a = 0; a < 3; ++a)
#pragma unroll
    for (int b = 0; b < 3; ++b) h[a * 3 + b] = tot[6 + a * 3 + b] - sx[a] * ref_sum_c(L.ref, b) * inv_n;
  const double gx = sxx - (sx[0] * sx[0] + sx[1] * sx[1] + sx[2] * sx[2]) * inv_n;
  const double gy = ref_gy(L.ref);
  const QcpOut q = qcp_lambda(h, 0.5 * (gx + gy));
  const double rmsd = sqrt(msd_from(gx, gy, q.lambda, n));
  if (L.out.rmsd) L.out.rmsd[f] = rmsd;
  if (L.refine && (L.out.rmsd || L.out.stats) && rmsd < kRefineScale * (gx + gy) * inv_n) {
    // near-zero RMSD: queue the frame for the explicit residual pass
    const unsigned slot = atomicAdd(L.refine_count, 1u);
    double* rec = L.refine + (size_t)slot * kStatDoubles;
    rec[0] = (double)f;
    rec[1] = sx[0] * inv_n; rec[2] = sx[1] * inv_n; rec[3] = sx[2] * inv_n;
#pragma unroll
    for (int e = 0; e < 9; ++e) rec[4 + e] = h[e];
    rec[13] = q.lambda;
  }
  if (L.out.stats) {
    double* st = L.out.stats + f * kStatDoubles;
    st[0] = sx[0] * inv_n; st[1] = sx[1] * inv_n; st[2] = sx[2] * inv_n;
#pragma unroll
    for (int e = 0; e < 9; ++e) st[3 + e] = h[e];
    st[12] = q.lambda; st[13] = rmsd; st[14] = n; st[15] = gx + gy;
  }
  if (L.out.cov) {
#pragma unroll
    for (int e = 0; e < 9; ++e) L.out.cov[f * 9 + e] = (float)h[e];
  }
  if (L.out.sum_x2) L.out.sum_x2[f] = (float)gx;
  if (L.out.sum_y2) L.out.sum_y2[f] = (float)gy;
}

// A frame's superposition onto the reference from its (weighted) sums: r starts as
// the identity and stays so with norotate or zero total weight; t = c_y - R c_x.
__device__ __forceinline__ void transform_from_totals(const RefInfo& ref, const double* tot, int norotate,
                                                      double (&r)[9], double (&t)[3]) {
  const double W = ref.wsum;
  double cx[3] = {0, 0, 0}, cy[3] = {0, 0, 0};
  if (W > 0.0 || W < 0.0) {
    const double inv_w = 1.0 / W;
    cx[0] = tot[0] * inv_w; cx[1] = tot[1] * inv_w; cx[2] = tot[2] * inv_w;
    for (int c = 0; c < 3; ++c) cy[c] = ref_mean(ref, c);
    if (!norotate) {
      double h[9];
      for (int a = 0; a < 3; ++a)
        for (int b = 0; b < 3; ++b) h[a * 3 + b] = tot[6 + a * 3 + b] - cx[a] * ref_sum_c(ref, b);
      const double gx = tot[3] + tot[4] + tot[5] - (tot[0] * cx[0] + tot[1] * cx[1] + tot[2] * cx[2]);
      const QcpOut q = qcp_lambda(h, 0.5 * (gx + ref_gy(ref)));
      rotation_from_qcp(h, q.lambda, r);
    }
  }
  for (int i = 0; i < 3; ++i) t[i] = cy[i] - (r[i * 3 + 0] * cx[0] + r[i * 3 + 1] * cx[1] + r[i * 3 + 2] * cx[2]);
}

// Positions per lane whose loads are in flight together in gather_item.
constexpr int kGatherDepth = 4;

// An atom's 12 bytes cost two loads, not three: an 8-byte load of the pair
// that starts on an 8-byte boundary (x,y or y,z) and a 4-byte load of the
// other coordinate.
__device__ __forceinline__ void load_xyz(const float* p, float& x, float& y, float& z) {
  const bool odd = (reinterpret_cast<uintptr_t>(p) & 7u) != 0;
  const float2 pr = __ldg(reinterpret_cast<const float2*>(p + (odd ? 1 : 0)));
  const float s = __ldg(p + (odd ? 0 : 2));
  x = odd ? s : pr.x;
  y = odd ? pr.x : pr.y;
  z = odd ? pr.y : s;
}

// One warp's sums over list positions [a0, a1) of a frame (L.sel's atoms, or the
// positions themselves; kDense: there is no list), in sub-chunks of 32 x kGatherJ positions with all of a
// sub-chunk's loads in flight before any use.  Returned as
// warp_reduce_scatter16 leaves them: lane 2e holds sum e.
template <int STRIDE, int MODE, int kGatherJ = kGatherDepth, bool kDense = false>
__device__ __forceinline__ double gather_item(const FrameLaunch& L, const float* __restrict__ frame, int64_t a0,
                                              int64_t a1, const double (&mean)[3], int lane) {
  double acc[16];
#pragma unroll
  for (int e = 0; e < 16; ++e) acc[e] = 0.0;
  // the next sub-chunk's indices are loaded a sub-chunk ahead, so that its atoms' loads
  // do not wait for them
  uint32_t next[kGatherJ];
  auto fetch = [&](int64_t c0) {
#pragma unroll
    for (int j = 0; j < kGatherJ; ++j) {
      const int64_t k = c0 + lane + 32 * j;
      if (!kDense && L.sel && k < a1) next[j] = __ldg(L.sel + k);
    }
  };
  fetch(a0);
#pragma unroll 1
  for (int64_t c0 = a0; c0 < a1; c0 += 32 * kGatherJ) {
    float x[kGatherJ][3];
    double y[kGatherJ][3];
    float wt[MODE == kFwdW ? kGatherJ : 1];
#pragma unroll
    for (int j = 0; j < kGatherJ; ++j) {
      const int64_t k = c0 + lane + 32 * j;
      if (k < a1) {
        int64_t idx = !kDense && L.sel ? (int64_t)next[j] : k;
        if (!kDense && idx >= L.n_atoms) {  // bad device-side selection: report, read atom 0
          atomicOr(L.status, kStatusBadIndex);
          idx = 0;
        }
        load_xyz(frame + idx * STRIDE, x[j][0], x[j][1], x[j][2]);
        const double* yp = L.ref.yc + k * 3;
        y[j][0] = __ldg(yp); y[j][1] = __ldg(yp + 1); y[j][2] = __ldg(yp + 2);
        if (MODE == kFwdW) wt[MODE == kFwdW ? j : 0] = __ldg(L.ref.w + k);
      } else {
        x[j][0] = x[j][1] = x[j][2] = 0.f;
        y[j][0] = y[j][1] = y[j][2] = 0.0;
        if (MODE == kFwdW) wt[MODE == kFwdW ? j : 0] = 0.f;
      }
    }
    fetch(c0 + 32 * kGatherJ);
#pragma unroll
    for (int j = 0; j < kGatherJ; ++j) {
      const double x0 = x[j][0], x1 = x[j][1], x2 = x[j][2];
      if (MODE == kFwdRaw) {
        if (c0 + lane + 32 * j < a1) {
          const double d0 = x0 - (y[j][0] + mean[0]);
          const double d1 = x1 - (y[j][1] + mean[1]);
          const double d2 = x2 - (y[j][2] + mean[2]);
          acc[0] = fma(d0, d0, acc[0]);
          acc[1] = fma(d1, d1, acc[1]);
          acc[2] = fma(d2, d2, acc[2]);
        }
      } else {
        if (MODE == kFwdW) {
          const double wj = wt[MODE == kFwdW ? j : 0];
          const double u0 = wj * x0, u1 = wj * x1, u2 = wj * x2;
          acc[0] += u0; acc[1] += u1; acc[2] += u2;
          acc[3] = fma(u0, x0, acc[3]); acc[4] = fma(u1, x1, acc[4]); acc[5] = fma(u2, x2, acc[5]);
        } else {
          acc[0] += x0; acc[1] += x1; acc[2] += x2;
          acc[3] = fma(x0, x0, acc[3]); acc[4] = fma(x1, x1, acc[4]); acc[5] = fma(x2, x2, acc[5]);
        }
        acc[6] = fma(x0, y[j][0], acc[6]);  acc[7] = fma(x0, y[j][1], acc[7]);  acc[8] = fma(x0, y[j][2], acc[8]);
        acc[9] = fma(x1, y[j][0], acc[9]);  acc[10] = fma(x1, y[j][1], acc[10]); acc[11] = fma(x1, y[j][2], acc[11]);
        acc[12] = fma(x2, y[j][0], acc[12]); acc[13] = fma(x2, y[j][1], acc[13]); acc[14] = fma(x2, y[j][2], acc[14]);
      }
    }
  }
  if (MODE == kFwdRaw) {
    acc[0] += acc[1] + acc[2];
    acc[1] = acc[2] = 0.0;
  }
  return warp_reduce_scatter16(acc);
}

}  // namespace wmd
