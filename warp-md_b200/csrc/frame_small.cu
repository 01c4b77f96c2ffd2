// frame_small.cu -- per-frame RMSD and its gradient for launches too small to fill
// the GPU: one CTA per frame, everything in one launch.
//
// The streaming path takes four launches (clear the residual queue, statistics,
// finalize, residual pass), and its gradient two; at these sizes each is a few
// microseconds of latency around next to no work.  Here a frame's 8 warps sum a
// slice of its atoms each (gather_item: plain loads, any selection, stride or
// alignment), warp 0 adds them in warp order and finishes the frame
// (finish_totals), and a frame that needs the explicit residuals gets them from
// the same CTA.  Bound by that chain's latency (loads, a reduction, QCP on one
// thread), so the rule (small_frames) keeps it to launches of a wave or two.
// 64 x 250: forward 19 -> 12 us a call, RMSD under autograd with its backward
// 186 -> 168 us (launches from Python).
#include <cuda_runtime.h>

#include <cstdint>

#include "frame_parts.cuh"
#include "frame_residual.cuh"
#include "wmd_internal.h"

namespace wmd {
namespace {

constexpr int kSmallWarps = 8;
constexpr int kSmallThreads = kSmallWarps * 32;

template <int STRIDE, int MODE>
__global__ void __launch_bounds__(kSmallThreads) rmsd_small_kernel(const FrameLaunch P) {
  __shared__ double red[kSmallWarps][16];
  __shared__ double rec[kStatDoubles];
  __shared__ unsigned queued;
  FrameLaunch L = P;
  depend_wait();  // for a reference centred just before (reference.cu)
  depend_read(L.ref.yc);
  depend_read(L.ref.scal);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t n = L.ref.n_sel;
  const double mean[3] = {MODE == kFwdRaw ? ref_mean(L.ref, 0) : 0.0, MODE == kFwdRaw ? ref_mean(L.ref, 1) : 0.0,
                          MODE == kFwdRaw ? ref_mean(L.ref, 2) : 0.0};
  const int64_t f = blockIdx.x;
  const float* frame = L.coords + (size_t)f * L.n_atoms * STRIDE;
  const double v = gather_item<STRIDE, MODE>(L, frame, n * warp / kSmallWarps, n * (warp + 1) / kSmallWarps, mean, lane);
  if ((lane & 1) == 0) red[warp][lane >> 1] = v;
  if (threadIdx.x == 0) queued = 0;
  __syncthreads();
  if (warp == 0) {
    double s = 0.0, tot[16];
#pragma unroll
    for (int w = 0; w < kSmallWarps; ++w) s += red[w][lane & 15];
#pragma unroll
    for (int e = 0; e < 16; ++e) tot[e] = __shfl_sync(0xffffffffu, s, e);
    if (lane == 0) {
      FrameLaunch K = L;  // a queue of one: this frame's record stays in the CTA
      K.refine = L.align ? rec : nullptr;
      K.refine_count = &queued;
      finish_totals(K, f, tot, MODE);
    }
  }
  if (MODE != kFwdFit) return;
  __syncthreads();
  if (queued) residual_rmsd<STRIDE>(L, rec, red[0]);
}

// Gradient: a frame's atoms over gridDim.y CTAs; each re-derives the rotation
// from the forward's record (as rmsd_bwd_prologue does) while its loads are in flight.
template <int STRIDE>
__global__ void __launch_bounds__(kSmallThreads)
    rmsd_small_grad_kernel(const FrameLaunch L, const double* __restrict__ stats, const float* __restrict__ grad_rmsd,
                           const double* __restrict__ grad_f64, int64_t grad_stride) {
  __shared__ double rot[kStatDoubles];
  const int64_t f = blockIdx.x;
  const int64_t k0 = (int64_t)blockIdx.y * kSmallThreads + threadIdx.x, step = (int64_t)gridDim.y * kSmallThreads;
  const int64_t n = L.ref.n_sel;
  const float* frame = L.coords + (size_t)f * L.n_atoms * STRIDE;
  float* gframe = L.grad + (size_t)f * L.n_atoms * 3;
  int64_t atom = 0;
  float x0 = 0.f, x1 = 0.f, x2 = 0.f;
  double y0 = 0.0, y1 = 0.0, y2 = 0.0;
  auto load = [&](int64_t k) {
    atom = L.sel ? (int64_t)__ldg(L.sel + k) : k;
    if (atom >= L.n_atoms) {  // bad device-side selection: report, use atom 0
      atomicOr(L.status, kStatusBadIndex);
      atom = 0;
    }
    load_xyz(frame + atom * STRIDE, x0, x1, x2);
    const double* y = L.ref.yc + k * 3;
    y0 = __ldg(y); y1 = __ldg(y + 1); y2 = __ldg(y + 2);
  };
  if (k0 < n) load(k0);
  if (threadIdx.x == 0) frame_rotation(stats, grad_rmsd, grad_f64, grad_stride, f, rot);
  __syncthreads();
  double R[9], c[3];
#pragma unroll
  for (int e = 0; e < 9; ++e) R[e] = rot[e];
  c[0] = rot[9]; c[1] = rot[10]; c[2] = rot[11];
  const double scale = rot[12];
  for (int64_t k = k0; k < n;) {
    const double t0 = R[0] * y0 + R[3] * y1 + R[6] * y2;
    const double t1 = R[1] * y0 + R[4] * y1 + R[7] * y2;
    const double t2 = R[2] * y0 + R[5] * y1 + R[8] * y2;
    float* g = gframe + atom * 3;
    g[0] = (float)(scale * (((double)x0 - c[0]) - t0));
    g[1] = (float)(scale * (((double)x1 - c[1]) - t1));
    g[2] = (float)(scale * (((double)x2 - c[2]) - t2));
    k += step;
    if (k < n) load(k);
  }
}

}  // namespace

// Measured whole calls, one CTA per frame against the streaming path (us):
//   frames x atoms   64 x 250   296 x 3,000   148 x 8,000   600 x 1,000   600 x 10,000 (every tenth)
//   one CTA each       12.0        12.2          14.4          12.3          22.7
//   streaming          19.0        19.0          19.0          19.2          44.0
// The lines: two resident CTAs an SM take a second pair of frames in the same time
// (1,200 x 1,000: 20.2 against 19.5), and a CTA's chain grows with the atoms
// (600 x 3,000: 20.8 against 20.4; 296 x 8,000: 21 against 23.6).
bool small_frames(const FrameLaunch& L) {
  return !L.wait.withhold &&  // the bounded waits' test needs the streaming kernels
         L.ref.n_sel >= 1 && L.ref.n_sel <= 8192 && L.n_frames <= 592 && L.n_frames * L.ref.n_sel <= 1200000;
}

cudaError_t launch_small_forward(const FrameLaunch& L, cudaStream_t s) {
  const unsigned grid = (unsigned)L.n_frames;
  if (L.stride == 4)
    return launch_dependent(L.align ? rmsd_small_kernel<4, kFwdFit> : rmsd_small_kernel<4, kFwdRaw>, grid, kSmallThreads,
                            0, s, L);
  return launch_dependent(L.align ? rmsd_small_kernel<3, kFwdFit> : rmsd_small_kernel<3, kFwdRaw>, grid, kSmallThreads, 0,
                          s, L);
}

cudaError_t launch_small_backward(const FrameLaunch& L, const double* stats, const float* grad_rmsd,
                                  const double* grad_f64, int64_t grad_stride, cudaStream_t s) {
  const dim3 grid((unsigned)L.n_frames, (unsigned)((L.ref.n_sel + kSmallThreads - 1) / kSmallThreads));
  if (L.stride == 4)
    rmsd_small_grad_kernel<4><<<grid, kSmallThreads, 0, s>>>(L, stats, grad_rmsd, grad_f64, grad_stride);
  else
    rmsd_small_grad_kernel<3><<<grid, kSmallThreads, 0, s>>>(L, stats, grad_rmsd, grad_f64, grad_stride);
  return cudaGetLastError();
}

}  // namespace wmd
