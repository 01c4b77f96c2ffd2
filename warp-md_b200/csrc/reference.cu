// reference.cu -- a device-resident reference structure centred on the device.
//
// wmd_reference_upload brings a device reference to the host, sums it there and
// copies the centred coordinates back: three synchronous copies and an
// allocation, ~85 us for 2,000 atoms against 53 us for the value-and-gradient
// kernel that follows.  Here one CTA does the same on the caller's stream,
// latency-bound (two passes, two block reductions): 6.5 us for 2,000 atoms (8.3 with
// the loads of one atom in flight), and
// nothing waits for it on the host (rmsd_value_and_grad of 4,096 x 2,000 with a
// new reference 141 -> 63 us).  More CTAs would need a grid barrier between the
// passes.
//
// Every sum carries the rounding error of its additions along (Knuth's TwoSum), as
// the host's Neumaier sums do, and is added in a fixed tree: the kernels correct
// H by the sum of the centred coordinates, which is all rounding.
#include <cuda_runtime.h>

#include <cstdint>

#include "device_util.cuh"
#include "wmd_internal.h"

namespace wmd {
namespace {

constexpr int kRefThreads = 512;

struct ExactSum {
  double s = 0.0, c = 0.0;
  __device__ __forceinline__ void add(double x) {
    const double t = s + x, b = t - s;
    c += (s - (t - b)) + (x - b);
    s = t;
  }
  __device__ __forceinline__ void merge(double s2, double c2) {
    add(s2);
    c += c2;
  }
};

__device__ __forceinline__ void tree_add(ExactSum& v, int o) {
  const double s2 = __shfl_xor_sync(0xffffffffu, v.s, o), c2 = __shfl_xor_sync(0xffffffffu, v.c, o);
  v.merge(s2, c2);
}

// fn(k, y) for this thread's atoms in order, kRefAhead of them loaded at a time.
constexpr int kRefAhead = 4;

template <int STRIDE, class Fn>
__device__ __forceinline__ void each_atom(const float* __restrict__ ref, int64_t n, Fn fn) {
  for (int64_t k0 = threadIdx.x; k0 < n; k0 += kRefAhead * kRefThreads) {
    float y[kRefAhead][3];
#pragma unroll
    for (int u = 0; u < kRefAhead; ++u)
#pragma unroll
      for (int c = 0; c < 3; ++c)
        y[u][c] = k0 + u * kRefThreads < n ? __ldg(ref + (k0 + u * kRefThreads) * STRIDE + c) : 0.f;
#pragma unroll
    for (int u = 0; u < kRefAhead; ++u)
      if (k0 + u * kRefThreads < n) fn(k0 + u * kRefThreads, y[u]);
  }
}

template <int STRIDE>
__global__ void __launch_bounds__(kRefThreads) ref_prep_kernel(const float* __restrict__ ref, int64_t n,
                                                               double* __restrict__ yc, double* __restrict__ scal) {
  constexpr int kWarps = kRefThreads / 32;
  __shared__ double red[kWarps][4][2];
  depend_launch();  // the kernel that reads yc starts meanwhile
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ExactSum m[3];
  each_atom<STRIDE>(ref, n, [&](int64_t, const float (&y)[3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) m[c].add((double)y[c]);
  });
#pragma unroll
  for (int c = 0; c < 3; ++c) {
#pragma unroll
    for (int o = 16; o; o >>= 1) tree_add(m[c], o);
    if (lane == 0) {
      red[warp][c][0] = m[c].s;
      red[warp][c][1] = m[c].c;
    }
  }
  __syncthreads();
  double mean[3];
#pragma unroll
  for (int c = 0; c < 3; ++c) {  // every warp adds the warps' sums in the same tree
    m[c].s = lane < kWarps ? red[lane][c][0] : 0.0;
    m[c].c = lane < kWarps ? red[lane][c][1] : 0.0;
#pragma unroll
    for (int o = kWarps / 2; o; o >>= 1) tree_add(m[c], o);
    mean[c] = n > 0 ? __shfl_sync(0xffffffffu, m[c].s + m[c].c, 0) / (double)n : 0.0;
  }
  __syncthreads();  // red is written again
  ExactSum e[4];  // sum of y_c, sum |y_c|^2
  each_atom<STRIDE>(ref, n, [&](int64_t k, const float (&y)[3]) {
#pragma unroll
    for (int c = 0; c < 3; ++c) {
      const double d = (double)y[c] - mean[c];
      yc[k * 3 + c] = d;
      e[c].add(d);
      e[3].add(d * d);
    }
  });
  // 32 zero atoms after the reference: the frames-across-lanes kernels copy
  // whole 32-atom blocks of it
  for (int64_t k = n * 3 + threadIdx.x; k < (n + 32) * 3; k += kRefThreads) yc[k] = 0.0;
#pragma unroll
  for (int c = 0; c < 4; ++c) {
#pragma unroll
    for (int o = 16; o; o >>= 1) tree_add(e[c], o);
    if (lane == 0) {
      red[warp][c][0] = e[c].s;
      red[warp][c][1] = e[c].c;
    }
  }
  __syncthreads();
  if (warp != 0) return;
  double t[4];
#pragma unroll
  for (int c = 0; c < 4; ++c) {
    e[c].s = lane < kWarps ? red[lane][c][0] : 0.0;
    e[c].c = lane < kWarps ? red[lane][c][1] : 0.0;
#pragma unroll
    for (int o = kWarps / 2; o; o >>= 1) tree_add(e[c], o);
    t[c] = e[c].s + e[c].c;
  }
  if (lane == 0) {
    for (int c = 0; c < 3; ++c) {
      scal[kRefMean + c] = mean[c];
      scal[kRefSumC + c] = t[c];
    }
    // sum |y_c - sum_c / n|^2
    scal[kRefGy] = n > 0 ? t[3] - (t[0] * t[0] + t[1] * t[1] + t[2] * t[2]) / (double)n : 0.0;
  }
}

}  // namespace

cudaError_t launch_ref_prep(const float* ref, int64_t n_sel, int stride, double* yc, double* scal, cudaStream_t s) {
  if (stride == 4) ref_prep_kernel<4><<<1, kRefThreads, 0, s>>>(ref, n_sel, yc, scal);
  else ref_prep_kernel<3><<<1, kRefThreads, 0, s>>>(ref, n_sel, yc, scal);
  return cudaGetLastError();
}

}  // namespace wmd
