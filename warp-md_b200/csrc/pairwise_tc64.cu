// pairwise_tc64.cu -- the FP64 mode of the all-pairs RMSD matrix on the
// tcgen05 int8 tensor cores.
//
// Arithmetic.  The FP64 matrix needs sum_k x_a(i,k) x_b(j,k) of every frame
// pair to FP64-like accuracy: 18 n FP64 operations a pair, which the SIMT tiles
// (pairwise.cu) run at 61 % of the FP64 pipe (3.39 ms for 4,000 frames x 500
// atoms).  Here each frame is centred in FP64 and written in 40-bit fixed point
// with a scale of its own, q = round((x - c) / s), |q| <= 127 * 2^32 (a step of
// 1.8e-12 of the frame's extent), split into five signed int8 digits
// q = sum_p a_p 2^(8p), and
//     H_ij = s_i s_j sum_{p + r >= 4} 2^(8(p+r)) sum_k a_p(i,k) a_r(j,k)
// takes 15 int8 products in five shift groups (p + r = 4..8), each accumulated
// exactly in int32 (5 n 128^2 < 2^31 for n <= 26,176 atoms) and combined exactly
// in int64.  The products left out (p + r < 4) are below 2^-38 of the extent
// squared; the frames' self-sums G leave out the same ones.  Splitting FP64
// operands over exact integer products is Ozaki, Ogita, Oishi & Rump 2012
// (Numer Algorithms 59:95); Ootomo, Ozaki & Yokota 2024 use int8 units.
//
// Error.  Against 64-bit sums the left-out products move the mean-square
// deviation by 3e-12 m^2 / sqrt(n) (RMS; m = the frame's extent; chains of 10
// to 5,000 atoms), the 40-bit rounding by 300 times less.  That is below 1e-8
// of the RMSD, a third of the float32 result's own rounding, unless the MSD is
// below 1.5e-4 m^2 / sqrt(n) (RMSD 0.14 A for 500 atoms of extent 54 A).
// Pairs below that bound are listed and recomputed in FP64 from the
// coordinates (pair_refine_kernel); when they are more than an eighth of all
// pairs the FP64 SIMT tiles recompute the matrix.  Relative error against
// 64-bit torch: 2.6e-8 (float32 rounding), as the SIMT tiles.
//
// Kernel.  The pipeline of pairwise_tc.cu: persistent CTAs, a TMA warp, an MMA
// warp, 12 warps that drain TMEM and 20 warps for the pair epilogue.  Tiles
// are 40 x 30 frames (M = 128, N = 96): five accumulators of 96 columns take
// 480 of the 512 TMEM columns.  K chunks of 32 atoms, 35 KB each (five digits
// of both operands), in a 4-stage ring; with the staged covariances (86 KB of
// FP64) that fills the 227 KB.  The MMA reads 7 KB of operands for 96 columns,
// 56 clocks of shared-memory bandwidth against 48 of tensor work (59.5 measured).
// 4,000 frames x 500 atoms take 0.76 ms with everything (SIMT tiles 3.46 ms),
// x 1,200 atoms 1.51 ms (7.81 ms).  What bounds it: per K chunk the 35 KB from
// L2 (0.68 us, 7.8 TB/s over all SMs; 0.49 us without the loads), and per tile
// ~4 us of the FP64 pair epilogue (qcp_gap, ~95 FP64 operations a pair) that the
// next tile's MMAs do not hide, since FP64 issues at a fraction of its rate
// beside them (math-pipe throttle is the top stall), and 2 us of TMEM drain.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <string>

#include "../../include/warpmd_rmsd.h"
#include "device_util.cuh"
#include "pairwise_tc.h"
#include "qcp.cuh"
#include "tcgen05.cuh"

namespace wmd {
namespace {

constexpr int kDigits = 5;
constexpr int kShift = 4;            // lowest shift group formed
constexpr int kGroups = 2 * kDigits - 1 - kShift;
constexpr int kGroupFrames = 10;     // frames per 32 GEMM rows (30 used)
constexpr int kTileM = 128, kTileN = 96;
constexpr int kFramesM = 40, kFramesN = 30;
constexpr int kSlices = kTileN / 32;
constexpr int kDrainWarps = 4 * kSlices;  // every (TMEM lane quarter, 32-column slice)
constexpr int kQcpWarps = 20;             // the drain warps and 8 more
constexpr int kThreads64 = 64 + 32 * kQcpWarps;
constexpr int kKPad = 32;                 // atoms are padded to whole K chunks
constexpr int kChunkK = 32;
constexpr int kStages64 = 4;
constexpr int kTmemCols = 512;
constexpr int kBlockPairs = kGroupFrames * kGroupFrames;  // frame pairs per drain warp
constexpr int kABytes = kDigits * kTileM * kChunkK;
constexpr int kBBytes = kDigits * kTileN * kChunkK;
constexpr int kStageBytes64 = kABytes + kBBytes;
// staged H, pair-major: entry e = 3a + b of pair p at [e][p]
constexpr int kHBytes = 9 * kBlockPairs * 8;
constexpr int kHOffset = kStages64 * kStageBytes64;
constexpr int kTermOffset = kHOffset + kDrainWarps * kHBytes;  // per-frame G, s, 1/s
constexpr int kTermFrames = kFramesM + kFramesN;
constexpr int kBarOffset64 = kTermOffset + 3 * kTermFrames * 8;
constexpr int kSmemBytes64 = kBarOffset64 + 16 * 8 + 32;
static_assert(kSmemBytes64 <= 227 * 1024, "shared memory");
static_assert(kBarOffset64 % 8 == 0 && kBBytes % 256 == 0 && kABytes % 256 == 0, "alignment");

constexpr double kQmax = 127.0 * 4294967296.0;  // 127 * 2^32
// n MSD, in units of the staged sums, below which a pair is recomputed:
// 1.5e-4 sqrt(n) (m_i^2 + m_j^2) / 2 with m = kQmax s, and s^2 * 2^32 the unit
constexpr double kFlagUnits = 1.5e-4 * 0.5 * 127.0 * 127.0 * 4294967296.0;

// kind::i8 instruction descriptor: D s32, A/B s8, both K-major, M=128, N=96.
constexpr uint32_t kIdesc64 = (2u << 4) | (1u << 7) | (1u << 10) | (uint32_t(kTileN >> 3) << 17) |
                              (uint32_t(kTileM >> 4) << 24);

using Tiles64 = TileWalk<kFramesM, kFramesN>;

struct Args64 {
  int64_t F;
  int n_k;             // K chunks
  double n;            // selected atoms
  float flag_units;    // kFlagUnits sqrt(n)
  int metric;
  const double* gsum;  // [F] self-sums, units of (s 2^16)^2
  const double* scale; // [F] s 2^16
  const double* inv;   // [F] 1 / (s 2^16)
  const double* cen;   // [F][3]
  float* out;          // [F][F]
  int* status;
  WaitCfg wait;
  uint2* flagged;
  unsigned* n_flagged;
  unsigned cap;
};

__global__ void __launch_bounds__(kThreads64, 1)
    pair_tc64_kernel(const __grid_constant__ CUtensorMap map_a, const __grid_constant__ CUtensorMap map_b,
                     const Args64 args, const Tiles64 walk, int64_t n_tiles) {
  extern __shared__ __align__(1024) unsigned char smem[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smem + kBarOffset64);
  uint64_t* empty = full + kStages64;
  uint64_t* tmem_full = empty + kStages64;
  uint64_t* tmem_empty = tmem_full + 1;
  uint64_t* drain = tmem_full + 2;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kBarOffset64 + 16 * 8);
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kBarOffset64 + 16 * 8 + 16);
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  Tiles64 tiles = walk;  // every role walks its own cursor

  if (threadIdx.x == 0) {
    for (int s = 0; s < kStages64; ++s) {
      mbar_init(&full[s], 1);
      mbar_init(&empty[s], 1);
    }
    mbar_init(tmem_full, 1);
    mbar_init(tmem_empty, kDrainWarps);
    mbar_init(drain, 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  if (warp == 1) tmem_alloc(tmem_slot, kTmemCols);
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem_base = *tmem_slot;

  if (warp == 0) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      const bool withheld = args.wait.withhold && blockIdx.x == 0;  // error-path test: first stage never armed
      uint32_t it = 0;
      bool ok = true;
      for (int64_t t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
        int bi, bj;
        if (!tiles.at(t, bi, bj)) continue;
        for (int kc = 0; kc < args.n_k; ++kc, ++it) {
          const int s = it % kStages64;
          if (!tc_wait(&empty[s], ((it / kStages64) & 1u) ^ 1u, args.status, abort_flag, args.wait.limit_ns)) {
            ok = false;
            break;
          }
          if (withheld && it == 0) continue;
          unsigned char* st = smem + s * kStageBytes64;
          mbar_arrive_expect_tx(&full[s], kStageBytes64);
          tma_load_3d(st, &map_a, kc * kChunkK, bi * kTileM, 0, &full[s]);
          tma_load_3d(st + kABytes, &map_b, kc * kChunkK, bj * kTileN, 0, &full[s]);
        }
      }
      // loads for MMAs that never ran (a wait ran out) must land before the CTA exits
      const uint32_t first = it > (uint32_t)kStages64 ? it - (uint32_t)kStages64 : 0u;
      for (uint32_t j = first; j < it; ++j)
        if (!(withheld && j == 0)) mbar_drain(&full[j % kStages64], (j / kStages64) & 1u, args.status);
    }
  } else if (warp == 1) {
    // ---------------- MMA issuer (the whole warp, see mma_i8) ----------------
    uint32_t it = 0, tc = 0;
    bool ok = true;
    const uint32_t on = elect_one();
    auto wait = [&](uint64_t* bar, uint32_t parity) {
      return __all_sync(0xffffffffu, tc_wait(bar, parity, args.status, abort_flag, args.wait.limit_ns)) != 0;
    };
    const uint64_t dbase = desc_sw<kChunkK>(smem);
    for (int64_t t = blockIdx.x; t < n_tiles && ok; t += gridDim.x) {
      int bi, bj;
      if (!tiles.at(t, bi, bj)) continue;
      if (!wait(tmem_empty, (tc & 1u) ^ 1u)) break;
      tc_fence_after();
      for (int kc = 0; kc < args.n_k; ++kc, ++it) {
        const int s = it % kStages64;
        if (!wait(&full[s], (it / kStages64) & 1u)) {
          ok = false;
          break;
        }
        const uint64_t dst = dbase + (uint64_t)((uint32_t)(s * kStageBytes64) >> 4);
        const uint32_t later = kc > 0 ? 1u : 0u;
#pragma unroll
        for (int p = 0; p < kDigits; ++p) {
#pragma unroll
          for (int r = 0; r < kDigits; ++r) {
            if (p + r < kShift) continue;
            // p ascends, so a group's first pair is the one with the top digit of B
            const uint32_t acc = r == kDigits - 1 ? later : 1u;
            mma_i8(tmem_base + (uint32_t)((p + r - kShift) * kTileN), dst + (uint64_t)((p * kTileM * kChunkK) >> 4),
                   dst + (uint64_t)((kABytes + r * kTileN * kChunkK) >> 4), kIdesc64, acc, on);
          }
        }
        tc_commit(&empty[s], on);
      }
      if (!ok) break;
      tc_commit(tmem_full, on);
      ++tc;
    }
    // all MMAs issued by this warp must finish before TMEM is freed
    tc_commit(drain, on);
    mbar_drain(drain, 0, args.status);
  } else {
    // ---------------- epilogue ----------------
    // the first 12 warps drain TMEM into shared memory, the others stage the
    // tile's per-frame terms; then all 20 run the tile's pairs, between two
    // named barriers (1 after staging, 2 before it is rewritten)
    const int wq = warp - 2;
    const bool drainer = wq < kDrainWarps;
    const int quarter = warp & 3;  // the TMEM lanes a warp may access
    const int slice = wq >> 2;
    const double inv_n = 1.0 / args.n;
    double* terms = reinterpret_cast<double*>(smem + kTermOffset);
    uint32_t tc = 0;
    for (int64_t t = blockIdx.x; t < n_tiles; t += gridDim.x) {
      int bi, bj;
      if (!tiles.at(t, bi, bj)) continue;
      if (drainer) {
        if (tc_wait(tmem_full, tc & 1u, args.status, abort_flag, args.wait.limit_ns)) {
          tc_fence_after();
          double* hs = reinterpret_cast<double*>(smem + kHOffset + wq * kHBytes);
#pragma unroll
          for (int half = 0; half < 2; ++half) {
            // columns [16 half, 16 half + 16) of the slice; 30 are frame columns
            long long acc[16];
#pragma unroll
            for (int c = 0; c < 16; ++c) acc[c] = 0;
#pragma unroll
            for (int g = 0; g < kGroups; ++g) {
              int32_t v[16];
              const uint32_t col = tmem_base + ((uint32_t)(quarter * 32) << 16) +
                                   (uint32_t)(g * kTileN + slice * 32 + 16 * half);
              tmem_ld8(col, v);
              tmem_ld8(col + 8, v + 8);
              tmem_wait_ld();
#pragma unroll
              for (int c = 0; c < 16; ++c) acc[c] += (long long)v[c] << (8 * g);
            }
            if (lane < 30) {
              // lane = 3 pi + a (row frame pi, component a); column 3 pj + b
              const int pi = lane / 3, a = lane - 3 * pi;
              double* row = hs + a * 3 * kBlockPairs + pi * kGroupFrames;
#pragma unroll
              for (int c = 0; c < 16; ++c) {
                const int cc = 16 * half + c;
                if (cc < 30) row[(cc % 3) * kBlockPairs + cc / 3] = (double)acc[c];
              }
            }
          }
          tc_fence_before();
          __syncwarp();
          if (lane == 0) mbar_arrive(tmem_empty);  // the next tile's MMAs may start
        }
      } else {
        for (int q = (wq - kDrainWarps) * 32 + lane; q < kTermFrames; q += (kQcpWarps - kDrainWarps) * 32) {
          const int64_t f = q < kFramesM ? (int64_t)bi * kFramesM + q : (int64_t)bj * kFramesN + (q - kFramesM);
          const bool in = f < args.F;
          terms[q] = in ? args.gsum[f] : 0.0;
          terms[kTermFrames + q] = in ? args.scale[f] : 1.0;
          terms[2 * kTermFrames + q] = in ? args.inv[f] : 1.0;
        }
      }
      ++tc;
      named_barrier_sync(1, 32 * kQcpWarps);
      if (*abort_flag) break;
      constexpr int kPairs = kDrainWarps * kBlockPairs;
#pragma unroll 1
      for (int gp = wq * 32 + lane; gp < kPairs; gp += kQcpWarps * 32) {
        const int blk = gp / kBlockPairs, pl = gp - blk * kBlockPairs;
        const int pi = pl / kGroupFrames, pj = pl - pi * kGroupFrames;
        // lane quarter and slice of drain warp blk (warp blk + 2 reads quarter (blk + 2) & 3)
        const int fi = ((blk + 2) & 3) * kGroupFrames + pi, fj = (blk >> 2) * kGroupFrames + pj;
        const int64_t i = (int64_t)bi * kFramesM + fi, j = (int64_t)bj * kFramesN + fj;
        if (!(i < j && j < args.F)) continue;
        const double* hs = reinterpret_cast<const double*>(smem + kHOffset + blk * kHBytes) + pl;
        double h[9];
#pragma unroll
        for (int e = 0; e < 9; ++e) h[e] = hs[e * kBlockPairs];
        const int ti = fi, tj = kFramesM + fj;
        const double si = terms[kTermFrames + ti], sj = terms[kTermFrames + tj];
        const double rho = si * terms[2 * kTermFrames + tj], rhoi = sj * terms[2 * kTermFrames + ti];
        // units of s_i s_j
        const double D = fma(terms[ti], rho, terms[tj] * rhoi);
        double gap;
        double far = 0.0;  // nofit: |c_i - c_j|^2
        if (args.metric == WMD_PAIR_NOFIT) {
          const double* ci = args.cen + i * 3;
          const double* cj = args.cen + j * 3;
          const double d0 = __ldg(ci) - __ldg(cj), d1 = __ldg(ci + 1) - __ldg(cj + 1), d2 = __ldg(ci + 2) - __ldg(cj + 2);
          far = d0 * d0 + d1 * d1 + d2 * d2;
          gap = D - 2.0 * (h[0] + h[4] + h[8]);
        } else if (!qcp_gap(h, D, &gap)) {  // a root that is not simple
          gap = 2.0 * (0.5 * D - qcp_lambda(h, 0.5 * D).lambda);
        }
        const bool low = (float)gap < args.flag_units * (float)(rho + rhoi);
        const double msd = fma(gap * (si * sj), inv_n, far);
        // Heron's step from the float32 root with the FP64 residual: rounded to float32 once
        float v = 0.0f;
        if (msd > 0.0) {
          const float r = sqrtf((float)msd);
          const double rd = (double)r;
          v = r > 1e-15f && r < 1e15f ? fmaf((float)fma(-rd, rd, msd), 0.5f / r, r) : (float)sqrt(msd);
        }
        args.out[(size_t)i * args.F + j] = v;
        args.out[(size_t)j * args.F + i] = v;
        if (low) {
          const unsigned k = atomicAdd(args.n_flagged, 1u);
          if (k < args.cap) args.flagged[k] = make_uint2((unsigned)i, (unsigned)j);
        }
      }
      named_barrier_sync(2, 32 * kQcpWarps);
    }
  }

  tc_fence_before();
  __syncthreads();
  if (warp == 1) {
    tc_fence_after();
    tmem_dealloc(tmem_base, kTmemCols);
  }
}

// One CTA per frame: FP64 centroid, the frame's extent and scale, the int8
// digits L[p][row(f, a)][k] (four atoms' digits per 32-bit store) and the
// self-sum over the products the tensor cores form.  Rows 30 and 31 of each
// 32-row group and rows past the last frame are left as they are: they only
// reach entries no pair reads.  Also zeroes out[f][f].
constexpr int kPrepThreads = 128;

__global__ void __launch_bounds__(kPrepThreads)
    tc64_prep(const float* __restrict__ coords, int64_t n_atoms, int stride, const uint32_t* __restrict__ sel,
              int64_t n_sel, int64_t n_pad, int64_t rows, double* __restrict__ cen, double* __restrict__ scale,
              double* __restrict__ inv_scale, double* __restrict__ gsum, int8_t* __restrict__ digits,
              float* __restrict__ out, int64_t F, int* status) {
  constexpr int kWarps = kPrepThreads / 32;
  __shared__ double red[kWarps][3];
  __shared__ double mred[kWarps];
  __shared__ long long gred[kWarps];
  const int64_t f = blockIdx.x;
  const float* fr = coords + (size_t)f * n_atoms * stride;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double s0 = 0, s1 = 0, s2 = 0;
  for (int64_t k = threadIdx.x; k < n_sel; k += kPrepThreads) {
    int64_t idx = sel ? (int64_t)sel[k] : k;
    if (idx >= n_atoms) {  // bad device-side selection: report, read atom 0
      atomicOr(status, kStatusBadIndex);
      idx = 0;
    }
    const float* p = fr + idx * stride;
    s0 += p[0]; s1 += p[1]; s2 += p[2];
  }
  for (int o = 16; o; o >>= 1) {
    s0 += __shfl_xor_sync(0xffffffffu, s0, o);
    s1 += __shfl_xor_sync(0xffffffffu, s1, o);
    s2 += __shfl_xor_sync(0xffffffffu, s2, o);
  }
  if (lane == 0) { red[warp][0] = s0; red[warp][1] = s1; red[warp][2] = s2; }
  __syncthreads();
  double c[3] = {0, 0, 0};
  for (int w = 0; w < kWarps; ++w) { c[0] += red[w][0]; c[1] += red[w][1]; c[2] += red[w][2]; }
  const double inv = 1.0 / (double)n_sel;
  c[0] *= inv; c[1] *= inv; c[2] *= inv;
  double m = 0.0;
  for (int64_t k = threadIdx.x; k < n_sel; k += kPrepThreads) {
    int64_t idx = sel ? (int64_t)sel[k] : k;
    if (idx >= n_atoms) idx = 0;
    const float* p = fr + idx * stride;
    for (int q = 0; q < 3; ++q) m = fmax(m, fabs((double)p[q] - c[q]));
  }
  for (int o = 16; o; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
  if (lane == 0) mred[warp] = m;
  __syncthreads();
  for (int w = 0; w < kWarps; ++w) m = fmax(m, mred[w]);
  const double s = m > 0.0 ? m / kQmax * (1.0 + 1e-14) : 1.0;
  const double inv_s = 1.0 / s;
  const int64_t row0 = (f / kGroupFrames) * 32 + (f % kGroupFrames) * 3;
  long long g = 0;
  for (int64_t k0 = 4 * (int64_t)threadIdx.x; k0 < n_pad; k0 += 4 * kPrepThreads) {
    uint32_t packed[3][kDigits];
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int l = 0; l < kDigits; ++l) packed[a][l] = 0;
#pragma unroll
    for (int u = 0; u < 4; ++u) {
      if (k0 + u >= n_sel) break;
      int64_t idx = sel ? (int64_t)sel[k0 + u] : k0 + u;
      if (idx >= n_atoms) idx = 0;
      const float* p = fr + idx * stride;
#pragma unroll
      for (int a = 0; a < 3; ++a) {
        long long q = llrint(((double)p[a] - c[a]) * inv_s);
        const long long qm = (long long)kQmax;
        q = q > qm ? qm : (q < -qm ? -qm : q);
        int d[kDigits];
#pragma unroll
        for (int l = 0; l < kDigits - 1; ++l) {
          d[l] = (int)(int8_t)(q & 255);  // balanced digit in [-128, 127]
          q = (q - d[l]) >> 8;
        }
        d[kDigits - 1] = (int)q;
#pragma unroll
        for (int l = 0; l < kDigits; ++l) packed[a][l] |= (uint32_t)(d[l] & 255) << (8 * u);
        g += (long long)(2 * (d[0] * d[4] + d[1] * d[3]) + d[2] * d[2]) + ((long long)(2 * (d[1] * d[4] + d[2] * d[3])) << 8) +
             ((long long)(2 * d[2] * d[4] + d[3] * d[3]) << 16) + ((long long)(2 * d[3] * d[4]) << 24) +
             ((long long)(d[4] * d[4]) << 32);
      }
    }
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
      for (int l = 0; l < kDigits; ++l)
        *reinterpret_cast<uint32_t*>(digits + ((size_t)l * rows + row0 + a) * n_pad + k0) = packed[a][l];
  }
  for (int o = 16; o; o >>= 1) g += __shfl_xor_sync(0xffffffffu, g, o);
  if (lane == 0) gred[warp] = g;
  __syncthreads();
  if (threadIdx.x == 0) {
    long long tot = 0;
    for (int w = 0; w < kWarps; ++w) tot += gred[w];
    gsum[f] = (double)tot;
    scale[f] = s * 65536.0;
    inv_scale[f] = inv_s * (1.0 / 65536.0);
    cen[f * 3 + 0] = c[0]; cen[f * 3 + 1] = c[1]; cen[f * 3 + 2] = c[2];
    out[(size_t)f * F + f] = 0.0f;
  }
}

}  // namespace

int pairwise_tc64_run(PairwiseWorkspace& w, int sm_count, const float* coords, int64_t F, int64_t n_atoms, int stride,
                      const uint32_t* sel, int64_t n_sel, int metric, float* out, int* status, cudaStream_t s,
                      std::string* msg, PairFlags* flags) {
  const int64_t n_pad = (n_sel + kKPad - 1) / kKPad * kKPad;
  // whole tiles of A (128 rows) and of B (96 rows)
  const int64_t row_groups = (F + kGroupFrames - 1) / kGroupFrames;
  const int64_t rows_pad = std::max((row_groups + 3) / 4 * 4, (row_groups + 2) / 3 * 3) * 32;
  const size_t digit_bytes = (size_t)kDigits * rows_pad * n_pad;
  const int64_t pairs = F * (F - 1) / 2;
  const unsigned cap = (unsigned)std::min<int64_t>(std::max<int64_t>(pairs / 8, 1), 1 << 20);
  const size_t head = 256 + (size_t)F * 6 * sizeof(double);
  const size_t digits_at = (head + 1023) & ~size_t(1023);
  const size_t list_at = (digits_at + digit_bytes + 15) & ~size_t(15);
  const size_t need = list_at + (size_t)cap * sizeof(uint2);
  if (!w.extra || w.extra_bytes < need) {
    if (w.extra) cudaFree(w.extra);
    w.extra = nullptr;
    w.extra_bytes = 0;
    cudaError_t e = cudaMalloc(&w.extra, need);
    if (e != cudaSuccess) {
      cudaGetLastError();
      *msg = std::string("cuda driver error: pairwise workspace allocation failed: ") + cudaGetErrorString(e);
      return WMD_ERR_OOM;
    }
    w.extra_bytes = need;
  }
  unsigned char* base = static_cast<unsigned char*>(w.extra);
  unsigned* n_flagged = reinterpret_cast<unsigned*>(base);
  double* gsum = reinterpret_cast<double*>(base + 256);
  double* scale = gsum + F;
  double* inv = scale + F;
  double* cen = inv + F;
  int8_t* digits = reinterpret_cast<int8_t*>(base + digits_at);
  uint2* list = reinterpret_cast<uint2*>(base + list_at);

  cudaError_t e = cudaMemsetAsync(base, 0, 256, s);
  if (e != cudaSuccess) {
    *msg = std::string("cuda driver error: ") + cudaGetErrorString(e);
    return WMD_ERR_CUDA;
  }
  tc64_prep<<<(unsigned)F, kPrepThreads, 0, s>>>(coords, n_atoms, stride, sel, n_sel, n_pad, rows_pad, cen, scale, inv,
                                                 gsum, digits, out, F, status);
  if ((e = cudaGetLastError()) != cudaSuccess) {
    *msg = std::string("cuda driver error: pairwise prep: ") + cudaGetErrorString(e);
    return WMD_ERR_CUDA;
  }
  CUtensorMap map_a, map_b;
  int rc = encode_digits(&map_a, digits, n_pad, rows_pad, kDigits, kChunkK, kTileM, msg);
  if (!rc) rc = encode_digits(&map_b, digits, n_pad, rows_pad, kDigits, kChunkK, kTileN, msg);
  if (rc) return rc;

  Args64 a;
  a.F = F;
  a.n_k = (int)(n_pad / kChunkK);
  a.n = (double)n_sel;
  a.flag_units = (float)(kFlagUnits * std::sqrt((double)n_sel));
  a.metric = metric;
  a.gsum = gsum;
  a.scale = scale;
  a.inv = inv;
  a.cen = cen;
  a.out = out;
  a.status = status;
  a.wait = w.wait;
  a.flagged = list;
  a.n_flagged = n_flagged;
  a.cap = cap;
  const Tiles64 tiles(F, w.part, w.parts);
  const int64_t n_tiles = tiles.count();
  if ((e = cudaFuncSetAttribute(pair_tc64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmemBytes64)) !=
      cudaSuccess) {
    *msg = std::string("cuda driver error: ") + cudaGetErrorString(e);
    return WMD_ERR_CUDA;
  }
  const int grid = (int)std::max<int64_t>(1, std::min<int64_t>(sm_count, n_tiles));
  pair_tc64_kernel<<<grid, kThreads64, kSmemBytes64, s>>>(map_a, map_b, a, tiles, n_tiles);
  if ((e = cudaGetLastError()) != cudaSuccess) {
    *msg = std::string("cuda driver error: pairwise tensor-core launch: ") + cudaGetErrorString(e);
    return WMD_ERR_CUDA;
  }
  flags->list = list;
  flags->count = n_flagged;
  flags->cap = cap;
  flags->cen = cen;
  return 0;
}

}  // namespace wmd
