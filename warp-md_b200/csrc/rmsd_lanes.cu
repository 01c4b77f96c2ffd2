// rmsd_lanes.cu -- per-frame RMSD statistics with frames across lanes.
//
// The atom-major streaming kernel (rmsd_frames.cu) gives every thread a few
// atoms of one frame, so each (tile, frame) item ends in a 15-value
// cross-lane reduction and a CTA barrier; those cost about as many
// instructions as the FP64 arithmetic itself.  Here the roles are swapped:
//
//   * A warp owns a run of stages; a stage is 32 frames x 32 atoms (lane l =
//     frame 32g + l).  The frames' coordinates arrive by 2-D TMA (boxes of 32
//     rows x 128 bytes, 128-byte swizzle, so that every lane reading "its"
//     row hits a different bank group), the 32 reference atoms (centred,
//     FP64) by a 1-D bulk copy next to them.  Two stages per warp, refilled
//     by lane 0 as soon as the warp is done with one.
//   * Each lane adds, in FP64 and in atom order, the 15 sums of its own frame
//     (sum x, sum x_a^2, sum x y_c^T): no shuffles, no barriers.
//   * The stages of all frame groups, group after group, are split over the
//     warp slots in equal runs (LaneSplit).  A group within one run is finished from
//     registers; otherwise each of its warps stores a record (15 sums x 32 frames,
//     coalesced, in L2) and the last to do so adds them in warp order and finishes
//     the group, a frame per lane, while other warps still stream.  The split depends
//     on the sizes and the device alone, so results are bitwise reproducible.
//     With more than kLaneFinishParts warps a group (few frames of many atoms),
//     lanes_finalize_kernel adds the records, a CTA a group.
//
// Whole (tile, group) units, tile after tile, used to be the warps' work: the last tile's
// few warps then finished every group (31 us for 2,400 x 1,000, whose stream takes
// 4.4), a warp had 1 or 2 units but not 1.5, and the records were a frame apart.
// Measured, us a call, then / with equal runs: 2,400 x 4,000 58 / 37; 5,000 x 8,000
// 119 / 94; 20,000 x 3,000 209 / 132; 5,001 x 3,001 62 / 50; 2,000 x 20,000 101 / 96.
// Bound by HBM for long runs (4,000 x 100,000: 6.5 TB/s); short ones by the launch,
// the first loads and the finish (~12 us together).
//
// Frames whose stride is not a multiple of 16 bytes (packed xyz with
// n_atoms % 4 != 0) cannot be rows of a tensor map; four consecutive frames
// can (48 n_atoms bytes).  Such launches (dense selections) read "quad rows":
// a stage is four boxes of [8 quad rows x 100 floats], box j holding frames
// 32g + 4i + j (i = 0..7).  Box j starts at the 16-byte boundary at or below
// frame position j's first atom of the stage, so lane 4i + j reads its 96
// floats at a fixed offset of (3 j n_atoms) mod 4 floats with 32-bit loads:
// rows of 400 bytes put the 32 lanes in distinct banks for odd n_atoms (two
// lanes per bank otherwise).  Atoms past the tile come from the next frame of
// the quad row and are masked.  The last n_frames mod 4 frames are no quad row:
// their tiles are summed with plain loads, atoms across lanes, by warps set aside
// for them.  As a launch behind this kernel they cost 12 us of 83 for 5,001
// frames x 3,001 atoms.
//
// Atoms streamed: a dense selection (the first n_sel atoms), or the span
// [lane_atom0, lane_atom0 + lane_atoms) of a sorted selection with the
// reference expanded onto it and per-atom weights (1 for selected atoms, 0
// for the rest; or the masses of a weighted reference).  The weights also
// serve weighted references over dense selections.  Requirements (else the
// atom-major kernel runs): a 16-byte aligned first streamed atom and a frame
// stride that is a multiple of 16 bytes (n_atoms % 4 == 0 for packed xyz).
// The reference values and weights must be padded with 32 zero atoms (the
// bulk copies of the last stage read past the span).
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <cstring>

#include "device_util.cuh"
#include "frame_parts.cuh"
#include "wmd_internal.h"

namespace wmd {

namespace {

constexpr int kLaneWarps = 4;   // warps per CTA
constexpr int kLaneStages = 2;  // stage ring per warp
constexpr int kLaneAtoms = 32;  // atoms per stage
constexpr int kLaneBlock = 16;  // stages added up in one chain
// The split of the stages over the warps (lanes_split): fewest stages a warp, most
// stages that runs of whole groups may add to the busiest warp, most parts of a group
// that the last of its warps adds up itself.
constexpr int kLaneMinStages = 4;
constexpr int kLaneWholeStages = 4;
constexpr int kLaneFinishParts = 16;

template <int STRIDE>
struct LaneGeo {
  static constexpr int kBoxes = kLaneAtoms * STRIDE / 32;  // [32 frames][32 floats] boxes per stage
  static constexpr int kXBytes = kBoxes * 32 * 32 * 4;
  static constexpr int kYBytes = kLaneAtoms * 3 * 8;
  static constexpr int kWBytes = kLaneAtoms * 4;  // per-atom weights (weighted / expanded launches)
  static constexpr int kStageBytes = (kXBytes + kYBytes + kWBytes + 1023) / 1024 * 1024;
  static constexpr int kBarOffset = kLaneWarps * kLaneStages * kStageBytes;
  static constexpr int kAbortOffset = kBarOffset + kLaneWarps * kLaneStages * 8;
  static constexpr int kSmemBytes = kAbortOffset + 16 + 1024;  // + slack to align the base to 1024
};

// quad rows (packed xyz, n_atoms % 4 != 0): 4 boxes of [8 quad rows x 100 floats], no swizzle
struct QuadGeo {
  static constexpr int kBoxRowBytes = 100 * 4;
  static constexpr int kBoxBytes = 8 * kBoxRowBytes;
  static constexpr int kXBytes = 4 * kBoxBytes;
  static constexpr int kYBytes = kLaneAtoms * 3 * 8;
  static constexpr int kWBytes = kLaneAtoms * 4;
  static constexpr int kStageBytes = (kXBytes + kYBytes + kWBytes + 127) / 128 * 128;
  static constexpr int kBarOffset = kLaneWarps * kLaneStages * kStageBytes;
  static constexpr int kAbortOffset = kBarOffset + kLaneWarps * kLaneStages * 8;
  static constexpr int kSmemBytes = kAbortOffset + 16 + 1024;
};

template <bool QUAD, int STRIDE>
struct PickGeo {
  using type = LaneGeo<STRIDE>;
};
template <int STRIDE>
struct PickGeo<true, STRIDE> {
  using type = QuadGeo;
};

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, int x, int y, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::
          "r"(smem_addr(dst)),
      "l"(reinterpret_cast<uint64_t>(map)), "r"(x), "r"(y), "r"(smem_addr(bar))
      : "memory");
}

// One lane's sums over the valid atoms of a stage (valid is warp-uniform).
// Packed xyz: 4 atoms = 3 swizzled 16-byte chunks; xyzw: 1 atom = 1 chunk.
template <int STRIDE, bool RAW, bool W>
__device__ __forceinline__ void stage_sums(double (&acc)[15], const unsigned char* st, int lane, int valid,
                                           const double (&mean)[3]) {
  const float* wb = reinterpret_cast<const float*>(st + LaneGeo<STRIDE>::kXBytes + LaneGeo<STRIDE>::kYBytes);
  const unsigned char* row = st + lane * 128;
  const int sw = lane & 7;
  auto chunk = [&](int c) -> float4 {
    return *reinterpret_cast<const float4*>(row + (c >> 3) * 4096 + (((c & 7) ^ sw) << 4));
  };
  const double2* yb = reinterpret_cast<const double2*>(st + LaneGeo<STRIDE>::kXBytes);
  // k: the atom's index within the stage (its weight; y is pre-multiplied)
  auto add_atom = [&](float fx, float fy, float fz, double y0, double y1, double y2, bool in, int k) {
    const double x0 = fx, x1 = fy, x2 = fz;
    if (W && RAW) in = in && wb[k] != 0.0f;  // expanded selection: unselected atoms have weight 0
    if (RAW) {
      const double d0 = x0 - (y0 + mean[0]);
      const double d1 = x1 - (y1 + mean[1]);
      const double d2 = x2 - (y2 + mean[2]);
      acc[0] = fma(d0, in ? d0 : 0.0, acc[0]);
      acc[1] = fma(d1, in ? d1 : 0.0, acc[1]);
      acc[2] = fma(d2, in ? d2 : 0.0, acc[2]);
    } else {
      if (W) {  // sum w x, sum w x_a^2 (the weighted forms of rmsd_frames_kernel)
        const double w = wb[k];
        const double u0 = w * x0, u1 = w * x1, u2 = w * x2;
        acc[0] += u0; acc[1] += u1; acc[2] += u2;
        acc[3] = fma(u0, x0, acc[3]); acc[4] = fma(u1, x1, acc[4]); acc[5] = fma(u2, x2, acc[5]);
      } else {
        acc[0] += x0; acc[1] += x1; acc[2] += x2;
        acc[3] = fma(x0, x0, acc[3]); acc[4] = fma(x1, x1, acc[4]); acc[5] = fma(x2, x2, acc[5]);
      }
      acc[6] = fma(x0, y0, acc[6]);  acc[7] = fma(x0, y1, acc[7]);  acc[8] = fma(x0, y2, acc[8]);
      acc[9] = fma(x1, y0, acc[9]);  acc[10] = fma(x1, y1, acc[10]); acc[11] = fma(x1, y2, acc[11]);
      acc[12] = fma(x2, y0, acc[12]); acc[13] = fma(x2, y1, acc[13]); acc[14] = fma(x2, y2, acc[14]);
    }
  };
  if (STRIDE == 3) {
#pragma unroll
    for (int m = 0; m < kLaneAtoms / 4; ++m) {
      if (4 * m >= valid) break;
      const float4 a = chunk(3 * m), b = chunk(3 * m + 1), c = chunk(3 * m + 2);
      const double2 y01 = yb[6 * m + 0], y23 = yb[6 * m + 1], y45 = yb[6 * m + 2];
      const double2 y67 = yb[6 * m + 3], y89 = yb[6 * m + 4], yab = yb[6 * m + 5];
      add_atom(a.x, a.y, a.z, y01.x, y01.y, y23.x, 4 * m + 0 < valid, 4 * m + 0);
      add_atom(a.w, b.x, b.y, y23.y, y45.x, y45.y, 4 * m + 1 < valid, 4 * m + 1);
      add_atom(b.z, b.w, c.x, y67.x, y67.y, y89.x, 4 * m + 2 < valid, 4 * m + 2);
      add_atom(c.y, c.z, c.w, y89.y, yab.x, yab.y, 4 * m + 3 < valid, 4 * m + 3);
    }
  } else {
#pragma unroll
    for (int m = 0; m < kLaneAtoms / 2; ++m) {
      if (2 * m >= valid) break;
      const float4 a = chunk(2 * m), b = chunk(2 * m + 1);
      const double2 y01 = yb[3 * m + 0], y23 = yb[3 * m + 1], y45 = yb[3 * m + 2];
      add_atom(a.x, a.y, a.z, y01.x, y01.y, y23.x, 2 * m + 0 < valid, 2 * m + 0);
      add_atom(b.x, b.y, b.z, y23.y, y45.x, y45.y, 2 * m + 1 < valid, 2 * m + 1);
    }
  }
}

// The quad-row form of stage_sums: lane 4i + j reads frame position j's box,
// row i, from float offset off; atoms at or past `valid` are masked.
template <bool RAW, bool W>
__device__ __forceinline__ void stage_sums_quad(double (&acc)[15], const unsigned char* st, int lane, int off,
                                                int valid, const double (&mean)[3]) {
  const float* wb = reinterpret_cast<const float*>(st + QuadGeo::kXBytes + QuadGeo::kYBytes);
  const float* row =
      reinterpret_cast<const float*>(st + (lane & 3) * QuadGeo::kBoxBytes + (lane >> 2) * QuadGeo::kBoxRowBytes) + off;
  const double* yb = reinterpret_cast<const double*>(st + QuadGeo::kXBytes);
#pragma unroll 4
  for (int k = 0; k < kLaneAtoms; ++k) {
    if (k >= valid) break;
    const double x0 = row[3 * k], x1 = row[3 * k + 1], x2 = row[3 * k + 2];
    const double y0 = yb[3 * k], y1 = yb[3 * k + 1], y2 = yb[3 * k + 2];
    if (RAW) {
      const bool in = !W || wb[k] != 0.0f;
      const double d0 = x0 - (y0 + mean[0]);
      const double d1 = x1 - (y1 + mean[1]);
      const double d2 = x2 - (y2 + mean[2]);
      acc[0] = fma(d0, in ? d0 : 0.0, acc[0]);
      acc[1] = fma(d1, in ? d1 : 0.0, acc[1]);
      acc[2] = fma(d2, in ? d2 : 0.0, acc[2]);
    } else {
      if (W) {
        const double w = wb[k];
        const double u0 = w * x0, u1 = w * x1, u2 = w * x2;
        acc[0] += u0; acc[1] += u1; acc[2] += u2;
        acc[3] = fma(u0, x0, acc[3]); acc[4] = fma(u1, x1, acc[4]); acc[5] = fma(u2, x2, acc[5]);
      } else {
        acc[0] += x0; acc[1] += x1; acc[2] += x2;
        acc[3] = fma(x0, x0, acc[3]); acc[4] = fma(x1, x1, acc[4]); acc[5] = fma(x2, x2, acc[5]);
      }
      acc[6] = fma(x0, y0, acc[6]);  acc[7] = fma(x0, y1, acc[7]);  acc[8] = fma(x0, y2, acc[8]);
      acc[9] = fma(x1, y0, acc[9]);  acc[10] = fma(x1, y1, acc[10]); acc[11] = fma(x1, y2, acc[11]);
      acc[12] = fma(x2, y0, acc[12]); acc[13] = fma(x2, y1, acc[13]); acc[14] = fma(x2, y2, acc[14]);
    }
  }
}

// How the frame groups' stages are split over the active warps: group-major, in
// equal runs (lane_whole: runs of whole groups).  A warp's run holds whole groups
// and at most two parts of groups, its first and its last, each with a record of
// 15 sums x 32 frames.
struct LaneSplit {
  int64_t nw, groups, total;
  int stages;
  bool whole;
  __device__ __forceinline__ explicit LaneSplit(const FrameLaunch& L)
      : nw(L.lane_warps), groups((L.n_frames + 31) / 32), stages((int)((L.lane_atoms + kLaneAtoms - 1) / kLaneAtoms)),
        whole(L.lane_whole) {
    total = groups * stages;
  }
  // first stage of warp w's run
  __device__ __forceinline__ int64_t first(int64_t w) const {
    return whole ? groups * w / nw * stages : total * w / nw;
  }
  // warp whose run holds stage j (not with whole)
  __device__ __forceinline__ int64_t owner(int64_t j) const { return ((j + 1) * nw - 1) / total; }
  __device__ __forceinline__ double* record(const FrameLaunch& L, int64_t w, int64_t g) const {
    return L.lane_rec + (2 * w + (first(w) >= g * stages ? 0 : 1)) * (16 * 32);
  }
  // tot = the records of group g of warps wa, wa + step, ... below wb, in that order
  template <int UNROLL>
  __device__ __forceinline__ void add_records(const FrameLaunch& L, int64_t g, int64_t wa, int64_t wb, int step, int lane,
                                              double (&tot)[16]) const {
#pragma unroll
    for (int e = 0; e < 16; ++e) tot[e] = 0.0;
#pragma unroll UNROLL
    for (int64_t w = wa; w < wb; w += step) {
      // the warp that holds the group's start may have another group's part first
      const double* rec = record(L, w, g) + lane;
#pragma unroll
      for (int e = 0; e < 15; ++e) tot[e] += __ldcg(rec + e * 32);
    }
  }
};

// A frame's outputs, or its sums for a caller that finishes the frames itself.
__device__ __forceinline__ void lane_finish(const FrameLaunch& L, int64_t f, const double (&tot)[16], int mode) {
  if (!L.lane_totals) {
    finish_totals(L, f, tot, mode);
    return;
  }
  double2* o = reinterpret_cast<double2*>(L.partial + f * kStatDoubles);
#pragma unroll
  for (int e = 0; e < 8; ++e) o[e] = make_double2(tot[2 * e], tot[2 * e + 1]);
}

template <int STRIDE, bool RAW, bool W, bool QUAD = false>
__global__ void __launch_bounds__(kLaneWarps * 32) rmsd_lanes_kernel(const __grid_constant__ CUtensorMap map,
                                                                     const FrameLaunch L) {
  using G = typename PickGeo<QUAD, STRIDE>::type;
  depend_launch();
  extern __shared__ unsigned char smem_raw[];
  unsigned char* smem = smem_raw + ((1024u - (smem_addr(smem_raw) & 1023u)) & 1023u);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  uint64_t* bars = reinterpret_cast<uint64_t*>(smem + G::kBarOffset);
  uint64_t* full = bars + warp * kLaneStages;
  volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + G::kAbortOffset);
  unsigned char* ring = smem + warp * kLaneStages * G::kStageBytes;

  // atoms streamed: the selection itself, or the atom span an expanded
  // selection covers (L.lane_atom0 is folded into the tensor map's base)
  const int64_t F = L.n_frames, n_sel = L.lane_atoms;
  const int64_t groups = (F + 31) / 32;
  const int64_t nw = L.lane_warps, gw = (int64_t)blockIdx.x * kLaneWarps + warp;
  const LaneSplit split(L);
  constexpr int kMode = RAW ? kFwdRaw : kFwdFit;
  const double mean[3] = {RAW ? ref_mean(L.ref, 0) : 0.0, RAW ? ref_mean(L.ref, 1) : 0.0, RAW ? ref_mean(L.ref, 2) : 0.0};

  if (threadIdx.x == 0) {
    for (int i = 0; i < kLaneWarps * kLaneStages; ++i) mbar_init(&bars[i], 1);
    *abort_flag = 0;
    fence_barrier_init();
  }
  __syncthreads();

  // counts this warp's stored records of one of `parts` parts: true for the last
  auto last_part = [&](int64_t counter, int parts) {
    __threadfence();
    __syncwarp();
    unsigned before = 0;
    if (lane == 0) before = atomicAdd(L.group_done + counter, 1u);
    before = __shfl_sync(0xffffffffu, before, 0);
    if (before + 1u != (unsigned)parts) return false;
    __threadfence();
    return true;
  };

  if (gw >= nw) {
    // the frames past the last quad row, by warps of their own: (frame, tile) items
    const int64_t item = gw - nw, tiles = (n_sel + L.lane_tail_tile - 1) / L.lane_tail_tile;
    if (!QUAD || item >= L.tail_frames * tiles) return;
    double* tail = L.lane_rec + 2 * nw * (16 * 32);  // [tail frame][tile][16]
    const int64_t t = item % tiles;
    const double v = gather_item<3, RAW ? kFwdRaw : (W ? kFwdW : kFwdFit), kGatherDepth, true>(
        L, L.coords + (size_t)(F + item / tiles) * L.n_atoms * 3, t * L.lane_tail_tile,
        min(n_sel, (t + 1) * L.lane_tail_tile), mean, lane);
    if ((lane & 1) == 0) tail[item * 16 + (lane >> 1)] = v;
    if (!last_part(groups, L.lane_tail_warps)) return;
    // a lane per (element, parity) adds the tiles of a frame, then lane k finishes frame k
    double tot[16];
#pragma unroll
    for (int e = 0; e < 16; ++e) tot[e] = 0.0;
    for (int k = 0; k < L.tail_frames; ++k) {
      double s = 0.0;
#pragma unroll 8
      for (int64_t i = lane >> 4; i < tiles; i += 2) s += __ldcg(tail + (k * tiles + i) * 16 + (lane & 15));
      s += __shfl_xor_sync(0xffffffffu, s, 16);
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const double v = __shfl_sync(0xffffffffu, s, e);
        if (lane == k) tot[e] = v;
      }
    }
    if (lane < L.tail_frames) lane_finish(L, F + lane, tot, kMode);
    return;
  }

  const int64_t w0 = split.first(gw), w1 = split.first(gw + 1);
  const int kst = split.stages;  // stages of a frame group
  if (w0 >= w1) return;
  // producer cursor (lane 0): stage pk of group pg; n_issued stages so far
  const int64_t total = w1 - w0;
  int64_t pg = w0 / kst;
  int pk = (int)(w0 - pg * kst);
  int64_t n_issued = 0;
  // under the error-path test the first stage of CTA 0's warp 0 is never armed
  const bool withheld = L.wait.withhold && blockIdx.x == 0 && warp == 0;
  auto issue_next = [&]() {  // lane 0
    const int slot = (int)(n_issued % kLaneStages);
    unsigned char* dst = ring + slot * G::kStageBytes;
    const int64_t a0 = (int64_t)pk * kLaneAtoms;
    if (!(withheld && n_issued == 0)) {
      // the warp's earlier generic reads of this slot before the async writes
      asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
      mbar_arrive_expect_tx(&full[slot], G::kXBytes + G::kYBytes + (W ? G::kWBytes : 0));
      if (QUAD) {
        // frame position j of the quad rows 8g .. 8g + 7: its atoms a0 .. a0 + 31
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          const int64_t e = (int64_t)j * 3 * L.n_atoms + 3 * a0;
          tma_load_2d(dst + j * QuadGeo::kBoxBytes, &map, (int)(e & ~int64_t(3)), (int)(pg * 8), &full[slot]);
        }
      } else {
#pragma unroll
        for (int b = 0; b < LaneGeo<STRIDE>::kBoxes; ++b)
          tma_load_2d(dst + b * 4096, &map, (int)(a0 * STRIDE + 32 * b), (int)(pg * 32), &full[slot]);
      }
      bulk_copy_g2s(dst + G::kXBytes, L.lane_y + a0 * 3, G::kYBytes, &full[slot]);
      if (W) bulk_copy_g2s(dst + G::kXBytes + G::kYBytes, L.lane_w + a0, G::kWBytes, &full[slot]);
    }
    ++n_issued;
    if (++pk == kst) {
      pk = 0;
      ++pg;
    }
  };
  if (lane == 0)
    while (n_issued < kLaneStages && n_issued < total) issue_next();

  // quad rows: this lane's float offset into its box row (stages start at
  // multiples of 32 atoms, so only the frame position matters)
  const int quad_off = QUAD ? (int)(((int64_t)(lane & 3) * 3 * L.n_atoms) & 3) : 0;
  int64_t n_done = 0;
  bool aborted = false;
  for (int64_t g = w0 / kst; g * kst < w1; ++g) {
    // this warp's part of group g: stages [k0, k1)
    const int k0 = (int)max((int64_t)0, w0 - g * kst), k1 = (int)min((int64_t)kst, w1 - g * kst);
    double acc[15], tot[16];
#pragma unroll
    for (int e = 0; e < 15; ++e) acc[e] = tot[e] = 0.0;
    tot[15] = 0.0;
    for (int k = k0; k < k1; ++k) {
      const int slot = (int)(n_done % kLaneStages);
      const uint32_t parity = (uint32_t)((n_done / kLaneStages) & 1);
      if (!mbar_wait(&full[slot], parity, L.status, kStatusTimeoutFull, abort_flag, L.wait.limit_ns)) {
        aborted = true;
        break;
      }
      const int valid = (int)min((int64_t)kLaneAtoms, n_sel - (int64_t)k * kLaneAtoms);
      if (QUAD)
        stage_sums_quad<RAW, W>(acc, ring + slot * G::kStageBytes, lane, quad_off, valid, mean);
      else
        stage_sums<STRIDE, RAW, W>(acc, ring + slot * G::kStageBytes, lane, valid, mean);
      ++n_done;
      __syncwarp();
      if (lane == 0 && n_issued < total) issue_next();
      // sums of kLaneBlock stages, then their sum: rounding grows with the longest chain
      if ((k + 1) % kLaneBlock == 0 || k + 1 == k1) {
#pragma unroll
        for (int e = 0; e < 15; ++e) {
          tot[e] += acc[e];
          acc[e] = 0.0;
        }
      }
    }
    if (aborted) break;
    if (RAW) {  // the no-fit record holds sum |x - y|^2 in its first word
      tot[0] += tot[1] + tot[2];
      tot[1] = tot[2] = 0.0;
    }
    if (k1 - k0 < kst) {  // other warps hold the rest of the group
      double* rec = split.record(L, gw, g) + lane;
#pragma unroll
      for (int e = 0; e < 15; ++e) __stcg(rec + e * 32, tot[e]);
      if (!L.lane_fused) continue;
      const int64_t wa = split.owner(g * kst), wb = split.owner((g + 1) * kst - 1);
      if (!last_part(g, (int)(wb - wa) + 1)) continue;
      split.add_records<4>(L, g, wa, wb + 1, 1, lane, tot);
    }
    const int64_t f = g * 32 + lane;
    if (f < F) lane_finish(L, f, tot, kMode);
    __syncwarp();
  }

  // after an abort, copies this warp issued may still be landing (a withheld
  // stage has none)
  if (aborted && lane == 0) {
    for (int64_t j = n_done; j < n_issued; ++j)
      if (!(withheld && j == 0)) mbar_drain(&full[j % kLaneStages], (uint32_t)((j / kLaneStages) & 1), L.status);
  }
}

// Frame groups spread over more warps than one of them should add up: a CTA per
// group, its warps adding every kFinalizeWarps-th record, then a lane per frame.
constexpr int kFinalizeWarps = 16;

template <int MODE>
__global__ void __launch_bounds__(kFinalizeWarps * 32) lanes_finalize_kernel(const FrameLaunch L) {
  extern __shared__ double red[];  // [kFinalizeWarps][15][32]
  depend_wait();
  depend_launch();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const LaneSplit split(L);
  const int64_t g = blockIdx.x;
  const int64_t wa = split.owner(g * split.stages), wb = split.owner((g + 1) * split.stages - 1);
  if (wa == wb) return;  // one warp had the whole group
  double tot[16];
  split.add_records<4>(L, g, wa + warp, wb + 1, kFinalizeWarps, lane, tot);
#pragma unroll
  for (int e = 0; e < 15; ++e) red[(warp * 15 + e) * 32 + lane] = tot[e];
  __syncthreads();
  // element e of every frame by warp e
  if (warp < 15) {
    double s = 0.0;
#pragma unroll
    for (int w = 0; w < kFinalizeWarps; ++w) s += red[(w * 15 + warp) * 32 + lane];
    red[warp * 32 + lane] = s;  // slot (0, e): read by this warp alone
  }
  __syncthreads();
  const int64_t f = g * 32 + lane;
  if (warp != 0 || f >= L.n_frames) return;
#pragma unroll
  for (int e = 0; e < 15; ++e) tot[e] = red[e * 32 + lane];
  tot[15] = 0.0;
  lane_finish(L, f, tot, MODE);
}

using EncodeTiled = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                                 const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                                 CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeTiled encode_fn() {
  static EncodeTiled fn = nullptr;
  if (fn) return fn;
  void* p = nullptr;
  cudaDriverEntryPointQueryResult qr;
  if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &qr) != cudaSuccess ||
      qr != cudaDriverEntryPointSuccess || !p) {
    cudaGetLastError();
    return nullptr;
  }
  fn = reinterpret_cast<EncodeTiled>(p);
  return fn;
}

template <int STRIDE, bool RAW, bool QUAD = false>
int lanes_occupancy() {
  using G = typename PickGeo<QUAD, STRIDE>::type;
  auto kern = rmsd_lanes_kernel<STRIDE, RAW, false, QUAD>;
  cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, G::kSmemBytes);
  int b = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, kern, kLaneWarps * 32, G::kSmemBytes) != cudaSuccess) b = 1;
  return std::max(b, 1);
}

// QUAD: L.n_frames is a multiple of 4 and the rows of the tensor map are
// quad rows of 4 frames (packed xyz, dense selection).
template <int STRIDE, bool RAW, bool W, bool QUAD = false>
cudaError_t launch_lanes(const FrameLaunch& L, cudaStream_t s) {
  using G = typename PickGeo<QUAD, STRIDE>::type;
  EncodeTiled enc = encode_fn();
  if (!enc) return cudaErrorNotSupported;
  CUtensorMap map;
  CUresult r;
  if (QUAD) {
    const cuuint64_t dims[2] = {(cuuint64_t)(L.n_atoms * 12), (cuuint64_t)(L.n_frames / 4)};
    const cuuint64_t strides[1] = {(cuuint64_t)(L.n_atoms * 48)};
    const cuuint32_t box[2] = {100, 8};
    const cuuint32_t estr[2] = {1, 1};
    r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, const_cast<float*>(L.coords), dims, strides, box, estr,
            CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
            CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  } else {
    const cuuint64_t dims[2] = {(cuuint64_t)(L.lane_atoms * STRIDE), (cuuint64_t)L.n_frames};
    const cuuint64_t strides[1] = {(cuuint64_t)(L.n_atoms * STRIDE * 4)};
    const cuuint32_t box[2] = {32, 32};
    const cuuint32_t estr[2] = {1, 1};
    float* base = const_cast<float*>(L.coords) + L.lane_atom0 * STRIDE;
    r = enc(&map, CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 2, base, dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
            CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  }
  if (r != CUDA_SUCCESS) return cudaErrorInvalidValue;
  auto kern = rmsd_lanes_kernel<STRIDE, RAW, W, QUAD>;
  static bool attr_done[64] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev < 0 || dev >= 64) return cudaErrorInvalidDevice;
  if (!attr_done[dev]) {
    cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, G::kSmemBytes);
    if (e != cudaSuccess) return e;
    attr_done[dev] = true;
  }
  const int grid = (L.lane_warps + L.lane_tail_warps + kLaneWarps - 1) / kLaneWarps;
  kern<<<grid, kLaneWarps * 32, G::kSmemBytes, s>>>(map, L);
  cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess || L.lane_fused) return e;
  auto fin = lanes_finalize_kernel<RAW ? kFwdRaw : kFwdFit>;
  constexpr int kFinBytes = kFinalizeWarps * 15 * 32 * 8;
  static bool fin_done[64] = {};
  if (!fin_done[dev]) {
    if ((e = cudaFuncSetAttribute(fin, cudaFuncAttributeMaxDynamicSharedMemorySize, kFinBytes)) != cudaSuccess) return e;
    fin_done[dev] = true;
  }
  return launch_dependent(fin, (unsigned)((L.n_frames + 31) / 32), kFinalizeWarps * 32, kFinBytes, s, L);
}

// Packed xyz frames whose stride is not a multiple of 16 bytes, streamed as
// quad rows: a dense selection only (the tensor map covers whole frames).
bool lanes_quad(const FrameLaunch& L) {
  return L.stride == 3 && (L.n_atoms & 3) != 0 && L.sel == nullptr && L.lane_atom0 == 0 &&
         L.lane_atoms == L.ref.n_sel && L.lane_y == L.ref.yc && L.lane_w == L.ref.w;
}

// y_exp[(sel[i] - a0)][c] = yc[i][c], w_exp[sel[i] - a0] = w ? w[i] : 1 (the
// buffers were zeroed; selection indices are strictly increasing)
__global__ void lanes_expand_kernel(const uint32_t* __restrict__ sel, int64_t n_sel, int64_t a0,
                                    const double* __restrict__ yc, const float* __restrict__ w,
                                    double* __restrict__ y_exp, float* __restrict__ w_exp) {
  for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n_sel; i += (int64_t)gridDim.x * blockDim.x) {
    const int64_t k = (int64_t)sel[i] - a0;
    y_exp[k * 3 + 0] = yc[i * 3 + 0];
    y_exp[k * 3 + 1] = yc[i * 3 + 1];
    y_exp[k * 3 + 2] = yc[i * 3 + 2];
    w_exp[k] = w ? w[i] : 1.0f;
  }
}

}  // namespace

cudaError_t launch_lanes_expand(const uint32_t* sel, int64_t n_sel, int64_t a0, const double* yc, const float* w,
                                double* y_exp, float* w_exp, cudaStream_t s) {
  if (n_sel <= 0) return cudaSuccess;
  const unsigned grid = (unsigned)std::min<int64_t>((n_sel + 255) / 256, 4096);
  lanes_expand_kernel<<<grid, 256, 0, s>>>(sel, n_sel, a0, yc, w, y_exp, w_exp);
  return cudaGetLastError();
}

bool lanes_eligible(const FrameLaunch& L) {
  static int mode = -1;
  if (mode < 0) {
    // WMD_FRAMES_KERNEL=atoms: always the atom-major kernel; =noquad: not for
    // packed frames whose stride is not a multiple of 16 bytes
    const char* e = std::getenv("WMD_FRAMES_KERNEL");
    mode = (e && std::strcmp(e, "atoms") == 0) ? 0 : (e && std::strcmp(e, "noquad") == 0) ? 2 : 1;
  }
  if (!mode || L.lane_atoms <= 0 || L.n_frames <= 0) return false;
  if ((reinterpret_cast<uintptr_t>(L.coords + L.lane_atom0 * L.stride) & 15u) != 0) return false;
  if (L.stride != 4 && (L.n_atoms & 3) != 0) {
    // quad rows of 4 frames: whole frames of a dense selection, and enough
    // frames that the gathered tail (n_frames mod 4) stays small
    if (mode == 2 || !lanes_quad(L) || L.n_frames < 32) return false;
    return L.n_atoms * 12 < (int64_t(1) << 31) && L.n_frames < (int64_t(1) << 31);
  }
  if ((L.lane_atom0 + L.lane_atoms) * L.stride >= (int64_t(1) << 31) || L.n_frames >= (int64_t(1) << 31))
    return false;
  return true;
}

static int lanes_slots(const FrameLaunch& L, int sm_count) {
  static int occ[3] = {0, 0, 0};
  const int which = L.stride == 4 ? 1 : lanes_quad(L) ? 2 : 0;
  int& o = occ[which];
  if (o == 0) o = which == 1 ? lanes_occupancy<4, false>() : which == 2 ? lanes_occupancy<3, false, true>()
                                                                        : lanes_occupancy<3, false>();
  return sm_count * o * kLaneWarps;
}

// Against the atom-major kernel, whose cost is its (1,024-atom tile, frame) items
// and its finalize launch (us, lanes / atom-major): 8,000 x 128 15.5 / 39; 4,000 x 500
// 18.4 / 26.6; 1,500 x 2,000 23.3 / 24.7; 5,001 x 3,001 50 / 59; 600 x 4,000 22.7 / 21.5;
// 2,400 x 1,000 21.6 / 20.9.  Few groups leave lanes empty and many parts to add:
// 256 x 40,000 41.9 / 44.1, but 160 x 20,000 29.3 / 25.0, 64 x 400,000 102 / 94.
// With weights it is ahead at every size measured (300 x 100,000, superposition
// with masses: 211 / 265; 2,000 x 2,000 47 / 49); an expanded selection's
// alternative is the gathered kernel.
bool lanes_worthwhile(const FrameLaunch& L, int sm_count) {
  const int64_t groups = (L.n_frames + 31) / 32;
  if (L.lane_w) return groups * ((L.lane_atoms + 255) / 256) >= 2 * (int64_t)sm_count;
  return groups >= 8 && L.n_frames * ((L.lane_atoms + 1023) / 1024) >= 20 * (int64_t)sm_count;
}

int lanes_grid(const FrameLaunch& L, int sm_count) { return lanes_slots(L, sm_count) / kLaneWarps; }

// Two records per warp and the tail frames' tiles.
size_t lane_record_bytes(const FrameLaunch& L, int sm_count) {
  return (size_t)lanes_slots(L, sm_count) * (2 * 16 * 32 + 3 * 16) * sizeof(double);
}

// Splits L's frames over `slots` warps.
static void lanes_split(FrameLaunch& L, int64_t slots) {
  if (L.tail_frames > 0) {
    // warps for the tail frames by their share of the work (a warp streams ~16 times
    // as many atom-frames across lanes as it gathers along one frame)
    const int64_t part = 16 * L.tail_frames;
    const int64_t d = std::min(std::max<int64_t>(1, slots / 2 / L.tail_frames),
                               (slots * 16 + L.n_frames + part - 1) / (L.n_frames + part));  // per frame
    L.lane_tail_tile = ((L.lane_atoms + d - 1) / d + 127) / 128 * 128;
    L.lane_tail_warps = (int)(L.tail_frames * ((L.lane_atoms + L.lane_tail_tile - 1) / L.lane_tail_tile));
    slots -= L.lane_tail_warps;
  }
  const int64_t groups = (L.n_frames + 31) / 32, stages = (L.lane_atoms + kLaneAtoms - 1) / kLaneAtoms;
  const int64_t total = groups * stages;
  int64_t nw = std::max<int64_t>(1, std::min(slots, total / kLaneMinStages));
  // whole groups where that costs the busiest warp only a few stages
  const int64_t runs = std::min(groups, nw);
  const int64_t longest = (groups + runs - 1) / runs * stages;
  L.lane_whole = longest <= (total + nw - 1) / nw + kLaneWholeStages;
  if (L.lane_whole) nw = runs;
  L.lane_warps = (int)nw;
  L.lane_fused = L.lane_whole || (nw + groups - 1) / groups + 1 <= kLaneFinishParts;
}

cudaError_t launch_lanes_forward(const FrameLaunch& L, bool raw, cudaStream_t s) {
  FrameLaunch K = L;
  const bool w = L.lane_w != nullptr, quad = lanes_quad(L);
  if (quad) {  // whole quad rows, and the last n_frames mod 4 frames with plain loads
    K.n_frames = L.n_frames & ~int64_t(3);
    K.tail_frames = (int)(L.n_frames - K.n_frames);
  }
  lanes_split(K, std::max<int64_t>(2, (int64_t)L.grid * kLaneWarps));
  cudaError_t e = cudaSuccess;
  if (!L.done_cleared && ((K.lane_fused && !K.lane_whole) || K.tail_frames > 0)) {
    e = cudaMemsetAsync(K.group_done, 0, (size_t)frame_groups(K.n_frames) * sizeof(unsigned), s);
    if (e != cudaSuccess) return e;
  }
  if (quad)
    return w ? (raw ? launch_lanes<3, true, true, true>(K, s) : launch_lanes<3, false, true, true>(K, s))
             : (raw ? launch_lanes<3, true, false, true>(K, s) : launch_lanes<3, false, false, true>(K, s));
  if (L.stride == 4) {
    if (w) return raw ? launch_lanes<4, true, true>(K, s) : launch_lanes<4, false, true>(K, s);
    return raw ? launch_lanes<4, true, false>(K, s) : launch_lanes<4, false, false>(K, s);
  }
  if (w) return raw ? launch_lanes<3, true, true>(K, s) : launch_lanes<3, false, true>(K, s);
  return raw ? launch_lanes<3, true, false>(K, s) : launch_lanes<3, false, false>(K, s);
}

}  // namespace wmd
