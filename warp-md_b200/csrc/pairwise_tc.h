// pairwise_tc.h -- tensor-core (tcgen05) forms of the pairwise RMSD matrix.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>

#include <cstdint>
#include <string>

#include "device_util.cuh"
#include "pairwise.h"

namespace wmd {

// limbs = 3 (24-bit fixed point) or 2 (16-bit); see pairwise_tc.cu.
int pairwise_tc_run(PairwiseWorkspace& w, int sm_count, const float* coords, int64_t n_frames, int64_t n_atoms,
                    int stride, const uint32_t* sel, int64_t n_sel, int metric, int limbs, float* out, int* status,
                    const WaitCfg& wait, cudaStream_t s, std::string* msg);

// Pairs a tensor-core kernel listed for recomputation (device memory; count may
// exceed cap, then the list is incomplete) and the frames' centroids.
struct PairFlags {
  const uint2* list = nullptr;
  const unsigned* count = nullptr;
  unsigned cap = 0;
  const double* cen = nullptr;  // [F][3]
};

// The FP64 mode on the tensor cores (pairwise_tc64.cu): fills every entry of
// this part's pairs and the diagonal, and lists in *flags the pairs to
// recompute in FP64.  At most kTc64MaxAtoms selected atoms.
constexpr int64_t kTc64MaxAtoms = 26176;  // 5 n 128^2 < 2^31, a multiple of 32
int pairwise_tc64_run(PairwiseWorkspace& w, int sm_count, const float* coords, int64_t n_frames, int64_t n_atoms,
                      int stride, const uint32_t* sel, int64_t n_sel, int metric, float* out, int* status,
                      cudaStream_t s, std::string* msg, PairFlags* flags);

// Recomputes the listed pairs in FP64 from the coordinates; scan: when the list
// overflowed, finds the pairs below 0.01 A in the matrix instead.
cudaError_t launch_pair_refine(const PairFlags& flags, int sm_count, const float* coords, int64_t n_atoms, int stride,
                               const uint32_t* sel, int64_t n_sel, int64_t n_frames, int metric, float* out, int part,
                               int parts, bool scan, int* status, cudaStream_t s);

int encode_digits(CUtensorMap* map, const int8_t* digits, int64_t n_pad, int64_t rows, int limbs, int chunk,
                  int tile_rows, std::string* msg);

}  // namespace wmd
