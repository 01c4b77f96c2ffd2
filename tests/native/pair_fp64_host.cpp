// Host build of the tensor-core pairwise kernels' tile walk and of the FP64
// pair epilogue, for CPU unit tests (test-only).
#include "qcp.cuh"
#include "tile_walk.h"

extern "C" {
int t_qcp_gap(const double* h, double d, double* gap) { return wmd::qcp_gap(h, d, gap) ? 1 : 0; }

// Walks the tiles `stride` apart from every start below it, as the CTAs of a
// launch do; counts each visited tile that holds a pair in seen[bi * nj + bj].
long long t_walk(int wide, long long frames, int part, int parts, int stride, int nj, int* seen, long long* empty) {
  auto go = [&](auto proto) {
    const long long n = proto.count();
    for (int c = 0; c < stride; ++c) {
      auto w = proto;
      for (long long t = c; t < n; t += stride) {
        int bi, bj;
        if (w.at(t, bi, bj)) ++seen[(long long)bi * nj + bj];
        else ++*empty;
      }
    }
    return n;
  };
  return wide ? go(wmd::TileWalk<40, 40>(frames, part, parts)) : go(wmd::TileWalk<40, 30>(frames, part, parts));
}
}
