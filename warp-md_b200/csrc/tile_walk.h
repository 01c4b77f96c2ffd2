// tile_walk.h -- the order in which the tensor-core pairwise kernels visit the
// tiles of the frame x frame matrix (plain C++: the host counts the tiles, the
// kernels walk them).
#pragma once

#include <cstdint>

#if defined(__CUDACC__)
#define WMD_WALK_HD __host__ __device__
#else
#define WMD_WALK_HD
#endif

namespace wmd {

// Tiles of FM x FN frames over the pairs i < j, for the I blocks bi = part (mod
// parts) of this launch.  They are enumerated in groups of kRowGroup of those
// tile rows, column after column inside a group, so that the ~148 tiles in
// flight at once share a few A rows and B columns and their limbs stay in L2.
// (Row after row, they would share one A row but stream 148 B columns,
// rereading each column from DRAM for every row once the limbs outgrow L2:
// 196 MB for 20,000 frames x 1,000 atoms.)  A group starts at the first column
// its first row needs, so a CTA's stride through the list meets almost only
// tiles with work (enumerating all columns left half of the list empty and up
// to 3 % more tiles on some CTAs than on others).
constexpr int kRowGroup = 8;

template <int FM, int FN>
struct TileWalk {
  int ni, nj;  // I blocks (FM frames) x J blocks (FN frames)
  int64_t F;
  int part, parts;
  int g;               // cursor: the group holding the last position asked for,
  int64_t base, size;  // its first position, its tiles,
  int g_rows, g_col0;  // tile rows and first column

  WMD_WALK_HD TileWalk() {}
  WMD_WALK_HD TileWalk(int64_t frames, int part_, int parts_)
      : ni((int)((frames + FM - 1) / FM)), nj((int)((frames + FN - 1) / FN)), F(frames), part(part_), parts(parts_),
        g(-1), base(0), size(0), g_rows(1), g_col0(0) {}
  WMD_WALK_HD int rows_total() const { return part < ni ? (ni - part + parts - 1) / parts : 0; }
  WMD_WALK_HD int rows(int grp) const {
    const int r = rows_total() - grp * kRowGroup;
    return r < kRowGroup ? r : kRowGroup;
  }
  // first column of a group: the block holding frame i0 + 1 of its first row
  // (the partners of frame i0 start there)
  WMD_WALK_HD int col0(int grp) const {
    const int64_t j = ((int64_t)grp * kRowGroup * parts + part) * FM + 1;
    const int64_t c = j / FN;
    return c < nj ? (int)c : nj;
  }
  WMD_WALK_HD int64_t count() const {
    int64_t n = 0;
    for (int grp = 0; grp * kRowGroup < rows_total(); ++grp) n += (int64_t)rows(grp) * (nj - col0(grp));
    return n;
  }
  // Tile at position t (not below any position asked for before); false when
  // it holds no pair i < j.
  WMD_WALK_HD bool at(int64_t t, int& bi, int& bj) {
    while (t >= base + size) {
      base += size;
      ++g;
      g_rows = rows(g);
      g_col0 = col0(g);
      size = (int64_t)g_rows * (nj - g_col0);
    }
    const unsigned r = (unsigned)(t - base);  // < kRowGroup nj
    const unsigned c = r / (unsigned)g_rows;
    bj = g_col0 + (int)c;
    bi = (g * kRowGroup + (int)(r - c * (unsigned)g_rows)) * parts + part;
    const int64_t i0 = (int64_t)bi * FM;
    const int64_t jend = (int64_t)(bj + 1) * FN;
    return i0 < (jend < F ? jend : F) - 1;
  }
};

}  // namespace wmd
