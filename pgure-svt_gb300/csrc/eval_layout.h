// eval_layout.h — dynamic shared memory of k_eval (eval.cu): what the host
// allocates for a launch and where the kernel puts things in it, from one set of
// functions (host C++ alone can check one against the other).
//
// A launch allocates for `points` lambda values, the most that a round of the
// search can hold; the round at hand may hold fewer (`nl`).  In 4-byte words:
//   left vectors  patches of at most 16 rows: [NC][kEvalPatches][kUStride]
//   g of copy 0   [nl][NC][kEvalPatches]
//   linear terms  [nl][4][kEvalPatches]
//   tiles         [nwin][2][eval_tile()]
#ifndef PGSVT_EVAL_LAYOUT_H
#define PGSVT_EVAL_LAYOUT_H

#ifdef __CUDACC__
#define PGSVT_HD __host__ __device__
#else
#define PGSVT_HD
#endif

namespace pgsvt {

constexpr int kEvalPatches = 32;  // kept patches per block

// floats of a staged left vector: 16-byte vectors that start on different banks
PGSVT_HD constexpr int eval_ustride(int M) { return M == 16 ? 20 : M; }

// words before g: the staged left vectors (patch side bs; 0: any side above 8)
PGSVT_HD constexpr int eval_staged(int bs, int NC) {
  return bs >= 1 && bs <= 4 ? NC * kEvalPatches * eval_ustride(bs * bs) : 0;
}
// words before the tiles of a round of nl values
PGSVT_HD constexpr int eval_tiles_at(int bs, int NC, int nl) {
  return eval_staged(bs, NC) + nl * (NC + 4) * kEvalPatches;
}
// words of a round of nl values with tiles of T pixels
PGSVT_HD constexpr int eval_words(int bs, int NC, int nwin, int nl, int T) {
  return eval_tiles_at(bs, NC, nl) + nwin * 2 * T;
}

// Pixels of a tile: the 32 blocks of an 8 x 4 half tile cover (7 + side) x (3 +
// side) pixels when they move together, and a few more rows and columns as a
// rule (simulated on the benchmark's trajectories: 4 x 4 patches fit 256 pixels
// in 85% of the cases and 384 in 98%, 8 x 8 ones 256 in 62% and 512 in 97%; the
// rest straddle two columns of tiles).  A footprint that does not fit costs a
// global atomic per pixel and patch.  The int64 accumulators (wide) round values
// of the tile and others differently, so they keep one size.
// Patches of at most 16 rows with more than 8 lambda values have no room for
// more than 256 at two blocks per SM.
PGSVT_HD constexpr int eval_alloc_tile(int bs, bool wide, int points) {
  return wide ? 256 : (bs >= 1 && bs <= 4 ? (points <= 8 ? 384 : 256) : 512);
}
// words that a launch allocates
PGSVT_HD constexpr int eval_alloc_words(int bs, bool wide, int NC, int nwin, int points) {
  return eval_words(bs, NC, nwin, points, eval_alloc_tile(bs, wide, points));
}
// The most values of a round that leave room for the larger tile of short launches
// (the whole launch, where that is its tile).
PGSVT_HD constexpr int eval_large_rounds(int bs, bool wide, int NC, int nwin, int points) {
  const int words = eval_alloc_words(bs, wide, NC, nwin, points);
  int nl = points;
  while (nl > 0 && eval_words(bs, NC, nwin, nl, eval_alloc_tile(bs, wide, 1)) > words) --nl;
  return nl;
}
// The tile of a round of nl <= points values.
PGSVT_HD constexpr int eval_tile(int bs, bool wide, int large_rounds, int nl) {
  return eval_alloc_tile(bs, wide, nl <= large_rounds ? 1 : 16);
}

}  // namespace pgsvt

#endif
