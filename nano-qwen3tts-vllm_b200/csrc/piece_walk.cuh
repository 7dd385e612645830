// piece_walk.cuh - which (row, piece of the row) a thread of a streaming pass has next.  A pass over rows of `pieces` pieces gives thread i the pieces
// i, i + stride, i + 2 stride, ... of all rows one behind another; a division for each of them costs as much as what is done with it, so a step is kept as whole rows
// and pieces.  Rows are counted in 64 bits: a row behind the last one, or a step from one near 2^31, stays above it.
#pragma once
#include <stdint.h>

#ifdef __CUDACC__
#define PIECE_WALK_FN __host__ __device__ __forceinline__
#else
#define PIECE_WALK_FN inline
#endif

namespace b2 {

struct PieceStep { int rows, pieces; };            // of `stride` pieces
PIECE_WALK_FN PieceStep piece_step(unsigned stride, int pieces) {
  return {static_cast<int>(stride / static_cast<unsigned>(pieces)), static_cast<int>(stride % static_cast<unsigned>(pieces))};
}

struct PieceWalk {
  int64_t row;
  int piece;
};
PIECE_WALK_FN PieceWalk piece_at(unsigned i, int pieces) {
  return {static_cast<int64_t>(i / static_cast<unsigned>(pieces)), static_cast<int>(i % static_cast<unsigned>(pieces))};
}
PIECE_WALK_FN PieceWalk piece_next(PieceWalk w, PieceStep s, int pieces) {
  w.row += s.rows;
  w.piece += s.pieces;                             // both below `pieces`, which is at most 2^28
  if (w.piece >= pieces) { w.piece -= pieces; ++w.row; }
  return w;
}

}  // namespace b2
