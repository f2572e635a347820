// What a kernel asks L2 for before it waits for the kernel in front: which rows, and which part of them. Plain arithmetic without
// the CUDA headers, so that its bounds are tested on the host.
#pragma once

#ifdef __CUDACC__
#define DJV_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define DJV_HOST_DEVICE inline
#endif

namespace djv {

constexpr int AHEAD_PIECE = 8192;  // bytes of a bulk prefetch at most

// Whether a row that a list names is asked for: a list that is still being written can hold anything.
DJV_HOST_DEVICE bool ahead_takes(long long row, int rows) { return row >= 0 && row < rows; }

struct AheadSpan {
  int row, offset, bytes;  // offset and bytes: multiples of 16, as row_bytes is; bytes <= 0: nothing
};

// Piece p of rows of row_bytes that follow one another, each cut every AHEAD_PIECE bytes.
DJV_HOST_DEVICE int ahead_pieces(int row_bytes) { return (row_bytes + AHEAD_PIECE - 1) / AHEAD_PIECE; }
DJV_HOST_DEVICE AheadSpan ahead_piece(int p, int row_bytes) {
  const int pieces = ahead_pieces(row_bytes), offset = p % pieces * AHEAD_PIECE, left = row_bytes - offset;
  return {p / pieces, offset, left < AHEAD_PIECE ? left : AHEAD_PIECE};
}

// Share `at` of a row that `shares` blocks of a cluster read together, AHEAD_PIECE bytes of it at most.
DJV_HOST_DEVICE AheadSpan ahead_share(int at, int shares, int row_bytes) {
  int bytes = ((row_bytes + shares - 1) / shares + 15) / 16 * 16;
  if (bytes > AHEAD_PIECE) bytes = AHEAD_PIECE;
  const int offset = at * bytes, left = row_bytes - offset;
  return {0, offset, left < bytes ? left : bytes};
}

}  // namespace djv
