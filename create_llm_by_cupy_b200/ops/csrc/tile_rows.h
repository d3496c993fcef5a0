// Which rows of a key tile the decode attention copies; no CUDA calls in here, so that it is tested on the host.
#pragma once

#ifdef __CUDACC__
#define B200_TILE_ROWS_FN __host__ __device__ __forceinline__
#else
#define B200_TILE_ROWS_FN inline
#endif

namespace b200 {

// Rows [0, first) and, behind one that is left out, [first + 1, first + 1 + rest).
struct TileRows {
  int first, rest;
};

// The valid rows (keys below `len`) of the `tile` keys from key0 < len on, without key `pos`, whose row is being written
// (-1: none is).
B200_TILE_ROWS_FN TileRows tile_rows(int key0, int tile, int len, int pos) {
  const int n = len - key0 < tile ? len - key0 : tile, at = pos - key0;
  if (pos < 0 || at < 0 || at >= n) return {n, 0};
  return {at, n - 1 - at};
}

}  // namespace b200
