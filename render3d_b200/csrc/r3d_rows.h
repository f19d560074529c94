/* How a row of bytes is read four at a time at any address. */
#ifndef R3D_ROWS_H
#define R3D_ROWS_H

#include <stdint.h>

#if defined(__CUDACC__)
#define R3D_ROW_HD __host__ __device__ __forceinline__
#else
#define R3D_ROW_HD static inline
#endif

/* Bytes [x, x + 4) of a row of n bytes (x < n), byte x lying `off` bytes past
 * a multiple of four: the number of aligned words, from byte x - off, that
 * hold them and lie inside the row -- one (off 0), two, or 0 when a word would
 * reach outside it (the first row of a caller's volume starts its buffer, the
 * last one ends it). */
R3D_ROW_HD uint32_t r3d_row_words(uint32_t off, uint32_t x, uint32_t n) {
  const uint32_t left = n - x;
  if (off == 0u) return left >= 4u ? 1u : 0u;
  return x >= off && left >= 8u - off ? 2u : 0u;
}

#endif /* R3D_ROWS_H */
