// Builders of the LOD brick cache (r3d_build.cu) and the byte-row loads that
// device-side builders share.
#pragma once

#include "r3d_march.cuh"
#include "r3d_rows.h"

namespace r3d {

// Bytes [x, x + 4) of a row of n bytes, zero past its end.  VEC: the row and
// x are 4-byte aligned and n a multiple of 4; else two aligned words are
// shifted together, which may hold up to three bytes beyond either end of the
// row.  `inner` says that those lie in the same buffer; where they may not (the
// first and last row of a caller's volume: inner_row), such words are read
// byte by byte.  (Byte by byte at every row's ends the builders of volumes with
// odd rows lost 10 to 20 %, the section fills 5 %.)
template <bool VEC>
__device__ __forceinline__ uint32_t load4(const uint8_t *__restrict__ row, uint32_t x, uint32_t n,
                                          bool inner = true) {
  if (x >= n) return 0u;
  if (VEC) return __ldg(reinterpret_cast<const uint32_t *>(row + x));
  const uint32_t left = n - x, off = (uint32_t)((uintptr_t)(row + x) & 3u);
  uint32_t v = 0;
  if (inner || r3d_row_words(off, x, n)) {
    const uint32_t *w = reinterpret_cast<const uint32_t *>(row + x - off);
    const uint32_t lo = __ldg(w), hi = left + off > 4u && (inner || off) ? __ldg(w + 1) : 0u;
    v = __funnelshift_r(lo, hi, 8u * off);
  } else {
    for (uint32_t k = 0; k < 4u && k < left; k++) v |= (uint32_t)__ldg(row + x + k) << (8u * k);
  }
  return left >= 4u ? v : v & (0xFFFFFFFFu >> (8u * (4u - left)));
}
// Whether three bytes on either side of row (y, z) of a volume of ny x nz rows
// of n bytes are in its buffer.
__device__ __forceinline__ bool inner_row(uint32_t y, uint32_t z, uint32_t n, uint32_t ny, uint32_t nz) {
  return n >= 4u && (y | z) != 0u && (y + 1u != ny || z + 1u != nz);
}

// Bytes [x, x + 8) likewise (VEC: 8-byte aligned, n a multiple of 8).
template <bool VEC>
__device__ __forceinline__ uint2 load8(const uint8_t *__restrict__ row, uint32_t x, uint32_t n,
                                       bool inner = true) {
  if (VEC)
    return x < n ? __ldg(reinterpret_cast<const uint2 *>(row + x)) : make_uint2(0u, 0u);
  return make_uint2(load4<false>(row, x, n, inner), load4<false>(row, x + 4u, n, inner));
}

// A warp writes dst[0, n): byte i is row[x0 + i], row[0] left of the row, and
// past its nx bytes row[nx - 1] (CLAMP) or 0.  Words of dst are stored whole
// and read as two aligned words of the row; only its unaligned ends and the
// words that leave the row go byte by byte.  (The rows are the context's own:
// three bytes past the last one are in its buffer.)
template <bool CLAMP>
__device__ __forceinline__ uint32_t row_byte(const uint8_t *__restrict__ row, int64_t x, uint32_t nx) {
  if (x >= (int64_t)nx) return CLAMP ? row[nx - 1u] : 0u;
  return row[x < 0 ? 0 : x];
}
template <bool CLAMP>
__device__ __forceinline__ void warp_row(uint8_t *__restrict__ dst, uint32_t n,
                                         const uint8_t *__restrict__ row, int64_t x0, uint32_t nx) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint32_t head = min((uint32_t)(-(uintptr_t)dst & 3u), n), words = (n - head) / 4u;
  const uint32_t tail = head + words * 4u;
  if (lane < head) dst[lane] = (uint8_t)row_byte<CLAMP>(row, x0 + lane, nx);
  if (tail + lane < n) dst[tail + lane] = (uint8_t)row_byte<CLAMP>(row, x0 + tail + lane, nx);
  for (uint32_t k = lane; k < words; k += 32u) {
    const int64_t x = x0 + head + 4u * k;
    uint32_t v = 0;
    if (x >= 0 && x + 4 <= (int64_t)nx) {
      v = load4<false>(row, (uint32_t)x, nx);
    } else {
#pragma unroll
      for (int b = 0; b < 4; b++) v |= row_byte<CLAMP>(row, x + b, nx) << (8 * b);
    }
    *reinterpret_cast<uint32_t *>(dst + head + 4u * k) = v;
  }
}

// the largest of the four bytes of w
__device__ __forceinline__ uint32_t max_byte(uint32_t w) {
  w = __vmaxu4(w, w >> 16);
  return max(w & 0xFFu, (w >> 8) & 0xFFu);
}

// One pyramid level as a source of bricks: its bytes and extent, its brick
// grid, and the first job of the level in the job list.
struct LevelSrc {
  const uint8_t *p;
  uint32_t ex, ey, ez;
  uint32_t bdx, bdy;
  uint32_t job0;
};

// 2x box reduction of a level (sx, sy, sz) to dst (dx, dy, dz: multiples of
// 128, dst null: none) and, with vmax (zeroed by the caller), the maximum of
// every 128^3 brick of the source (bdx * bdy * ... entries).
cudaError_t launch_level_down(const uint8_t *src, uint32_t sx, uint32_t sy, uint32_t sz,
                              uint8_t *dst, uint32_t dx, uint32_t dy, uint32_t dz, uint32_t *vmax,
                              uint32_t bdx, uint32_t bdy, cudaStream_t st);
// Slots from bricks of pyramid levels: job j puts brick brick[j] of the level
// whose job range holds j into slot slot[j] (null: j): its bytes (pool), quad
// words and block maxima, each left out when null.
cudaError_t launch_slot_fill(const LevelSrc *lev, uint32_t nlev, const uint32_t *brick,
                             const uint32_t *slot, uint32_t njobs, uint8_t *pool, uint32_t *quad,
                             uint8_t *bmax, cudaStream_t st);
// The cube's and the shard atlas's tables, of levels of any extent (x
// fastest, no padding): the next mip (clamped source coordinates, (sum + 4) /
// 8), the maxima of 8^3 blocks, and the quad words of DevCube::quad.
cudaError_t launch_mip(const uint8_t *src, uint32_t sx, uint32_t sy, uint32_t sz, uint8_t *dst,
                       uint32_t dx, uint32_t dy, uint32_t dz, cudaStream_t st);
cudaError_t launch_occ_raw(const uint8_t *vox, uint32_t nx, uint32_t ny, uint32_t nz, uint8_t *raw,
                           cudaStream_t st);
cudaError_t launch_level_quads(const uint8_t *src, uint32_t dx, uint32_t dy, uint32_t dz,
                               uint32_t *quad, cudaStream_t st);
// Bytes of the quad words of a cube whose extents are set (0 past
// kQuadVoxels), setting c.qoff; and the words themselves, at `at` (null:
// none, the bytes are sampled), setting c.quad.
size_t cube_quad_bytes(DevCube &c);
// Whether `words` bytes of quad words may be taken with `bytes` bytes of
// levels, `back` bytes being given back for them.  The words make a volume five
// times as large, and what a program allocates after it should fit as it does
// beside the bytes alone: so words of more than a gibibyte are taken only where
// a quarter of the device's memory stays free (asking takes 0.09 ms, a fifth of
// a small volume's first upload; without the words a view takes up to twice
// as long).
bool words_fit(size_t bytes, size_t words, size_t back);
cudaError_t build_cube_quads(DevCube &c, uint32_t *at, cudaStream_t st);

// Quad words and block maxima of slots slot[0..njobs) (null: 0..njobs) of a
// pool; the source slots may be another pool than the tables' (same index).
cudaError_t launch_slot_tables(const uint8_t *pool, const uint32_t *slot, uint32_t njobs,
                               uint32_t *quad, uint8_t *bmax, cudaStream_t st);

}  // namespace r3d
