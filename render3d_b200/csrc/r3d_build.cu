// Device-side builders of the LOD brick cache: the box pyramid with its
// per-brick maxima, and the slots' derived tables (quad words and dilated
// 8^3 block maxima).  All of them move bytes: the design is one pass over
// each level, four to sixteen bytes a lane, and every table of a slot made
// from the words that are already in registers.
#include "r3d_build.cuh"

namespace r3d {

// 2x box reduction of one pyramid level, zeros outside the source, and the
// maximum of every 128^3 source brick in the same pass: dst voxel = (sum of
// its 2^3 source voxels + 4) / 8 (tools/lodpack/main.c:203-230).  dst may be
// null (the coarsest level: maxima only), vmax too.
//
// Bound by DRAM: 1 byte read and 1/8 written per source voxel.  A lane makes
// four outputs from four rows of 8 source bytes (two words, summed as 16-bit
// pairs); a warp covers 128 outputs, that is two source bricks along x, and
// walks rows and planes of one brick, so that the maxima cost one reduction
// over 16 lanes and one atomic per warp.  The level-0 pass of a 1024^3
// volume with its brick maxima took 0.90 + 4.31 ms as two byte-wise kernels
// (one thread per voxel; one row per thread) and takes 0.27 ms (4.5 TB/s);
// two output planes a block, since eight left the small levels with too few
// blocks (0.32, 0.09 and 0.09 ms for levels 0, 1 and 2; now 0.27, 0.05, 0.02).
constexpr uint32_t kDownY = 64u, kDownZ = 2u;  // output rows and planes of a block

template <bool VEC>
__global__ void __launch_bounds__(256) k_level_down(const uint8_t *__restrict__ src, uint32_t sx,
                                                    uint32_t sy, uint32_t sz,
                                                    uint8_t *__restrict__ dst, uint32_t dx,
                                                    uint32_t dy, uint32_t *__restrict__ vmax,
                                                    uint32_t bdx, uint32_t bdy) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t ox = blockIdx.x * 128u + lane * 4u;  // first output of the lane
  uint32_t m = 0;
  for (uint32_t zi = 0; zi < kDownZ; zi++) {
    const uint32_t oz = blockIdx.z * kDownZ + zi;
#pragma unroll 4
    for (uint32_t yi = 0; yi < kDownY / 8u; yi++) {
      const uint32_t oy = blockIdx.y * kDownY + yi * 8u + warp;
      uint32_t s0 = 0x00040004u, s1 = 0x00040004u;  // pair sums of outputs 0, 1 and 2, 3
#pragma unroll
      for (uint32_t k = 0; k < 4u; k++) {
        const uint32_t y = 2u * oy + (k & 1u), z = 2u * oz + (k >> 1);
        uint2 w = make_uint2(0u, 0u);
        if (y < sy && z < sz)
          w = load8<VEC>(src + ((size_t)z * sy + y) * sx, 2u * ox, sx, VEC || inner_row(y, z, sx, sy, sz));
        s0 += (w.x & 0x00FF00FFu) + ((w.x >> 8) & 0x00FF00FFu);
        s1 += (w.y & 0x00FF00FFu) + ((w.y >> 8) & 0x00FF00FFu);
        m = __vmaxu4(m, __vmaxu4(w.x, w.y));
      }
      if (dst) {
        s0 = (s0 >> 3) & 0x00FF00FFu;
        s1 = (s1 >> 3) & 0x00FF00FFu;
        *reinterpret_cast<uint32_t *>(dst + ((size_t)oz * dy + oy) * dx + ox) =
            __byte_perm(s0, s1, 0x6420);
      }
    }
  }
  if (!vmax) return;
  m = max_byte(m);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
  // source brick: x 256 * blockIdx.x + 8 * lane, y and z likewise halved
  const uint32_t bx = blockIdx.x * 2u + (lane >> 4), by = blockIdx.y * kDownY / 64u,
                 bz = blockIdx.z * kDownZ / 64u;
  if ((lane & 15u) == 0u && m) atomicMax(vmax + ((size_t)bz * bdy + by) * bdx + bx, m);
}

cudaError_t launch_level_down(const uint8_t *src, uint32_t sx, uint32_t sy, uint32_t sz,
                              uint8_t *dst, uint32_t dx, uint32_t dy, uint32_t dz, uint32_t *vmax,
                              uint32_t bdx, uint32_t bdy, cudaStream_t st) {
  const dim3 grid(dx / 128u, dy / kDownY, dz / kDownZ);
  // vector loads: every row of the source starts on 8 bytes
  if (sx % 8u == 0u && ((uintptr_t)src & 7u) == 0u)
    k_level_down<true><<<grid, 256, 0, st>>>(src, sx, sy, sz, dst, dx, dy, vmax, bdx, bdy);
  else
    k_level_down<false><<<grid, 256, 0, st>>>(src, sx, sy, sz, dst, dx, dy, vmax, bdx, bdy);
  return cudaGetLastError();
}

// The slots' bytes, quad words (DevBricks::quad) and dilated 8^3 block
// maxima (DevBricks::bmax: max over voxels [8b, min(8b + 8, 127)] per axis)
// in one pass.  SRC 0: from the slots of a pool; 1: from the bricks of
// pyramid levels (zero outside a level's extent), the slot bytes written on
// the way.  Null outputs are left out.
//
// Bound by the DRAM writes: 4 bytes of quad word per voxel beside 1 read
// (and 1 written with SRC 1).  A block makes the 8 planes of one z block of
// a slot, a warp 16 rows of each (two y blocks), a lane 4 voxels: the
// plane's 17 row words are loaded together, the word's right neighbour comes
// from the next lane by shuffle, and a lane stores its four quad words as 16
// bytes, 512 contiguous bytes a warp.  The block maxima fold the same words
// over rows and planes (the ninth plane is loaded for them alone, 1/8 more
// reads, mostly from L2) and over lane pairs at the end.  The 585 slots of a
// 1024^3 cache took 1.20 ms (copy) + 2.45 ms (quad words) + 0.78 ms (maxima)
// as three byte-wise kernels and take 1.24 ms (5.9 TB/s).
struct FillJobs {
  LevelSrc lev[kMaxLevels];
  uint32_t nlev;
  const uint32_t *brick, *slot;  // per job: brick of its level (SRC 1), slot (null: the job)
  uint32_t job0;                 // first job of the launch
};

template <int SRC, bool VEC>
__global__ void __launch_bounds__(256) k_slot_fill(const __grid_constant__ FillJobs f,
                                                   const uint8_t *__restrict__ from,
                                                   uint8_t *__restrict__ pool,
                                                   uint32_t *__restrict__ quad,
                                                   uint8_t *__restrict__ bmax) {
  const uint32_t lane = threadIdx.x & 31u, warp = threadIdx.x >> 5;
  const uint32_t bz = blockIdx.x, job = f.job0 + blockIdx.y;
  const uint32_t slot = f.slot ? f.slot[job] : job;
  const size_t base = (size_t)slot * (128u * 128u * 128u);
  // SRC 1: origin and extent of the job's brick in its level
  const uint8_t *g = nullptr;
  uint32_t ex = 128u, ey = 128u, ez = 128u, x0 = 0u, y0 = 0u, z0 = 0u;
  if (SRC == 0) {
    g = from + base;
  } else {
    uint32_t l = 0;
    while (l + 1u < f.nlev && job >= f.lev[l + 1u].job0) l++;
    const LevelSrc &L = f.lev[l];
    const uint32_t b = f.brick[job];
    g = L.p;
    ex = L.ex, ey = L.ey, ez = L.ez;
    x0 = (b % L.bdx) * 128u, y0 = (b / L.bdx % L.bdy) * 128u, z0 = (b / L.bdx / L.bdy) * 128u;
  }
  const uint32_t yr = warp * 16u;
  uint32_t m0 = 0, m1 = 0;  // maxima of y blocks 2 warp and 2 warp + 1
#pragma unroll 1
  for (uint32_t zi = 0; zi < 9u; zi++) {
    const uint32_t z = bz * 8u + zi;
    if (z > 127u || (zi == 8u && !bmax)) break;
    uint32_t r[17];
#pragma unroll
    for (uint32_t i = 0; i < 17u; i++) {
      const uint32_t y = min(yr + i, 127u);
      r[i] = 0u;
      if (z0 + z < ez && y0 + y < ey) {
        const uint8_t *row = g + ((size_t)(z0 + z) * ey + (y0 + y)) * ex;
        r[i] = load4<VEC>(row, x0 + lane * 4u, ex, VEC || inner_row(y0 + y, z0 + z, ex, ey, ez));
      }
    }
#pragma unroll
    for (uint32_t i = 0; i < 9u; i++) m0 = __vmaxu4(m0, r[i]);
#pragma unroll
    for (uint32_t i = 8; i < 17u; i++) m1 = __vmaxu4(m1, r[i]);
    if (zi == 8u) break;
    const size_t at = base + ((size_t)z << 14) + (yr << 7) + lane * 4u;
    uint32_t lo, hi;  // (v0, v1, v1, v2) and (v2, v3, v3, v4) of row i: pairs (x, x + 1)
    {
      const uint32_t n = __shfl_down_sync(0xffffffffu, r[0], 1);
      const uint32_t nb = lane == 31u ? r[0] >> 24 : n;
      lo = __byte_perm(r[0], 0u, 0x2110);
      hi = __byte_perm(r[0], nb, 0x4332);
    }
#pragma unroll
    for (uint32_t i = 0; i < 16u; i++) {
      const uint32_t n = __shfl_down_sync(0xffffffffu, r[i + 1], 1);
      const uint32_t nb = lane == 31u ? r[i + 1] >> 24 : n;
      const uint32_t lo1 = __byte_perm(r[i + 1], 0u, 0x2110), hi1 = __byte_perm(r[i + 1], nb, 0x4332);
      if (quad)
        *reinterpret_cast<uint4 *>(quad + at + i * 128u) =
            make_uint4(__byte_perm(lo, lo1, 0x5410), __byte_perm(lo, lo1, 0x7632),
                       __byte_perm(hi, hi1, 0x5410), __byte_perm(hi, hi1, 0x7632));
      if (SRC == 1 && pool) *reinterpret_cast<uint32_t *>(pool + at + i * 128u) = r[i];
      lo = lo1;
      hi = hi1;
    }
  }
  if (!bmax) return;
#pragma unroll
  for (uint32_t k = 0; k < 2u; k++) {
    uint32_t m = k ? m1 : m0;
    const uint32_t r1 = __shfl_down_sync(0xffffffffu, m, 1), r2 = __shfl_down_sync(0xffffffffu, m, 2);
    m = max_byte(__vmaxu4(m, r1));
    if (lane < 30u) m = max(m, r2 & 0xFFu);
    if (!(lane & 1u))
      bmax[(size_t)slot * 4096u + bz * 256u + (2u * warp + k) * 16u + (lane >> 1)] = (uint8_t)m;
  }
}

cudaError_t launch_slot_fill(const LevelSrc *lev, uint32_t nlev, const uint32_t *brick,
                             const uint32_t *slot, uint32_t njobs, uint8_t *pool, uint32_t *quad,
                             uint8_t *bmax, cudaStream_t st) {
  FillJobs f;
  bool vec = true;
  for (uint32_t l = 0; l < nlev; l++) {
    f.lev[l] = lev[l];
    vec = vec && lev[l].ex % 4u == 0u && ((uintptr_t)lev[l].p & 3u) == 0u;
  }
  f.nlev = nlev;
  f.brick = brick;
  f.slot = slot;
  for (uint32_t j0 = 0; j0 < njobs; j0 += 65535u) {
    f.job0 = j0;
    const dim3 grid(16u, njobs - j0 < 65535u ? njobs - j0 : 65535u);
    if (vec)
      k_slot_fill<1, true><<<grid, 256, 0, st>>>(f, nullptr, pool, quad, bmax);
    else
      k_slot_fill<1, false><<<grid, 256, 0, st>>>(f, nullptr, pool, quad, bmax);
  }
  return cudaGetLastError();
}

cudaError_t launch_slot_tables(const uint8_t *pool, const uint32_t *slot, uint32_t njobs,
                               uint32_t *quad, uint8_t *bmax, cudaStream_t st) {
  FillJobs f;
  f.nlev = 0u;
  f.brick = nullptr;
  f.slot = slot;
  // a pool handed over by a caller may start at any byte
  const bool vec = ((uintptr_t)pool & 3u) == 0u;
  for (uint32_t j0 = 0; j0 < njobs; j0 += 65535u) {
    f.job0 = j0;
    const dim3 grid(16u, njobs - j0 < 65535u ? njobs - j0 : 65535u);
    if (vec)
      k_slot_fill<0, true><<<grid, 256, 0, st>>>(f, pool, nullptr, quad, bmax);
    else
      k_slot_fill<0, false><<<grid, 256, 0, st>>>(f, pool, nullptr, quad, bmax);
  }
  return cudaGetLastError();
}

// A warp per output row of the kernels below: words of four bytes a lane,
// loaded at whatever alignment the row has.
static unsigned row_blocks(uint64_t rows) {
  const uint64_t b = (rows + 7u) / 8u;
  return (unsigned)(b < 148u * 32u ? (b ? b : 1u) : 148u * 32u);
}

// Next mip: clamped coordinates matter only where the source has one texel
// (elsewhere 2 d <= s).  The mips of a 1024^3 cube took 0.77 ms a byte a
// thread; rows that start on 8 bytes are loaded in whole words (VEC), which
// took a 1024^3 shard build from 2.81 to 2.36 ms.
template <bool VEC>
__global__ void __launch_bounds__(256) k_mip(const uint8_t *__restrict__ src, uint32_t sx,
                                             uint32_t sy, uint32_t sz, uint8_t *__restrict__ dst,
                                             uint32_t dx, uint32_t dy, uint32_t dz) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t rows = (uint64_t)dy * dz;
  for (uint64_t r = blockIdx.x * 8ull + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8ull) {
    const uint32_t y = (uint32_t)(r % dy), z = (uint32_t)(r / dy);
    for (uint32_t x = lane * 4u; x < dx; x += 128u) {
      uint32_t s0 = 0x00040004u, s1 = 0x00040004u;
#pragma unroll
      for (uint32_t k = 0; k < 4u; k++) {
        const uint32_t yy = min(2u * y + (k & 1u), sy - 1u), zz = min(2u * z + (k >> 1), sz - 1u);
        uint2 w = load8<VEC>(src + ((size_t)zz * sy + yy) * sx, 2u * x, sx);
        if (sx == 1u) w.x |= w.x << 8;
        s0 += (w.x & 0x00FF00FFu) + ((w.x >> 8) & 0x00FF00FFu);
        s1 += (w.y & 0x00FF00FFu) + ((w.y >> 8) & 0x00FF00FFu);
      }
      const uint32_t v = __byte_perm((s0 >> 3) & 0x00FF00FFu, (s1 >> 3) & 0x00FF00FFu, 0x6420);
      uint8_t *o = dst + r * dx + x;
      if (!(dx & 3u)) {
        *reinterpret_cast<uint32_t *>(o) = v;
      } else {
        for (uint32_t k = 0; k < 4u && x + k < dx; k++) o[k] = (uint8_t)(v >> (8u * k));
      }
    }
  }
}

cudaError_t launch_mip(const uint8_t *src, uint32_t sx, uint32_t sy, uint32_t sz, uint8_t *dst,
                       uint32_t dx, uint32_t dy, uint32_t dz, cudaStream_t st) {
  const unsigned grid = row_blocks((uint64_t)dy * dz);
  if (sx % 8u == 0u && ((uintptr_t)src & 7u) == 0u)
    k_mip<true><<<grid, 256, 0, st>>>(src, sx, sy, sz, dst, dx, dy, dz);
  else
    k_mip<false><<<grid, 256, 0, st>>>(src, sx, sy, sz, dst, dx, dy, dz);
  return cudaGetLastError();
}

// 8^3 block maxima (src/vk/vkbackend.c:794-824), a lane per block: eight
// bytes of each of its 64 rows.
template <bool VEC>
__global__ void __launch_bounds__(256) k_occ_raw(const uint8_t *__restrict__ vox, uint32_t nx,
                                                 uint32_t ny, uint32_t nz,
                                                 uint8_t *__restrict__ raw, uint32_t ox,
                                                 uint32_t oy, uint32_t oz) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t rows = (uint64_t)oy * oz;
  for (uint64_t r = blockIdx.x * 8ull + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8ull) {
    const uint32_t y0 = (uint32_t)(r % oy) * 8u, z0 = (uint32_t)(r / oy) * 8u;
    const uint32_t y1 = min(y0 + 8u, ny), z1 = min(z0 + 8u, nz);
    for (uint32_t b = lane; b < ox; b += 32u) {
      uint32_t m = 0;
      for (uint32_t z = z0; z < z1; z++)
#pragma unroll 8
        for (uint32_t y = y0; y < y1; y++) {
          const uint2 w = load8<VEC>(vox + ((size_t)z * ny + y) * nx, 8u * b, nx);
          m = __vmaxu4(m, __vmaxu4(w.x, w.y));
        }
      raw[r * ox + b] = (uint8_t)max_byte(m);
    }
  }
}

cudaError_t launch_occ_raw(const uint8_t *vox, uint32_t nx, uint32_t ny, uint32_t nz, uint8_t *raw,
                           cudaStream_t st) {
  const uint32_t ox = (nx + 7u) / 8u, oy = (ny + 7u) / 8u, oz = (nz + 7u) / 8u;
  if (nx % 8u == 0u && ((uintptr_t)vox & 7u) == 0u)
    k_occ_raw<true><<<row_blocks((uint64_t)oy * oz), 256, 0, st>>>(vox, nx, ny, nz, raw, ox, oy, oz);
  else
    k_occ_raw<false><<<row_blocks((uint64_t)oy * oz), 256, 0, st>>>(vox, nx, ny, nz, raw, ox, oy, oz);
  return cudaGetLastError();
}

// Quad words of a level: bound by the 4 bytes written per texel.
__global__ void __launch_bounds__(256) k_level_quads(const uint8_t *__restrict__ src, uint32_t dx,
                                                     uint32_t dy, uint32_t dz,
                                                     uint32_t *__restrict__ quad) {
  const uint32_t lane = threadIdx.x & 31u;
  const uint64_t rows = (uint64_t)dy * dz;
  for (uint64_t r = blockIdx.x * 8ull + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8ull) {
    const uint8_t *row = src + r * dx, *next = r % dy + 1u < dy ? row + dx : row;
    for (uint32_t x = lane * 4u; x < dx; x += 128u) {
      // the row's bytes x .. x + 3 and, clamped, x + 4
      uint32_t a = load4<false>(row, x, dx), b = load4<false>(next, x, dx);
      const uint32_t left = dx - x;
      if (left < 4u) {  // the last texel's neighbour is itself
        a |= (a >> (8u * (left - 1u)) & 0xFFu) << (8u * left);
        b |= (b >> (8u * (left - 1u)) & 0xFFu) << (8u * left);
      }
      const uint32_t an = left > 4u ? row[x + 4u] : a >> 24, bn = left > 4u ? next[x + 4u] : b >> 24;
      const uint32_t alo = __byte_perm(a, 0u, 0x2110), ahi = __byte_perm(a, an, 0x4332);
      const uint32_t blo = __byte_perm(b, 0u, 0x2110), bhi = __byte_perm(b, bn, 0x4332);
      const uint32_t q[4] = {__byte_perm(alo, blo, 0x5410), __byte_perm(alo, blo, 0x7632),
                             __byte_perm(ahi, bhi, 0x5410), __byte_perm(ahi, bhi, 0x7632)};
      uint32_t *o = quad + r * dx + x;
      if (!(dx & 3u)) {
        *reinterpret_cast<uint4 *>(o) = make_uint4(q[0], q[1], q[2], q[3]);
      } else {
#pragma unroll
        for (uint32_t k = 0; k < 4u; k++)
          if (k < left) o[k] = q[k];
      }
    }
  }
}

cudaError_t launch_level_quads(const uint8_t *src, uint32_t dx, uint32_t dy, uint32_t dz,
                               uint32_t *quad, cudaStream_t st) {
  k_level_quads<<<row_blocks((uint64_t)dy * dz), 256, 0, st>>>(src, dx, dy, dz, quad);
  return cudaGetLastError();
}

size_t cube_quad_bytes(DevCube &c) {
  if ((uint64_t)c.dim[0][0] * c.dim[0][1] * c.dim[0][2] > kQuadVoxels) return 0;
  size_t words = 0;
  for (uint32_t m = 0; m < c.nlevels; m++) {
    c.qoff[m] = (uint32_t)words;
    words += ((size_t)c.dim[m][0] * c.dim[m][1] * c.dim[m][2] + 63u) & ~(size_t)63u;
  }
  return words * sizeof(uint32_t);
}

bool words_fit(size_t bytes, size_t words, size_t back) {
  size_t left = 0, all = 0;
  if (words <= (size_t)1 << 30) return true;
  if (cudaMemGetInfo(&left, &all) != cudaSuccess) {
    cudaGetLastError();
    return true;
  }
  return left + back >= bytes + words + all / 4u;
}

cudaError_t build_cube_quads(DevCube &c, uint32_t *at, cudaStream_t st) {
  c.quad = at;
  cudaError_t e = cudaSuccess;
  for (uint32_t m = 0; m < c.nlevels && at && e == cudaSuccess; m++)
    e = launch_level_quads(c.lev[m], c.dim[m][0], c.dim[m][1], c.dim[m][2], at + c.qoff[m], st);
  return e;
}

}  // namespace r3d
