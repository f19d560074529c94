// Virtual slab: a W x H x D window anywhere in a volume, rendered from
// world-anchored toroidal tile grids (render3d's vslab mode: src/core/vslab.h,
// src/vk/vkbackend.c:5675-6660).  The reference decodes cells from its shard
// store on a worker thread and uploads them layer by layer; here the volume
// lives on the device, a frame's fills run as kernels on the context's
// stream ahead of the frames that read them, and the validity table is
// published right after.  The fill writes the texels the reference's
// vs_fill / vs_scatter_depth write: the base tile with its one-texel apron
// (duplicated at the volume's near edges, zero past its far edges), and the
// pyramid strips (a 4x4 box of the payload, then 2x2 boxes, truncating)
// scattered into the up to four pyramid tiles they overlap, aprons included.
#include <string.h>

#include <algorithm>
#include <vector>

#include "r3d_build.cuh"
#include "r3d_internal.h"

namespace r3d {

// Fill jobs run together: kernels take a batch's jobs along grid y, each
// writing its own cell's texels (the host ends a batch where two cells would
// share a tile).  A frame that scrolls 56 cells by one slice took 56 launches
// of 4.5 us and takes two of 14 us.
constexpr uint32_t kVsBatch = 32u;
struct VsJobs {
  r3d_vslab_job j[kVsBatch];
  uint32_t nx, ny, px, wz, gx, gy;  // volume extent, payload, ring; the kernel's level grid
};

// Base tile of cell (cx, cy): texel (tx, ty) of world slice zs0 + k holds
// world voxel (cx * px - 1 + tx, cy * px - 1 + ty), clamped up to 0 and zero
// past the volume (vkbackend.c:6089-6111,5992-6010).  One warp per row.
__global__ void __launch_bounds__(256) k_vs_base(const uint8_t *__restrict__ vol,
                                                 const __grid_constant__ VsJobs f,
                                                 uint8_t *__restrict__ tiles) {
  const r3d_vslab_job &j = f.j[blockIdx.y];
  const uint32_t T = f.px + 2u, rows = T * j.nz;
  const size_t plane = (size_t)T * T;
  uint8_t *tile = tiles + (size_t)((uint32_t)(j.cy % f.gy) * f.gx + (uint32_t)(j.cx % f.gx)) * (plane * f.wz);
  for (uint32_t r = blockIdx.x * 8u + (threadIdx.x >> 5); r < rows; r += gridDim.x * 8u) {
    const uint32_t ty = r % T, k = r / T;
    const int64_t wx = j.cx * (int64_t)f.px - 1, wy = j.cy * (int64_t)f.px - 1 + ty, z = j.zs0 + k;
    // rows past the volume: a row of no voxels
    const bool in = wy < (int64_t)f.ny;
    warp_row<false>(tile + (size_t)(z % f.wz) * plane + (size_t)ty * T, T,
                    vol + ((size_t)z * f.ny + (size_t)(in ? max(wy, (int64_t)0) : 0)) * f.nx,
                    in ? wx : 0, in ? f.nx : 0u);
  }
}

// Pyramid level 1 strip of a cell: the truncating 4x4 box of its payload
// (vkbackend.c:5682-5696,6118-6121), n = px / 4 texels a side, per slice.
// Job b's strips start at strip + b * stride.
__global__ void k_vs_down4(const uint8_t *__restrict__ vol, const __grid_constant__ VsJobs f,
                           uint8_t *__restrict__ strip, size_t stride) {
  const r3d_vslab_job &j = f.j[blockIdx.y];
  const uint32_t n = f.px / 4u;
  const size_t plane = (size_t)n * n, total = plane * j.nz;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t x = (uint32_t)(i % n), y = (uint32_t)((i / n) % n), k = (uint32_t)(i / plane);
    const int64_t z = j.zs0 + k, wx = j.cx * (int64_t)f.px + 4u * x;
    uint32_t sum = 0;
    for (uint32_t yy = 0; yy < 4u; yy++) {
      const int64_t wy = j.cy * (int64_t)f.px + 4u * y + yy;
      if (wy >= (int64_t)f.ny || wx >= (int64_t)f.nx) continue;
      sum = __dp4a(load4<false>(vol + ((size_t)z * f.ny + (size_t)wy) * f.nx, (uint32_t)wx, f.nx),
                   0x01010101u, sum);
    }
    strip[blockIdx.y * stride + i] = (uint8_t)(sum / 16u);
  }
}

// Next pyramid strip: truncating 2x2 box of the previous one (n a side).
__global__ void k_vs_down2(const __grid_constant__ VsJobs f, const uint8_t *__restrict__ src,
                           uint32_t n, uint8_t *__restrict__ dst, size_t stride) {
  const uint32_t h = n / 2u;
  const size_t plane = (size_t)h * h, total = plane * f.j[blockIdx.y].nz;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t x = (uint32_t)(i % h), y = (uint32_t)((i / h) % h), k = (uint32_t)(i / plane);
    const uint8_t *s = src + blockIdx.y * stride + (size_t)k * n * n + (size_t)(2u * y) * n + 2u * x;
    dst[blockIdx.y * stride + i] = (uint8_t)((s[0] + s[1] + s[n] + s[n + 1]) / 4u);
  }
}

// Scatters a level strip (n x n texels at level texel (cx * n, cy * n)) into
// the level's tiles it overlaps (vkbackend.c:6032-6057): tile (p, q) holds
// level texels [p * px - 1, p * px + px + 1) of each axis at texel t - p * px
// + 1; tiles p in [max(0, (t0 - 1) / px), (t0 + n) / px].
__global__ void k_vs_scatter(const __grid_constant__ VsJobs f, const uint8_t *__restrict__ strip,
                             size_t stride, uint32_t n, uint32_t base, uint8_t *__restrict__ pool) {
  const r3d_vslab_job &j = f.j[blockIdx.y];
  const int64_t t0x = j.cx * (int64_t)n, t0y = j.cy * (int64_t)n;
  const uint32_t T = f.px + 2u;
  const size_t tplane = (size_t)T * T, tbytes = tplane * f.wz;
  const size_t plane = (size_t)n * n, total = plane * j.nz;
  const int64_t P = f.px;
  int64_t p0x = (t0x - 1) / P, p0y = (t0y - 1) / P;  // truncating, as the reference's
  if (p0x < 0) p0x = 0;
  if (p0y < 0) p0y = 0;
  const int64_t p1x = (t0x + n) / P, p1y = (t0y + n) / P;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total;
       i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t x = (uint32_t)(i % n), y = (uint32_t)((i / n) % n), k = (uint32_t)(i / plane);
    const int64_t tx = t0x + x, ty = t0y + y;
    const uint8_t v = strip[blockIdx.y * stride + i];
    const size_t layer = (size_t)((j.zs0 + k) % f.wz) * tplane;
    for (int64_t q = ty / P - 1; q <= ty / P + 1; q++) {
      if (q < p0y || q > p1y || ty < q * P - 1 || ty >= q * P + P + 1) continue;
      for (int64_t p = tx / P - 1; p <= tx / P + 1; p++) {
        if (p < p0x || p > p1x || tx < p * P - 1 || tx >= p * P + P + 1) continue;
        const uint32_t tile = base + (uint32_t)(q % f.gy) * f.gx + (uint32_t)(p % f.gx);
        pool[(size_t)tile * tbytes + layer + (size_t)(ty - q * P + 1) * T + (tx - p * P + 1)] = v;
      }
    }
  }
}

// Blocks along x for n elements (a thread each) of every job of nj.
static unsigned grid_for(size_t n, uint32_t nj) {
  return (unsigned)std::max<size_t>(
      std::min<size_t>((n + 255) / 256, std::max(148u * 16u / nj, 16u)), 1u);
}

// A batch of fill jobs on the context's stream.
static cudaError_t vs_fill(r3d_cuda_ctx *c, const r3d_vslab_job *jobs, uint32_t nj) {
  if (!nj) return cudaSuccess;
  const r3d_vslab_layout &v = c->vsl;
  const uint32_t P = v.px, T = P + 2u;
  cudaStream_t st = c->stream;
  VsJobs f;
  uint32_t nz = 0;
  for (uint32_t k = 0; k < nj; k++) {
    f.j[k] = jobs[k];
    nz = std::max(nz, jobs[k].nz);
  }
  f.nx = (uint32_t)v.nx, f.ny = (uint32_t)v.ny, f.px = P, f.wz = v.wz;
  const auto level = [&](uint32_t l) -> const VsJobs & {
    f.gx = v.gx[l], f.gy = v.gy[l];
    return f;
  };
  const size_t tbytes = (size_t)T * T * v.wz, stride = c->vs_strip_bytes;
  k_vs_base<<<dim3(grid_for((size_t)T * nz * 32u, nj), nj), 256, 0, st>>>(
      c->vs_src, level(0), c->vs_tiles + (size_t)v.base[0] * tbytes);
  if (v.gx[1]) {
    uint32_t n = P / 4u;
    k_vs_down4<<<dim3(grid_for((size_t)n * n * nz, nj), nj), 256, 0, st>>>(
        c->vs_src, level(0), c->vs_strip + c->vs_strip_off[1], stride);
    for (uint32_t l = 2; l < R3D_VS_LEVELS && v.gx[l]; l++) {
      k_vs_down2<<<dim3(grid_for((size_t)(n / 2u) * (n / 2u) * nz, nj), nj), 256, 0, st>>>(
          level(0), c->vs_strip + c->vs_strip_off[l - 1], n, c->vs_strip + c->vs_strip_off[l], stride);
      n /= 2u;
    }
    for (uint32_t l = 1; l < R3D_VS_LEVELS && v.gx[l]; l++) {
      const uint32_t m = P / v.s[l];
      k_vs_scatter<<<dim3(grid_for((size_t)m * m * nz, nj), nj), 256, 0, st>>>(
          level(l), c->vs_strip + c->vs_strip_off[l], stride, m, v.base[l], c->vs_tiles);
    }
  }
  return cudaGetLastError();
}

// Whether two cells would write the same tile of a level as different tiles
// of the plane (grids are toroidal; the scheduler's windows never do, and a
// batch ends before a job that would).
static bool vs_collide(const r3d_vslab_layout &v, const r3d_vslab_job &a, const r3d_vslab_job &b) {
  for (uint32_t l = 0; l < R3D_VS_LEVELS && v.gx[l]; l++) {
    const int64_t n = v.px / v.s[l], P = v.px;
    // tiles [lo, hi] a job writes along an axis: its cell's at the base, the
    // overlapped ones above
    const auto lo = [&](int64_t c) { return l ? std::max<int64_t>((c * n - 1) / P, 0) : c; };
    const auto hi = [&](int64_t c) { return l ? (c * n + n) / P : c; };
    bool same[2] = {false, false}, other[2] = {false, false};
    const int64_t ca[2] = {a.cx, a.cy}, cb[2] = {b.cx, b.cy}, g[2] = {v.gx[l], v.gy[l]};
    for (int x = 0; x < 2; x++)
      for (int64_t p = lo(ca[x]); p <= hi(ca[x]); p++)
        for (int64_t q = lo(cb[x]); q <= hi(cb[x]); q++) {
          same[x] = same[x] || p == q;
          other[x] = other[x] || (p != q && (p - q) % g[x] == 0);
        }
    if ((other[0] && (same[1] || other[1])) || (other[1] && same[0])) return true;
  }
  return false;
}

}  // namespace r3d

using namespace r3d;

void vslab_reset(r3d_cuda_ctx *c) {
  cudaFree(c->vs_src);
  cudaFree(c->vs_tiles);
  cudaFree(c->vs_strip);
  cudaFree(c->vs_table);
  c->vs_src = c->vs_tiles = c->vs_strip = nullptr;
  c->vs_table = nullptr;
  c->vs_table_host.clear();
  c->vs_cells.clear();
  c->vs_jobs.clear();
  c->have_vslab = false;
  c->vs = DevVslab{};
}

extern "C" {

int r3d_cuda_vslab_begin(r3d_cuda_ctx *c, const r3d_volume_desc *d, const uint8_t *voxels,
                         uint32_t W, uint32_t H, uint32_t D, uint32_t z_margin) {
  if (!c || !d || !voxels || !d->nx || !d->ny || !d->nz)
    return fail(c, R3D_E_INVALID, "vslab_begin: bad arguments");
  r3d_vslab_layout v;
  if (r3d_host_vslab_init(&v, d->nx, d->ny, d->nz, W, H, D, z_margin) != 0)
    return fail(c, R3D_E_INVALID, "vslab_begin: bad %ux%ux%u window (margin %u) for %ux%ux%u",
                W, H, D, z_margin, d->nx, d->ny, d->nz);
  if (v.gx[0] > 63u || v.gy[0] > 63u)
    return fail(c, R3D_E_INVALID, "vslab_begin: %ux%u base tiles exceed slab_grid", v.gx[0],
                v.gy[0]);
  for (uint32_t l = 1; l < R3D_VS_LEVELS; l++)
    if (v.gx[l] > 15u || v.gy[l] > 15u)
      return fail(c, R3D_E_INVALID, "vslab_begin: level %u grid exceeds brick_mode", l);
  cudaSetDevice(c->device);
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  vslab_reset(c);
  const size_t T = v.px + 2u, tbytes = T * T * v.wz;
  const size_t vbytes = (size_t)d->nx * d->ny * d->nz;
  size_t strip = 0;
  for (uint32_t l = 1; l < R3D_VS_LEVELS; l++) {
    const size_t n = v.px / v.s[l];
    c->vs_strip_off[l] = strip;
    strip += (n * n * v.wz + 255u) & ~(size_t)255u;
  }
  c->vs_strip_bytes = strip;
  const uint32_t nslot = v.gx[0] * v.gy[0];
  cudaError_t e = cudaMalloc(&c->vs_src, vbytes + 4u);  // + 4: load4
  if (e == cudaSuccess) e = cudaMalloc(&c->vs_tiles, tbytes * v.ntiles);
  c->vs_batch = v.gx[1] ? kVsBatch : 1u;  // strips of a whole batch, else of one job
  if (e == cudaSuccess && cudaMalloc(&c->vs_strip, strip * c->vs_batch) != cudaSuccess) {
    cudaGetLastError();
    c->vs_batch = 1u;
    e = cudaMalloc(&c->vs_strip, strip);
  }
  if (!v.gx[1]) c->vs_batch = kVsBatch;  // no pyramid: no strips
  if (e == cudaSuccess) e = cudaMalloc(&c->vs_table, (size_t)nslot * 16u);
  if (e == cudaSuccess) e = copy_sync(c->stream, c->vs_src, voxels, vbytes);
  if (e == cudaSuccess) e = cudaMemsetAsync(c->vs_tiles, 0, tbytes * v.ntiles, c->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(c->vs_table, 0, (size_t)nslot * 16u, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) {
    vslab_reset(c);
    return cuda_fail(c, e, "vslab_begin");
  }
  c->vsl = v;
  c->vs_cells.assign(nslot, r3d_vslab_cell{INT64_MIN, INT64_MIN, 0, 0});
  c->vs_table_host.assign((size_t)nslot * 4u, 0u);
  DevVslab dv{};
  dv.tiles = c->vs_tiles;
  dv.table = c->vs_table;
  dv.tile_bytes = tbytes;
  dv.px = v.px;
  dv.wz = v.wz;
  for (uint32_t l = 0; l < R3D_VS_LEVELS; l++) {
    dv.gx[l] = v.gx[l];
    dv.gy[l] = v.gy[l];
    dv.base[l] = v.base[l];
    dv.rg[l][0] = v.gx[l] ? 1.0f / (float)v.gx[l] : 0.0f;
    dv.rg[l][1] = v.gy[l] ? 1.0f / (float)v.gy[l] : 0.0f;
  }
  dv.rp = 1.0f / (float)v.px;
  dv.rt = 1.0f / ((float)v.px + 2.0f);
  dv.rwz = 1.0f / (float)v.wz;
  dv.nx = (float)v.W;
  c->vs = dv;
  c->have_vslab = true;
  return R3D_OK;
}

int r3d_cuda_vslab_frame(r3d_cuda_ctx *c, double fx, double fy, int64_t z0, uint32_t budget,
                         r3d_frame_params *p, r3d_vslab_stats *st) {
  if (!c) return R3D_E_INVALID;
  if (!c->have_vslab) return fail(c, R3D_E_STATE, "vslab_frame: no virtual slab");
  cudaSetDevice(c->device);
  r3d_vslab_layout &v = c->vsl;
  c->vs_jobs.resize(64u + 48u);
  const uint32_t nj = r3d_host_vslab_plan(&v, c->vs_cells.data(), fx, fy, z0, budget,
                                          c->vs_jobs.data(), (uint32_t)c->vs_jobs.size());
  c->vs_jobs.resize(nj);
  uint32_t slices = 0;
  for (uint32_t k = 0, k0 = 0; k < nj; k++) {
    const r3d_vslab_job &j = c->vs_jobs[k];
    slices += j.nz;
    const uint32_t slot = r3d_host_vslab_apply(&v, c->vs_cells.data(), &j, v.z0);
    const r3d_vslab_cell &cell = c->vs_cells[slot];
    uint32_t *w = &c->vs_table_host[(size_t)slot * 4u];
    w[0] = r3d_host_vslab_key(cell.cx, cell.cy);
    w[1] = (uint32_t)cell.za;
    w[2] = (uint32_t)cell.zb;
    // the batch of jobs [k0, k] goes out when it is full, last, or the next
    // job may not run beside one of it
    bool last = k + 1u == nj || k + 1u - k0 == c->vs_batch;
    for (uint32_t m = k0; m <= k && !last; m++) last = vs_collide(v, c->vs_jobs[m], c->vs_jobs[k + 1u]);
    if (last) {
      R3D_CUDA_TRY(c, vs_fill(c, &c->vs_jobs[k0], k + 1u - k0));
      k0 = k + 1u;
    }
  }
  // publish the table after the fills, in stream order (a pageable copy is
  // staged before this returns, so the host copy may change right after)
  if (nj)
    R3D_CUDA_TRY(c, cudaMemcpyAsync(c->vs_table, c->vs_table_host.data(),
                                    c->vs_table_host.size() * 4u, cudaMemcpyHostToDevice,
                                    c->stream));
  c->vs.x0 = (float)v.x0;
  c->vs.y0 = (float)v.y0;
  c->vs.z0 = (float)v.z0;
  if (st) {
    int64_t c0x, c1x, c0y, c1y;
    r3d_host_vslab_range(&v, 0, v.x0, v.nx, v.W, &c0x, &c1x);
    r3d_host_vslab_range(&v, 0, v.y0, v.ny, v.H, &c0y, &c1y);
    int64_t vis_end = v.z0 + (int64_t)v.D + 2;
    if (vis_end > (int64_t)v.nz) vis_end = (int64_t)v.nz;
    uint32_t pending = 0;
    for (int64_t cy = c0y; cy <= c1y; cy++)
      for (int64_t cx = c0x; cx <= c1x; cx++) {
        const r3d_vslab_cell &cell =
            c->vs_cells[(uint32_t)(cy % v.gy[0]) * v.gx[0] + (uint32_t)(cx % v.gx[0])];
        pending += !(cell.cx == cx && cell.cy == cy && cell.za <= v.z0 && cell.zb >= vis_end);
      }
    st->jobs = nj;
    st->slices = slices;
    st->pending = pending;
    st->pad = 0;
    st->origin[0] = v.x0;
    st->origin[1] = v.y0;
    st->origin[2] = v.z0;
  }
  if (p) r3d_cuda_vslab_params(c, p);
  return R3D_OK;
}

void r3d_cuda_vslab_params(const r3d_cuda_ctx *c, r3d_frame_params *p) {
  if (!c || !p || !c->have_vslab) return;
  const r3d_vslab_layout &v = c->vsl;
  // vkbackend.c:6628-6645
  p->slab_grid = v.gx[0] | (v.gy[0] << 6) | kVslabGrid;
  uint32_t bm = 0;
  for (uint32_t l = 1; l < R3D_VS_LEVELS; l++) bm |= (v.gx[l] | (v.gy[l] << 4)) << ((l - 1u) * 8u);
  p->brick_mode = bm;
  p->slab_wz = v.wz;
  p->slab_z0 = (float)(v.z0 < 0 ? 0 : v.z0);
  p->slab_nx = (float)v.W;
  p->slab_ny = (float)v.H;
  p->slab_px = (float)v.px;
  p->slab_py = (float)v.px;
  p->slab_depth = v.D;
  p->slab_x0 = (float)(v.x0 < 0 ? 0 : v.x0);
  p->slab_y0 = (float)(v.y0 < 0 ? 0 : v.y0);
  p->clip_valid = 0u;
}

int r3d_cuda_vslab_layout(const r3d_cuda_ctx *c, r3d_vslab_layout *out) {
  if (!c || !out) return R3D_E_INVALID;
  if (!c->have_vslab) return R3D_E_STATE;
  *out = c->vsl;
  return R3D_OK;
}

int r3d_cuda_vslab_read(r3d_cuda_ctx *c, uint32_t tile, uint8_t *out) {
  if (!c || !out) return R3D_E_INVALID;
  if (!c->have_vslab) return fail(c, R3D_E_STATE, "vslab_read: no virtual slab");
  if (tile >= c->vsl.ntiles) return fail(c, R3D_E_INVALID, "vslab_read: tile %u", tile);
  cudaSetDevice(c->device);
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  const size_t tb = c->vs.tile_bytes;
  R3D_CUDA_TRY(c, cudaMemcpy(out, c->vs_tiles + (size_t)tile * tb, tb, cudaMemcpyDeviceToHost));
  return R3D_OK;
}

int r3d_cuda_vslab_table(r3d_cuda_ctx *c, uint32_t *out) {
  if (!c || !out) return R3D_E_INVALID;
  if (!c->have_vslab) return fail(c, R3D_E_STATE, "vslab_table: no virtual slab");
  cudaSetDevice(c->device);
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  R3D_CUDA_TRY(c, cudaMemcpy(out, c->vs_table, c->vs_table_host.size() * 4u,
                             cudaMemcpyDeviceToHost));
  return R3D_OK;
}

}  // extern "C"
