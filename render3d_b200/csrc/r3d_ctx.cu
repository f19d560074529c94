// C-ABI entry points: context, scene uploads and device-side builders (mip
// chain, occupancy grid, LOD brick pyramid and page table), forward raycast.
#include <stdarg.h>
#include <stdio.h>
#include <string.h>

#include <algorithm>
#include <vector>

#include "r3d_build.cuh"
#include "r3d_internal.h"

namespace r3d {

int fail(r3d_cuda_ctx *c, int code, const char *fmt, ...) {
  char buf[512];
  va_list ap;
  va_start(ap, fmt);
  vsnprintf(buf, sizeof buf, fmt, ap);
  va_end(ap);
  if (c) c->err = buf;
  return code;
}

int cuda_fail(r3d_cuda_ctx *c, cudaError_t e, const char *what) {
  return fail(c, e == cudaErrorMemoryAllocation ? R3D_E_NOMEM : R3D_E_CUDA, "%s: %s (%s)", what,
              cudaGetErrorName(e), cudaGetErrorString(e));
}

bool is_device_ptr(const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice || a.type == cudaMemoryTypeManaged;
}

bool readable_in_place(const r3d_cuda_ctx *c, const void *p) {
  cudaPointerAttributes a;
  if (cudaPointerGetAttributes(&a, p) != cudaSuccess) {
    cudaGetLastError();
    return false;
  }
  return a.type == cudaMemoryTypeDevice && a.device == c->device;
}

cudaError_t idle_device(r3d_cuda_ctx *c) {
  if (!c->spare && cudaMalloc(&c->spare, 256u) != cudaSuccess) {
    cudaGetLastError();
    return cudaDeviceSynchronize();
  }
  const cudaError_t e = cudaFree(c->spare);
  if (e != cudaSuccess) return e;
  c->spare = nullptr;
  if (cudaMalloc(&c->spare, 256u) != cudaSuccess) cudaGetLastError();  // taken next time
  return cudaSuccess;
}

// ------------------------------------------------------------- builders

// 26-neighbour max dilation (src/vk/vkbackend.c:845-860)
__global__ void k_occ_dilate(const uint8_t *__restrict__ raw, uint8_t *__restrict__ dil,
                             uint32_t ox, uint32_t oy, uint32_t oz) {
  size_t n = (size_t)ox * oy * oz;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    int x = (int)(i % ox), y = (int)((i / ox) % oy), z = (int)(i / ox / oy);
    uint32_t m = 0;
    for (int dz = -1; dz <= 1; dz++)
      for (int dy = -1; dy <= 1; dy++)
        for (int dx = -1; dx <= 1; dx++) {
          int zz = z + dz, yy = y + dy, xx = x + dx;
          if (zz < 0 || yy < 0 || xx < 0 || zz >= (int)oz || yy >= (int)oy || xx >= (int)ox)
            continue;
          m = max(m, (uint32_t)raw[((size_t)zz * oy + yy) * ox + xx]);
        }
    dil[i] = (uint8_t)m;
  }
}


template <class T>
static cudaError_t reserve(r3d_cuda_ctx *c, T *&p, size_t &cap, size_t need) {
  if (keeps(p, cap, need)) return idle_device(c);
  cudaFree(p);
  p = nullptr;
  cap = 0;
  const cudaError_t e = cudaMalloc(&p, need);
  if (e == cudaSuccess) cap = need;
  return e;
}

static unsigned grid_for(size_t n) {
  size_t b = (n + 255) / 256;
  return (unsigned)(b < 148u * 64u ? (b ? b : 1) : 148u * 64u);
}

}  // namespace r3d

using namespace r3d;

r3d::DevScene r3d_cuda_ctx::scene() const {
  DevScene s;
  memset(&s, 0, sizeof s);
  s.cube = cube;
  s.br = br;
  s.sh = sh;
  s.sl = sl;
  s.cl = cl;
  s.vs = vs;
  s.status = status;
  s.alpha_cutoff = alpha_cutoff;
  s.tf_zero_t = tf_zero_t;
  s.slot_bits = slot_bits;
  return s;
}

extern "C" {

int r3d_cuda_create(int device, r3d_cuda_ctx **out) {
  if (!out) return R3D_E_INVALID;
  *out = nullptr;
  int n = 0;
  if (cudaGetDeviceCount(&n) != cudaSuccess || device < 0 || device >= n) {
    cudaGetLastError();
    return R3D_E_CUDA;
  }
  r3d_cuda_ctx *c = new (std::nothrow) r3d_cuda_ctx();
  if (!c) return R3D_E_NOMEM;
  c->device = device;
  if (cudaSetDevice(device) != cudaSuccess ||
      cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking) != cudaSuccess ||
      cudaMalloc(&c->status, sizeof(uint32_t)) != cudaSuccess ||
      cudaMalloc(&c->lut, 256 * sizeof(uchar4)) != cudaSuccess ||
      cudaMalloc(&c->spare, 256u) != cudaSuccess ||
      cudaMalloc(&c->total, (R3D_COUNTERS + 1) * sizeof(unsigned long long)) != cudaSuccess ||
      cudaEventCreate(&c->ev0) != cudaSuccess || cudaEventCreate(&c->ev1) != cudaSuccess ||
      cudaMallocHost(&c->ring_host, sizeof(DevView) * kMaxBatchViews * r3d_cuda_ctx::kRing) !=
          cudaSuccess ||
      cudaMalloc(&c->ring_dev, sizeof(DevView) * kMaxBatchViews * r3d_cuda_ctx::kRing) !=
          cudaSuccess ||
      cudaMalloc(&c->ring_queue, sizeof(uint32_t) * 2 * kMaxBatchViews * r3d_cuda_ctx::kRing) !=
          cudaSuccess ||
      cudaMalloc(&c->diff_words, sizeof(uint32_t) * 2 * (r3d_cuda_ctx::kRing +
                                                         r3d_cuda_ctx::kCapturedCalls)) !=
          cudaSuccess) {
    cudaGetLastError();
    r3d_cuda_destroy(c);
    return R3D_E_CUDA;
  }
  if (cudaMemsetAsync(c->status, 0, sizeof(uint32_t), c->stream) != cudaSuccess ||
      cudaStreamSynchronize(c->stream) != cudaSuccess) {
    cudaGetLastError();
    r3d_cuda_destroy(c);
    return R3D_E_CUDA;
  }
  for (int k = 0; k < r3d_cuda_ctx::kRing; k++)
    if (cudaEventCreateWithFlags(&c->ring_ev[k], cudaEventDisableTiming) != cudaSuccess ||
        cudaEventCreateWithFlags(&c->ring_march_ev[k], cudaEventDisableTiming) != cudaSuccess) {
      r3d_cuda_destroy(c);
      return R3D_E_CUDA;
    }
  // default transfer function: grey ramp with alpha = value
  // (src/vk/vkbackend.c:1100-1114)
  uint8_t ramp[256][4];
  for (int i = 0; i < 256; i++) ramp[i][0] = ramp[i][1] = ramp[i][2] = ramp[i][3] = (uint8_t)i;
  if (r3d_cuda_set_transfer(c, ramp) != R3D_OK) {
    r3d_cuda_destroy(c);
    return R3D_E_CUDA;
  }
  *out = c;
  return R3D_OK;
}

void r3d_cuda_destroy(r3d_cuda_ctx *c) {
  if (!c) return;
  cudaSetDevice(c->device);
  if (c->stream) cudaStreamSynchronize(c->stream);
  cudaFree(c->cube_buf);
  cudaFree(c->cube_quad);
  cudaFree(c->shard_quad);
  cudaFree(c->page);
  cudaFree(c->pool);
  cudaFree(c->bmax);
  cudaFree(c->quad);
  for (int i = 0; i < 4; i++) cudaFree(c->ovl_quad[i]);
  cudaFreeHost(c->ovl_stage);
  cudaFree(c->ovl_stage_dev);
  cudaFree(c->shard_buf);
  cudaFree(c->shard_page);
  cudaFree(c->lut);
  cudaFree(c->spare);
  cudaFree(c->status);
  cudaFree(c->img);
  cudaFree(c->aux_buf);
  cudaFree(c->total);
  stream_reset(c);
  slab_reset(c);
  clip_reset(c);
  vslab_reset(c);
  surf_reset(c);
  postfilter_reset(c);
  if (c->page_ev) cudaEventDestroy(c->page_ev);
  cudaFree(c->diff_q);
  cudaFree(c->tape);
  cudaFree(c->diff_quad);
  cudaFree(c->tape_n);
  if (c->ev0) cudaEventDestroy(c->ev0);
  if (c->ev1) cudaEventDestroy(c->ev1);
  for (int k = 0; k < r3d_cuda_ctx::kRing; k++) {
    if (c->ring_ev[k]) cudaEventDestroy(c->ring_ev[k]);
    if (c->ring_march_ev[k]) cudaEventDestroy(c->ring_march_ev[k]);
  }
  cudaFreeHost(c->ring_host);
  cudaFree(c->ring_dev);
  cudaFree(c->ring_queue);
  cudaFree(c->diff_words);
  if (c->stream) cudaStreamDestroy(c->stream);
  delete c;
}

const char *r3d_cuda_last_error(const r3d_cuda_ctx *c) { return c ? c->err.c_str() : "no ctx"; }

void *r3d_cuda_stream(r3d_cuda_ctx *c) { return c ? (void *)c->stream : nullptr; }

int r3d_cuda_status(r3d_cuda_ctx *c, uint32_t *bits, int clear) {
  if (!c) return R3D_E_INVALID;
  cudaSetDevice(c->device);
  uint32_t v = 0;
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  R3D_CUDA_TRY(c, cudaMemcpy(&v, c->status, 4, cudaMemcpyDeviceToHost));
  if (clear) R3D_CUDA_TRY(c, cudaMemsetAsync(c->status, 0, 4, c->stream));
  if (bits) *bits = v;
  return R3D_OK;
}

int r3d_cuda_upload_volume(r3d_cuda_ctx *c, const r3d_volume_desc *d, const uint8_t *voxels) {
  if (!c || !d || !voxels || !d->nx || !d->ny || !d->nz)
    return fail(c, R3D_E_INVALID, "upload_volume: bad arguments");
  cudaSetDevice(c->device);
  uint32_t nx = d->nx, ny = d->ny, nz = d->nz;
  uint32_t maxdim = max(nx, max(ny, nz));
  if (maxdim > 65535u) return fail(c, R3D_E_INVALID, "upload_volume: dimension > 65535");
  uint32_t mips = 1;
  while ((maxdim >> mips) >= 1u && mips < 16u) mips++;
  DevCube cube;
  memset(&cube, 0, sizeof cube);
  cube.nlevels = mips;
  cube.maxdim = maxdim;
  size_t off[17];
  off[0] = 0;
  for (uint32_t m = 0; m < mips; m++) {
    cube.dim[m][0] = nx >> m ? nx >> m : 1u;
    cube.dim[m][1] = ny >> m ? ny >> m : 1u;
    cube.dim[m][2] = nz >> m ? nz >> m : 1u;
    size_t b = (size_t)cube.dim[m][0] * cube.dim[m][1] * cube.dim[m][2];
    off[m + 1] = off[m] + ((b + 255) & ~(size_t)255);
  }
  for (int a = 0; a < 3; a++) cube.odim[a] = ((a == 0 ? nx : a == 1 ? ny : nz) + 7u) / 8u;
  size_t onb = (size_t)cube.odim[0] * cube.odim[1] * cube.odim[2];
  size_t total = off[mips] + ((onb + 255) & ~(size_t)255);
  uint8_t *buf = nullptr, *raw = nullptr;
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  // bytes, occupancy (and its raw grid) and quad words in one allocation,
  // kept when about this size as the brick cache's are; the words stand alone
  // when the whole does not fit beside the volume it replaces
  const size_t base = (total + onb + 255) & ~(size_t)255;
  size_t qbytes = cube_quad_bytes(cube);
  if (!keeps(c->cube_buf, c->cube_cap, base + qbytes) && !words_fit(base, qbytes, c->cube_cap))
    qbytes = 0;
  const bool kept = keeps(c->cube_buf, c->cube_cap, base + qbytes);
  bool whole = true;
  cudaError_t e = kept ? idle_device(c) : cudaMalloc(&buf, base + qbytes);
  if (e == cudaErrorMemoryAllocation && qbytes) {
    cudaGetLastError();
    whole = false;
    e = cudaMalloc(&buf, base);
  }
  if (e != cudaSuccess) return cuda_fail(c, e, "upload_volume: cudaMalloc");
  if (kept) buf = c->cube_buf;
  raw = buf + total;
  // (a copy that is refused leaves a kept buffer, and its volume, as it was)
  e = cudaMemcpyAsync(buf, voxels, (size_t)nx * ny * nz, cudaMemcpyDefault, c->stream);
  if (kept && e == cudaSuccess) c->have_cube = false;
  for (uint32_t m = 0; m < mips; m++) cube.lev[m] = buf + off[m];
  cube.occ = buf + off[mips];
  for (uint32_t m = 1; m < mips && e == cudaSuccess; m++)
    e = launch_mip(cube.lev[m - 1], cube.dim[m - 1][0], cube.dim[m - 1][1], cube.dim[m - 1][2],
                   buf + off[m], cube.dim[m][0], cube.dim[m][1], cube.dim[m][2], c->stream);
  if (e == cudaSuccess) e = launch_occ_raw(buf, nx, ny, nz, raw, c->stream);
  if (e == cudaSuccess) {
    k_occ_dilate<<<grid_for(onb), 256, 0, c->stream>>>(raw, buf + off[mips], cube.odim[0],
                                                       cube.odim[1], cube.odim[2]);
    e = cudaGetLastError();
  }
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) {
    if (!kept) cudaFree(buf);
    return cuda_fail(c, e, "upload_volume");
  }
  if (!kept) {
    cudaFree(c->cube_buf);
    c->cube_buf = buf;
    c->cube_cap = whole ? base + qbytes : base;
  }
  c->have_cube = false;
  c->cube.quad = nullptr;
  cudaFree(c->cube_quad);
  c->cube_quad = nullptr;
  uint32_t *words = whole && qbytes ? (uint32_t *)(buf + base) : nullptr;
  if (!whole && cudaMalloc(&c->cube_quad, qbytes) == cudaSuccess) words = c->cube_quad;
  if (!whole) cudaGetLastError();
  e = build_cube_quads(cube, words, c->stream);
  if (e == cudaSuccess) e = cudaStreamSynchronize(c->stream);
  if (e != cudaSuccess) return cuda_fail(c, e, "upload_volume: quad words");
  c->cube_bytes = total;
  c->have_cube = true;
  c->cube = cube;
  return R3D_OK;
}

int r3d_cuda_set_transfer(r3d_cuda_ctx *c, const uint8_t rgba[256][4]) {
  if (!c || !rgba) return fail(c, R3D_E_INVALID, "set_transfer: bad arguments");
  cudaSetDevice(c->device);
  memcpy(c->lut_host, rgba, sizeof c->lut_host);
  int imin = 256;
  for (int i = 0; i < 256; i++)
    if (rgba[i][3]) {
      imin = i;
      break;
    }
  // TF coordinate t < imin - 1 interpolates two zero-alpha texels
  c->tf_zero_t = (float)(imin - 1);
  R3D_CUDA_TRY(c, cudaMemcpyAsync(c->lut, c->lut_host, sizeof c->lut_host, cudaMemcpyHostToDevice,
                                  c->stream));
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  return R3D_OK;
}

int r3d_cuda_set_quality(r3d_cuda_ctx *c, uint32_t quality) {
  if (!c || quality >= R3D_QUALITY_COUNT) return fail(c, R3D_E_INVALID, "set_quality: %u", quality);
  c->quality = quality;
  return R3D_OK;
}

int r3d_cuda_set_slot_trace(r3d_cuda_ctx *c, uint32_t *bits) {
  if (!c) return R3D_E_INVALID;
  if (bits && !is_device_ptr(bits)) return fail(c, R3D_E_INVALID, "set_slot_trace: not device");
  c->slot_bits = bits;
  return R3D_OK;
}

int r3d_cuda_set_alpha_cutoff(r3d_cuda_ctx *c, float cutoff) {
  if (!c || !(cutoff > 0.0f && cutoff <= 1.0f))
    return fail(c, R3D_E_INVALID, "set_alpha_cutoff: %g not in (0, 1]", (double)cutoff);
  c->alpha_cutoff = cutoff;
  return R3D_OK;
}

}  // extern "C"

// Validates a LOD page-table header and decodes it into the kernel's form.
static int decode_header(r3d_cuda_ctx *c, const uint32_t *page, uint32_t words, uint32_t nslots,
                         DevBricks &b) {
  memset(&b, 0, sizeof b);
  if (words < R3D_BRICK_PAGE_HEADER) return fail(c, R3D_E_INVALID, "page table < 64 words");
  uint32_t nlev = page[0];
  if (nlev < 1u || nlev > 15u) return fail(c, R3D_E_INVALID, "page header: %u levels", nlev);
  if (!page[1] || !page[2] || !page[3] || page[1] > 65535u || page[2] > 65535u ||
      page[3] > 65535u)
    return fail(c, R3D_E_INVALID, "page header: bad base shape");
  b.nlev = nlev;
  for (int a = 0; a < 3; a++) b.bs[a] = (float)page[1 + a];
  b.md = fmaxf(b.bs[0], fmaxf(b.bs[1], b.bs[2]));
  for (int a = 0; a < 3; a++) b.bs_hi[a] = fmaxf(b.bs[a] - 0.001f, 0.0f);
  for (uint32_t l = 0; l < nlev; l++) {
    uint32_t off = page[4 + 4 * l], packed = page[5 + 4 * l], scale = page[6 + 4 * l];
    uint32_t bd[3] = {packed & 1023u, (packed >> 10) & 1023u, packed >> 20};
    if (!scale || (scale & (scale - 1u)) || scale > (1u << 20))
      return fail(c, R3D_E_INVALID, "page header: level %u scale %u not a power of two", l, scale);
    if (!bd[0] || !bd[1] || !bd[2] || bd[2] > 1023u)
      return fail(c, R3D_E_INVALID, "page header: level %u empty brick grid", l);
    uint64_t end = (uint64_t)off + (uint64_t)bd[0] * bd[1] * bd[2];
    if (off < R3D_BRICK_PAGE_HEADER || end > words)
      return fail(c, R3D_E_INVALID, "page header: level %u entries out of range", l);
    b.off[l] = off;
    b.scale[l] = scale;
    b.inv_scale[l] = 1.0f / (float)scale;
    for (int a = 0; a < 3; a++) b.bd[l][a] = bd[a];
  }
  b.page_words = words;
  b.nslots = nslots;
  return R3D_OK;
}

// Room for the per-slot tables (block maxima, quad words) of c->nslots
// slots; overlays follow the old slot assignment and go.
static int reserve_tables(r3d_cuda_ctx *c) {
  for (int i = 0; i < 4; i++) {
    cudaFree(c->ovl_quad[i]);
    c->ovl_quad[i] = nullptr;
    c->br.ovl[i] = nullptr;
    c->ovl_src_on[i] = false;  // a new cache detaches CPU-sourced atlases
    c->ovl_key[i].clear();
  }
  c->br.bmax = nullptr;
  c->br.quad = nullptr;
  const size_t n = c->nslots ? c->nslots : 1u;
  R3D_CUDA_TRY(c, reserve(c, c->bmax, c->bmax_cap, n * 4096u));
  R3D_CUDA_TRY(c, reserve(c, c->quad, c->quad_cap, n * (128u * 128u * 128u) * sizeof(uint32_t)));
  if (!c->nslots) R3D_CUDA_TRY(c, cudaMemsetAsync(c->bmax, 0, 4096u, c->stream));
  return R3D_OK;
}

// (Re)builds the per-slot tables of the context's slot pool.
int build_blockmax(r3d_cuda_ctx *c) {
  if (c->defer_tables) return R3D_OK;
  const int rc = reserve_tables(c);
  if (rc != R3D_OK) return rc;
  R3D_CUDA_TRY(c, launch_slot_tables(c->pool, nullptr, c->nslots, c->quad, c->bmax, c->stream));
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  c->br.bmax = c->bmax;
  c->br.quad = c->quad;
  return R3D_OK;
}

int replace_pool(r3d_cuda_ctx *c, uint32_t nslots) {
  c->br.pool = nullptr;
  R3D_CUDA_TRY(c, reserve(c, c->pool, c->pool_cap, (size_t)(nslots ? nslots : 1u) * (128u * 128u * 128u)));
  c->br.pool = c->pool;
  return R3D_OK;
}

uint32_t atlas_bpa(uint32_t nslots) {
  uint32_t a = 1;
  while ((uint64_t)a * a * a < nslots) a++;
  return a;
}

extern "C" {

int r3d_cuda_bricks_build(r3d_cuda_ctx *c, const r3d_volume_desc *d, const uint8_t *voxels,
                          uint32_t nlev, uint32_t min_max) {
  if (!c || !d || !voxels || !d->nx || !d->ny || !d->nz || nlev < 1u || nlev > 15u)
    return fail(c, R3D_E_INVALID, "bricks_build: bad arguments");
  uint32_t nx = d->nx, ny = d->ny, nz = d->nz;
  if (max(nx, max(ny, nz)) > 65535u) return fail(c, R3D_E_INVALID, "bricks_build: too large");
  cudaSetDevice(c->device);
  stream_reset(c);
  cudaStream_t st = c->stream;
  R3D_CUDA_TRY(c, cudaStreamSynchronize(st));
  // level extents: level 0 is the volume itself, level l >= 1 the zero-
  // padded brick grid 128 * ceil(ceil(n / 2^l) / 128)
  uint32_t E[16][3], bd[16][3];
  size_t lev_off[16] = {0}, lev_total = 0;
  uint32_t nb_total = 0;
  for (uint32_t l = 0; l < nlev; l++) {
    uint32_t n3[3] = {nx, ny, nz};
    for (int a = 0; a < 3; a++) {
      uint32_t dl = (n3[a] + (1u << l) - 1u) >> l;
      bd[l][a] = (dl + 127u) / 128u;
      E[l][a] = l == 0 ? n3[a] : bd[l][a] * 128u;
    }
    if (bd[l][0] > 1023u || bd[l][1] > 1023u || bd[l][2] > 1023u)
      return fail(c, R3D_E_INVALID, "bricks_build: brick grid too large");
    lev_off[l] = lev_total;
    lev_total += ((size_t)E[l][0] * E[l][1] * E[l][2] + 255) & ~(size_t)255;
    nb_total += bd[l][0] * bd[l][1] * bd[l][2];
  }
  // the level buffer holds levels 1.. and, when the voxels are not on this
  // device, level 0; a device volume is read where it is
  const bool dev_in = readable_in_place(c, voxels);
  if (dev_in) {
    const size_t skip = nlev > 1u ? lev_off[1] : lev_total;
    for (uint32_t l = 1; l < nlev; l++) lev_off[l] -= skip;
    lev_total -= skip;
  }
  uint32_t words = R3D_BRICK_PAGE_HEADER + nb_total;
  uint8_t *lev = nullptr;
  uint32_t *dmax = nullptr, *jobs = nullptr;
  uint8_t *pool = nullptr;
  uint32_t *page = nullptr;
  size_t pool_bytes = 0;
  std::vector<uint32_t> hmax(nb_total), hpage(words, R3D_BRICK_ABSENT);
  std::vector<uint32_t> src_brick;
  LevelSrc src[16];
  int rc = R3D_OK;
  // level buffer, brick maxima, brick list: one allocation
  const size_t max_off = (lev_total + 255) & ~(size_t)255, job_off = max_off + (size_t)nb_total * 4;
  cudaError_t e = cudaMalloc(&lev, job_off + (size_t)nb_total * 4);
  if (e != cudaSuccess) {
    rc = cuda_fail(c, e, "bricks_build: cudaMalloc levels");
    goto out;
  }
  dmax = (uint32_t *)(lev + max_off);
  jobs = (uint32_t *)(lev + job_off);
  e = cudaMemsetAsync(dmax, 0, (size_t)nb_total * 4, st);
  if (e == cudaSuccess && !dev_in)
    e = cudaMemcpyAsync(lev, voxels, (size_t)nx * ny * nz, cudaMemcpyDefault, st);
  {
    // each level is read once: the next one and the level's brick maxima
    uint32_t moff = 0;
    for (uint32_t l = 0; l < nlev; l++) {
      src[l] = {l == 0 && dev_in ? voxels : lev + lev_off[l], E[l][0], E[l][1], E[l][2],
                bd[l][0], bd[l][1], 0u};
      uint32_t o[3];
      for (int a = 0; a < 3; a++) o[a] = l + 1u < nlev ? E[l + 1][a] : (bd[l][a] + 1u) / 2u * 128u;
      if (e == cudaSuccess)
        e = launch_level_down(src[l].p, E[l][0], E[l][1], E[l][2],
                              l + 1u < nlev ? lev + lev_off[l + 1] : nullptr, o[0], o[1], o[2],
                              dmax + moff, bd[l][0], bd[l][1], st);
      moff += bd[l][0] * bd[l][1] * bd[l][2];
    }
  }
  if (e == cudaSuccess)
    e = cudaMemcpyAsync(hmax.data(), dmax, (size_t)nb_total * 4, cudaMemcpyDeviceToHost, st);
  if (e == cudaSuccess) e = cudaStreamSynchronize(st);
  if (e != cudaSuccess) {
    rc = cuda_fail(c, e, "bricks_build: pyramid");
    goto out;
  }
  {
    // page table in render3d's format (src/vk/vkbackend.c:4184-4206)
    memset(hpage.data(), 0, R3D_BRICK_PAGE_HEADER * 4);
    hpage[0] = nlev;
    hpage[1] = nx;
    hpage[2] = ny;
    hpage[3] = nz;
    uint32_t off = 0, slot = 0;
    for (uint32_t l = 0; l < nlev; l++) {
      uint32_t nb = bd[l][0] * bd[l][1] * bd[l][2];
      hpage[4 + 4 * l] = R3D_BRICK_PAGE_HEADER + off;
      hpage[5 + 4 * l] = bd[l][0] | (bd[l][1] << 10) | (bd[l][2] << 20);
      hpage[6 + 4 * l] = 1u << l;
      src[l].job0 = slot;
      for (uint32_t bi = 0; bi < nb; bi++) {
        uint32_t m = hmax[off + bi];
        if (m >= min_max) {
          hpage[R3D_BRICK_PAGE_HEADER + off + bi] = slot | (m << 24);
          src_brick.push_back(bi);
          slot++;
        }
      }
      off += nb;
    }
    if (slot >= (1u << 24)) {
      rc = fail(c, R3D_E_INVALID, "bricks_build: %u slots exceed the 24-bit slot field", slot);
      goto out;
    }
    uint32_t nslots = slot;
    DevBricks b;
    rc = decode_header(c, hpage.data(), words, nslots, b);
    if (rc != R3D_OK) goto out;
    // the pool and the page table: kept when about this size, else allocated
    // before the old ones go
    pool_bytes = (size_t)(nslots ? nslots : 1u) * (128u * 128u * 128u);
    e = keeps(c->pool, c->pool_cap, pool_bytes) ? idle_device(c) : cudaMalloc(&pool, pool_bytes);
    if (e == cudaSuccess) e = cudaMalloc(&page, (size_t)words * 4);
    if (e != cudaSuccess) {
      rc = cuda_fail(c, e, "bricks_build: cudaMalloc pool");
      goto out;
    }
    c->have_bricks = false;
    if (pool) {
      cudaFree(c->pool);
      c->pool = pool;
      c->pool_cap = pool_bytes;
      pool = nullptr;
    }
    cudaFree(c->page);
    c->page = page;
    page = nullptr;
    b.page = c->page;
    b.pool = c->pool;
    c->page_words = words;
    c->nslots = nslots;
    c->abpa = atlas_bpa(nslots);
    c->shape[0] = nx;
    c->shape[1] = ny;
    c->shape[2] = nz;
    c->br = b;
    // the display filter comes before the tables that derive from the slots
    // (a build whose pool becomes a streaming store stays unfiltered: its
    // bricks are filtered when uploaded); without it one pass over the
    // levels fills the slots and their tables
    const bool filter = !c->defer_tables && postfilter_on(c, 0u), fused = !c->defer_tables && !filter;
    if (fused) {
      rc = reserve_tables(c);
      if (rc != R3D_OK) goto out;
    }
    if (e == cudaSuccess && nslots)
      e = cudaMemcpyAsync(jobs, src_brick.data(), (size_t)nslots * 4, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess && nslots)
      e = launch_slot_fill(src, nlev, jobs, nullptr, nslots, c->pool, fused ? c->quad : nullptr,
                           fused ? c->bmax : nullptr, st);
    if (e == cudaSuccess)
      e = cudaMemcpyAsync(c->page, hpage.data(), (size_t)words * 4, cudaMemcpyHostToDevice, st);
    if (e == cudaSuccess) e = cudaStreamSynchronize(st);
    if (e != cudaSuccess) {
      rc = cuda_fail(c, e, "bricks_build: slots");
      goto out;
    }
    if (fused) {
      c->br.bmax = c->bmax;
      c->br.quad = c->quad;
    }
    if (filter) {
      std::vector<uint32_t> all(nslots);
      for (uint32_t s = 0; s < nslots; s++) all[s] = s;
      rc = postfilter_slots(c, 0u, c->pool, all.data(), nslots);
      if (rc != R3D_OK) goto out;
    }
    if (!fused) rc = build_blockmax(c);
    if (rc != R3D_OK) goto out;
    c->have_bricks = true;
  }
out:
  cudaFree(lev);
  cudaFree(pool);
  cudaFree(page);
  return rc;
}

int r3d_cuda_bricks_load(r3d_cuda_ctx *c, const uint32_t *page, uint32_t page_words,
                         const uint8_t *slots, uint32_t nslots) {
  if (!c || !page || (!slots && nslots)) return fail(c, R3D_E_INVALID, "bricks_load: bad args");
  if (nslots >= (1u << 24)) return fail(c, R3D_E_INVALID, "bricks_load: too many slots");
  stream_reset(c);
  DevBricks b;
  int rc = decode_header(c, page, page_words, nslots, b);
  if (rc != R3D_OK) return rc;
  cudaSetDevice(c->device);
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  uint32_t *dpage = nullptr;
  uint8_t *dpool = nullptr;
  size_t pool_bytes = (size_t)(nslots ? nslots : 1u) * (128u * 128u * 128u);
  cudaError_t e = cudaMalloc(&dpage, (size_t)page_words * 4);
  if (e == cudaSuccess) e = cudaMalloc(&dpool, pool_bytes);
  if (e == cudaSuccess) e = copy_sync(c->stream, dpage, page, (size_t)page_words * 4);
  if (e == cudaSuccess && nslots)
    e = copy_sync(c->stream, dpool, slots, (size_t)nslots * (128u * 128u * 128u));
  if (e != cudaSuccess) {
    cudaFree(dpage);
    cudaFree(dpool);
    return cuda_fail(c, e, "bricks_load");
  }
  b.page = dpage;
  b.pool = dpool;
  cudaFree(c->page);
  cudaFree(c->pool);
  c->page = dpage;
  c->pool = dpool;
  c->pool_cap = pool_bytes;
  c->page_words = page_words;
  c->nslots = nslots;
  c->abpa = atlas_bpa(nslots);
  c->shape[0] = page[1];
  c->shape[1] = page[2];
  c->shape[2] = page[3];
  c->br = b;
  c->have_bricks = false;
  rc = build_blockmax(c);
  if (rc != R3D_OK) return rc;
  c->have_bricks = true;
  return R3D_OK;
}

uint32_t r3d_cuda_brick_mode(const r3d_cuda_ctx *c) {
  if (!c || !c->have_bricks) return 0u;
  return c->abpa | (c->br.nlev << 8) | R3D_BRICK_LOD_FLAG;
}

int r3d_cuda_bricks_info(const r3d_cuda_ctx *c, uint32_t *page_words, uint32_t *nslots,
                         uint32_t shape[3], uint32_t *nlev) {
  if (!c) return R3D_E_INVALID;
  if (!c->have_bricks) return R3D_E_STATE;
  if (page_words) *page_words = c->page_words;
  if (nslots) *nslots = c->nslots;
  if (shape) memcpy(shape, c->shape, sizeof c->shape);
  if (nlev) *nlev = c->br.nlev;
  return R3D_OK;
}

int r3d_cuda_bricks_read(r3d_cuda_ctx *c, uint32_t *page, uint8_t *slots) {
  if (!c) return R3D_E_INVALID;
  if (!c->have_bricks) return fail(c, R3D_E_STATE, "bricks_read: no bricks");
  cudaSetDevice(c->device);
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  if (page) R3D_CUDA_TRY(c, cudaMemcpy(page, c->page, (size_t)c->page_words * 4, cudaMemcpyDefault));
  if (slots && c->nslots)
    R3D_CUDA_TRY(c, cudaMemcpy(slots, c->pool, (size_t)c->nslots * (128u * 128u * 128u),
                               cudaMemcpyDefault));
  return R3D_OK;
}

int r3d_cuda_cube_read(r3d_cuda_ctx *c, int level, uint8_t *out, uint32_t dims[3]) {
  if (!c) return R3D_E_INVALID;
  if (!c->have_cube) return fail(c, R3D_E_STATE, "cube_read: no volume");
  const DevCube &cb = c->cube;
  const uint8_t *src;
  uint32_t d[3];
  if (level < 0) {
    src = cb.occ;
    memcpy(d, cb.odim, sizeof d);
  } else {
    if ((uint32_t)level >= cb.nlevels) return fail(c, R3D_E_INVALID, "cube_read: level");
    src = cb.lev[level];
    memcpy(d, cb.dim[level], sizeof d);
  }
  if (dims) memcpy(dims, d, sizeof d);
  if (out) {
    cudaSetDevice(c->device);
    R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
    R3D_CUDA_TRY(c, cudaMemcpy(out, src, (size_t)d[0] * d[1] * d[2], cudaMemcpyDefault));
  }
  return R3D_OK;
}

}  // extern "C"

// The view's rectangle clipped to the image (src/vk/vkbackend.c:6871-6900):
// 1 to render, 0 when nothing of it is inside.
static int view_rect(const r3d_frame_params &in, uint32_t out_w, uint32_t out_h,
                     r3d_frame_params &pc) {
  uint32_t ox = in.view_org & 0xffffu, oy = (in.view_org >> 16) & 0xffffu;
  uint32_t vw = in.viewport[0] ? in.viewport[0] : out_w;
  uint32_t vh = in.viewport[1] ? in.viewport[1] : out_h;
  bool ok = ox < out_w && oy < out_h;
  if (ok) {
    vw = min(vw, out_w - ox);
    vh = min(vh, out_h - oy);
    ok = vw && vh;
  }
  pc.view_org = ox | (oy << 16);
  pc.viewport[0] = ok ? vw : 0u;
  pc.viewport[1] = ok ? vh : 0u;
  return ok ? 1 : 0;
}

// Validates and sanitizes one view against the image.  Returns 1 to render,
// 0 to skip, < 0 error.
int prepare_view(r3d_cuda_ctx *c, const r3d_frame_params &in, uint32_t out_w,
                        uint32_t out_h, r3d_frame_params &pc) {
  pc = in;
  if (in.mode >= R3D_MODE_COUNT) return fail(c, R3D_E_INVALID, "view: mode %u", in.mode);
  if (in.view_flags & R3D_VIEW_SURF) {  // flattened segment: the view must describe the window
    if (!c->sv_vol || !c->sv_baked)
      return fail(c, R3D_E_STATE, "view: no baked surface volume (r3d_cuda_surfvol_window)");
    r3d_frame_params ref = in;
    r3d_cuda_surfvol_params(c, &ref);
    if (in.slab_x0 != ref.slab_x0 || in.slab_y0 != ref.slab_y0 || in.slab_px != ref.slab_px ||
        in.slab_nx != ref.slab_nx || in.slab_ny != ref.slab_ny || in.slab_wz != ref.slab_wz ||
        in.slab_grid != ref.slab_grid || in.max_mip != ref.max_mip ||
        in.vol_tx != ref.vol_tx || in.vol_ty != ref.vol_ty)
      return fail(c, R3D_E_INVALID, "view: surface parameters do not match the baked window "
                                    "(r3d_cuda_surfvol_params)");
    if (!(in.step_voxels > 0.0f)) return fail(c, R3D_E_INVALID, "view: step_voxels must be > 0");
    return view_rect(in, out_w, out_h, pc);
  }
  if (in.clip_valid) {  // clipmap: the view must describe the loaded levels
    if (!c->have_clip) return fail(c, R3D_E_STATE, "view: no clipmap loaded");
    r3d_frame_params ref;
    memset(&ref, 0, sizeof ref);
    r3d_cuda_clip_params(c, &ref);
    if (in.clip_valid != ref.clip_valid || in.slab_z0 != ref.slab_z0 ||
        in.slab_nx != ref.slab_nx || in.slab_ny != ref.slab_ny || in.slab_wz != ref.slab_wz ||
        memcmp(in.clip_orig, ref.clip_orig, sizeof ref.clip_orig) || in.brick_mode ||
        in.slab_grid)
      return fail(c, R3D_E_INVALID, "view: clipmap parameters do not match the loaded levels "
                                    "(r3d_cuda_clip_params)");
    if (in.slab_depth < 1u || in.slab_depth > in.slab_wz)
      return fail(c, R3D_E_INVALID, "view: slab_depth %u not in [1, %u]", in.slab_depth,
                  in.slab_wz);
    if (in.overlay_flags & kOvlAtlases)
      return fail(c, R3D_E_UNSUPPORTED, "view: overlay atlases need the LOD brick cache");
  } else if (in.slab_grid & kVslabGrid) {  // virtual slab: the view must describe the window
    if (!c->have_vslab) return fail(c, R3D_E_STATE, "view: no virtual slab loaded");
    r3d_frame_params ref;
    memset(&ref, 0, sizeof ref);
    r3d_cuda_vslab_params(c, &ref);
    if (in.slab_grid != ref.slab_grid || in.brick_mode != ref.brick_mode ||
        in.slab_wz != ref.slab_wz || in.slab_z0 != ref.slab_z0 || in.slab_nx != ref.slab_nx ||
        in.slab_ny != ref.slab_ny || in.slab_px != ref.slab_px || in.slab_py != ref.slab_py ||
        in.slab_x0 != ref.slab_x0 || in.slab_y0 != ref.slab_y0)
      return fail(c, R3D_E_INVALID, "view: virtual-slab parameters do not match the loaded "
                                    "window (r3d_cuda_vslab_params)");
    if (in.slab_depth < 1u || in.slab_depth > c->vsl.D)
      return fail(c, R3D_E_INVALID, "view: slab_depth %u not in [1, %u]", in.slab_depth,
                  c->vsl.D);
    if (in.overlay_flags & kOvlAtlases)
      return fail(c, R3D_E_UNSUPPORTED, "view: overlay atlases need the LOD brick cache");
  } else if (in.slab_grid) {  // tiled slab: the view must describe the loaded window
    if (!c->have_slab) return fail(c, R3D_E_STATE, "view: no slab loaded");
    r3d_frame_params ref;
    memset(&ref, 0, sizeof ref);
    r3d_cuda_slab_params(c, &ref);
    if (in.slab_grid != ref.slab_grid || in.slab_wz != ref.slab_wz ||
        in.slab_z0 != ref.slab_z0 || in.slab_nx != ref.slab_nx || in.slab_ny != ref.slab_ny ||
        in.slab_px != ref.slab_px || in.slab_py != ref.slab_py || in.brick_mode)
      return fail(c, R3D_E_INVALID, "view: slab parameters do not match the loaded window "
                                    "(r3d_cuda_slab_params)");
    if (in.slab_depth < 1u || in.slab_depth > in.slab_wz - 1u)
      return fail(c, R3D_E_INVALID, "view: slab_depth %u not in [1, %u]", in.slab_depth,
                  in.slab_wz - 1u);
    if (in.overlay_flags & kOvlAtlases)
      return fail(c, R3D_E_UNSUPPORTED, "view: overlay atlases need the LOD brick cache");
  }
  if (in.overlay_flags & kOvlAtlases) {
    if (!(in.brick_mode & R3D_BRICK_LOD_FLAG))
      return fail(c, R3D_E_UNSUPPORTED, "view: overlay atlases need the LOD brick cache");
    static const char *names[4] = {"ink", "3D ink", "labels", "registration"};
    const uint32_t bit[4] = {kOvlInk, kOvlInk3d, kOvlLabels, kOvlReg};
    for (int i = 0; i < 4; i++)
      if ((in.overlay_flags & bit[i]) && !c->ovl_quad[i])
        return fail(c, R3D_E_STATE, "view: overlay atlas '%s' is not loaded", names[i]);
  }
  if (!(in.max_mip >= 0.0f)) return fail(c, R3D_E_INVALID, "view: max_mip must be >= 0");
  if (!(in.step_voxels > 0.0f)) return fail(c, R3D_E_INVALID, "view: step_voxels must be > 0");
  if (in.slab_grid & kVslabGrid) {
    // brick_mode holds the pyramid grids (checked above)
  } else if (in.brick_mode & R3D_BRICK_LOD_FLAG) {
    if (!c->have_bricks) return fail(c, R3D_E_STATE, "view: no brick cache loaded");
  } else if (in.brick_mode) {
    if (!c->have_shard) return fail(c, R3D_E_STATE, "view: no single-level brick atlas loaded");
    if (in.brick_mode != r3d_cuda_shard_mode(c))
      return fail(c, R3D_E_INVALID, "view: brick_mode 0x%x does not match the atlas (0x%x)",
                  in.brick_mode, r3d_cuda_shard_mode(c));
  } else if (!in.slab_grid && !in.clip_valid && !c->have_cube) {
    return fail(c, R3D_E_STATE, "view: no volume uploaded");
  }
  return view_rect(in, out_w, out_h, pc);
}

// Persistent launches for the renderable views of one call: views sharing a
// sampling path and mode go into one launch (template parameters of the
// kernel), in order of first appearance.
static int launch_views_persistent(r3d_cuda_ctx *c, uint32_t persistent,
                                   const r3d_frame_params *pcs, const int *render,
                                   uint32_t nviews, uint8_t *const *imgs,
                                   const uint32_t *strides, uint32_t *steps, uint32_t *mip,
                                   unsigned long long *total, unsigned long long *counters,
                                   cudaStream_t st) {
  const int k = c->ring_next;
  c->ring_next = (k + 1) % r3d_cuda_ctx::kRing;
  if (c->ring_used[k]) R3D_CUDA_TRY(c, cudaEventSynchronize(c->ring_ev[k]));
  DevView *hv = c->ring_host + (size_t)k * kMaxBatchViews;
  DevView *dv = c->ring_dev + (size_t)k * kMaxBatchViews;
  uint32_t *queue = c->ring_queue + (size_t)k * 2 * kMaxBatchViews;  // two words per group
  const r3d_cuda_schedule &sc = c->sched;
  // group views by (path, mode)
  uint32_t order[64], group_of[64], ngroups = 0, gkey[64], gstart[65], gcount[64];
  uint32_t n = 0;
  for (uint32_t v = 0; v < nviews; v++) {
    if (!render[v]) continue;
    uint32_t key = (uint32_t)path_of_view(pcs[v]) * 8u | pcs[v].mode;
    uint32_t g = 0;
    while (g < ngroups && gkey[g] != key) g++;
    if (g == ngroups) {
      gkey[ngroups] = key;
      gcount[ngroups] = 0;
      ngroups++;
    }
    group_of[n] = g;
    order[n++] = v;
    gcount[g]++;
  }
  if (!n) return R3D_OK;
  gstart[0] = 0;
  for (uint32_t g = 0; g < ngroups; g++) gstart[g + 1] = gstart[g] + gcount[g];
  uint32_t fill[64] = {0}, ntiles[64] = {0};
  for (uint32_t i = 0; i < n; i++) {
    uint32_t g = group_of[i], slot = gstart[g] + fill[g]++;
    DevView &d = hv[slot];
    memset(&d, 0, sizeof d);
    d.pc = pcs[order[i]];
    d.img = (uchar4 *)imgs[order[i]];
    d.stride = strides[order[i]];
    d.tile_begin = ntiles[g];
    ntiles[g] += view_tiles(d, persistent == 2u ? 0u : sc.tile_shape);
  }
  R3D_CUDA_TRY(c, cudaMemcpyAsync(dv, hv, sizeof(DevView) * n, cudaMemcpyHostToDevice, st));
  R3D_CUDA_TRY(c, cudaEventRecord(c->ring_ev[k], st));
  c->ring_used[k] = true;
  R3D_CUDA_TRY(c, cudaMemsetAsync(queue, 0, sizeof(uint32_t) * 2 * ngroups, st));
  int dev_sms = 148;
  cudaDeviceGetAttribute(&dev_sms, cudaDevAttrMultiProcessorCount, c->device);
  const DevScene s = c->scene();
  if (persistent == 2u) {  // whole tiles, the views as launch parameters
    for (uint32_t g = 0; g < ngroups; g++) {
      TilesLaunch T;
      memset(&T, 0, sizeof T);
      T.views = hv + gstart[g];
      T.nviews = gcount[g];
      T.ntiles = ntiles[g];
      T.scenes = &s;
      T.luts = &c->lut;
      T.nscenes = 1u;
      T.queue = queue + 2 * g;
      T.steps = steps;
      T.mip = mip;
      T.total = total;
      T.counters = counters;
      T.blocks = sc.blocks_per_sm * (uint32_t)dev_sms;
      T.mode = gkey[g] & 7u;
      T.fast = c->quality == R3D_QUALITY_FAST;
      T.path = (int)(gkey[g] >> 3);
      cudaError_t e = launch_tiles(T, st);
      if (e != cudaSuccess) return cuda_fail(c, e, "raycast_fwd: whole-tile launch");
    }
    return R3D_OK;
  }
  for (uint32_t g = 0; g < ngroups; g++) {
    PersistLaunch L;
    memset(&L, 0, sizeof L);
    L.views = dv + gstart[g];
    L.nviews = gcount[g];
    L.ntiles = ntiles[g];
    L.lut = c->lut;
    L.queue = queue + 2 * g;
    L.refill_min = sc.refill_min;
    L.shape = sc.tile_shape;
    L.unroll = sc.unroll;
    L.steps = steps;
    L.mip = mip;
    L.total = total;
    L.counters = counters;
    L.mode = gkey[g] & 7u;
    L.fast = c->quality == R3D_QUALITY_FAST;
    L.path = (int)(gkey[g] >> 3);
    int per_sm = sc.blocks_per_sm
                     ? (int)sc.blocks_per_sm
                     : persist_blocks_per_sm(L, s);
    // no more blocks than there are tiles for their warps
    uint32_t want = (uint32_t)per_sm * (uint32_t)dev_sms;
    uint32_t cap = (L.ntiles + 3u) / 4u;
    L.blocks = want < cap ? want : (cap ? cap : 1u);
    cudaError_t e = launch_persist(L, s, st);
    if (e != cudaSuccess) return cuda_fail(c, e, "raycast_fwd: persistent launch");
  }
  return R3D_OK;
}

// One colour into every pixel of an RGBA8 image (grid-stride).
__global__ void k_fill_rgba(uchar4 *__restrict__ img, size_t npix, uchar4 col) {
  for (size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x; i < npix;
       i += (size_t)gridDim.x * blockDim.x)
    img[i] = col;
}

extern "C" {

int r3d_cuda_set_schedule(r3d_cuda_ctx *c, const r3d_cuda_schedule *sc) {
  if (!c || !sc || sc->persistent > 3u || sc->staging > 1u || sc->refill_min < 1u || sc->refill_min > 32u ||
      sc->tile_shape > 2u || (sc->unroll != 1u && sc->unroll != 2u) || sc->shade_group > 32u ||
      sc->blocks_per_sm > 32u)
    return fail(c, R3D_E_INVALID, "set_schedule: bad schedule");
  c->sched = *sc;
  return R3D_OK;
}

int r3d_cuda_get_schedule(const r3d_cuda_ctx *c, r3d_cuda_schedule *sc) {
  if (!c || !sc) return R3D_E_INVALID;
  *sc = c->sched;
  return R3D_OK;
}

int r3d_cuda_raycast_rows(r3d_cuda_ctx *c, const r3d_frame_params *view, uint8_t *rgba_out,
                          uint32_t out_w, uint32_t out_h, uint32_t row0, uint32_t row1,
                          void *stream) {
  if (!c || !view || !rgba_out || !out_w || !out_h || out_w > 65535u || out_h > 65535u)
    return fail(c, R3D_E_INVALID, "raycast_rows: bad arguments");
  if (!is_device_ptr(rgba_out))
    return fail(c, R3D_E_INVALID, "raycast_rows: the image must be device memory");
  if (view->view_flags & R3D_VIEW_SURF)
    return fail(c, R3D_E_UNSUPPORTED, "raycast_rows: surface views render whole");
  cudaSetDevice(c->device);
  r3d_frame_params pc;
  const int rc = prepare_view(c, *view, out_w, out_h, pc);
  if (rc <= 0) return rc;
  Rows rows;
  rows.row0 = row0;
  rows.row1 = row1;
  R3D_CUDA_TRY(c, launch_view(c, pc, rgba_out, out_w, nullptr, nullptr, nullptr, nullptr,
                              stream ? (cudaStream_t)stream : c->stream, rows));
  return R3D_OK;
}

int r3d_cuda_raycast_fwd(r3d_cuda_ctx *c, const r3d_frame_params *views, uint32_t nviews,
                         uint8_t *rgba_out, uint32_t out_w, uint32_t out_h,
                         const r3d_cuda_aux *aux, void *stream) {
  if (!c || !views || !nviews || nviews > 64u || !rgba_out || !out_w || !out_h ||
      out_w > 65535u || out_h > 65535u)
    return fail(c, R3D_E_INVALID, "raycast_fwd: bad arguments");
  cudaSetDevice(c->device);
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  r3d_frame_params pcs[64];
  int render[64];
  for (uint32_t v = 0; v < nviews; v++) {
    render[v] = prepare_view(c, views[v], out_w, out_h, pcs[v]);
    if (render[v] < 0) return render[v];
  }
  bool host = !is_device_ptr(rgba_out);
  size_t npix = (size_t)out_w * out_h;
  uint8_t *img = rgba_out;
  uint32_t *steps = aux ? aux->steps : nullptr, *mip = aux ? aux->mip_index : nullptr;
  unsigned long long *total = aux ? aux->total_steps : nullptr;
  unsigned long long *counters = aux ? aux->counters : nullptr;
  if (host) {
    if (c->img_cap < npix * 4) {
      cudaFree(c->img);
      c->img = nullptr;
      c->img_cap = 0;
      R3D_CUDA_TRY(c, cudaMalloc(&c->img, npix * 4));
      c->img_cap = npix * 4;
    }
    img = c->img;
    // pixels outside every view keep the caller's contents
    R3D_CUDA_TRY(c, cudaMemcpyAsync(img, rgba_out, npix * 4, cudaMemcpyHostToDevice, st));
    if (steps || mip) {
      if (c->aux_cap < npix * 2) {
        cudaFree(c->aux_buf);
        c->aux_buf = nullptr;
        c->aux_cap = 0;
        R3D_CUDA_TRY(c, cudaMalloc(&c->aux_buf, npix * 2 * 4));
        c->aux_cap = npix * 2;
      }
      steps = steps ? c->aux_buf : nullptr;
      mip = mip ? c->aux_buf + npix : nullptr;
      if (steps)
        R3D_CUDA_TRY(c, cudaMemcpyAsync(steps, aux->steps, npix * 4, cudaMemcpyHostToDevice, st));
      if (mip)
        R3D_CUDA_TRY(c,
                     cudaMemcpyAsync(mip, aux->mip_index, npix * 4, cudaMemcpyHostToDevice, st));
    }
    if (total || counters) {
      R3D_CUDA_TRY(c, cudaMemsetAsync(c->total, 0, (R3D_COUNTERS + 1) * 8, st));
      total = total ? c->total : nullptr;
      counters = counters ? c->total + 1 : nullptr;
    }
  }
  R3D_CUDA_TRY(c, cudaEventRecord(c->ev0, st));
  // views with overlay atlases and flattened-segment views render through
  // their own grid kernels
  bool any_ovl = false;
  for (uint32_t v = 0; v < nviews; v++)
    any_ovl = any_ovl || (render[v] && ((pcs[v].overlay_flags & kOvlAtlases) ||
                                        (pcs[v].view_flags & R3D_VIEW_SURF)));
  uint32_t nrender = 0;
  for (uint32_t v = 0; v < nviews; v++) nrender += render[v] ? 1u : 0u;
  const uint32_t persistent = resolved_persistent(c->sched, nrender);
  if (persistent && !any_ovl) {
    uint8_t *imgs[64];
    uint32_t strides[64];
    for (uint32_t v = 0; v < nviews; v++) {
      imgs[v] = img;
      strides[v] = out_w;
    }
    int rc = launch_views_persistent(c, persistent, pcs, render, nviews, imgs, strides, steps,
                                     mip, total, counters, st);
    if (rc != R3D_OK) return rc;
  } else {
    for (uint32_t v = 0; v < nviews; v++) {
      if (!render[v]) continue;
      cudaError_t e = launch_view(c, pcs[v], img, out_w, steps, mip, total, counters, st);
      if (e != cudaSuccess) return cuda_fail(c, e, "raycast_fwd: launch");
    }
  }
  R3D_CUDA_TRY(c, cudaEventRecord(c->ev1, st));
  c->timed = true;
  if (host) {
    R3D_CUDA_TRY(c, cudaMemcpyAsync(rgba_out, img, npix * 4, cudaMemcpyDeviceToHost, st));
    if (steps)
      R3D_CUDA_TRY(c, cudaMemcpyAsync(aux->steps, steps, npix * 4, cudaMemcpyDeviceToHost, st));
    if (mip)
      R3D_CUDA_TRY(c, cudaMemcpyAsync(aux->mip_index, mip, npix * 4, cudaMemcpyDeviceToHost, st));
    unsigned long long tsum[R3D_COUNTERS + 1] = {0};
    if (total || counters)
      R3D_CUDA_TRY(c, cudaMemcpyAsync(tsum, c->total, sizeof tsum, cudaMemcpyDeviceToHost, st));
    R3D_CUDA_TRY(c, cudaStreamSynchronize(st));
    if (total) *aux->total_steps += tsum[0];
    if (counters)
      for (int k = 0; k < R3D_COUNTERS; k++) aux->counters[k] += tsum[1 + k];
  }
  return R3D_OK;
}

int r3d_cuda_fill_rgba(r3d_cuda_ctx *c, uint8_t *img, size_t npix, const uint8_t rgba[4],
                       void *stream) {
  if (!c || !img || !rgba) return fail(c, R3D_E_INVALID, "fill_rgba: bad arguments");
  if (!npix) return R3D_OK;
  R3D_CUDA_TRY(c, cudaSetDevice(c->device));
  if (!is_device_ptr(img)) return fail(c, R3D_E_INVALID, "fill_rgba: the image must be device memory");
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  const uchar4 col = make_uchar4(rgba[0], rgba[1], rgba[2], rgba[3]);
  const uint32_t blocks = (uint32_t)std::min<size_t>((npix + 255u) / 256u, 148u * 16u);
  k_fill_rgba<<<blocks, 256, 0, st>>>((uchar4 *)img, npix, col);
  R3D_CUDA_TRY(c, cudaGetLastError());
  return R3D_OK;
}

int r3d_cuda_raycast_batch(r3d_cuda_ctx *c, const r3d_cuda_request *reqs, uint32_t n,
                           unsigned long long *total_steps, void *stream) {
  if (!c || !reqs || !n || n > kMaxBatchViews)
    return fail(c, R3D_E_INVALID, "raycast_batch: 1..%u requests", kMaxBatchViews);
  R3D_CUDA_TRY(c, cudaSetDevice(c->device));
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  r3d_frame_params pcs[kMaxBatchViews];
  int render[kMaxBatchViews];
  uint8_t *imgs[kMaxBatchViews];
  uint32_t strides[kMaxBatchViews];
  bool any_ovl = false;
  for (uint32_t i = 0; i < n; i++) {
    const r3d_frame_params &v = reqs[i].view;
    if (!reqs[i].rgba || !v.viewport[0] || !v.viewport[1] || v.view_org)
      return fail(c, R3D_E_INVALID, "raycast_batch: request %u needs an image, a viewport and "
                                    "view_org 0", i);
    if (!is_device_ptr(reqs[i].rgba))
      return fail(c, R3D_E_INVALID, "raycast_batch: request %u image is not device memory", i);
    render[i] = prepare_view(c, v, v.viewport[0], v.viewport[1], pcs[i]);
    if (render[i] < 0) return render[i];
    imgs[i] = reqs[i].rgba;
    strides[i] = pcs[i].viewport[0];
    any_ovl = any_ovl || (pcs[i].overlay_flags & kOvlAtlases) || (pcs[i].view_flags & R3D_VIEW_SURF);
  }
  uint32_t nrender = 0;
  for (uint32_t i = 0; i < n; i++) nrender += render[i] ? 1u : 0u;
  const uint32_t persistent = resolved_persistent(c->sched, nrender);
  if (persistent && !any_ovl)
    return launch_views_persistent(c, persistent, pcs, render, n, imgs, strides, nullptr,
                                   nullptr, total_steps, nullptr, st);
  for (uint32_t i = 0; i < n; i++) {
    if (!render[i]) continue;
    cudaError_t e = launch_view(c, pcs[i], imgs[i], strides[i], nullptr, nullptr, total_steps,
                                nullptr, st);
    if (e != cudaSuccess) return cuda_fail(c, e, "raycast_batch: launch");
  }
  return R3D_OK;
}

int r3d_cuda_last_kernel_ns(r3d_cuda_ctx *c, uint64_t *ns) {
  if (!c || !ns) return R3D_E_INVALID;
  if (!c->timed) return fail(c, R3D_E_STATE, "last_kernel_ns: nothing timed");
  cudaSetDevice(c->device);
  R3D_CUDA_TRY(c, cudaEventSynchronize(c->ev1));
  float ms = 0.0f;
  R3D_CUDA_TRY(c, cudaEventElapsedTime(&ms, c->ev0, c->ev1));
  *ns = (uint64_t)((double)ms * 1e6);
  return R3D_OK;
}

}  // extern "C"

