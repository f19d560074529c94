// Differentiable emission-absorption raycast: forward and adjoint.
//
// The render is render3d's compositing without shading (FLAT mode,
// src/shaders/raycast.slang:894-1017) over an FP32 density grid and an FP32
// 256x4 transfer function: ray setup of the cube path, trilinear density at
// texel centres (level 0, clamp to edge, no empty-space skip), TF lookup at
// v*256-0.5, alpha clamped to [0, 1], opacity correction
// a = 1 - (1 - alpha)^(density * step * lod_step), samples with a <= 0.003
// ignored, front-to-back compositing with termination at the cutoff, then
// the background.  The forward kernel writes an FP32 RGB image per view;
// its arithmetic equals the CPU oracle's bit for bit.  A sample whose
// density falls in the TF's leading run of zero-alpha texels (both texels
// alpha 0) has opacity exactly 0; it is skipped before the TF lookup.
//
// The adjoint kernel (one thread per ray) returns the gradients of
// L = sum(dL/drgb * rgb) with respect to every voxel, every LUT entry and the
// density scale.  It first marches the ray forward, keeping a checkpoint
// (position and accumulated opacity) every K samples in local memory, the
// number of contributing samples of each K-sample segment, and the last 64
// contributing samples.  It then walks the segments with contributions from
// last to first: a segment whose samples are still among the remembered ones
// uses them, any other is recomputed from its checkpoint; the samples are
// visited in reverse with the colour behind them S (S <- a c + (1 - a) S,
// starting from the background).  Transmittance is never divided out, which
// would be unstable as alpha approaches 1.
//
// Gradients: voxel contributions are summed per trilinear cell in registers
// while consecutive samples stay in one cell, then flushed with global
// atomics; LUT contributions go to a per-block shared-memory table flushed
// once per block; the density-scale gradient is reduced per warp.  Atomic
// mode adds FP32 (order-dependent rounding).  Deterministic mode adds
// fixed-point integers (value * 2^32, rounded, in int64; mod 2^64 as two
// 32-bit words in the shared table): integer addition is associative, so
// the result is identical for any execution order.
#include <string.h>

#include "r3d_internal.h"

namespace r3d {

constexpr double kFix = 4294967296.0;  // 2^32, deterministic fixed point

struct DiffView {
  r3d_frame_params pc;
  unsigned long long out_off;  // first float of the view's RGB image
  uint32_t tile_begin;         // first of the view's 8x4 ray tiles in the call's
  uint32_t pad;
};

struct DiffGrid {
  const float *dens;
  // per voxel (x, y, z): the densities at (x, y), (x1, y), (x, y1), (x1, y1)
  // of its z plane, x1 = min(x + 1, nx - 1) and y1 likewise, so that a
  // trilinear sample reads two float4 instead of eight floats
  const float4 *quad;
  // the call's own words (call_words): [0] the TF's first texel with alpha not
  // 0 (256: none), [1] the next ray tile
  uint32_t *zc;
  uint32_t n[3];
  uint32_t nmax;
  uint32_t wide;  // an axis of more than 2^23 voxels (floor_frac's range)
  const float *lut;  // 256 x 4
  float cutoff;
};

struct DiffRay {
  float ro[3], dir[3];
  float t0, tf, dt, span;
  bool hit;
};

// ray setup of the cube path (raycast.slang:640-748)
__device__ __forceinline__ void diff_setup(const r3d_frame_params &pc, const DiffGrid &g,
                                           uint32_t px, uint32_t py, DiffRay &r) {
  const bool ortho = (pc.view_flags & R3D_VIEW_ORTHO) != 0u;
  float ux = ((float)px + 0.5f) / (float)pc.viewport[0];
  float uy = ((float)py + 0.5f) / (float)pc.viewport[1];
  float nx = ux * 2.0f - 1.0f, ny = 1.0f - uy * 2.0f;
  float3 fw = make_float3(pc.cam_forward[0], pc.cam_forward[1], pc.cam_forward[2]);
  float3 rt = make_float3(pc.cam_right[0], pc.cam_right[1], pc.cam_right[2]);
  float3 up = make_float3(pc.cam_up[0], pc.cam_up[1], pc.cam_up[2]);
  float3 d = ortho ? fw
                   : make_float3(fmaf(ny, up.x, fmaf(nx, rt.x, fw.x)),
                                 fmaf(ny, up.y, fmaf(nx, rt.y, fw.y)),
                                 fmaf(ny, up.z, fmaf(nx, rt.z, fw.z)));
  d = norm3(d);
  float3 o = make_float3(pc.cam_origin[0], pc.cam_origin[1], pc.cam_origin[2]);
  if (ortho)
    o = make_float3(fmaf(ny, up.x, fmaf(nx, rt.x, o.x)), fmaf(ny, up.y, fmaf(nx, rt.y, o.y)),
                    fmaf(ny, up.z, fmaf(nx, rt.z, o.z)));
  const float c = 0.5f;
  float q[3] = {(o.x - pc.vol_tx) - c, (o.y - pc.vol_ty) - c, (o.z - pc.vol_tz) - c};
  float dv[3] = {d.x, d.y, d.z};
  const float *r0 = pc.vol_r0, *r1 = pc.vol_r1, *r2 = pc.vol_r2;
#pragma unroll
  for (int a = 0; a < 3; a++) {
    r.ro[a] = fmaf(r2[a], q[2], fmaf(r1[a], q[1], r0[a] * q[0])) + c;
    r.dir[a] = fmaf(r2[a], dv[2], fmaf(r1[a], dv[1], r0[a] * dv[0]));
  }
  float tmn[3], tmx[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    float iv = 1.0f / r.dir[a];
    float t0 = (0.0f - r.ro[a]) * iv, t1 = (1.0f - r.ro[a]) * iv;
    tmn[a] = fminf(t0, t1);
    tmx[a] = fmaxf(t0, t1);
  }
  float tn = fmaxf(fmaxf(fmaxf(tmn[0], tmn[1]), tmn[2]), 0.0f);
  float tf = fminf(fminf(fminf(tmx[0], tmx[1]), tmx[2]), 1e30f);
  r.hit = !(tn >= tf);
  float voxel = 1.0f / (float)g.nmax;
  r.dt = pc.step_voxels * voxel;
  r.t0 = fmaf(hash12(px, py, pc.frame_index), r.dt, tn);
  r.tf = tf;
  r.span = fmaxf((tf - tn) / (4096.0f * r.dt), 1.0f);
}


// One sample: density, TF, opacity.  Fills the trilinear cell for scatters.
struct DiffSample {
  float v, tt, f, s[4], alpha, a;
  uint32_t i0, i1;
  uint32_t base, sx, sy, sz;  // corner (x0,y0,z0) and strides to x1/y1/z1 (0 at edges)
  float fx, fy, fz;
};

// The trilinear cell of the sample at t: corner, strides, fractions.
__device__ __forceinline__ void diff_cell(const DiffGrid &g, const DiffRay &r, float t,
                                          DiffSample &o) {
  float p[3] = {fmaf(t, r.dir[0], r.ro[0]), fmaf(t, r.dir[1], r.ro[1]),
                fmaf(t, r.dir[2], r.ro[2])};
  uint32_t i0[3];
  float fr[3];
  bool up[3];
#pragma unroll
  for (int a = 0; a < 3; a++) {
    float tc = clamp_(fmaf(p[a], (float)g.n[a], -0.5f), 0.0f, (float)(g.n[a] - 1u));
    if (g.wide) {
      i0[a] = (uint32_t)tc;
      fr[a] = tc - (float)i0[a];
    } else {  // the same without the conversion unit
      i0[a] = floor_frac(tc, fr[a]);
    }
    up[a] = i0[a] + 1u < g.n[a];
  }
  const uint32_t nx = g.n[0], nxy = g.n[0] * g.n[1];
  o.base = i0[0] + i0[1] * nx + i0[2] * nxy;
  o.sx = up[0] ? 1u : 0u;
  o.sy = up[1] ? nx : 0u;
  o.sz = up[2] ? nxy : 0u;
  o.fx = fr[0];
  o.fy = fr[1];
  o.fz = fr[2];
}

// Density of a sample whose cell is known.
__device__ __forceinline__ void diff_value(float4 q0, float4 q1, DiffSample &o) {
  const float c00 = lerp_(q0.x, q0.y, o.fx), c10 = lerp_(q0.z, q0.w, o.fx);
  const float c01 = lerp_(q1.x, q1.y, o.fx), c11 = lerp_(q1.z, q1.w, o.fx);
  o.v = lerp_(lerp_(c00, c10, o.fy), lerp_(c01, c11, o.fy), o.fz);
}

// TF coordinate, texels and fraction of a sample
__device__ __forceinline__ void diff_texel(DiffSample &o) {
  o.tt = clamp_(fmaf(o.v, 256.0f, -0.5f), 0.0f, 255.0f);
  o.i0 = floor_frac(o.tt, o.f);
  o.i1 = min(o.i0 + 1u, 255u);
}

// and its colour and alpha (FP32, as the oracle)
__device__ __forceinline__ void diff_tf_color(const float4 *lut, DiffSample &o) {
  const float4 l0 = lut[o.i0], l1 = lut[o.i1];
  o.s[0] = lerp_(l0.x, l1.x, o.f);
  o.s[1] = lerp_(l0.y, l1.y, o.f);
  o.s[2] = lerp_(l0.z, l1.z, o.f);
  o.s[3] = lerp_(l0.w, l1.w, o.f);
  o.alpha = clamp_(o.s[3], 0.0f, 1.0f);
}

// TF and opacity of a sample whose density is known; false when it cannot
// contribute: under the low cut, both TF texels with alpha 0 (z = the TF's
// first texel whose alpha is not 0: then alpha = lerp(0, 0, f) = 0 and the
// opacity is 1 - 1^k = 0), or at most the 0.003 floor.
__device__ __forceinline__ bool diff_live(const float4 *lut, uint32_t z, float threshold, float k,
                                          DiffSample &o) {
  if (o.v < threshold) return false;
  diff_texel(o);
  if (o.i1 < z) return false;
  diff_tf_color(lut, o);
  o.a = 1.0f - r3d_powf(1.0f - o.alpha, k);
  return o.a > 0.003f;
}

// Steps [step, last) of a ray from position t: visit(step, t, sample) for
// each sample that can contribute, until it returns false; returns the steps
// taken.  No step depends on what a sample holds, only whether the march goes
// on, so the cells of the next kAhead samples are loaded before any of them
// is used (one past the end reads a clamped cell).  The march waits on those
// loads (each takes about 12 wavefronts of the L1 pipe, 70 % of its rate):
// 64 views of 256^2 over 256^3 forward 1.63 ms with one sample at a time,
// 1.53 / 1.50 / 1.55 with 2 / 3 / 4; keeping the words of a repeated cell in
// registers gained nothing (1.57).
constexpr int kAhead = 3;
template <class F>
__device__ __forceinline__ uint32_t diff_march(const DiffGrid &g, const DiffRay &r,
                                               const float4 *lut, uint32_t z, float threshold,
                                               float k, float t, uint32_t step, uint32_t last,
                                               F visit) {
  while (true) {
    DiffSample s[kAhead];
    float4 q0[kAhead], q1[kAhead];
    float at[kAhead];
#pragma unroll
    for (int i = 0; i < kAhead; i++) {
      at[i] = t;
      diff_cell(g, r, t, s[i]);
      q0[i] = __ldg(g.quad + s[i].base);
      q1[i] = __ldg(g.quad + s[i].base + s[i].sz);
      t = fmaf(r.dt, r.span, t);
    }
#pragma unroll
    for (int i = 0; i < kAhead; i++) {
      if (!(at[i] < r.tf && step < last)) return step;
      step++;
      diff_value(q0[i], q1[i], s[i]);
      if (diff_live(lut, z, threshold, k, s[i]) && !visit(step, at[i], s[i])) return step;
    }
  }
}

// The quad grid of DiffGrid::quad from the density grid.
__global__ void k_diff_quads(const float *__restrict__ d, uint32_t nx, uint32_t ny, uint32_t nz,
                             float4 *__restrict__ q) {
  const size_t n = (size_t)nx * ny * nz;
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x) {
    const uint32_t x = (uint32_t)(i % nx), y = (uint32_t)((i / nx) % ny);
    const size_t dx = x + 1u < nx ? 1u : 0u, dy = y + 1u < ny ? nx : 0u;
    q[i] = make_float4(__ldg(d + i), __ldg(d + i + dx), __ldg(d + i + dy), __ldg(d + i + dy + dx));
  }
}

// The call's words (DiffGrid::zc): the TF's first texel with alpha, and the
// tile counter at 0 (one block).
__global__ void k_diff_tf_clear(const float *__restrict__ lut, uint32_t *__restrict__ zc) {
  __shared__ uint32_t z;
  if (threadIdx.x == 0) z = 256u;
  __syncthreads();
  for (uint32_t i = threadIdx.x; i < 256u; i += blockDim.x)
    if (__ldg(lut + 4u * i + 3u) != 0.0f) atomicMin(&z, i);
  __syncthreads();
  if (threadIdx.x == 0) {
    zc[0] = z;
    zc[1] = 0u;
  }
}

// Tape of a training forward: per ray, the first kTape contributing samples
// and their count.  An entry holds t, the accumulated opacity before the
// sample, and the sample's density and opacity (x, y, z, w), so that the
// backward needs neither the density fetch nor the opacity's power again.
// A backward over the same views and scene walks these in reverse instead
// of marching the ray again; rays with more contributions take the
// checkpoint path.  Entry i of ray tile k's lane l stands at (k * kTape + i) *
// 32 + l, so that a warp's entries i are 512 contiguous bytes.
constexpr uint32_t kTape = 64;
using TapeEntry = float4;

// The march kernels' ray tiles: a warp takes the next 8x4 tile of the call's
// views from a counter until none is left, so a launch holds only resident
// blocks, a warp whose rays end early takes the next tile at once, and the
// blocks' shared tables are cleared and flushed once per resident block.
struct DiffTile {
  uint32_t view, px, py;
  uint32_t k;  // the tile's index in the call
};
__device__ __forceinline__ bool next_tile(const DiffView *__restrict__ views, uint32_t nviews,
                                          uint32_t ntiles, uint32_t *queue, DiffTile &t) {
  const uint32_t lane = threadIdx.x & 31u;
  uint32_t k = 0;
  if (lane == 0u) k = atomicAdd(queue, 1u);
  k = __shfl_sync(0xffffffffu, k, 0);
  if (k >= ntiles) return false;
  while (t.view + 1u < nviews && views[t.view + 1u].tile_begin <= k) t.view++;  // tiles only move on
  const uint32_t tiles_x = (views[t.view].pc.viewport[0] + 7u) / 8u;
  const uint32_t r = k - views[t.view].tile_begin;
  t.px = (r % tiles_x) * 8u + ((lane & 1u) | ((lane >> 1) & 2u) | ((lane >> 2) & 4u));
  t.py = (r / tiles_x) * 4u + (((lane >> 1) & 1u) | ((lane >> 2) & 2u));
  t.k = k;
  return true;
}

template <bool TAPE>
__global__ void __launch_bounds__(128) k_diff_fwd(const DiffView *__restrict__ views,
                                                  uint32_t nviews, uint32_t ntiles,
                                                  const __grid_constant__ DiffGrid g,
                                                  float *__restrict__ rgb,
                                                  unsigned long long *__restrict__ total,
                                                  TapeEntry *__restrict__ tape,
                                                  uint32_t *__restrict__ tape_n) {
  const float4 *lut = (const float4 *)g.lut;
  const uint32_t zc = __ldg(g.zc);
  const uint32_t lane = threadIdx.x & 31u;
  unsigned long long all_steps = 0;
  DiffTile tile = {0u, 0u, 0u, 0u};
  while (next_tile(views, nviews, ntiles, g.zc + 1, tile)) {
    const DiffView &vw = views[tile.view];
    const r3d_frame_params &pc = vw.pc;
    const uint32_t px = tile.px, py = tile.py;
    if (px >= pc.viewport[0] || py >= pc.viewport[1]) continue;
    TapeEntry *rec = TAPE ? tape + (size_t)tile.k * (kTape * 32u) + lane : nullptr;
    DiffRay r;
    diff_setup(pc, g, px, py, r);
    float acc_r = 0.0f, acc_g = 0.0f, acc_b = 0.0f, acc_a = 0.0f;
    uint32_t nc = 0, steps = 0;
    if (r.hit) {
      const float k = (pc.density * pc.step_voxels) * r.span;
      steps = diff_march(g, r, lut, zc, pc.threshold, k, r.t0, 0u, 4096u,
                         [&](uint32_t, float t, const DiffSample &s) {
        if (TAPE && nc < kTape) rec[nc * 32u] = make_float4(t, acc_a, s.v, s.a);
        nc++;
        float w = (1.0f - acc_a) * s.a;
        acc_r = fmaf(w, s.s[0], acc_r);
        acc_g = fmaf(w, s.s[1], acc_g);
        acc_b = fmaf(w, s.s[2], acc_b);
        acc_a = acc_a + w;
        return acc_a < g.cutoff;
      });
    }
    if (TAPE) tape_n[(size_t)tile.k * 32u + lane] = nc;
    float tr = 1.0f - acc_a;
    float *o = rgb + vw.out_off + ((size_t)py * pc.viewport[0] + px) * 3u;
    o[0] = fmaf(tr, 0.02f, acc_r);
    o[1] = fmaf(tr, 0.02f, acc_g);
    o[2] = fmaf(tr, 0.03f, acc_b);
    all_steps += steps;
  }
  if (total) {
    for (int off = 16; off > 0; off >>= 1) all_steps += __shfl_xor_sync(0xffffffffu, all_steps, off);
    if (lane == 0 && all_steps) atomicAdd(total, all_steps);
  }
}

// x * 2^32 rounded to the nearest int64: the product is exact in FP32 (a
// power-of-two scale), so converting it directly equals converting
// (double)x * 2^32
__device__ __forceinline__ long long fix32(float x) {
  return __float2ll_rn(x * 4294967296.0f);
}

// voxel gradient sink: FP32 atomics or 2^32 fixed point
template <bool DET>
__device__ __forceinline__ void vox_add(float *gf, unsigned long long *gq, uint32_t i, float x) {
  if (x == 0.0f) return;
  if (DET)
    atomicAdd(gq + i, (unsigned long long)fix32(x));
  else
    atomicAdd(gf + i, x);
}

// The block's LUT-gradient table in shared memory.  Deterministic sums are
// kept mod 2^64 as two 32-bit words per entry: the low word takes the low
// half of each addend, and a carry out of it goes to the high word with the
// high half, so that every update is two native 32-bit shared atomics.
// An FP32 shared atomic is a compare-and-swap loop, which repeats for each
// lane of the warp that meets the same word, and neighbouring rays often pass
// the same few texels (air, the sheet's mean).  So the FP32 table is kept
// four times, a lane in four using each (every sample lit: 0.92 -> 0.83 ms a
// backward; the integer table gains nothing, 0.74 and 0.81 ms); the stride
// keeps the copies of a texel in different banks.
template <bool DET>
constexpr uint32_t kLutCopies = DET ? 1u : 4u;
constexpr uint32_t kLutStride = 1024u + 4u;
template <bool DET>
struct LutGrad {
  uint32_t w[kLutCopies<DET> * kLutStride * (DET ? 2u : 1u)];  // deterministic: low words, then high words
};

template <bool DET>
__device__ __forceinline__ void lut_add(LutGrad<DET> &lg, uint32_t i, float x) {
  i += (threadIdx.x & (kLutCopies<DET> - 1u)) * kLutStride;
  if (DET) {
    const long long q = fix32(x);
    if (!q) return;
    const uint32_t ql = (uint32_t)q, qh = (uint32_t)((unsigned long long)q >> 32);
    const uint32_t old = atomicAdd(&lg.w[i], ql);
    const uint32_t h = qh + (old + ql < old ? 1u : 0u);
    if (h) atomicAdd(&lg.w[kLutCopies<DET> * kLutStride + i], h);
  } else {
    if (x != 0.0f) atomicAdd(reinterpret_cast<float *>(&lg.w[i]), x);
  }
}

template <bool DET>
__device__ __forceinline__ void lut_clear(LutGrad<DET> &lg) {
  for (uint32_t i = threadIdx.x; i < sizeof lg.w / 4u; i += blockDim.x) lg.w[i] = 0u;  // 0.0f too
}

template <bool DET>
__device__ __forceinline__ void lut_flush(const LutGrad<DET> &lg, float *g_lut,
                                          unsigned long long *q_lut) {
  for (uint32_t i = threadIdx.x; i < 1024u; i += blockDim.x) {
    if (DET) {
      unsigned long long q = 0;
#pragma unroll
      for (uint32_t c = 0; c < kLutCopies<DET>; c++) {
        const uint32_t k = c * kLutStride + i;
        q += ((unsigned long long)lg.w[kLutCopies<DET> * kLutStride + k] << 32) | lg.w[k];
      }
      if (q) atomicAdd(q_lut + i, q);
    } else {
      float x = 0.0f;
#pragma unroll
      for (uint32_t c = 0; c < kLutCopies<DET>; c++) x += __uint_as_float(lg.w[c * kLutStride + i]);
      if (x != 0.0f) atomicAdd(g_lut + i, x);
    }
  }
}

constexpr int kRing = 64;  // contributing samples remembered by the forward sweep

// State of one ray's reverse sweep: the colour behind the current sample,
// the trilinear cell whose voxel gradients are being summed, and the
// density-scale gradient.
struct BwdRay {
  float gr, gg, gb;  // dL/drgb of the pixel
  float k, kstep;
  float S_r, S_g, S_b;
  uint32_t cell, csx, csy, csz;
  float cw[8];
  float g_density;
};

template <bool DET>
__device__ __forceinline__ void bwd_flush(BwdRay &b, float *g_dens, unsigned long long *q_dens) {
  if (b.cell == 0xffffffffu) return;
#pragma unroll
  for (int c = 0; c < 8; c++)
    vox_add<DET>(g_dens, q_dens,
                 b.cell + ((c & 1) ? b.csx : 0u) + ((c & 2) ? b.csy : 0u) + ((c & 4) ? b.csz : 0u),
                 b.cw[c]);
}

// Adjoint of one contributing sample s (density, TF and opacity filled) with
// accumulated opacity acc_a before it, visited in reverse order (suffix
// colour S <- a c + (1 - a) S).
template <bool DET>
__device__ __forceinline__ void bwd_contrib(const float4 *lut, const DiffSample &s, float acc_a,
                                            BwdRay &b, LutGrad<DET> &lg, float *g_dens,
                                            unsigned long long *q_dens) {
  const float tprev = 1.0f - acc_a;
  const float dc_r = b.gr * tprev * s.a, dc_g = b.gg * tprev * s.a, dc_b = b.gb * tprev * s.a;
  const float da = b.gr * tprev * (s.s[0] - b.S_r) + b.gg * tprev * (s.s[1] - b.S_g) +
                   b.gb * tprev * (s.s[2] - b.S_b);
  b.S_r = fmaf(s.a, s.s[0] - b.S_r, b.S_r);
  b.S_g = fmaf(s.a, s.s[1] - b.S_g, b.S_g);
  b.S_b = fmaf(s.a, s.s[2] - b.S_b, b.S_b);
  float dalpha = 0.0f;
  const bool alpha_free = s.s[3] > 0.0f && s.s[3] < 1.0f;  // implies alpha < 1
  if (s.alpha < 1.0f) {
    const float x = 1.0f - s.alpha, l2 = r3d_log2f(x);
    if (alpha_free) {  // r3d_powf(x, k - 1) with the logarithm shared (x > 0 here)
      const float y = b.k - 1.0f;
      dalpha = da * b.k * (y == 0.0f || x == 1.0f ? 1.0f : r3d_exp2f(y * l2));
    }
    b.g_density += da * (-(1.0f - s.a) * (l2 * 0.693147181f)) * b.kstep;
  }
  const float ds[4] = {dc_r, dc_g, dc_b, dalpha};
  const float lf0 = 1.0f - s.f;
  const float4 l0 = lut[s.i0];
  const float4 l1 = lut[s.i1];
  const float dl[4] = {l1.x - l0.x, l1.y - l0.y, l1.z - l0.z, l1.w - l0.w};
  float dvv = 0.0f;
#pragma unroll
  for (int c = 0; c < 4; c++) {
    lut_add<DET>(lg, s.i0 * 4u + c, ds[c] * lf0);
    lut_add<DET>(lg, s.i1 * 4u + c, ds[c] * s.f);
    dvv = fmaf(ds[c], dl[c], dvv);
  }
  const bool tt_free = s.tt > 0.0f && s.tt < 255.0f;
  const float dv = tt_free ? dvv * 256.0f : 0.0f;
  // trilinear scatter, aggregated per cell
  if (s.base != b.cell || s.sx != b.csx || s.sy != b.csy || s.sz != b.csz) {
    bwd_flush<DET>(b, g_dens, q_dens);
    b.cell = s.base;
    b.csx = s.sx;
    b.csy = s.sy;
    b.csz = s.sz;
#pragma unroll
    for (int c = 0; c < 8; c++) b.cw[c] = 0.0f;
  }
  const float wx[2] = {1.0f - s.fx, s.fx}, wy[2] = {1.0f - s.fy, s.fy},
              wz[2] = {1.0f - s.fz, s.fz};
#pragma unroll
  for (int c = 0; c < 8; c++)
    b.cw[c] = fmaf(dv, (wx[c & 1] * wy[(c >> 1) & 1]) * wz[c >> 2], b.cw[c]);
}

// The adjoint of a contributing sample whose march position, accumulated
// opacity, density and opacity are known.
template <bool DET>
__device__ __forceinline__ void bwd_known(const DiffGrid &g, const float4 *lut, const DiffRay &r,
                                          float4 e, BwdRay &b, LutGrad<DET> &lg, float *g_dens,
                                          unsigned long long *q_dens) {
  DiffSample s;
  diff_cell(g, r, e.x, s);
  s.v = e.z;
  diff_texel(s);
  diff_tf_color(lut, s);
  s.a = e.w;
  bwd_contrib<DET>(lut, s, e.y, b, lg, g_dens, q_dens);
}

// One ray per lane.  Bound by issue and by the chains of each contribution
// (logarithm, power, TF loads); five blocks a SM (96 registers; 116 with four
// lose 5 %, 80 with six 10 %).  64 views of 256^2 over 256^3 from the tape,
// deterministic: 1.54 ms with a block per 16 x 8 rays and a tape of a ray's
// entries in a row, 1.19 ms.  Without a tape, every sample lit (5 views of
// 151 x 117): 2.97 -> 0.83 ms, of which the reverse sweep's common loops give
// all but 0.5.
template <int K, bool DET>
__global__ void __launch_bounds__(128, 5) k_diff_bwd(const DiffView *__restrict__ views,
                                                  uint32_t nviews, uint32_t ntiles,
                                                  const __grid_constant__ DiffGrid g,
                                                  const float *__restrict__ dl_drgb,
                                                  float *__restrict__ g_dens,
                                                  unsigned long long *__restrict__ q_dens,
                                                  float *__restrict__ g_lut,
                                                  unsigned long long *__restrict__ q_lut,
                                                  float *__restrict__ g_scale,
                                                  unsigned long long *__restrict__ q_scale,
                                                  const TapeEntry *__restrict__ tape,
                                                  const uint32_t *__restrict__ tape_n) {
  constexpr int kMaxCk = (4096 + K - 1) / K;
  __shared__ LutGrad<DET> lg;
  lut_clear<DET>(lg);
  __syncthreads();
  const float4 *lut = (const float4 *)g.lut;
  const uint32_t zc = __ldg(g.zc);
  constexpr uint32_t kAll = 0xffffffffu;
  const uint32_t lane = threadIdx.x & 31u;
  long long q_sum = 0;  // density scale: the lane's rays
  float f_sum = 0.0f;
  DiffTile tile = {0u, 0u, 0u, 0u};
  while (next_tile(views, nviews, ntiles, g.zc + 1, tile)) {
    const DiffView &vw = views[tile.view];
    const r3d_frame_params &pc = vw.pc;
    const uint32_t px = tile.px, py = tile.py;
    const bool inside = px < pc.viewport[0] && py < pc.viewport[1];
    BwdRay b;
    b.g_density = 0.0f;
    DiffRay r;
    diff_setup(pc, g, px, py, r);
    b.gr = b.gg = b.gb = 0.0f;
    if (inside) {
      const float *gp = dl_drgb + vw.out_off + ((size_t)py * pc.viewport[0] + px) * 3u;
      b.gr = gp[0];
      b.gg = gp[1];
      b.gb = gp[2];
    }
    b.k = (pc.density * pc.step_voxels) * r.span;
    b.kstep = pc.step_voxels * r.span;
    b.S_r = 0.02f;
    b.S_g = 0.02f;
    b.S_b = 0.03f;
    b.cell = 0xffffffffu;
    b.csx = b.csy = b.csz = 0u;
#pragma unroll
    for (int c = 0; c < 8; c++) b.cw[c] = 0.0f;
    const bool go = inside && r.hit && (b.gr != 0.0f || b.gg != 0.0f || b.gb != 0.0f);
    const uint32_t taped = go && tape ? tape_n[(size_t)tile.k * 32u + lane] : 0xffffffffu;
    // The lanes of a warp take their n-th last contribution together (loops
    // of the warp's largest count, lanes without one idle): written as loops
    // of each lane's own counts the reverse sweep ran at 8 of 32 lanes.
    const uint32_t ntape = go && taped <= kTape ? taped : 0u;  // every contribution is on the tape
    const TapeEntry *rec = tape + (size_t)tile.k * (kTape * 32u) + lane;
    for (uint32_t n = __reduce_max_sync(kAll, ntape); n-- > 0u;)
      if (n < ntape) bwd_known<DET>(g, lut, r, __ldg(rec + n * 32u), b, lg, g_dens, q_dens);
    const bool march = go && taped > kTape;
    if (__any_sync(kAll, march)) {
      // forward sweep: checkpoints (t, accumulated opacity) before steps
      // 1, K+1, 2K+1, ..., the number of contributing samples of each
      // segment, and the last kRing contributing samples themselves
      float ck_t[kMaxCk], ck_a[kMaxCk];
      uint8_t ck_n[kMaxCk];
      float4 ring[kRing];
      uint32_t nsteps = 0, ncontrib = 0;
      const float threshold = pc.threshold;
      if (march) {
        float t = r.t0, acc_a = 0.0f;
        bool more = true;
        while (more && t < r.tf && nsteps < 4096u) {  // a segment
          const uint32_t j = nsteps / K, n0 = ncontrib, s_end = nsteps + K;
          ck_t[j] = t;
          ck_a[j] = acc_a;
          nsteps = diff_march(g, r, lut, zc, threshold, b.k, t, nsteps, s_end,
                              [&](uint32_t, float at, const DiffSample &s) {
            ring[ncontrib % kRing] = make_float4(at, acc_a, s.v, s.a);
            ncontrib++;
            acc_a = acc_a + (1.0f - acc_a) * s.a;
            more = acc_a < g.cutoff;
            return more;
          });
          ck_n[j] = (uint8_t)(ncontrib - n0);
          for (int i = 0; i < K; i++) t = fmaf(r.dt, r.span, t);
        }
      }
      __syncwarp();
      // reverse sweep over each ray's segments, the last one first
      float4 seg[K];
      const uint32_t nck = (nsteps + K - 1u) / K;
      uint32_t end = ncontrib;  // contributions of the segments left: [0, end)
      const uint32_t rounds = __reduce_max_sync(kAll, nck);
      for (uint32_t i = 1; i <= rounds; i++) {
        const bool have = i <= nck;
        const uint32_t j = have ? nck - i : 0u;
        const uint32_t nj = have ? ck_n[j] : 0u, start = end - nj;
        const bool in_ring = ncontrib - start <= (uint32_t)kRing;
        if (nj && !in_ring) {  // recompute segment j from its checkpoint
          float acc_a = ck_a[j];
          int nseg = 0;
          diff_march(g, r, lut, zc, threshold, b.k, ck_t[j], j * K, min(nsteps, (j + 1u) * K),
                     [&](uint32_t, float t, const DiffSample &s) {
            seg[nseg++] = make_float4(t, acc_a, s.v, s.a);
            acc_a = acc_a + (1.0f - acc_a) * s.a;
            return true;
          });
        }
        __syncwarp();
        for (uint32_t n = __reduce_max_sync(kAll, nj); n-- > 0u;)
          if (n < nj)
            bwd_known<DET>(g, lut, r, in_ring ? ring[(start + n) % kRing] : seg[n], b, lg, g_dens,
                           q_dens);
        end = start;
      }
    }
    bwd_flush<DET>(b, g_dens, q_dens);
    if (DET)
      q_sum += fix32(b.g_density);
    else
      f_sum += b.g_density;
  }
  // density scale: warp reduction, one global add per warp
  if (DET) {
    for (int off = 16; off > 0; off >>= 1) q_sum += __shfl_xor_sync(0xffffffffu, q_sum, off);
    if (lane == 0 && q_sum) atomicAdd(q_scale, (unsigned long long)q_sum);
  } else {
    for (int off = 16; off > 0; off >>= 1) f_sum += __shfl_xor_sync(0xffffffffu, f_sum, off);
    if (lane == 0 && f_sum != 0.0f) atomicAdd(g_scale, f_sum);
  }
  __syncthreads();
  lut_flush<DET>(lg, g_lut, q_lut);
}

// Blocks of 128 threads of a march kernel over ntiles tiles: the resident
// ones, and no more warps than tiles.
template <class F>
static unsigned march_blocks(F kernel, uint32_t ntiles) {
  int dev = 0, sms = 148, per = 1;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, kernel, 128, 0) != cudaSuccess || per < 1)
    per = 1;
  return max(min((unsigned)(per * sms), (ntiles + 3u) / 4u), 1u);
}

static unsigned grid_blocks(size_t n) {
  size_t b = (n + 255) / 256;
  return (unsigned)(b < 148u * 32u ? (b ? b : 1) : 148u * 32u);
}

// fixed point -> float
__global__ void k_fix_to_float(const unsigned long long *__restrict__ q, float *__restrict__ out,
                               size_t n) {
  for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n;
       i += (size_t)gridDim.x * blockDim.x)
    out[i] = (float)((double)(long long)q[i] / kFix);
}

}  // namespace r3d

using namespace r3d;

// A call's words (DiffGrid::zc).  Calls of one context may overlap on several
// streams, and each drains its own tile counter, so the words go with the view
// table's ring slot: the call that takes a slot again waits, on its stream, for
// the march of the one that had it.  A call that is being captured can not
// wait for work outside its graph, and its graph may run at any later time:
// it takes words that only captured calls use, others for each call until
// kCapturedCalls have been captured.
static int call_words(r3d_cuda_ctx *c, int slot, DiffGrid &g, bool &captured, cudaStream_t st) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  R3D_CUDA_TRY(c, cudaStreamIsCapturing(st, &cs));
  captured = cs != cudaStreamCaptureStatusNone;
  if (!captured) {
    g.zc = c->diff_words + 2 * slot;
    if (c->ring_marched[slot]) R3D_CUDA_TRY(c, cudaStreamWaitEvent(st, c->ring_march_ev[slot], 0));
  } else {
    g.zc = c->diff_words + 2 * (r3d_cuda_ctx::kRing + c->captured_next);
    c->captured_next = (c->captured_next + 1u) % r3d_cuda_ctx::kCapturedCalls;
  }
  return R3D_OK;
}

// After the march: the slot may be taken again.
static int call_marched(r3d_cuda_ctx *c, int slot, bool captured, cudaStream_t st) {
  if (captured) return R3D_OK;
  R3D_CUDA_TRY(c, cudaEventRecord(c->ring_march_ev[slot], st));
  c->ring_marched[slot] = true;
  return R3D_OK;
}

// Validates the grid and views, takes the call's words and uploads the view
// table; returns the grid descriptor, total output floats and ring slot.
static int diff_prepare(r3d_cuda_ctx *c, const r3d_cuda_diff_scene *sc,
                        const r3d_frame_params *views, uint32_t nviews, DiffGrid &g,
                        DiffView *&dviews, uint32_t &ntiles, size_t &nfloats, int &slot,
                        bool &captured, cudaStream_t st) {
  if (!sc || !sc->density || !sc->lut || !sc->nx || !sc->ny || !sc->nz || !views || !nviews ||
      nviews > kMaxBatchViews)
    return fail(c, R3D_E_INVALID, "diff: bad arguments");
  if ((uint64_t)sc->nx * sc->ny * sc->nz >= (1ull << 32))
    return fail(c, R3D_E_INVALID, "diff: grid too large for 32-bit voxel indices");
  g.dens = sc->density;
  g.n[0] = sc->nx;
  g.n[1] = sc->ny;
  g.n[2] = sc->nz;
  g.nmax = max(sc->nx, max(sc->ny, sc->nz));
  g.wide = g.nmax > (1u << 23) ? 1u : 0u;
  g.lut = sc->lut;
  g.cutoff = c->alpha_cutoff;
  const int k = c->ring_next;
  c->ring_next = (k + 1) % r3d_cuda_ctx::kRing;
  if (c->ring_used[k]) R3D_CUDA_TRY(c, cudaEventSynchronize(c->ring_ev[k]));
  static_assert(sizeof(DiffView) <= sizeof(DevView), "ring slot size");
  DiffView *hv = (DiffView *)(c->ring_host + (size_t)k * kMaxBatchViews);
  dviews = (DiffView *)(c->ring_dev + (size_t)k * kMaxBatchViews);
  nfloats = 0;
  uint64_t tiles = 0;
  for (uint32_t v = 0; v < nviews; v++) {
    const r3d_frame_params &p = views[v];
    if (!p.viewport[0] || !p.viewport[1] || p.viewport[0] > 16384u || p.viewport[1] > 16384u)
      return fail(c, R3D_E_INVALID, "diff: view %u needs an explicit viewport", v);
    if (p.brick_mode || p.slab_grid || p.clip_valid || p.overlay_flags ||
        (p.view_flags & ~R3D_VIEW_ORTHO))
      return fail(c, R3D_E_UNSUPPORTED, "diff: view %u uses a feature the differentiable "
                                        "render does not have", v);
    if (!(p.step_voxels > 0.0f)) return fail(c, R3D_E_INVALID, "diff: step_voxels");
    memset(&hv[v], 0, sizeof hv[v]);
    hv[v].pc = p;
    hv[v].out_off = nfloats;
    hv[v].tile_begin = (uint32_t)tiles;
    nfloats += (size_t)p.viewport[0] * p.viewport[1] * 3u;
    tiles += (uint64_t)((p.viewport[0] + 7u) / 8u) * ((p.viewport[1] + 3u) / 4u);
  }
  ntiles = (uint32_t)tiles;  // at most 64 views of 2048 x 4096 tiles: 2^29
  slot = k;
  const int rc = call_words(c, slot, g, captured, st);
  if (rc != R3D_OK) return rc;
  R3D_CUDA_TRY(c, cudaMemcpyAsync(dviews, hv, sizeof(DiffView) * nviews, cudaMemcpyHostToDevice,
                                  st));
  R3D_CUDA_TRY(c, cudaEventRecord(c->ring_ev[k], st));
  c->ring_used[k] = true;
  return R3D_OK;
}

// Fills g.quad: the context's quad grid, rebuilt from the density unless
// `reuse` and it was last built from this density buffer.
static int diff_quads(r3d_cuda_ctx *c, const r3d_cuda_diff_scene *sc, DiffGrid &g, bool reuse,
                      cudaStream_t st) {
  const size_t nvox = (size_t)sc->nx * sc->ny * sc->nz;
  const size_t need = nvox * sizeof(float4);
  if (c->diff_quad_bytes < need) {  // grow; earlier work on the old buffer must finish first
    R3D_CUDA_TRY(c, cudaDeviceSynchronize());
    cudaFree(c->diff_quad);
    c->diff_quad = nullptr;
    c->diff_quad_bytes = 0;
    c->quad_src = nullptr;
    R3D_CUDA_TRY(c, cudaMalloc(&c->diff_quad, need));
    c->diff_quad_bytes = need;
  }
  g.quad = (const float4 *)c->diff_quad;
  // the TF may change between calls that share the density
  k_diff_tf_clear<<<1, 256, 0, st>>>(sc->lut, g.zc);
  R3D_CUDA_TRY(c, cudaGetLastError());
  if (reuse && c->quad_src == sc->density) return R3D_OK;
  k_diff_quads<<<grid_blocks(nvox), 256, 0, st>>>(sc->density, sc->nx, sc->ny, sc->nz,
                                                  (float4 *)c->diff_quad);
  R3D_CUDA_TRY(c, cudaGetLastError());
  c->quad_src = sc->density;
  return R3D_OK;
}

// Identity of a tape: the views, the scene's buffers and sizes and the
// cutoff of the forward that wrote it.
static bool tape_matches(const r3d_cuda_ctx *c, const r3d_cuda_diff_scene *sc,
                         const r3d_frame_params *views, uint32_t nviews) {
  return c->tape_valid && c->tape_nviews == nviews && c->tape_density == sc->density &&
         c->tape_lut == sc->lut && c->tape_dims[0] == sc->nx && c->tape_dims[1] == sc->ny &&
         c->tape_dims[2] == sc->nz && c->tape_cutoff == c->alpha_cutoff &&
         memcmp(c->tape_views, views, sizeof(r3d_frame_params) * nviews) == 0;
}

static int diff_forward(r3d_cuda_ctx *c, const r3d_cuda_diff_scene *sc,
                        const r3d_frame_params *views, uint32_t nviews, float *rgb_out,
                        unsigned long long *total_steps, void *stream, bool tape) {
  if (!c || !rgb_out) return fail(c, R3D_E_INVALID, "diff_forward: bad arguments");
  cudaSetDevice(c->device);
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  if (!is_device_ptr(rgb_out)) return fail(c, R3D_E_INVALID, "diff_forward: rgb_out not device");
  DiffGrid g;
  DiffView *dv;
  uint32_t nt;
  size_t nf;
  int slot = 0;
  bool captured = false;
  int rc = diff_prepare(c, sc, views, nviews, g, dv, nt, nf, slot, captured, st);
  if (rc != R3D_OK) return rc;
  rc = diff_quads(c, sc, g, false, st);
  if (rc != R3D_OK) return rc;
  TapeEntry *tp = nullptr;
  uint32_t *tn = nullptr;
  if (tape) {
    const size_t rays = (size_t)nt * 32u;  // whole tiles
    c->tape_valid = false;
    if (c->tape_rays < rays) {  // grow; earlier work on the old buffers must finish first
      R3D_CUDA_TRY(c, cudaDeviceSynchronize());
      cudaFree(c->tape);
      cudaFree(c->tape_n);
      c->tape = nullptr;
      c->tape_n = nullptr;
      c->tape_rays = 0;
      R3D_CUDA_TRY(c, cudaMalloc(&c->tape, rays * kTape * sizeof(TapeEntry)));
      R3D_CUDA_TRY(c, cudaMalloc(&c->tape_n, rays * sizeof(uint32_t)));
      c->tape_rays = rays;
    }
    tp = (TapeEntry *)c->tape;
    tn = c->tape_n;
  }
  R3D_CUDA_TRY(c, cudaEventRecord(c->ev0, st));
  if (tape)
    k_diff_fwd<true><<<march_blocks(k_diff_fwd<true>, nt), 128, 0, st>>>(dv, nviews, nt, g, rgb_out,
                                                                         total_steps, tp, tn);
  else
    k_diff_fwd<false><<<march_blocks(k_diff_fwd<false>, nt), 128, 0, st>>>(
        dv, nviews, nt, g, rgb_out, total_steps, nullptr, nullptr);
  R3D_CUDA_TRY(c, cudaGetLastError());
  rc = call_marched(c, slot, captured, st);
  if (rc != R3D_OK) return rc;
  R3D_CUDA_TRY(c, cudaEventRecord(c->ev1, st));
  c->timed = true;
  if (tape) {
    memcpy(c->tape_views, views, sizeof(r3d_frame_params) * nviews);
    c->tape_nviews = nviews;
    c->tape_density = sc->density;
    c->tape_lut = sc->lut;
    c->tape_dims[0] = sc->nx;
    c->tape_dims[1] = sc->ny;
    c->tape_dims[2] = sc->nz;
    c->tape_cutoff = c->alpha_cutoff;
    c->tape_valid = true;
  }
  return R3D_OK;
}

extern "C" int r3d_cuda_diff_forward(r3d_cuda_ctx *c, const r3d_cuda_diff_scene *sc,
                                     const r3d_frame_params *views, uint32_t nviews,
                                     float *rgb_out, unsigned long long *total_steps,
                                     void *stream) {
  return diff_forward(c, sc, views, nviews, rgb_out, total_steps, stream, false);
}

extern "C" int r3d_cuda_diff_forward_tape(r3d_cuda_ctx *c, const r3d_cuda_diff_scene *sc,
                                          const r3d_frame_params *views, uint32_t nviews,
                                          float *rgb_out, unsigned long long *total_steps,
                                          void *stream) {
  return diff_forward(c, sc, views, nviews, rgb_out, total_steps, stream, true);
}

template <int K, bool DET>
static cudaError_t launch_bwd(uint32_t nviews, uint32_t nt, cudaStream_t st, const DiffView *dv, const DiffGrid &g,
                              const float *dl, float *gd, unsigned long long *qd, float *gl,
                              unsigned long long *ql, float *gs, unsigned long long *qs,
                              const TapeEntry *tp, const uint32_t *tn) {
  k_diff_bwd<K, DET><<<march_blocks(k_diff_bwd<K, DET>, nt), 128, 0, st>>>(
      dv, nviews, nt, g, dl, gd, qd, gl, ql, gs, qs, tp, tn);
  return cudaGetLastError();
}

extern "C" int r3d_cuda_raycast_bwd(r3d_cuda_ctx *c, const r3d_cuda_diff_scene *sc,
                                    const r3d_frame_params *views, uint32_t nviews,
                                    const float *dl_drgb, const r3d_cuda_grads *out,
                                    uint32_t ckpt_k, int deterministic, void *stream) {
  if (!c || !dl_drgb || !out || !out->density || !out->lut || !out->density_scale)
    return fail(c, R3D_E_INVALID, "raycast_bwd: bad arguments");
  if (ckpt_k != 32u && ckpt_k != 64u && ckpt_k != 128u)
    return fail(c, R3D_E_INVALID, "raycast_bwd: checkpoint interval %u not 32, 64 or 128",
                ckpt_k);
  if (deterministic & ~(int)(R3D_BWD_DETERMINISTIC | R3D_BWD_TAPE))
    return fail(c, R3D_E_INVALID, "raycast_bwd: unknown flags 0x%x", deterministic);
  const bool det = (deterministic & (int)R3D_BWD_DETERMINISTIC) != 0;
  cudaSetDevice(c->device);
  cudaStream_t st = stream ? (cudaStream_t)stream : c->stream;
  DiffGrid g;
  DiffView *dv;
  uint32_t nt;
  size_t nf;
  int slot = 0;
  bool captured = false;
  int rc = diff_prepare(c, sc, views, nviews, g, dv, nt, nf, slot, captured, st);
  if (rc != R3D_OK) return rc;
  const size_t nvox = (size_t)sc->nx * sc->ny * sc->nz;
  unsigned long long *qd = nullptr, *ql = nullptr, *qs = nullptr;
  if (det) {
    const size_t need = (nvox + 1024u + 1u) * sizeof(unsigned long long);
    if (c->diff_q_bytes < need) {
      cudaFree(c->diff_q);
      c->diff_q = nullptr;
      c->diff_q_bytes = 0;
      R3D_CUDA_TRY(c, cudaMalloc(&c->diff_q, need));
      c->diff_q_bytes = need;
    }
    qd = c->diff_q;
    ql = qd + nvox;
    qs = ql + 1024;
    R3D_CUDA_TRY(c, cudaMemsetAsync(c->diff_q, 0, need, st));
  } else {
    R3D_CUDA_TRY(c, cudaMemsetAsync(out->density, 0, nvox * sizeof(float), st));
    R3D_CUDA_TRY(c, cudaMemsetAsync(out->lut, 0, 1024 * sizeof(float), st));
    R3D_CUDA_TRY(c, cudaMemsetAsync(out->density_scale, 0, sizeof(float), st));
  }
  // the tape of the matching training forward, when asked for
  const bool use_tape = (deterministic & (int)R3D_BWD_TAPE) != 0;
  if (use_tape && !tape_matches(c, sc, views, nviews))
    return fail(c, R3D_E_STATE, "raycast_bwd: no tape of a training forward over these views "
                                "and this scene");
  const TapeEntry *tp = use_tape ? (const TapeEntry *)c->tape : nullptr;
  const uint32_t *tn = use_tape ? c->tape_n : nullptr;
  // the tape's forward built the quads from this (unchanged) density
  rc = diff_quads(c, sc, g, use_tape, st);
  if (rc != R3D_OK) return rc;
  R3D_CUDA_TRY(c, cudaEventRecord(c->ev0, st));
  cudaError_t e;
  float *gd = out->density, *gl = out->lut, *gs = out->density_scale;
  if (det) {
    e = ckpt_k == 32u ? launch_bwd<32, true>(nviews, nt, st, dv, g, dl_drgb, gd, qd, gl, ql, gs, qs, tp, tn)
        : ckpt_k == 64u ? launch_bwd<64, true>(nviews, nt, st, dv, g, dl_drgb, gd, qd, gl, ql, gs, qs, tp, tn)
                        : launch_bwd<128, true>(nviews, nt, st, dv, g, dl_drgb, gd, qd, gl, ql, gs, qs, tp, tn);
  } else {
    e = ckpt_k == 32u ? launch_bwd<32, false>(nviews, nt, st, dv, g, dl_drgb, gd, qd, gl, ql, gs, qs, tp, tn)
        : ckpt_k == 64u ? launch_bwd<64, false>(nviews, nt, st, dv, g, dl_drgb, gd, qd, gl, ql, gs, qs, tp, tn)
                        : launch_bwd<128, false>(nviews, nt, st, dv, g, dl_drgb, gd, qd, gl, ql, gs, qs, tp, tn);
  }
  if (e != cudaSuccess) return cuda_fail(c, e, "raycast_bwd: launch");
  rc = call_marched(c, slot, captured, st);
  if (rc != R3D_OK) return rc;
  if (det) {
    k_fix_to_float<<<grid_blocks(nvox), 256, 0, st>>>(qd, gd, nvox);
    k_fix_to_float<<<4, 256, 0, st>>>(ql, gl, 1024);
    k_fix_to_float<<<1, 32, 0, st>>>(qs, gs, 1);
    R3D_CUDA_TRY(c, cudaGetLastError());
  }
  R3D_CUDA_TRY(c, cudaEventRecord(c->ev1, st));
  c->timed = true;
  return R3D_OK;
}
