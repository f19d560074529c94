// Flattened-segment (surf) views: render3d's segment pane.  A segment is a
// grid of surface points (xyz + valid) and unit normals; the bake resamples
// the LOD brick cache into a W x H x L "flattened volume" over (u, v,
// layer): texel (x, y, l) holds the volume at surface(u, v) + normal(u, v) *
// (zoff0 + (l - nback) * lstep) (src/shaders/surfvol.comp), R = CT, G = an
// overlay atlas.  The surf raycast then marches each pixel's column of
// layers (src/shaders/raycast.slang:515-638): composite or MIP, gradient
// shading in flattened space, overlay tint, the flattening-distortion
// heatmap and the supervision-mask tint.  The reference bakes in row bands
// spread over frames and shifts the window in place on integer moves; here
// a bake covers the whole window in one launch on the context's stream.
#include <string.h>

#include "r3d_internal.h"

namespace r3d {

// GLSL mix(x, y, a) = x * (1 - a) + y * a
__device__ __forceinline__ float mixf(float x, float y, float a) {
  return fmaf(y, a, x * (1.0f - a));
}

struct SurfBake {
  const float4 *coords, *normals;  // gw x gh grids, row-major
  uint32_t gw, gh;
  float u0, v0, step, zoff0, sx, sy, lstep;
  uint32_t W, H, L, nback, lod;
  int ovl;       // overlay atlas baked into G, or -1
  uint8_t *vol;  // W x H x L texels of (R, G), x fastest
  const float *pred;  // live ink prediction, pw x ph, or null
  uint32_t pw, ph;
  float pg0u, pg0v, pppg;  // texel (0, 0) in grid coordinates; texels per grid unit
};

// The prediction texture, clamp-to-edge bilinear at texel-space position
// (px, py), sampled as textureLod(inkpred, (pp + 0.5) / size)
// (surfvol.comp:131-136).
__device__ __forceinline__ float pred_sample(const SurfBake &b, float px, float py) {
  const float u = (px + 0.5f) / (float)b.pw, v = (py + 0.5f) / (float)b.ph;
  const float tx = clamp_(fmaf(u, (float)b.pw, -0.5f), 0.0f, (float)(b.pw - 1u));
  const float ty = clamp_(fmaf(v, (float)b.ph, -0.5f), 0.0f, (float)(b.ph - 1u));
  const uint32_t x0 = (uint32_t)tx, y0 = (uint32_t)ty;
  const uint32_t x1 = min(x0 + 1u, b.pw - 1u), y1 = min(y0 + 1u, b.ph - 1u);
  const float fx = tx - (float)x0, fy = ty - (float)y0;
  const float *r0 = b.pred + (size_t)y0 * b.pw, *r1 = b.pred + (size_t)y1 * b.pw;
  return lerp_(lerp_(__ldg(r0 + x0), __ldg(r0 + x1), fx), lerp_(__ldg(r1 + x0), __ldg(r1 + x1), fx), fy);
}

// Per-column brick cache of the bake (surfvol.comp:40-52): the cached brick
// by its float origin lo = 128 * brick in its level's voxels (no brick: lo =
// +inf, which no position reaches; see lod_cache_hit) and its scale.
struct ColCache {
  float inv_scale, lo[3];
  uint32_t slot;
};

// The brick under a base-level position bv: at the column's level, else the
// next two coarser levels, else the coarsest (surfvol.comp:66-96).
__device__ __forceinline__ void surf_locate(const DevScene &s, uint32_t lod, const float (&bv)[3],
                                            ColCache &c) {
  const DevBricks &br = s.br;
  const int desired = (int)min(lod, br.nlev - 1u), last = (int)br.nlev - 1;
  c.lo[0] = c.lo[1] = c.lo[2] = R3D_FM_INF;
#pragma unroll 1
  for (int stp = 0; stp < 4; stp++) {
    const int li = stp < 3 ? desired + stp : last;
    if (li > last || (stp == 3 && li <= desired + 2)) continue;
    uint32_t bc[3];
#pragma unroll
    for (int a = 0; a < 3; a++)
      bc[a] = min((uint32_t)(bv[a] * br.inv_scale[li]) >> 7, br.bd[li][a] - 1u);
    const uint32_t e =
        page_entry(s, br.off[li] + (bc[2] * br.bd[li][1] + bc[1]) * br.bd[li][0] + bc[0]);
    if (e == 0xFFFFFFFFu) continue;
    if ((e & 0xFFFFFFu) >= br.nslots) {
      atomicOr(s.status, R3D_STATUS_PAGE_RANGE);
      continue;
    }
    c.inv_scale = br.inv_scale[li];
    c.slot = e & 0xFFFFFFu;
#pragma unroll
    for (int a = 0; a < 3; a++) c.lo[a] = (float)(bc[a] << 7);
    break;
  }
}

// One thread per (u, v) column (surfvol.comp:98-153); OVL: an overlay atlas
// or the live prediction goes into G.
//
// Bound by issue (a texel costs about 60 instructions; 2 bytes written and 8
// read of it).  The column keeps its brick as the raycast does (origin and
// reciprocal scale, both exact; no division or conversion while it stays in
// the brick), a texel is stored as one 16-bit word, and a warp covers 16 x 2
// columns so that its stores fill whole sectors.  1536^2 x 80 texels at a
// pitch of half a voxel: 0.69 -> 0.42 ms (450 G texels/s).
template <bool OVL>
__global__ void __launch_bounds__(128) k_surf_bake(const __grid_constant__ DevScene s,
                                                   const __grid_constant__ SurfBake b) {
  const uint32_t x = blockIdx.x * 16u + (threadIdx.x & 15u), y = blockIdx.y * 8u + (threadIdx.x >> 4);
  if (x >= b.W || y >= b.H) return;
  const float fu = fmaf((float)x + 0.5f, b.step, b.u0), fv = fmaf((float)y + 0.5f, b.step, b.v0);
  const float gx = fu * b.sx, gy = fv * b.sy;  // grid coordinates
  bool ok = false;
  float3 wp0 = make_float3(0.0f, 0.0f, 0.0f), nrm = wp0;
  if (gx >= 0.0f && gy >= 0.0f && gx <= (float)(b.gw - 1u) && gy <= (float)(b.gh - 1u)) {
    const uint32_t ix = min((uint32_t)gx, b.gw - 2u), iy = min((uint32_t)gy, b.gh - 2u);
    const float fx = gx - (float)ix, fy = gy - (float)iy;
    const size_t i00 = (size_t)iy * b.gw + ix;
    const float4 c00 = b.coords[i00], c10 = b.coords[i00 + 1], c01 = b.coords[i00 + b.gw],
                 c11 = b.coords[i00 + b.gw + 1];
    if (fminf(fminf(c00.w, c10.w), fminf(c01.w, c11.w)) >= 0.5f) {
      wp0 = make_float3(mixf(mixf(c00.x, c10.x, fx), mixf(c01.x, c11.x, fx), fy),
                        mixf(mixf(c00.y, c10.y, fx), mixf(c01.y, c11.y, fx), fy),
                        mixf(mixf(c00.z, c10.z, fx), mixf(c01.z, c11.z, fx), fy));
      const float4 n00 = b.normals[i00], n10 = b.normals[i00 + 1], n01 = b.normals[i00 + b.gw],
                   n11 = b.normals[i00 + b.gw + 1];
      nrm = make_float3(mixf(mixf(n00.x, n10.x, fx), mixf(n01.x, n11.x, fx), fy),
                        mixf(mixf(n00.y, n10.y, fx), mixf(n01.y, n11.y, fx), fy),
                        mixf(mixf(n00.z, n10.z, fx), mixf(n01.z, n11.z, fx), fy));
      const float nl = sqrtf(dot3(nrm, nrm));
      if (nl > 1e-4f) {
        nrm = make_float3(nrm.x / nl, nrm.y / nl, nrm.z / nl);
        ok = true;
      }
    }
  }
  // one prediction per column, painted over every layer (surfvol.comp:127-150)
  float pred = -1.0f;
  if (OVL && b.pred) {
    const float px = (gx - b.pg0u) * b.pppg, py = (gy - b.pg0v) * b.pppg;
    if (px >= 0.0f && py >= 0.0f && px < (float)b.pw && py < (float)b.ph) pred = pred_sample(b, px, py);
  }
  const uint32_t pred8 = pred >= 0.0f ? unorm8(pred) : 0u;
  uint16_t *o = reinterpret_cast<uint16_t *>(b.vol) + (size_t)y * b.W + x;
  const size_t plane = (size_t)b.W * b.H;
  ColCache c = {1.0f, {R3D_FM_INF, R3D_FM_INF, R3D_FM_INF}, 0u};
  float zf = -(float)b.nback;  // (float)z - (float)nback: whole numbers, exact
#pragma unroll 1
  for (uint32_t z = 0; z < b.L; z++, zf += 1.0f, o += plane) {
    uint32_t v = 0u, g = 0u;
    if (ok) {
      const float k = fmaf(zf, b.lstep, b.zoff0);
      const float3 wp = make_float3(fmaf(nrm.x, k, wp0.x), fmaf(nrm.y, k, wp0.y), fmaf(nrm.z, k, wp0.z));
      if (wp.x >= 0.0f && wp.y >= 0.0f && wp.z >= 0.0f && wp.x < s.br.bs[0] && wp.y < s.br.bs[1] &&
          wp.z < s.br.bs[2]) {
        const float bv[3] = {fminf(wp.x, s.br.bs_hi[0]), fminf(wp.y, s.br.bs_hi[1]),
                             fminf(wp.z, s.br.bs_hi[2])};
        float bl[3];
        bool in = true;
#pragma unroll
        for (int a = 0; a < 3; a++) {
          bl[a] = bv[a] * c.inv_scale - c.lo[a];
          in = in && bl[a] >= 0.0f && bl[a] < 128.0f;
        }
        if (!in) {
          surf_locate(s, b.lod, bv, c);
          in = c.lo[0] < R3D_FM_INF;
#pragma unroll
          for (int a = 0; a < 3; a++) bl[a] = bv[a] * c.inv_scale - c.lo[a];
        }
        if (in) {
          const SlotCoord q = slot_coord(make_float3(bl[0], bl[1], bl[2]));
          v = unorm8(slot_sample(s, c.slot, q));
          if (OVL && b.ovl >= 0) g = unorm8(ovl_fetch(s, b.ovl, c.slot, q));
        }
      }
    }
    if (OVL && pred >= 0.0f) g = pred8;
    *o = (uint16_t)(v | (g << 8));
  }
}

struct DevSurfView {
  const uint8_t *vol;  // W x H x L (R, G) texels
  uint32_t W, H, L;
  const float4 *coords;  // segment grid (heatmap taps)
  uint32_t gw, gh;
  const uint8_t *mask;  // supervision mask, or null
  uint32_t mw, mh;
  float ix, iy, iz;  // 1 / W, 1 / H, 1 / L as the view's parameters give them
};

// Clamp-to-edge trilinear of the (R, G) volume at normalized uvw.
__device__ __forceinline__ float2 surf_tex(const DevSurfView &v, float u, float w_, float t) {
  const float tx = clamp_(fmaf(u, (float)v.W, -0.5f), 0.0f, (float)(v.W - 1u));
  const float ty = clamp_(fmaf(w_, (float)v.H, -0.5f), 0.0f, (float)(v.H - 1u));
  const float tz = clamp_(fmaf(t, (float)v.L, -0.5f), 0.0f, (float)(v.L - 1u));
  const uint32_t x0 = (uint32_t)tx, y0 = (uint32_t)ty, z0 = (uint32_t)tz;
  const float fx = tx - (float)x0, fy = ty - (float)y0, fz = tz - (float)z0;
  const uint32_t x1 = min(x0 + 1u, v.W - 1u), y1 = min(y0 + 1u, v.H - 1u), z1 = min(z0 + 1u, v.L - 1u);
  const uchar2 *g = reinterpret_cast<const uchar2 *>(v.vol);
  const size_t sy = v.W, sz = (size_t)v.W * v.H;
  const uchar2 a00 = __ldg(g + z0 * sz + y0 * sy + x0), a10 = __ldg(g + z0 * sz + y0 * sy + x1);
  const uchar2 a01 = __ldg(g + z0 * sz + y1 * sy + x0), a11 = __ldg(g + z0 * sz + y1 * sy + x1);
  const uchar2 b00 = __ldg(g + z1 * sz + y0 * sy + x0), b10 = __ldg(g + z1 * sz + y0 * sy + x1);
  const uchar2 b01 = __ldg(g + z1 * sz + y1 * sy + x0), b11 = __ldg(g + z1 * sz + y1 * sy + x1);
  const float r = lerp_(lerp_(lerp_(a00.x, a10.x, fx), lerp_(a01.x, a11.x, fx), fy),
                        lerp_(lerp_(b00.x, b10.x, fx), lerp_(b01.x, b11.x, fx), fy), fz);
  const float gch = lerp_(lerp_(lerp_(a00.y, a10.y, fx), lerp_(a01.y, a11.y, fx), fy),
                          lerp_(lerp_(b00.y, b10.y, fx), lerp_(b01.y, b11.y, fx), fy), fz);
  return make_float2(r * kInv255, gch * kInv255);
}

// flat_overlay_color (raycast.slang:76-81)
__device__ __forceinline__ float3 flat_overlay_color(uint32_t f) {
  if (f & 16u) return make_float3(1.0f, 0.25f, 1.0f);
  if (f & 2u) return make_float3(0.25f, 1.0f, 0.55f);
  if (f & 4u) return make_float3(1.0f, 0.30f, 0.22f);
  return ((f >> 8) & 0xffu) == 1u ? make_float3(0.3f, 0.72f, 1.0f) : make_float3(0.25f, 1.0f, 0.55f);
}

// One axis of surf_tex: base texel, step to its clamped neighbour, fraction.
struct SurfAxis {
  uint32_t i0, d;
  float f;
};
__device__ __forceinline__ SurfAxis surf_axis(float u, uint32_t n) {
  SurfAxis a;
  a.i0 = floor_frac(clamp_(fmaf(u, (float)n, -0.5f), 0.0f, (float)(n - 1u)), a.f);
  a.d = a.i0 + 1u < n ? 1u : 0u;
  return a;
}

// The four texels of a column at one layer.
struct SurfTexels {
  uint32_t a, b, c, d;
};
__device__ __forceinline__ SurfTexels surf_texels(const uint16_t *__restrict__ vol, size_t plane,
                                                  uint32_t W, uint32_t l, const SurfAxis &x,
                                                  const SurfAxis &y) {
  const uint16_t *r0 = vol + l * plane + (size_t)y.i0 * W + x.i0, *r1 = r0 + (y.d ? W : 0u);
  return {__ldg(r0), __ldg(r0 + x.d), __ldg(r1), __ldg(r1 + x.d)};
}

// The (x, y) lerps of surf_tex at one layer: a column's value there, in
// 0..255 space (R; with OVL also G).
template <bool G>
__device__ __forceinline__ float2 surf_lerp(const SurfTexels &t, const SurfAxis &x, const SurfAxis &y) {
  float2 v;
  v.x = lerp_(lerp_raw(qraw(t.a, 0), qraw(t.b, 0), x.f), lerp_raw(qraw(t.c, 0), qraw(t.d, 0), x.f), y.f);
  v.y = G ? lerp_(lerp_raw(qraw(t.a, 1), qraw(t.b, 1), x.f), lerp_raw(qraw(t.c, 1), qraw(t.d, 1), x.f), y.f)
          : 0.0f;
  return v;
}
template <bool G>
__device__ __forceinline__ float2 surf_layer(const uint16_t *__restrict__ vol, size_t plane,
                                             uint32_t W, uint32_t l, const SurfAxis &x,
                                             const SurfAxis &y) {
  return surf_lerp<G>(surf_texels(vol, plane, W, l, x, y), x, y);
}

enum SurfKind { kSurfFull = 0, kSurfFlat = 1, kSurfMip = 2, kSurfStretch = 3 };

// One pixel of the surf branch of the raycast (raycast.slang:515-638): where
// it lies on the segment, and its ray along the layers.
struct SurfRay {
  float fu, fv;  // segment coordinates
  float tx, ty;  // window texels
  float t, hi, dt, center, lo;
};

// False: background.
__device__ __forceinline__ bool surf_begin(const r3d_frame_params &pc, uint32_t px, uint32_t py,
                                           SurfRay &r) {
  const float ux = ((float)px + 0.5f) / (float)pc.viewport[0];
  const float uy = ((float)py + 0.5f) / (float)pc.viewport[1];
  const float nx = ux * 2.0f - 1.0f, ny = 1.0f - uy * 2.0f;
  r.fu = fmaf(ny, pc.cam_up[0], fmaf(nx, pc.cam_right[0], pc.cam_origin[0]));
  r.fv = fmaf(ny, pc.cam_up[1], fmaf(nx, pc.cam_right[1], pc.cam_origin[1]));
  r.tx = (r.fu - pc.slab_x0) / pc.slab_px;
  r.ty = (r.fv - pc.slab_y0) / pc.slab_px;
  if (r.tx < 0.0f || r.ty < 0.0f || r.tx >= pc.slab_nx || r.ty >= pc.slab_ny) return false;
  const float L = (float)pc.slab_wz;
  r.center = (pc.slab_z0 - pc.max_mip) + (float)(pc.slab_grid & 0xffffu);
  const float halfd = 0.5f * fmaxf((float)pc.slab_depth, 1.0f);
  r.lo = clamp_(r.center - halfd, 0.0f, L);
  r.hi = clamp_(r.center + halfd, 0.0f, L);
  if (r.lo >= r.hi) return false;
  r.dt = fmaxf(pc.step_voxels, 0.25f);  // layers per step
  r.t = fmaf(hash12(px, py, pc.frame_index), r.dt, r.lo);
  return true;
}

// The flattening-distortion heatmap (:540-570).
__device__ __forceinline__ float3 surf_stretch(const r3d_frame_params &pc, const DevSurfView &v,
                                               const SurfRay &r) {
  const float ix = v.ix, iy = v.iy, iz = v.iz;
  const float gx = r.fu * pc.vol_tx, gy = r.fv * pc.vol_ty;
  const int gix = (int)clamp_(gx, 1.0f, (float)v.gw - 2.0f);
  const int giy = (int)clamp_(gy, 1.0f, (float)v.gh - 2.0f);
  const float4 cu0 = v.coords[(size_t)giy * v.gw + gix - 1], cu1 = v.coords[(size_t)giy * v.gw + gix + 1];
  const float4 cv0 = v.coords[(size_t)(giy - 1) * v.gw + gix], cv1 = v.coords[(size_t)(giy + 1) * v.gw + gix];
  if (fminf(fminf(cu0.w, cu1.w), fminf(cv0.w, cv1.w)) < 0.5f) return make_float3(0.02f, 0.02f, 0.03f);
  const float3 du = make_float3(cu1.x - cu0.x, cu1.y - cu0.y, cu1.z - cu0.z);
  const float3 dv = make_float3(cv1.x - cv0.x, cv1.y - cv0.y, cv1.z - cv0.z);
  const float su = sqrtf(dot3(du, du)) * 0.5f * pc.vol_tx;
  const float sv = sqrtf(dot3(dv, dv)) * 0.5f * pc.vol_ty;
  const float x = clamp_(r3d_log2f(fmaxf(0.5f * (su + sv), 1e-4f)) / 0.35f, -1.0f, 1.0f);
  const float m = r3d_powf(fabsf(x), 0.6f);
  const float3 tint = x < 0.0f ? make_float3(0.0f, 0.35f, 1.0f) : make_float3(1.0f, 0.15f, 0.0f);
  const float ct = surf_tex(v, r.tx * ix, r.ty * iy, clamp_(r.center, r.lo, r.hi) * iz).x;
  const float k = fmaf(0.5f, ct, 0.5f);
  return make_float3(lerp_(0.95f, tint.x, m) * k, lerp_(0.95f, tint.y, m) * k,
                     lerp_(0.95f, tint.z, m) * k);
}

// The supervision mask over a pixel's colour, nearest (:619-635).
__device__ __forceinline__ float3 surf_mask(const r3d_frame_params &pc, const DevSurfView &v,
                                            const SurfRay &r, float3 col) {
  if (!(pc.overlay_flags & 32u) || !v.mask) return col;
  const float gx = r.fu * pc.vol_tx, gy = r.fv * pc.vol_ty;
  const float upx = (float)v.mw / fmaxf((float)v.gw - 1.0f, 1.0f);
  const float upy = (float)v.mh / fmaxf((float)v.gh - 1.0f, 1.0f);
  const float mxf = gx * upx, myf = gy * upy;
  // int(g * up) truncates toward zero, so (-1, 0) lands on texel 0
  if (mxf > -1.0f && myf > -1.0f && mxf < (float)v.mw && myf < (float)v.mh) {
    const int mx = (int)mxf, my = (int)myf;
    const uint32_t mc = v.mask[(size_t)my * v.mw + mx];
    if (mc == 1u)
      col = make_float3(lerp_(col.x, 0.25f, 0.45f), lerp_(col.y, 0.45f, 0.45f), lerp_(col.z, 1.0f, 0.45f));
    else if (mc >= 2u)
      col = make_float3(lerp_(col.x, 1.0f, 0.55f), lerp_(col.y, 0.55f, 0.55f), lerp_(col.z, 0.10f, 0.55f));
  }
  return col;
}

// The column of a ray, layer by layer.  The ray runs along the layers at
// fixed (u, v), and a trilinear sample lerps x, then y, then z: so the (x, y)
// lerps of a layer are shared by every sample between it and its neighbours.
// The column's values at the two layers of the sample are kept and shifted
// as the ray passes a layer, and its texels at the layer after those are
// loaded one layer ahead of use.
template <bool G>
struct SurfColumn {
  SurfAxis x, y;
  uint32_t have = 0xffffffffu;  // the lower layer held
  float2 e0, e1;
  SurfTexels ahead;
  __device__ __forceinline__ void move(const uint16_t *__restrict__ vol, size_t plane, uint32_t W,
                                       uint32_t L, const SurfAxis &z) {
    if (z.i0 == have) return;
    const bool next = z.i0 == have + 1u && have != 0xffffffffu;
    e0 = next ? e1 : surf_layer<G>(vol, plane, W, z.i0, x, y);
    if (!next) ahead = surf_texels(vol, plane, W, z.i0 + z.d, x, y);
    e1 = surf_lerp<G>(ahead, x, y);  // (the last layer: e0 again)
    have = z.i0;
    ahead = surf_texels(vol, plane, W, min(have + 2u, L - 1u), x, y);
  }
};

// The shading queue of a warp (see ShadeQueue): per entry the sample's z, TF
// coordinate, weight and ink, then its colour and weight.
struct SurfQueue {
  float4 a[64];
  uint8_t ray[64];
  uint32_t own[32];
};

// R of the texels at p[x], as 2^23 + byte
__device__ __forceinline__ float surf_raw(const uint16_t *__restrict__ p, int x) {
  return qraw(__ldg(p + x), 0);
}

// The cross of a sample at one layer, away from the volume's edges: the
// values of its column and of the columns one texel along x and y, from the
// twelve texels that they read between them (20 column by column).
struct SurfCross {
  float c, xp, xm, yp, ym;
};
struct SurfFrac {  // fractions of the sample and of its taps
  float x, xp, xm, y, yp, ym;
};
__device__ __forceinline__ SurfCross surf_cross(const uint16_t *__restrict__ p, int W,
                                                const SurfFrac &f) {
  const uint16_t *r1 = p + W, *rm = p - W, *r2 = r1 + W;
  const float a0 = surf_raw(p, -1), b0 = surf_raw(p, 0), c0 = surf_raw(p, 1), d0 = surf_raw(p, 2);
  const float a1 = surf_raw(r1, -1), b1 = surf_raw(r1, 0), c1 = surf_raw(r1, 1), d1 = surf_raw(r1, 2);
  const float bm = surf_raw(rm, 0), cm = surf_raw(rm, 1), b2 = surf_raw(r2, 0), c2 = surf_raw(r2, 1);
  const float x0 = lerp_raw(b0, c0, f.x), x1 = lerp_raw(b1, c1, f.x);
  SurfCross s;
  s.c = lerp_(x0, x1, f.y);
  s.xp = lerp_(lerp_raw(c0, d0, f.xp), lerp_raw(c1, d1, f.xp), f.y);
  s.xm = lerp_(lerp_raw(a0, b0, f.xm), lerp_raw(a1, b1, f.xm), f.y);
  s.yp = lerp_(x1, lerp_raw(b2, c2, f.x), f.yp);
  s.ym = lerp_(lerp_raw(bm, cm, f.x), x0, f.ym);
  return s;
}

// Colour of the contributing sample at (u, w, z): TF colour, shading by
// 1-texel taps in flattened space, ink tint.  A tap is a trilinear lookup;
// the four in-plane ones share the sample's layers and fraction along them,
// the two along the layers its column.
template <bool OVL>
__device__ __forceinline__ float3 surf_shade(const r3d_frame_params &pc, const DevSurfView &v,
                                             const float4 *tf, float u, float w, float z, float tt,
                                             float ink) {
  const float ix = v.ix, iy = v.iy, iz = v.iz;
  const uint16_t *vol = reinterpret_cast<const uint16_t *>(v.vol);
  const size_t plane = (size_t)v.W * v.H;
  const SurfAxis x = surf_axis(u, v.W), y = surf_axis(w, v.H), c = surf_axis(z, v.L);
  const SurfAxis zp = surf_axis(z + iz, v.L), zm = surf_axis(z - iz, v.L);
  const auto at = [&](uint32_t l, const SurfAxis &ax, const SurfAxis &ay) {
    return surf_layer<false>(vol, plane, v.W, l, ax, ay).x;
  };
  const auto tap = [&](const SurfAxis &ax, const SurfAxis &ay, const SurfAxis &az) {
    return lerp_(at(az.i0, ax, ay), at(az.i0 + az.d, ax, ay), az.f) * kInv255;
  };
  const SurfAxis xp = surf_axis(u + ix, v.W), xm = surf_axis(u - ix, v.W);
  const SurfAxis yp = surf_axis(w + iy, v.H), ym = surf_axis(w - iy, v.H);
  float g0, g1, g2;
  // every tap exactly one texel off, none clamped at an edge (a tap's own
  // rounding can put it in the sample's texel, or two off)
  if (x.i0 - 1u < v.W - 3u && y.i0 - 1u < v.H - 3u && c.i0 - 1u < v.L - 3u && v.W > 3u &&
      v.H > 3u && v.L > 3u && xp.i0 == x.i0 + 1u && xm.i0 + 1u == x.i0 && yp.i0 == y.i0 + 1u &&
      ym.i0 + 1u == y.i0 && zp.i0 == c.i0 + 1u && zm.i0 + 1u == c.i0) {
    const uint16_t *p = vol + c.i0 * plane + (size_t)y.i0 * v.W + x.i0;
    const SurfFrac f = {x.f, xp.f, xm.f, y.f, yp.f, ym.f};
    const SurfCross s0 = surf_cross(p, (int)v.W, f), s1 = surf_cross(p + plane, (int)v.W, f);
    const auto column = [&](const uint16_t *q) {
      const uint16_t *q1 = q + v.W;
      return lerp_(lerp_raw(surf_raw(q, 0), surf_raw(q, 1), f.x),
                   lerp_raw(surf_raw(q1, 0), surf_raw(q1, 1), f.x), f.y);
    };
    g0 = lerp_(s0.xp, s1.xp, c.f) * kInv255 - lerp_(s0.xm, s1.xm, c.f) * kInv255;
    g1 = lerp_(s0.yp, s1.yp, c.f) * kInv255 - lerp_(s0.ym, s1.ym, c.f) * kInv255;
    g2 = lerp_(s1.c, column(p + 2u * plane), zp.f) * kInv255 -
         lerp_(column(p - plane), s0.c, zm.f) * kInv255;
  } else {
    g0 = tap(xp, y, c) - tap(xm, y, c);
    g1 = tap(x, yp, c) - tap(x, ym, c);
    g2 = tap(x, y, zp) - tap(x, y, zm);
  }
  const float4 sm = tf_sample(tf, tt);
  float cr = sm.x, cg = sm.y, cb = sm.z;
  const float gm = sqrtf(fmaf(g2, g2, fmaf(g1, g1, g0 * g0)));
  if (gm > 1e-4f) {
    const float diff = fmaf(0.7f, fabsf(g2 / gm), 0.3f);  // headlight along the layers
    const float lit = fmaf(0.75f, diff, 0.25f);
    const float lm = lerp_(1.0f, lit, sat_(gm * 6.0f));
    cr *= lm, cg *= lm, cb *= lm;
  }
  if (OVL) {
    const float3 oc = flat_overlay_color(pc.overlay_flags);
    const float kk = sat_(ink * pc.overlay_gain);
    cr = lerp_(cr, oc.x, kk), cg = lerp_(cg, oc.y, kk), cb = lerp_(cb, oc.z, kk);
  }
  return make_float3(cr, cg, cb);
}

// A warp's 32 pixels (`inside` says whether the lane has one).
template <int KIND, bool OVL>
__device__ __forceinline__ float3 surf_pixel(const r3d_frame_params &pc, const DevSurfView &v,
                                             const float4 *tf, float alpha_cutoff, float tf_zero_t,
                                             uint32_t px, uint32_t py, bool inside, SurfQueue &sq) {
  constexpr uint32_t kAll = 0xffffffffu;
  const float3 bg = make_float3(0.02f, 0.02f, 0.03f);
  SurfRay r;
  const bool hit = inside && surf_begin(pc, px, py, r);
  if (KIND == kSurfStretch) return hit ? surf_stretch(pc, v, r) : bg;
  constexpr bool composite = KIND != kSurfMip, queued = KIND == kSurfFull;
  const uint32_t lane = threadIdx.x & 31u, below = (1u << lane) - 1u;
  const float iz = v.iz;
  const float u = hit ? r.tx * v.ix : 0.0f, w = hit ? r.ty * v.iy : 0.0f;
  const float3 oc = flat_overlay_color(pc.overlay_flags);
  const float opac_k = pc.density * pc.step_voxels;
  const uint16_t *vol = reinterpret_cast<const uint16_t *>(v.vol);
  const size_t plane = (size_t)v.W * v.H;
  SurfColumn<OVL> col;
  col.x = surf_axis(u, v.W);
  col.y = surf_axis(w, v.H);
  float mip_max = 0.0f, ink_max = 0.0f;
  float acc_r = 0.0f, acc_g = 0.0f, acc_b = 0.0f, acc_a = 0.0f;
  float t = hit ? r.t : 0.0f;
  const float hi = hit ? r.hi : 0.0f;
  uint32_t head = 0, n = 0;  // the queue's waiting entries: [head, head + n), mod 64
  const auto shade = [&](uint32_t k) {
    const uint32_t e = (head + lane) & 63u;
    const float4 A = sq.a[e];
    const uint32_t ray = sq.ray[e] & 31u;
    const float ru = __shfl_sync(kAll, u, ray), rw = __shfl_sync(kAll, w, ray);
    if (lane < k) {
      const float3 c = surf_shade<OVL>(pc, v, tf, ru, rw, A.x, A.y, A.w);
      sq.a[e] = make_float4(c.x, c.y, c.z, A.z);
    }
    shade_fold(sq.a, sq.own, head, k, ray, acc_r, acc_g, acc_b);
    head += k;
    n -= k;
  };
  bool active = hit;
  uint32_t k = 0;
  while (queued ? __any_sync(kAll, active) : active) {
    bool push = false;
    float z = 0.0f, tt = 0.0f, wgt = 0.0f, ink = 0.0f;
    if (active && !(k < 512u && t < hi)) active = false;
    if (active) {
      z = t * iz;
      const SurfAxis cz = surf_axis(z, v.L);
      col.move(vol, plane, v.W, v.L, cz);
      const float val = lerp_(col.e0.x, col.e1.x, cz.f) * kInv255;
      ink = OVL ? lerp_(col.e0.y, col.e1.y, cz.f) * kInv255 : 0.0f;
      if (OVL && ink > ink_max) ink_max = ink;
      if (!(val < pc.threshold)) {
        if (!composite && val > mip_max) mip_max = val;
        tt = clamp_(fmaf(val, 256.0f, -0.5f), 0.0f, 255.0f);
        // below tf_zero_t both TF texels have alpha 0: the opacity is 1 - 1^k = 0
        if (composite && !(tt < tf_zero_t)) {
          const float4 sm = tf_sample(tf, tt);
          const float a = 1.0f - r3d_powf(1.0f - sm.w, opac_k);
          if (a > 0.003f) {
            wgt = (1.0f - acc_a) * a;
            if (!queued) {
              float cr = sm.x, cg = sm.y, cb = sm.z;
              if (OVL) {
                const float kk = sat_(ink * pc.overlay_gain);
                cr = lerp_(cr, oc.x, kk), cg = lerp_(cg, oc.y, kk), cb = lerp_(cb, oc.z, kk);
              }
              acc_r = fmaf(wgt, cr, acc_r);
              acc_g = fmaf(wgt, cg, acc_g);
              acc_b = fmaf(wgt, cb, acc_b);
            }
            push = true;
            acc_a = acc_a + wgt;
            if (acc_a >= alpha_cutoff) active = false;
          }
        }
      }
      k++;
      t += r.dt;
    }
    if (queued) {
      const uint32_t add = __ballot_sync(kAll, push);
      if (add) {
        if (push) {
          const uint32_t e = (head + n + (uint32_t)__popc(add & below)) & 63u;
          sq.a[e] = make_float4(z, tt, wgt, ink);
          sq.ray[e] = (uint8_t)lane;
        }
        n += (uint32_t)__popc(add);
        __syncwarp();
        if (n >= 32u) shade(32u);
      }
    }
  }
  if (queued && n) shade(n);  // at most 31 are left
  if (!hit) return bg;
  float3 c;
  if (composite) {
    const float tr = 1.0f - acc_a;
    c = make_float3(fmaf(tr, bg.x, acc_r), fmaf(tr, bg.y, acc_g), fmaf(tr, bg.z, acc_b));
  } else {
    const float m = mip_max * pc.density;
    c = make_float3(m, m, m);
    if (OVL) {
      const float kk = sat_(ink_max * pc.overlay_gain);
      c = make_float3(lerp_(c.x, oc.x, kk), lerp_(c.y, oc.y, kk), lerp_(c.z, oc.z, kk));
    }
  }
  return surf_mask(pc, v, r, c);
}

// One thread per pixel, 8x4 Morton warp tiles.  Bound by issue: at 1600x900
// over a 1536^2 x 80 window, FULL, 1.45 ms with eight texels per sample and
// tap, 0.88 ms with the column's layers kept, 0.83 ms with the next layer's
// texels loaded ahead, 0.68 ms with the taps through the warp's queue and
// their texels shared (0.83 with the queue alone; FLAT, without taps: 0.33).
template <int KIND, bool OVL>
__global__ void __launch_bounds__(128) k_surf_raycast(const __grid_constant__ r3d_frame_params pc,
                                                      const __grid_constant__ DevSurfView v,
                                                      const uchar4 *__restrict__ lut,
                                                      float alpha_cutoff, float tf_zero_t,
                                                      uchar4 *__restrict__ img, uint32_t out_w,
                                                      uint32_t *__restrict__ steps_out,
                                                      uint32_t *__restrict__ mip_out) {
  __shared__ float4 tf[256];
  __shared__ SurfQueue sq[KIND == kSurfFull ? 4 : 1];
  for (uint32_t i = threadIdx.x; i < 256u; i += blockDim.x) {
    const uchar4 u = lut[i];
    tf[i] = make_float4((float)u.x, (float)u.y, (float)u.z, (float)u.w);
  }
  __syncthreads();
  const bool half = (pc.view_flags & R3D_VIEW_HALF) != 0u;
  const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
  const uint32_t tx = blockIdx.x * 16u + (warp & 1u) * 8u +
                      ((lane & 1u) | ((lane >> 1) & 2u) | ((lane >> 2) & 4u));
  const uint32_t ty = blockIdx.y * 8u + (warp >> 1) * 4u + (((lane >> 1) & 1u) | ((lane >> 2) & 2u));
  const uint32_t px = half ? tx * 2u : tx, py = half ? ty * 2u : ty;
  const uint32_t vw = pc.viewport[0], vh = pc.viewport[1];
  const bool inside = px < vw && py < vh;
  const float3 c = surf_pixel<KIND, OVL>(pc, v, tf, alpha_cutoff, tf_zero_t, px, py, inside,
                                         sq[KIND == kSurfFull ? warp : 0u]);
  if (!inside) return;
  const uchar4 col = make_uchar4(unorm8(c.x), unorm8(c.y), unorm8(c.z), 255);
  const uint32_t ox = pc.view_org & 0xffffu, oy = pc.view_org >> 16;
  for (uint32_t k = 0; k < (half ? 4u : 1u); k++) {
    const uint32_t ax = px + (k & 1u), ay = py + (k >> 1);
    if (ax >= vw || ay >= vh) continue;
    const size_t i = (size_t)(oy + ay) * out_w + (ox + ax);
    img[i] = col;
    if (steps_out) steps_out[i] = 0u;  // no ray-march step counts in this view
    if (mip_out) mip_out[i] = 0u;
  }
}

cudaError_t launch_surf(const r3d_cuda_ctx *c, const r3d_frame_params &pc, uint8_t *img,
                        uint32_t out_w, uint32_t *steps, uint32_t *mip, cudaStream_t st) {
  DevSurfView v;
  v.vol = c->sv_vol;
  v.W = c->sv_W, v.H = c->sv_H, v.L = c->sv_L;
  v.coords = c->surf_coords;
  v.gw = c->surf_gw, v.gh = c->surf_gh;
  v.mask = c->surf_mask;
  v.mw = c->surf_mw, v.mh = c->surf_mh;
  v.ix = 1.0f / pc.slab_nx, v.iy = 1.0f / pc.slab_ny, v.iz = 1.0f / (float)pc.slab_wz;
  const bool half = (pc.view_flags & R3D_VIEW_HALF) != 0u;
  const uint32_t gw = half ? (pc.viewport[0] + 1u) / 2u : pc.viewport[0];
  const uint32_t gh = half ? (pc.viewport[1] + 1u) / 2u : pc.viewport[1];
  const dim3 grid((gw + 15u) / 16u, (gh + 7u) / 8u);
  const bool ovl = (pc.overlay_flags & 1u) != 0u;
#define R3D_SURF(K, O)                                                                           \
  k_surf_raycast<K, O><<<grid, 128, 0, st>>>(pc, v, c->lut, c->alpha_cutoff, c->tf_zero_t,        \
                                             (uchar4 *)img, out_w, steps, mip)
  if (pc.view_flags & R3D_VIEW_STRETCH)
    R3D_SURF(kSurfStretch, false);
  else if (pc.mode == R3D_MODE_MIP)
    ovl ? R3D_SURF(kSurfMip, true) : R3D_SURF(kSurfMip, false);
  else if (pc.mode == R3D_MODE_FULL)
    ovl ? R3D_SURF(kSurfFull, true) : R3D_SURF(kSurfFull, false);
  else
    ovl ? R3D_SURF(kSurfFlat, true) : R3D_SURF(kSurfFlat, false);
#undef R3D_SURF
  return cudaGetLastError();
}

}  // namespace r3d

using namespace r3d;

void surf_reset(r3d_cuda_ctx *c) {
  cudaFree(c->surf_coords);
  cudaFree(c->surf_normals);
  cudaFree(c->sv_vol);
  cudaFree(c->surf_mask);
  cudaFree(c->sv_pred);
  c->sv_pred = nullptr;
  c->sv_pw = c->sv_ph = 0;
  c->surf_coords = c->surf_normals = nullptr;
  c->sv_vol = nullptr;
  c->surf_mask = nullptr;
  c->surf_gw = c->surf_gh = c->surf_mw = c->surf_mh = 0;
  c->sv_W = c->sv_H = c->sv_L = 0;
  c->sv_step = 0.0f;
  c->sv_baked = false;
}

static int surf_bake(r3d_cuda_ctx *c) {
  if (!c->sv_vol || c->sv_step <= 0.0f) return R3D_OK;
  if (!c->have_bricks)
    return fail(c, R3D_E_STATE, "surfvol: the bake samples the LOD brick cache");
  if (c->sv_ovl >= 0 && !c->ovl_quad[c->sv_ovl])
    return fail(c, R3D_E_STATE, "surfvol: overlay atlas %d is not loaded", c->sv_ovl);
  SurfBake b;
  b.coords = c->surf_coords;
  b.normals = c->surf_normals;
  b.gw = c->surf_gw, b.gh = c->surf_gh;
  b.u0 = c->sv_u0, b.v0 = c->sv_v0, b.step = c->sv_step, b.zoff0 = c->sv_zoff0;
  b.sx = c->sv_sx, b.sy = c->sv_sy, b.lstep = 1.0f;  // depth stays native-res (vkbackend.c:7026)
  b.W = c->sv_W, b.H = c->sv_H, b.L = c->sv_L, b.nback = c->sv_nback;
  // level of the xy pitch: one per halving down to a 2-voxel step (:7013-7014)
  uint32_t lodq = 0;
  for (float s = c->sv_step; s >= 2.0f && lodq + 1u < c->br.nlev; s *= 0.5f) lodq++;
  b.lod = lodq;
  b.ovl = c->sv_ovl;
  b.vol = c->sv_vol;
  b.pred = c->sv_pred;
  b.pw = c->sv_pw, b.ph = c->sv_ph;
  b.pg0u = c->sv_pg0u, b.pg0v = c->sv_pg0v, b.pppg = c->sv_pppg;
  const dim3 grid((b.W + 15u) / 16u, (b.H + 7u) / 8u);
  if (b.ovl >= 0 || b.pred)
    k_surf_bake<true><<<grid, 128, 0, c->stream>>>(c->scene(), b);
  else
    k_surf_bake<false><<<grid, 128, 0, c->stream>>>(c->scene(), b);
  R3D_CUDA_TRY(c, cudaGetLastError());
  c->sv_baked = true;
  return R3D_OK;
}

extern "C" {

int r3d_cuda_surf_begin(r3d_cuda_ctx *c, uint32_t w, uint32_t h, const float *coords_rgba,
                        const float *normals_rgba) {
  if (!c || w < 3u || h < 3u || !coords_rgba || !normals_rgba)
    return fail(c, R3D_E_INVALID, "surf_begin: a grid of at least 3 x 3 points and both grids");
  cudaSetDevice(c->device);
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  const size_t bytes = (size_t)w * h * sizeof(float4);
  float4 *cd = nullptr, *nd = nullptr;
  cudaError_t e = cudaMalloc(&cd, bytes);
  if (e == cudaSuccess) e = cudaMalloc(&nd, bytes);
  if (e == cudaSuccess) e = copy_sync(c->stream, cd, coords_rgba, bytes);
  if (e == cudaSuccess) e = copy_sync(c->stream, nd, normals_rgba, bytes);
  if (e != cudaSuccess) {
    cudaFree(cd);
    cudaFree(nd);
    return cuda_fail(c, e, "surf_begin");
  }
  cudaFree(c->surf_coords);
  cudaFree(c->surf_normals);
  c->surf_coords = cd;
  c->surf_normals = nd;
  c->surf_gw = w, c->surf_gh = h;
  return surf_bake(c);  // a window already set re-bakes from the new grids
}

int r3d_cuda_surfvol_begin(r3d_cuda_ctx *c, uint32_t w, uint32_t h, uint32_t layers,
                           uint32_t nback, float sx, float sy) {
  if (!c || !w || !h || !layers || !(sx > 0.0f) || !(sy > 0.0f))
    return fail(c, R3D_E_INVALID, "surfvol_begin: bad arguments");
  if (!c->surf_coords) return fail(c, R3D_E_STATE, "surfvol_begin: no surface grids");
  if (w > 16384u || h > 16384u || layers > 2048u)
    return fail(c, R3D_E_INVALID, "surfvol_begin: %ux%ux%u window too large", w, h, layers);
  if (nback >= layers) nback = layers / 2u;  // vkbackend.c:1765
  cudaSetDevice(c->device);
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  cudaFree(c->sv_vol);
  c->sv_vol = nullptr;
  const size_t bytes = (size_t)w * h * layers * 2u;
  R3D_CUDA_TRY(c, cudaMalloc(&c->sv_vol, bytes));
  R3D_CUDA_TRY(c, cudaMemsetAsync(c->sv_vol, 0, bytes, c->stream));
  c->sv_W = w, c->sv_H = h, c->sv_L = layers, c->sv_nback = nback;
  c->sv_sx = sx, c->sv_sy = sy;
  c->sv_step = 0.0f;  // no window yet
  c->sv_baked = false;
  return R3D_OK;
}

int r3d_cuda_surfvol_window(r3d_cuda_ctx *c, double u0, double v0, float step, float zoff0) {
  if (!c) return R3D_E_INVALID;
  if (!c->sv_vol) return fail(c, R3D_E_STATE, "surfvol_window: no surface volume");
  if (!(step > 0.0f)) return fail(c, R3D_E_INVALID, "surfvol_window: step must be > 0");
  cudaSetDevice(c->device);
  c->sv_u0 = (float)u0, c->sv_v0 = (float)v0, c->sv_step = step, c->sv_zoff0 = zoff0;
  return surf_bake(c);
}

int r3d_cuda_surfvol_overlay(r3d_cuda_ctx *c, int atlas) {
  if (!c || atlas < -1 || atlas > 3 || atlas == 2)
    return fail(c, R3D_E_INVALID, "surfvol_overlay: atlas %d (ink 0, 3D ink 1, registration 3, "
                                  "none -1)", atlas);
  cudaSetDevice(c->device);
  c->sv_ovl = atlas;
  return surf_bake(c);
}

int r3d_cuda_surfvol_inkpred(r3d_cuda_ctx *c, const float *pred, uint32_t w, uint32_t h, float g0u,
                             float g0v, float px_per_grid) {
  if (!c) return R3D_E_INVALID;
  if (!c->sv_vol) return fail(c, R3D_E_STATE, "surfvol_inkpred: no surface volume");
  cudaSetDevice(c->device);
  if (!pred) {  // clear (vkbackend.c:1963-1968): re-bake without it
    if (!c->sv_pred) return R3D_OK;
    R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
    cudaFree(c->sv_pred);
    c->sv_pred = nullptr;
    c->sv_pw = c->sv_ph = 0;
    return surf_bake(c);
  }
  if (!w || !h || !(px_per_grid > 0.0f))
    return fail(c, R3D_E_INVALID, "surfvol_inkpred: a %ux%u prediction at %g texels per grid unit",
                w, h, (double)px_per_grid);
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  const size_t bytes = (size_t)w * h * sizeof(float);
  if (c->sv_pw != w || c->sv_ph != h) {  // size change: a new buffer
    cudaFree(c->sv_pred);
    c->sv_pred = nullptr;
    c->sv_pw = c->sv_ph = 0;
    R3D_CUDA_TRY(c, cudaMalloc(&c->sv_pred, bytes));
  }
  R3D_CUDA_TRY(c, copy_sync(c->stream, c->sv_pred, pred, bytes));
  c->sv_pw = w, c->sv_ph = h;
  c->sv_pg0u = g0u, c->sv_pg0v = g0v, c->sv_pppg = px_per_grid;
  return surf_bake(c);  // repaint the window with the new probabilities
}

int r3d_cuda_surfvol_mark(r3d_cuda_ctx *c) {
  if (!c) return R3D_E_INVALID;
  cudaSetDevice(c->device);
  return surf_bake(c);
}

void r3d_cuda_surfvol_params(const r3d_cuda_ctx *c, r3d_frame_params *p) {
  if (!c || !p || !c->sv_vol) return;
  // vkbackend.c:2054-2066
  p->slab_x0 = c->sv_u0;
  p->slab_y0 = c->sv_v0;
  p->slab_px = c->sv_step;
  p->slab_nx = (float)c->sv_W;
  p->slab_ny = (float)c->sv_H;
  p->slab_wz = c->sv_L;
  p->slab_grid = c->sv_nback;
  p->max_mip = c->sv_zoff0;
  p->vol_tx = c->sv_sx;
  p->vol_ty = c->sv_sy;
  p->view_flags |= R3D_VIEW_SURF;
}

int r3d_cuda_surfvol_read(r3d_cuda_ctx *c, uint8_t *out) {
  if (!c || !out) return R3D_E_INVALID;
  if (!c->sv_vol) return fail(c, R3D_E_STATE, "surfvol_read: no surface volume");
  cudaSetDevice(c->device);
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  R3D_CUDA_TRY(c, cudaMemcpy(out, c->sv_vol, (size_t)c->sv_W * c->sv_H * c->sv_L * 2u,
                             cudaMemcpyDeviceToHost));
  return R3D_OK;
}

int r3d_cuda_surfmask(r3d_cuda_ctx *c, const uint8_t *m, uint32_t w, uint32_t h) {
  if (!c) return R3D_E_INVALID;
  cudaSetDevice(c->device);
  R3D_CUDA_TRY(c, cudaStreamSynchronize(c->stream));
  cudaFree(c->surf_mask);
  c->surf_mask = nullptr;
  c->surf_mw = c->surf_mh = 0;
  if (!m || !w || !h) return R3D_OK;  // cleared
  R3D_CUDA_TRY(c, cudaMalloc(&c->surf_mask, (size_t)w * h));
  R3D_CUDA_TRY(c, copy_sync(c->stream, c->surf_mask, m, (size_t)w * h));
  c->surf_mw = w, c->surf_mh = h;
  return R3D_OK;
}

}  // extern "C"
