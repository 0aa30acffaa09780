// shade.cuh — the shading policies of the four renderers and the shared
// primary-ray loop (ShadeSample and main() of each reference shader).
// Included by march.cu (the marchers) and surrogate.cu (training targets and
// the surrogate-shaded marcher reuse the ground-truth light rays).
#pragma once

#include <algorithm>

#include <cuda_fp16.h>

#include "march.cuh"
#include "sampler.cuh"

namespace cvr {

// Iteration bounds of the secondary loops.  Validated parameters stay far
// below them (a cone walk has at most 0.75*diagonal/interval boxes, a light
// ray distance/step samples); they only stop a loop whose position stopped
// advancing from spinning forever.
constexpr int kMaxConeBoxes = 1 << 16;
constexpr int kMaxLightSteps = 1 << 20;

// ============================================= gradient Blinn-Phong terms
// texture(TexVolumeGradient, Tpos / VolumeGridSize).xyz: GL_LINEAR,
// clamp-to-edge on the voxel grid (the texture copy when there is one).
__device__ __forceinline__ float3 sample_gradient(const GradView& g, float3 p) {
  if (g.tex) {
    const float4 r = tex3D<float4>(g.tex, p.x * g.inv_grid.x, p.y * g.inv_grid.y, p.z * g.inv_grid.z);
    return f3(r.x, r.y, r.z);
  }
  const Tap a = axis_tap(fmaf(p.x, g.inv_spacing.x, -0.5f), g.nx);
  const Tap b = axis_tap(fmaf(p.y, g.inv_spacing.y, -0.5f), g.ny);
  const Tap c = axis_tap(fmaf(p.z, g.inv_spacing.z, -0.5f), g.nz);
  const size_t sy = (size_t)g.nx, sz = (size_t)g.nx * g.ny;
  auto at = [&](int x, int y, int z) {
    const uint2 q = __ldg(g.g + (size_t)x + sy * y + sz * z);
    const float2 xy = __half22float2(*reinterpret_cast<const __half2*>(&q.x));
    return f3(xy.x, xy.y, __low2float(*reinterpret_cast<const __half2*>(&q.y)));
  };
  auto lerp = [](float t, float3 u, float3 v) {
    return f3(fmaf(t, v.x - u.x, u.x), fmaf(t, v.y - u.y, u.y), fmaf(t, v.z - u.z, u.z));
  };
  const float3 c00 = lerp(a.t, at(a.i0, b.i0, c.i0), at(a.i1, b.i0, c.i0));
  const float3 c10 = lerp(a.t, at(a.i0, b.i1, c.i0), at(a.i1, b.i1, c.i0));
  const float3 c01 = lerp(a.t, at(a.i0, b.i0, c.i1), at(a.i1, b.i0, c.i1));
  const float3 c11 = lerp(a.t, at(a.i0, b.i1, c.i1), at(a.i1, b.i1, c.i1));
  return lerp(c.t, lerp(b.t, c00, c10), lerp(b.t, c01, c11));
}

// The terms every gradient branch shares (ray_marching_1p.comp:50-70 and its
// copies in the other shaders): false when the interpolated gradient is the
// zero vector, where the sample keeps its unshaded colour.
struct BlinnTerms {
  float diff;  // max(0, dot(N, L))
  float spec;  // pow(max(0, dot(H, N)), shininess)
};
__device__ __forceinline__ bool blinn_terms(const FrameArgs& f, float3 tx, BlinnTerms& t) {
  float3 n = sample_gradient(f.grad, tx);
  if (n.x == 0.0f && n.y == 0.0f && n.z == 0.0f) return false;
  n = normalize3(n);
  const float3 w = tx - f.vol.grid * 0.5f;
  const float3 l = normalize3(f.grad.light_pos - w);
  const float3 e = normalize3(f.cam.eye - w);
  const float3 hv = normalize3(e + l);
  t.diff = fmaxf(0.0f, dot3(n, l));
  // pow(x, N) = exp2(N log2 x) on the special-function unit (relative error
  // ~1e-6 for N = 30; 0 at x = 0 as GLSL's pow gives for N > 0)
  t.spec = __powf(fmaxf(0.0f, dot3(hv, n)), f.grad.shininess);
  return true;
}

// ShadeBlinnPhong (ray_marching_1p.comp:48-81):
// clr * (Ka + Kd * diff) + Ispecular * Ks * spec.
__device__ __forceinline__ float4 phong_plain(const FrameArgs& f, float4 L, float3 tx) {
  BlinnTerms t;
  if (!blinn_terms(f, tx, t)) return L;
  const float m = f.grad.ka + f.grad.kd * t.diff;
  const float s = f.grad.ks * t.spec;
  L.x = L.x * m + f.grad.ispec.x * s;
  L.y = L.y * m + f.grad.ispec.y * s;
  L.z = L.z * m + f.grad.ispec.z * s;
  return L;
}

// Extinction / light cache (ebs_ray_bbox_marching.comp:524-546,
// obj_ray_marching.comp:111-129):
// (1/(ka+kd)) * (L*Io*ka + Is*(L*kd*diff)) + Is*(ks*Ispecular*spec).
__device__ __forceinline__ float4 phong_ext(const FrameArgs& f, float4 L, float3 tx, float io, float ka, float is,
                                            float kd) {
  BlinnTerms t;
  if (!blinn_terms(f, tx, t)) return L;
  const float kk = 1.0f / (ka + kd);
  const float s = is * (f.grad.ks * t.spec);
  L.x = kk * (L.x * io * ka + is * (L.x * kd * t.diff)) + s * f.grad.ispec.x;
  L.y = kk * (L.y * io * ka + is * (L.y * kd * t.diff)) + s * f.grad.ispec.y;
  L.z = kk * (L.z * io * ka + is * (L.z * kd * t.diff)) + s * f.grad.ispec.z;
  return L;
}

// Cone and ground truth (ray_bbox_marching.comp:630-648, gt_ray_marching.comp:
// 277-295, whose specular colour is 1): L * ((1/(ka+kd)) * (Io*ka + Is*kd*diff))
// + Ispecular * (Is*ks*spec).
__device__ __forceinline__ float4 phong_cone(const FrameArgs& f, float4 L, float3 tx, float io, float ka, float is,
                                             float kd) {
  BlinnTerms t;
  if (!blinn_terms(f, tx, t)) return L;
  const float m = (1.0f / (ka + kd)) * (io * ka + is * kd * t.diff);
  const float s = is * f.grad.ks * t.spec;
  L.x = L.x * m + f.grad.ispec.x * s;
  L.y = L.y * m + f.grad.ispec.y * s;
  L.z = L.z * m + f.grad.ispec.z * s;
  return L;
}

// The weights of ShadeSample's occlusion and shadow terms and the colour of a
// sample from its (occlusion, shadow); EXT: the extinction renderer's gradient
// branch, else the cone's and the ground truth's.
struct LightTerms {
  float ka, kd;
  template <bool EXT>
  __device__ __forceinline__ float4 apply(const FrameArgs& f, float4 src, float3 tx, float2 l) const {
    if (f.grad.g) return EXT ? phong_ext(f, src, tx, l.x, ka, l.y, kd) : phong_cone(f, src, tx, l.x, ka, l.y, kd);
    const float k = 1.0f / (ka + kd);
    src.x = k * (src.x * l.x * ka + src.x * l.y * kd);
    src.y = k * (src.y * l.x * ka + src.y * l.y * kd);
    src.z = k * (src.z * l.x * ka + src.z * l.y * kd);
    return src;
  }
};
__host__ __device__ __forceinline__ LightTerms light_terms(int occ, int sdw, float ka, float kd) {
  return LightTerms{occ ? ka : 0.0f, sdw ? kd : 0.0f};
}

// ============================================================ plain (rc1pass)
struct PlainShade {
  __device__ __forceinline__ bool shades() const { return true; }
  struct Ray {};
  __device__ __forceinline__ void begin(Ray&, float3) const {}
  // ShadeSample is the identity unless gradient shading is on
  // (ApplyGradientPhongShading, ray_marching_1p.comp:143-145).
  __device__ __forceinline__ float4 shade(float4 src, float3 tx, const Ray&, const FrameArgs& f, unsigned&) const {
    return f.grad.g ? phong_plain(f, src, tx) : src;
  }
};

// ====================================================== extinction (rc1pextbsd)
// COMPACT: the frame's SAT box queries read the 32-bit table (SatView::sat32).
// ALIGNED: every AO box and every box of the directional shadow table has
// integer texel widths, so every query is the equal-fraction one
// (sat_box_aligned, sat_box_aligned64); the kernel then always has a table
// (ttx set).  ExtBoxShade below reads the same frames from box tables.

// SAT texel coordinate of a texture-space position: (tx + spacing) / spacing - 0.5.
__device__ __forceinline__ float3 sat_texel(const SatView& S, float3 tx) {
  return f3(fmaf(tx.x, S.inv_spacing.x, 0.5f), fmaf(tx.y, S.inv_spacing.y, 0.5f), fmaf(tx.z, S.inv_spacing.z, 0.5f));
}
// Texels between consecutive boxes of an aligned walk: the packed widths' one
// along the axis (the sample interval), with the walk's sign.
__device__ __forceinline__ int walk_step(int widths, int axis, float interval) {
  const int w = (widths >> (10 * axis)) & 1023;
  return interval < 0.0f ? -w : w;
}

// Cell and fraction of a directional walk's boxes along its axis: the boxes'
// low corners are a whole number of texels (dw) apart, so the first box's
// serve them all.
struct WalkStart {
  int cell;
  float frac;
};

// ExtinctionAmbientOcclusion from the box tables; g: the sample's SAT texel coordinate.
__device__ __forceinline__ float box_occlusion(const ExtArgs& e, float3 g) {
  const BoxView& B = e.box;
  float t = 0.0f, last = 0.0f;
  for (int i = 0; i < e.n_shells; ++i) {
    const float r = e.radii[i];
    const BoxGrid& G = B.ao_grid[i];
    const int pad = __float2int_rn(2.0f * r) + 1;
    float3 q;
    const unsigned x = min((unsigned)(cell_of(g.x - r, q.x) + pad), (unsigned)G.na - 1u);
    const unsigned y = min((unsigned)(cell_of(g.y - r, q.y) + pad), (unsigned)G.nb - 1u);
    const unsigned z = min((unsigned)(cell_of(g.z - r, q.z) + pad), (unsigned)G.nc - 1u);
    const BoxCorners c = box_corners(B.ao, B.ao_cell[i] + x + y * (unsigned)G.row + z * G.nab, G.row, G.nab);
    const float b = aligned_weigh(c.v00.x, c.v00.y, c.v01.x, c.v01.y, c.v10.x, c.v10.y, c.v11.x, c.v11.y, q);
    t = i == 0 ? b * (1.0f / (r * r)) : t + (b - last) * (1.0f / (r * r));
    last = b;
  }
  const float rk = e.radii[e.n_shells - 1];
  return expf(-((1.0f / (rk * rk)) * t));
}

template <bool COMPACT = false, bool ALIGNED = false>
struct ExtShadeT {
  const ExtArgs* e;
  // Per-frame box table of a directional light (shared memory), or nullptr.
  const float4* tlo = nullptr;
  const float4* thi = nullptr;
  // the table's texel offsets and packed integer widths (compact table only), or nullptr
  const float4* ttx = nullptr;
  int tn = 0, tax = 0;
  float tiw = 0.0f, tvmin = 0.0f, tvmax = 0.0f;
  struct Ray {};
  __device__ __forceinline__ void begin(Ray&, float3) const {}

  // EvaluateAmbientOcclusionSAT3D (ebs_ray_bbox_marching.comp:102-110).
  __device__ __forceinline__ float ao_box(float3 p1, float3 p2, const FrameArgs& f) const {
    const SatView& S = e->sat;
    p1 = clamp3(p1 + f.vol.spacing, S.min_pos, S.max_pos);
    p2 = clamp3(p2 + f.vol.spacing, S.min_pos, S.max_pos);
    return sat_box<COMPACT>(S, p1, p2);
  }

  static __device__ __forceinline__ float aligned_box(const SatView& S, int3 a, float3 t, int wx, int wy, int wz) {
    if constexpr (COMPACT) return sat_box_aligned(S, a, t, wx, wy, wz);
    else return sat_box_aligned64(S, a, t, wx, wy, wz);
  }

  // ExtinctionAmbientOcclusion (ebs_ray_bbox_marching.comp:112-146), with the
  // shell radii taken from a list (reference: AmbOccRadius * (i + 1)).
  __device__ float ambient_occlusion(float3 tx, const FrameArgs& f) const {
    if (ALIGNED || e->ao_aligned) {
      const float3 g = sat_texel(e->sat, tx);
      if (!ALIGNED && e->box.ao) return box_occlusion(*e, g);
      // the box [tx - r, tx + r] (voxels) starts at texel coordinate
      // (tx + spacing) / spacing - 0.5 - r = g - r and is 2 r texels wide
      const SatView& S = e->sat;
      float t = 0.0f, sat_i = 0.0f;
      for (int i = 0; i < e->n_shells; ++i) {
        const float ri = e->radii[i];
        const int wi = __float2int_rn(2.0f * ri);
        float3 q;
        const int3 a = make_int3(cell_of(g.x - ri, q.x), cell_of(g.y - ri, q.y), cell_of(g.z - ri, q.z));
        const float sat_n = aligned_box(S, a, q, wi, wi, wi);
        t = i == 0 ? sat_n * (1.0f / (ri * ri)) : t + (sat_n - sat_i) * (1.0f / (ri * ri));
        sat_i = sat_n;
      }
      const float rk = e->radii[e->n_shells - 1];
      return expf(-((1.0f / (rk * rk)) * t));
    }
    float3 sc = f.vol.spacing;
    float r0 = e->radii[0];
    float sat0 = ao_box(tx - sc * r0, tx + sc * r0, f);
    float t = sat0 * (1.0f / (r0 * r0));
    float sat_i = sat0;
    for (int i = 1; i < e->n_shells; ++i) {
      float ri = e->radii[i];
      float sat_n = ao_box(tx - sc * ri, tx + sc * ri, f);
      t = t + (sat_n - sat_i) * (1.0f / (ri * ri));
      sat_i = sat_n;
    }
    float rk = e->radii[e->n_shells - 1];
    float wa = 1.0f / (rk * rk);
    return expf(-(wa * t));
  }

  // EvaluateShadowSAT3D, texture() branch (ebs_ray_bbox_marching.comp:173-187).
  __device__ __forceinline__ float shadow_box(float3 p1, float3 p2, const FrameArgs& f) const {
    float3 sc = f.vol.spacing;
    float volq = (fabsf(p1.x - p2.x) / sc.x) * (fabsf(p1.y - p2.y) / sc.y) * (fabsf(p1.z - p2.z) / sc.z);
    const SatView& S = e->sat;
    p1 = clamp3(p1 + sc, S.min_pos, S.max_pos);
    p2 = clamp3(p2 + sc, S.min_pos, S.max_pos);
    return (sat_box<COMPACT>(S, p1, p2) / volq) * e->ui_weight;
  }

  // ConeZAxis / ConeYAxis / ConeXAxis (ebs_ray_bbox_marching.comp:190-430):
  // the walk of a cone c along its dominant axis.  The cone's edges in the
  // planes of the walk axis m and a lateral axis are straight lines through
  // the sample, so their slopes are formed once and a box's lateral extent is
  // [lo, hi] times its depth, rounded up to whole voxels about its middle.
  // With a whole interval every width is whole: the equal-fraction query, the
  // walk axis stepping whole cells.  Products that meet a sum are fused or
  // rounded explicitly, so that every kernel that inlines this rounds alike.
  template <int AXIS>
  __device__ float cone_walk(float3 pos, float3 c, const FrameArgs& f, unsigned& aux) const {
    const SatView& S = e->sat;
    const float3 sc = f.vol.spacing;
    auto pick = [](float3 v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); };
    constexpr int A = AXIS == 0 ? 1 : 0, B = AXIS == 2 ? 1 : 2;
    const float cm = pick(c, AXIS), scm = pick(sc, AXIS), pm = pick(pos, AXIS);
    // edge slopes in texels of the lateral axis per world unit of depth
    float lo[2], hi[2];
#pragma unroll
    for (int l = 0; l < 2; ++l) {
      const float ca = pick(c, l == 0 ? A : B), inv = pick(S.inv_spacing, l == 0 ? A : B);
      const float as = __fmul_rn(ca, e->cone_sin), ms = __fmul_rn(cm, e->cone_sin);
      const float s1 = fmaf(ca, e->cone_cos, ms) / fabsf(fmaf(cm, e->cone_cos, -as));
      const float s2 = fmaf(ca, e->cone_cos, -ms) / fabsf(fmaf(cm, e->cone_cos, as));
      lo[l] = fminf(s1, s2) * inv;
      hi[l] = fmaxf(s1, s2) * inv;
    }
    const float signal = cm < 0.0f ? -1.0f : 1.0f;
    const float interval = e->interval * signal * scm;
    float mp = e->initial * signal * scm;
    const float vmin = scm * 0.5f, vmax = pick(f.vol.grid, AXIS) - scm * 0.5f;
    const float inv_c = 1.0f / cm;
    const float3 g = sat_texel(S, pos);
    float tw;
    int aw = cell_of(fmaf(fminf(mp, mp + interval), pick(S.inv_spacing, AXIS), pick(g, AXIS)), tw);
    const int ww = __float2int_rn(e->interval), dw = cm < 0.0f ? -ww : ww;
    float st = 0.0f;
    for (int guard = 0; guard < kMaxConeBoxes && mp * inv_c < e->max_dist &&
                        (pm + (mp + interval) > vmin && pm + (mp + interval) < vmax); ++guard) {
      const float zm = fabsf(mp + interval * 0.5f);
      // widths rounded up (ceil by a round-up add), low corners about the middle
      float w[2], u[2];
#pragma unroll
      for (int l = 0; l < 2; ++l) {
        const float a = __fmul_rn(lo[l], zm), b = __fmul_rn(hi[l], zm);
        w[l] = __fadd_ru(b - a, 12582912.0f) - 12582912.0f;
        u[l] = 0.5f * ((a + b) - w[l]);
      }
      if (e->whole_interval) {
        float ta, tb;
        const int ia = cell_of(pick(g, A) + u[0], ta), ib = cell_of(pick(g, B) + u[1], tb);
        const int wa = __float2int_rn(w[0]), wb = __float2int_rn(w[1]);
        int3 at, wd;
        float3 q;
        if constexpr (AXIS == 2) { at = make_int3(ia, ib, aw); wd = make_int3(wa, wb, ww); q = f3(ta, tb, tw); }
        else if constexpr (AXIS == 1) { at = make_int3(ia, aw, ib); wd = make_int3(wa, ww, wb); q = f3(ta, tw, tb); }
        else { at = make_int3(aw, ia, ib); wd = make_int3(ww, wa, wb); q = f3(tw, ta, tb); }
        st = fmaf(aligned_box(S, at, q, wd.x, wd.y, wd.z) / (w[0] * w[1] * e->interval), e->ui_weight, st);
      } else {
        const float a0 = u[0] * pick(sc, A), b0 = u[1] * pick(sc, B);
        const float a1 = a0 + w[0] * pick(sc, A), b1 = b0 + w[1] * pick(sc, B);
        const float m0 = fminf(mp, mp + interval), m1 = fmaxf(mp, mp + interval);
        if constexpr (AXIS == 2) st += shadow_box(pos + f3(a0, b0, m0), pos + f3(a1, b1, m1), f);
        else if constexpr (AXIS == 1) st += shadow_box(pos + f3(a0, m0, b0), pos + f3(a1, m1, b1), f);
        else st += shadow_box(pos + f3(m0, a0, b0), pos + f3(m1, a1, b1), f);
      }
      ++aux;
      mp = mp + interval;
      aw += dw;
    }
    return st;
  }

  // The Cone*Axis walk over the precomputed boxes of a directional light:
  // same boxes, same CUT_WHEN_AWAY_FROM_VOLUME test, same sum.
  __device__ float shadow_table(float3 tx, const FrameArgs& f, unsigned& aux) const {
    const SatView& S = e->sat;
    const float3 sc = f.vol.spacing;
    const float pm = tax == 0 ? tx.x : (tax == 1 ? tx.y : tx.z);
    float st = 0.0f;
    if constexpr (ALIGNED) {
      // every box has integer widths: the equal-fraction query
      if (tn == 0) return 1.0f;
      const float3 g = sat_texel(S, tx);
      const float4 o0 = ttx[0];
      WalkStart ws;
      ws.cell = cell_of(tax == 0 ? g.x + o0.x : (tax == 1 ? g.y + o0.y : g.z + o0.z), ws.frac);
      const int dw = walk_step(__float_as_int(o0.w), tax, tiw);
      for (int k = 0; k < tn; ++k) {
        const float nxt = pm + (tlo[k].w + tiw);
        if (!(nxt > tvmin && nxt < tvmax)) break;
        const float4 o = ttx[k];
        const int w = __float_as_int(o.w);
        float3 q;
        int3 a = make_int3(cell_of(g.x + o.x, q.x), cell_of(g.y + o.y, q.y), cell_of(g.z + o.z, q.z));
        const int aw = ws.cell + k * dw;
        if (tax == 0) { a.x = aw; q.x = ws.frac; }
        else if (tax == 1) { a.y = aw; q.y = ws.frac; }
        else { a.z = aw; q.z = ws.frac; }
        float b;
        if (COMPACT && e->walk.oct) b = sat_box_walk(S, e->walk, a, q, w & 1023, (w >> 10) & 1023, w >> 20);
        else b = aligned_box(S, a, q, w & 1023, (w >> 10) & 1023, w >> 20);
        st = fmaf(b, thi[k].w, st);
        ++aux;
      }
      return expf(-st);
    }
    for (int k = 0; k < tn; ++k) {
      const float4 lo = tlo[k];
      const float nxt = pm + (lo.w + tiw);
      if (!(nxt > tvmin && nxt < tvmax)) break;
      const float4 hi = thi[k];
      float3 p1 = clamp3(tx + f3(lo.x, lo.y, lo.z) + sc, S.min_pos, S.max_pos);
      float3 p2 = clamp3(tx + f3(hi.x, hi.y, hi.z) + sc, S.min_pos, S.max_pos);
      st = fmaf(sat_box<COMPACT>(S, p1, p2), hi.w, st);
      ++aux;
    }
    return expf(-st);
  }

  // ExtinctionDirectionalShadows (ebs_ray_bbox_marching.comp:432-456).
  __device__ float shadow(float3 tx, const FrameArgs& f, unsigned& aux) const {
    float3 realpos = tx - f.vol.grid * 0.5f;
    float3 c = (e->shadow_type == 0) ? normalize3(e->light_pos - realpos) : normalize3(e->light_fwd);
    float3 a = abs3(c);
    float st;
    if (a.z > a.x && a.z > a.y) st = cone_walk<2>(tx, c, f, aux);
    else if (a.y > a.x) st = cone_walk<1>(tx, c, f, aux);
    else st = cone_walk<0>(tx, c, f, aux);
    return expf(-st);
  }

  // ShadeSample (ebs_ray_bbox_marching.comp:500-551): the light terms, and
  // the colour from them.
  __device__ __forceinline__ float2 light(float3 tx, const Ray&, const FrameArgs& f, unsigned& aux) const {
    float io = 0.0f, is = 0.0f;
    if (e->apply_occ) { io = ambient_occlusion(tx, f); aux += e->n_shells; }
    if (e->apply_sdw) {
      if constexpr (ALIGNED) is = shadow_table(tx, f, aux);
      else is = tlo ? shadow_table(tx, f, aux) : shadow(tx, f, aux);
    }
    return make_float2(io, is);
  }
  __device__ __forceinline__ float4 shade(float4 src, float3 tx, const Ray& r, const FrameArgs& f, unsigned& aux) const {
    return light_terms(e->apply_occ, e->apply_sdw, e->ka, e->kd).apply<true>(f, src, tx, light(tx, r, f, aux));
  }
};
using ExtShade = ExtShadeT<false>;

// Extinction shading from box tables (BoxView): the frames of ExtShadeT<.,
// true>, each box one trilinear lookup of its width's table.  Same images, bit
// for bit.  so[k] = (texel offset of box k's low corner along the fastest and
// the middle table axis; weight; first cell of its table plus k boxes' steps
// along the walk axis, as int bits), scut[k] = the axis offset its
// CUT_WHEN_AWAY_FROM_VOLUME test adds to the sample.
struct ExtBoxShade {
  const ExtArgs* e;
  const float4* so;
  const float* scut;
  int n, axis, pad_a, pad_b, pad_w;  // boxes; walk axis; pads of the tables
  float first;             // texel offset of the first box's low corner along it
  float vmin, vmax, per;   // the cut interval, 1 / signed box step (world units)
  struct Ray {};
  __device__ __forceinline__ void begin(Ray&, float3) const {}

  // Boxes of the walk from a sample at pm along the axis: the index of the
  // first that fails the cut test.  The test is monotone in k once the first
  // box passes (the boxes move towards one face), so the index is computed
  // from the step and corrected by the test itself; a known trip count lets
  // the loop run with several boxes' loads in flight.
  __device__ __forceinline__ int boxes(float pm) const {
    auto in = [&](int k) {
      const float nxt = pm + scut[k];
      return nxt > vmin && nxt < vmax;
    };
    if (n == 0 || !in(0)) return 0;
    int k = min(max((int)(((per > 0.0f ? vmax : vmin) - pm - scut[0]) * per) + 1, 1), n);
    while (k < n && in(k)) ++k;
    while (k > 1 && !in(k - 1)) --k;
    return k;
  }

  // AXIS 2: table axes (x, y, z), 1: (x, z, y), 0: (y, z, x), walk axis last.
  template <int AXIS>
  __device__ __forceinline__ float walk(float ga, float gb, float gw, int m) const {
    const BoxGrid& G = e->box.sdw_grid;
    const float* __restrict__ tab = e->box.sdw;
    const int row = G.row;
    const unsigned nab = G.nab, ma = (unsigned)G.na - 1u, mb = (unsigned)G.nb - 1u;
    float tw;
    const unsigned cw = (unsigned)(cell_of(gw + first, tw) + pad_w) * nab;
    float st = 0.0f;
#pragma unroll 4
    for (int k = 0; k < m; ++k) {
      const float4 o = so[k];
      float ta, tb;
      const unsigned a = min((unsigned)(cell_of(ga + o.x, ta) + pad_a), ma);
      const unsigned b = min((unsigned)(cell_of(gb + o.y, tb) + pad_b), mb);
      const BoxCorners c = box_corners(tab, (__float_as_uint(o.w) + cw) + (a + b * (unsigned)row), row, nab);
      float v;  // corners as (x, y, z) bits, so that the lerp order is z, y, x
      if constexpr (AXIS == 2)
        v = aligned_weigh(c.v00.x, c.v00.y, c.v01.x, c.v01.y, c.v10.x, c.v10.y, c.v11.x, c.v11.y, f3(ta, tb, tw));
      else if constexpr (AXIS == 1)
        v = aligned_weigh(c.v00.x, c.v00.y, c.v10.x, c.v10.y, c.v01.x, c.v01.y, c.v11.x, c.v11.y, f3(ta, tw, tb));
      else
        v = aligned_weigh(c.v00.x, c.v10.x, c.v00.y, c.v10.y, c.v01.x, c.v11.x, c.v01.y, c.v11.y, f3(tw, ta, tb));
      st = fmaf(v, o.z, st);
    }
    return expf(-st);
  }

  __device__ __forceinline__ float shadow(float3 tx, float3 g, unsigned& aux) const {
    const int m = boxes(axis == 0 ? tx.x : (axis == 1 ? tx.y : tx.z));
    aux += m;
    if (axis == 2) return walk<2>(g.x, g.y, g.z, m);
    if (axis == 1) return walk<1>(g.x, g.z, g.y, m);
    return walk<0>(g.y, g.z, g.x, m);
  }

  // ShadeSample (ebs_ray_bbox_marching.comp:500-551).
  __device__ __forceinline__ float2 light(float3 tx, const Ray&, const FrameArgs& f, unsigned& aux) const {
    const float3 g = sat_texel(e->sat, tx);
    float io = 0.0f, is = 0.0f;
    if (e->apply_occ) { io = box_occlusion(*e, g); aux += e->n_shells; }
    if (e->apply_sdw) is = shadow(tx, g, aux);
    return make_float2(io, is);
  }
  __device__ __forceinline__ float4 shade(float4 src, float3 tx, const Ray& r, const FrameArgs& f, unsigned& aux) const {
    return light_terms(e->apply_occ, e->apply_sdw, e->ka, e->kd).apply<true>(f, src, tx, light(tx, r, f, aux));
  }
};

// ==================================================== cone DOS (rc1pdosct)
// Pyramid taps of the cones at a section's lod: by FP32 lookups, through the
// texture unit, or from the quad copy with the section's levels laid out.
struct TapsFp32 {
  const DosArgs* d;
  using Section = float;
  __device__ __forceinline__ Section section(const float4* s, int i) const { return s[i].y; }
  __device__ __forceinline__ float operator()(Section lod, float3 p) const { return pyr_sample(d->pyr, lod, p); }
};

// pyr_sample's GL_LINEAR_MIPMAP_LINEAR lookup on the level textures: hardware
// trilinear within a level (normalised coordinates, all levels span the
// grid), linear between the two levels of a fractional lod.
struct TapsTex {
  const DosArgs* d;
  using Section = float;
  __device__ __forceinline__ Section section(const float4* s, int i) const { return s[i].y; }
  __device__ __forceinline__ float operator()(Section lod, float3 p) const {
    const PyramidView& P = d->pyr;
    lod = fminf(fmaxf(lod, 0.0f), float(P.n_levels - 1));
    const float fl = floorf(lod);
    const int l0 = int(fl);
    const float t = lod - fl;
    const float u = p.x * P.inv_grid.x, v = p.y * P.inv_grid.y, w = p.z * P.inv_grid.z;
    const float a = tex3D<float>(d->ptex[l0], u, v, w);
    if (t == 0.0f) return a;
    const float b = tex3D<float>(d->ptex[min(l0 + 1, P.n_levels - 1)], u, v, w);
    return fmaf(t, b - a, a);
  }
};

// A section's two levels for TapsQuads: extents as floats (and less one), the
// levels' first cells and pitches, the lod's fraction.
struct QuadSection {
  float4 x, y, z;    // d0, d1, d0 - 1, d1 - 1
  uint4 cell;        // first cell 0, 1; row 0, 1
  uint2 plane;
  float t;
  float pad;
};
// One lookup of both levels: their coordinates and cells as packed pairs, a
// coordinate clamped to [0, d - 1] as a float (both taps are the edge value
// beyond it).  pyr_sample's values, bit for bit.
struct TapsQuads {
  const float4* quads;
  const float4* first;           // the section tables this view's sections are numbered from
  const QuadSection* sections;
  float3 inv_grid;
  using Section = const QuadSection*;
  __device__ __forceinline__ Section section(const float4* s, int i) const { return sections + (s - first) + i; }
  static __device__ __forceinline__ uint2 cells(float q, float4 d, f2& t) {
    const float2 u = un2(fma2(dup2(q), mk2(d.x, d.y), dup2(-0.5f)));
    const int2 c = cell_of2(mk2(fminf(fmaxf(u.x, 0.0f), d.z), fminf(fmaxf(u.y, 0.0f), d.w)), t);
    return make_uint2((unsigned)(c.x + 1), (unsigned)(c.y + 1));  // past the border cell
  }
  static __device__ __forceinline__ float level(float4 a, float4 e, float tx, float ty, float tz) {
    const f2 t = dup2(tx);
    const float2 c0 = un2(lerp2(t, mk2(a.x, a.y), mk2(a.z, a.w))), c1 = un2(lerp2(t, mk2(e.x, e.y), mk2(e.z, e.w)));
    const float z0 = fmaf(ty, c0.y - c0.x, c0.x), z1 = fmaf(ty, c1.y - c1.x, c1.x);
    return fmaf(tz, z1 - z0, z0);
  }
  __device__ __forceinline__ float operator()(Section s, float3 p) const {
    f2 tx, ty, tz;
    const uint2 x = cells(p.x * inv_grid.x, s->x, tx), y = cells(p.y * inv_grid.y, s->y, ty),
                z = cells(p.z * inv_grid.z, s->z, tz);
    const float2 fx = un2(tx), fy = un2(ty), fz = un2(tz);
    const uint4 o = s->cell;
    const uint2 pl = s->plane;
    const float4* q = quads + (o.x + x.x + o.z * y.x + pl.x * z.x);
    const float4 a = __ldg(q), b = __ldg(q + pl.x);
    if (s->t == 0.0f) return level(a, b, fx.x, fy.x, fz.x);
    const float4* r = quads + (o.y + x.y + o.w * y.y + pl.y * z.y);
    const float4 c = __ldg(r), e = __ldg(r + pl.y);
    const float v0 = level(a, b, fx.x, fy.x, fz.x);
    return fmaf(s->t, level(c, e, fx.y, fy.y, fz.y) - v0, v0);
  }
};
// The QuadSection of a lod.
__device__ __forceinline__ QuadSection quad_section(const PyramidView& P, float lod) {
  lod = fminf(fmaxf(lod, 0.0f), float(P.n_levels - 1));
  const float fl = floorf(lod);
  const int a = int(fl), b = min(a + 1, P.n_levels - 1);
  auto axis = [&](int k) {
    const float da = (float)P.dims[a][k], db = (float)P.dims[b][k];
    return make_float4(da, db, da - 1.0f, db - 1.0f);
  };
  return QuadSection{axis(0), axis(1), axis(2), make_uint4(P.qoff[a], P.qoff[b], P.quad_row(a), P.quad_row(b)),
                     make_uint2(P.quad_plane(a), P.quad_plane(b)), lod - fl, 0.0f};
}

template <class Taps>
struct DosShadeT {
  const DosArgs* d;
  const float4* occ_tab;  // shared-memory copies of the section tables
  const float4* sdw_tab;
  Taps taps;
  struct Ray { float3 v_up, v_right; };

  // main(), ray_bbox_marching.comp:682-684.
  __device__ __forceinline__ void begin(Ray& r, float3 dir) const {
    r.v_right = normalize3(cross3(dir, f3(0.0f, 1.0f, 0.0f)));
    r.v_up = normalize3(cross3(-dir, r.v_right));
  }

  // GetGaussianExtinction with CONSIDER_BORDERS (ray_bbox_marching.comp:92-112).
  __device__ __forceinline__ float gauss_ext(float3 p, typename Taps::Section sec, float level, const FrameArgs& f) const {
    float rg = taps(sec, p);
    float3 S = f.vol.grid;
    if (p.x < 0.0f || p.x > S.x || p.y < 0.0f || p.y > S.y || p.z < 0.0f || p.z > S.z) {
      float sg = exp2f(level);
      float3 c = clamp3(p, f3(0.0f, 0.0f, 0.0f), S) - p;
      float dist = c.x * c.x + c.y * c.y + c.z * c.z;
      rg = rg * expf(-(dist) / (2.0f * sg * sg));
    }
    return rg;
  }

  // Cone1/3/7Ray{Occlusion,Shadow} (ray_bbox_marching.comp:124-322, 345-531):
  // the same three-stage integration for both cones, parameterised by table.
  __device__ float cone(const float4* tab, const ConeTableDev& T, float3 pos, float3 k, float3 u, float3 v,
                        const FrameArgs& f, unsigned& aux) const {
    aux += T.n1 + 3 * T.n3 + 7 * T.n7;
    float rays[7], last[7];
    float track = T.initial_step;
    rays[0] = 0.0f; last[0] = 0.0f;
    // Cone1Ray*: one sample per section.
    for (int i = 0; i < T.n1; ++i) {
      float4 s = tab[i];
      float tau = gauss_ext(pos + k * track, taps.section(tab, i), s.y, f);
      float amptau = tau * s.w;
      rays[0] += (last[0] + amptau) * s.z * T.ui_weight;
      last[0] = amptau;
      track += s.x;
    }
    if (T.n3 + T.n7 == 0) return expf(-rays[0]);
    // Cone3Ray*: transform 1 -> 3.
    rays[2] = rays[0]; rays[1] = rays[0];
    last[2] = last[0]; last[1] = last[0];
    {
      float3 vk[3];
#pragma unroll
      for (int r = 0; r < 3; ++r) vk[r] = k * T.axes[r].z + u * T.axes[r].y + v * T.axes[r].x;
      for (int i = 0; i < T.n3; ++i) {
        float4 s = tab[T.n1 + i];
        const typename Taps::Section sec = taps.section(tab, T.n1 + i);
#pragma unroll
        for (int r = 0; r < 3; ++r) {
          float tau = gauss_ext(pos + vk[r] * track, sec, s.y, f);
          float amptau = tau * s.w;
          rays[r] += (last[r] + amptau) * s.z * T.ui_weight;
          last[r] = amptau;
        }
        track += s.x;
      }
    }
    if (T.n7 == 0) return (expf(-rays[0]) + expf(-rays[1]) + expf(-rays[2])) / 3.0f;
    // Cone7Ray*: transform 3 -> 7.
    rays[6] = rays[5] = rays[2];
    rays[4] = rays[3] = rays[1];
    float avg = (rays[2] + rays[1] + rays[0]) / 3.0f;
    rays[2] = rays[1] = rays[0];
    rays[0] = avg;
    last[6] = last[5] = last[2];
    last[4] = last[3] = last[1];
    float avgt = (last[2] + last[1] + last[0]) / 3.0f;
    last[2] = last[1] = last[0];
    last[0] = avgt;
    float3 vk[7];
#pragma unroll
    for (int r = 0; r < 7; ++r) vk[r] = k * T.axes[3 + r].z + u * T.axes[3 + r].y + v * T.axes[3 + r].x;
    int step0 = T.n1 + T.n3;
    for (int i = 0; i < T.n7; ++i) {
      float4 s = tab[step0 + i];
      const typename Taps::Section sec = taps.section(tab, step0 + i);
#pragma unroll
      for (int r = 0; r < 7; ++r) {
        float tau = gauss_ext(pos + vk[r] * track, sec, s.y, f);
        float amptau = tau * s.w;
        rays[r] += (last[r] + amptau) * s.z * T.ui_weight;
        last[r] = amptau;
      }
      track += s.x;
    }
    return (expf(-rays[0]) + (expf(-rays[1]) + expf(-rays[2]) + expf(-rays[3]) + expf(-rays[4]) +
                              expf(-rays[5]) + expf(-rays[6])) * T.w7) / (1.0f + T.w7 * 6.0f);
  }

  // OcclusionEvaluationKernel (ray_bbox_marching.comp:324-333).
  __device__ __forceinline__ float occlusion(float3 tx, const Ray& r, const FrameArgs& f, unsigned& aux) const {
    float3 realpos = tx - f.vol.grid * 0.5f;
    float3 k = normalize3(f.cam.eye - realpos);
    return cone(occ_tab, d->occ, tx, k, r.v_up, r.v_right, f, aux);
  }

  // ShadowEvaluationKernel (ray_bbox_marching.comp:533-562).  Cone1RayShadow
  // declares its parameters as (pos, k, v, u) and is called with (pos, k, u, v),
  // so the shadow cone works in the swapped frame; that is kept.
  __device__ __forceinline__ float shadow(float3 tx, const FrameArgs& f, unsigned& aux) const {
    float3 k, u, v;
    if (d->shadow_type == 0 || d->shadow_type == 1) {
      k = normalize3(d->light_pos - (tx - f.vol.grid * 0.5f));
      u = normalize3(cross3(k, d->light_right));
      v = normalize3(cross3(k, u));
      if (d->shadow_type == 1 && dot3(k, d->light_fwd) < d->spot_cos_max) return 0.0f;
    } else {
      k = d->light_fwd; v = d->light_up; u = d->light_right;
    }
    return cone(sdw_tab, d->sdw, tx, k, v, u, f, aux);
  }

  // ShadeSample (ray_bbox_marching.comp:607-656).
  __device__ __forceinline__ float2 light(float3 tx, const Ray& r, const FrameArgs& f, unsigned& aux) const {
    float io = 0.0f, is = 0.0f;
    if (d->apply_occ) io = occlusion(tx, r, f, aux);
    if (d->apply_sdw) is = shadow(tx, f, aux);
    return make_float2(io, is);
  }
  __device__ __forceinline__ float4 shade(float4 src, float3 tx, const Ray& r, const FrameArgs& f, unsigned& aux) const {
    return light_terms(d->apply_occ, d->apply_sdw, d->ka, d->kd).apply<false>(f, src, tx, light(tx, r, f, aux));
  }
};
using DosShade = DosShadeT<TapsFp32>;


// ================================================= ground truth (rc1pcrtgt)
// S: the volume sampler; alpha: the transfer function's extinction.
template <class S>
struct GtShadeT {
  const GtArgs* g;
  S sample;
  TfAlpha alpha;
  const float3* occ_vec;  // shared-memory copies
  const float3* sdw_vec;
  struct Ray { float3 dir, v_up, v_right; };

  // main(), gt_ray_marching.comp:396-399.
  __device__ __forceinline__ void begin(Ray& r, float3 dir) const {
    r.dir = dir;
    r.v_right = normalize3(cross3(dir, f3(0.0f, 1.0f, 0.0f)));
    r.v_up = normalize3(cross3(-dir, r.v_right));
  }

  // One light ray of ConeOcclusion/ShadowsEvaluationRayCasting
  // (gt_ray_marching.comp:125-159 and 209-242): trapezoidal transmittance.
  // The samples' positions do not depend on the transmittance, only the ray's
  // end does, so kAhead samples are fetched together and then taken one by
  // one until the ray ends: kAhead loads in flight instead of one, for at
  // most kAhead - 1 samples fetched past the end of a ray.  The steps' optical
  // depths are summed and exponentiated once, at the end of the ray: where
  // kAhead whole steps remain, all inside, they take one test for the ray's
  // end between them (256^3 -> 512^2: 45.8 -> 37.7 ms against an exponential and
  // three tests a step).
  static constexpr int kAhead = 4;
  static constexpr float kOpaque = 4.60517f;  // -ln(0.01): 1 - transmittance > 0.99
  __device__ float light_ray(float3 tx, float3 w, float dist, const FrameArgs& f, unsigned& aux) const {
    float tau = 0.0f;
    ++aux;
    float s = g->gap;
    const float3 B = f.vol.grid;
    float st0 = alpha(sample(tx + w * s));
    float ta = 0.0f, tb = -1.0f;  // the samples that need no box test and no clamp
    if constexpr (S::kInside) inside_part(f.vol, tx, w, ta, tb);
    const float step = g->lstep, half = 0.5f * step;
    const float whole = dist - (kAhead + 0.5f) * step;  // kAhead whole steps remain up to here
    for (int guard = 0; guard < kMaxLightSteps && s < dist; guard += kAhead) {
      float at[kAhead], st[kAhead];
      if (S::kInside && s < whole) {
        float sj = s;
#pragma unroll
        for (int j = 0; j < kAhead; ++j) at[j] = sj = sj + step;
        if (at[0] >= ta && sj <= tb) {
#pragma unroll
          for (int j = 0; j < kAhead; j += 2) {
            const float2 a = un2(alpha.two(sample.two_inside(along2(tx, w, mk2(at[j], at[j + 1])))));
            st[j] = a.x;
            st[j + 1] = a.y;
          }
          float t[kAhead];
#pragma unroll
          for (int j = 0; j < kAhead; ++j) {
            tau = fmaf(st0 + st[j], half, tau);
            t[j] = tau;
            st0 = st[j];
          }
          if (fmaxf(fmaxf(t[0], t[1]), fmaxf(t[2], t[3])) > kOpaque) {
            const int n = t[0] > kOpaque ? 0 : (t[1] > kOpaque ? 1 : (t[2] > kOpaque ? 2 : 3));
            aux += n + 1;
            return expf(-(n == 0 ? t[0] : (n == 1 ? t[1] : (n == 2 ? t[2] : t[3]))));
          }
          aux += kAhead;
          s = sj;
          continue;
        }
      }
      float h[kAhead];
      bool in[kAhead];
      float sj = s;
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        h[j] = fminf(step, dist - sj);
        in[j] = sj < dist;
        sj = sj + h[j];
        at[j] = sj;
      }
#pragma unroll
      for (int j = 0; j < kAhead; j += 2) {
        const pos2 p = along2(tx, w, mk2(at[j], at[j + 1]));
        const float2 x = un2(p.x), y = un2(p.y), z = un2(p.z);
        in[j] = in[j] && !(x.x < 0.0f || x.x > B.x || y.x < 0.0f || y.x > B.y || z.x < 0.0f || z.x > B.z);
        in[j + 1] = in[j + 1] && !(x.y < 0.0f || x.y > B.x || y.y < 0.0f || y.y > B.y || z.y < 0.0f || z.y > B.z);
        const float2 a = un2(alpha.two(sample.two(p)));
        st[j] = a.x;
        st[j + 1] = a.y;
      }
#pragma unroll
      for (int j = 0; j < kAhead; ++j) {
        if (!in[j]) return expf(-tau);
        ++aux;
        tau = fmaf((st0 + st[j]) * 0.5f, h[j], tau);
        if (tau > kOpaque) return expf(-tau);
        st0 = st[j];
      }
      s = sj;
    }
    return expf(-tau);
  }

  // ConeOcclusionEvaluationRayCasting (gt_ray_marching.comp:109-169).
  __device__ float occlusion(float3 tx, const Ray& r, const FrameArgs& f, unsigned& aux) const {
    float socc = 0.0f, swgt = 0.0f;
    float3 vd = normalize3(-r.dir);
    for (int i = 0; i < g->n_occ; ++i) {
      float3 c = occ_vec[i];
      float3 w = normalize3(r.v_right * c.x + r.v_up * c.y + vd * c.z);
      float vt = light_ray(tx, w, g->occ_dist, f, aux);
      float rw = dot3(vd, w);
      socc += vt * rw;
      swgt += rw;
    }
    return socc / swgt;
  }

  // ConeShadowsEvaluationRayCasting (gt_ray_marching.comp:171-252).
  __device__ float shadow(float3 tx, const FrameArgs& f, unsigned& aux) const {
    float3 wpos = tx - f.vol.grid * 0.5f;
    float3 vd, vu, vr;
    if (g->shadow_type == 0 || g->shadow_type == 1) {
      vd = normalize3(g->light_pos - wpos);
      vu = normalize3(cross3(vd, g->light_right));
      vr = normalize3(cross3(vd, vu));
      // The reference compares a cosine against 30.0 here, so spot lights always return 0.
      if (g->shadow_type == 1 && dot3(vd, g->light_fwd) < 30.0f) return 0.0f;
    } else {
      vd = g->light_fwd; vu = g->light_up; vr = g->light_right;
    }
    float ssdw = 0.0f, swgt = 0.0f;
    for (int i = 0; i < g->n_sdw; ++i) {
      float3 c = sdw_vec[i];
      float3 w = normalize3(vr * c.x + vu * c.y + vd * c.z);
      float vt = light_ray(tx, w, g->sdw_dist, f, aux);
      float rw = dot3(vd, w);
      ssdw += vt * rw;
      swgt += rw;
    }
    return ssdw / swgt;
  }

  // ShadeSample (gt_ray_marching.comp:254-303).
  __device__ __forceinline__ float2 light(float3 tx, const Ray& r, const FrameArgs& f, unsigned& aux) const {
    float io = 0.0f, is = 0.0f;
    if (g->apply_occ) io = occlusion(tx, r, f, aux);
    if (g->apply_sdw) is = shadow(tx, f, aux);
    return make_float2(io, is);
  }
  __device__ __forceinline__ float4 shade(float4 src, float3 tx, const Ray& r, const FrameArgs& f, unsigned& aux) const {
    return light_terms(g->apply_occ, g->apply_sdw, g->ka, g->kd).apply<false>(f, src, tx, light(tx, r, f, aux));
  }
};

// ============================================================ primary loop
// The warp's log2 width in pixels (warps of 4x8, 8x4 or 16x2 pixels).
__device__ __forceinline__ int warp_shift(int warp_w) { return warp_w == 4 ? 2 : (warp_w == 16 ? 4 : 3); }

__device__ __forceinline__ void pixel_of(const FrameArgs& f, int& px, int& py) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, wl = warp_shift(f.warp_w);
  const int warps_x = f.tile_w >> wl;
  px = blockIdx.x * f.tile_w + (warp % warps_x) * (1 << wl) + (lane & ((1 << wl) - 1));
  py = blockIdx.y * f.tile_h + (warp / warps_x) * (32 >> wl) + (lane >> wl);
}

__device__ __forceinline__ void add_stats(const FrameArgs& f, unsigned int n, unsigned int shaded, unsigned int aux) {
  if (!f.stats) return;  // nobody asked: no shuffles, no atomics on three addresses
  unsigned long long a = n, b = shaded, c = aux;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_down_sync(0xffffffffu, a, o);
    b += __shfl_down_sync(0xffffffffu, b, o);
    c += __shfl_down_sync(0xffffffffu, c, o);
  }
  if ((threadIdx.x & 31) == 0) {
    atomicAdd(f.stats + 0, a);
    atomicAdd(f.stats + 1, b);
    atomicAdd(f.stats + 2, c);
  }
}

// One step's opacity, and its colour composited front to back.  Which samples a
// ray shades and where it ends follow from these and the primary ray alone; the
// passes of a deferred frame (deferred.cuh) and its methods' direct marchers work
// them out in different kernels, so every rounding is spelled out.
__device__ __forceinline__ float step_opacity(float sigma, float h) {
  return __fsub_rn(1.0f, expf(__fmul_rn(-sigma, h)));
}
__device__ __forceinline__ float over(float dst, float left, float src) { return fmaf(left, src, dst); }
__device__ __forceinline__ void composite(float4& dst, float4 src, float h) {
  const float a = step_opacity(src.w, h), left = __fsub_rn(1.0f, dst.w);
  dst.x = over(dst.x, left, __fmul_rn(src.x, a));
  dst.y = over(dst.y, left, __fmul_rn(src.y, a));
  dst.z = over(dst.z, left, __fmul_rn(src.z, a));
  dst.w = over(dst.w, left, a);
}

// The a5 loop (ray_marching_1p.comp:170-247): h = min(StepSize, D - s),
// sample at s + h/2, skip transparent samples, alpha = 1 - exp(-sigma h),
// front-to-back composite, stop once alpha > 0.99.
template <class S, class Tf, class Shade>
__device__ __forceinline__ void march_ray_with(const FrameArgs& f, const S& sample, const Tf& tf, const Shade& sh,
                                               int px, int py) {
  bool inside = px < f.W && py < f.H;
  unsigned int n = 0, shaded = 0, aux = 0;
  if (inside) {
    float3 dir = primary_dir(f.cam, px, py, f.W, f.H);
    float tnear, tfar;
    float4 dst = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (ray_aabb(f.cam.eye, dir, f.vol.grid, tnear, tfar)) {
      typename Shade::Ray ray;
      sh.begin(ray, dir);
      float D = fabsf(tfar - tnear);
      float3 tex0 = f.cam.eye + dir * tnear + f.vol.grid * 0.5f;
      // Bound on the step count (never reached for validated step sizes):
      // keeps a loop whose s stops advancing from spinning forever.
      const unsigned max_iter = (unsigned)fminf(D / f.step, 1.0e9f) + 4u;
      for (float s = 0.0f; s < D && n < max_iter;) {
        float h = fminf(f.step, D - s);
        float3 p = tex0 + dir * (s + h * 0.5f);
        float4 src = tf(sample(p));
        ++n;
        if (src.w > 0.0f) {
          ++shaded;
          src = sh.shade(src, p, ray, f, aux);
          composite(dst, src, h);
          if (dst.w > 0.99f) break;
        }
        s = s + h;
      }
    }
    size_t o = (size_t)py * f.W + px;
    f.out[o] = dst;
    if (f.counts) f.counts[o] = n;
  }
  add_stats(f, n, shaded, aux);
}

// The transfer function as staged by stage_tf.
struct TfStaged {
  const float4* e;
  int n;
  __device__ __forceinline__ float4 operator()(float density) const { return tf_lookup(e, n, density); }
};

// The same loop two samples at a time, their positions, cells and lerps in
// packed pairs (their positions do not depend on the compositing): for the
// marchers whose step is mostly the sample itself.
template <class S, class Shade>
__device__ __forceinline__ void march_ray_pairs(const FrameArgs& f, const S& sample, const TfTable& tf,
                                                const Shade& sh, int px, int py) {
  const bool inside = px < f.W && py < f.H;
  unsigned int n = 0, shaded = 0, aux = 0;
  if (inside) {
    const float3 dir = primary_dir(f.cam, px, py, f.W, f.H);
    float tnear, tfar;
    float4 dst = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (ray_aabb(f.cam.eye, dir, f.vol.grid, tnear, tfar)) {
      typename Shade::Ray ray;
      sh.begin(ray, dir);
      const float D = fabsf(tfar - tnear);
      const float3 tex0 = f.cam.eye + dir * tnear + f.vol.grid * 0.5f;
      const unsigned max_iter = (unsigned)fminf(D / f.step, 1.0e9f) + 4u;
      // one step; false when it ends the ray
      auto take = [&](float4 src, float3 p, float h) {
        ++n;
        if (src.w > 0.0f && sh.shades()) {
          ++shaded;
          src = sh.shade(src, p, ray, f, aux);
          src.w = 1.0f - expf(-src.w * h);
          src.x *= src.w; src.y *= src.w; src.z *= src.w;
          const float r = 1.0f - dst.w;
          dst.x += r * src.x; dst.y += r * src.y; dst.z += r * src.z; dst.w += r * src.w;
          if (dst.w > 0.99f) return false;
        }
        return true;
      };
      for (float s = 0.0f; s < D && n < max_iter;) {
        const float h0 = fminf(f.step, D - s);
        const float s1 = s + h0;
        const float h1 = fminf(f.step, D - s1);
        const pos2 p = along2(tex0, dir, mk2(s + h0 * 0.5f, s1 + h1 * 0.5f));
        float4 src0, src1;
        tf.two(sample.two(p), src0, src1);
        if (!take(src0, pos_lo(p), h0)) break;
        s = s1;
        if (!(s < D && n < max_iter)) break;
        if (!take(src1, pos_hi(p), h1)) break;
        s = s + h1;
      }
    }
    const size_t o = (size_t)py * f.W + px;
    f.out[o] = dst;
    if (f.counts) f.counts[o] = n;
  }
  add_stats(f, n, shaded, aux);
}

template <class Shade>
__device__ __forceinline__ void march_ray(const FrameArgs& f, const float4* tf, const Shade& sh, int px, int py) {
  march_ray_with(f, SampleAny(f.vol), TfStaged{tf, f.tf_n}, sh, px, py);
}

// One CTA-tile pixel per thread (pixel_of).
template <class Shade>
__device__ __forceinline__ void march_pixel(const FrameArgs& f, const float4* tf, const Shade& sh) {
  int px, py;
  pixel_of(f, px, py);
  march_ray(f, tf, sh, px, py);
}

// ============================================ persistent marcher, ray refill
// Next ray index for every active lane of a warp with one atomic.
__device__ __forceinline__ unsigned take_ray(unsigned int* work) {
  const unsigned m = __activemask();
  const int lane = threadIdx.x & 31;
  const int leader = __ffs(m) - 1;
  unsigned base = 0;
  if (lane == leader) base = atomicAdd(work, (unsigned)__popc(m));
  base = __shfl_sync(m, base, leader);
  return base + (unsigned)__popc(m & ((1u << lane) - 1u));
}

// Square spiral of 8x4-pixel tiles around the tile (cx, cy): sequence number
// k -> ring r = ceil((sqrt(k+1) - 1) / 2), then the position on that ring.
// Tiles near the projected volume centre (the longest rays) come first and
// consecutive tiles are neighbours, so the CTAs' working sets overlap.
__device__ __forceinline__ void spiral_tile(unsigned k, int& dx, int& dy) {
  if (k == 0) { dx = dy = 0; return; }
  int r = (int)((sqrtf((float)k + 1.0f) - 1.0f) * 0.5f);
  while ((unsigned)(2 * r + 1) * (unsigned)(2 * r + 1) <= k) ++r;  // fix float rounding
  while (r > 0 && (unsigned)(2 * r - 1) * (unsigned)(2 * r - 1) > k) --r;
  const int m = (int)(k - (unsigned)(2 * r - 1) * (unsigned)(2 * r - 1));
  const int side = m / (2 * r), off = m % (2 * r);
  switch (side) {
    case 0: dx = r; dy = -r + 1 + off; break;
    case 1: dx = r - 1 - off; dy = r; break;
    case 2: dx = -r; dy = r - 1 - off; break;
    default: dx = -r + 1 + off; dy = -r; break;
  }
}


// Ray order of the persistent marchers: 8x4-pixel tiles in the square spiral
// around the tile of the projected volume centre (long rays first,
// neighbouring tiles together); total = 32 x the tiles of the spiral's
// bounding square (positions outside the image are skipped).
struct RayOrder {
  int cx, cy, tiles_x, tiles_y;
  unsigned total;
};

// The a5 loop with persistent ray refill and warp-ballot control flow: each
// lane advances its own ray to its next shaded sample, then the lanes with a
// pending sample run ShadeSample together (the expensive light integrals run
// with the warp's lanes aligned); a lane whose ray ends (front-to-back
// termination or the far side of the box) writes its pixel and takes the
// next ray of the frame from *work, so no lane idles until the longest ray of
// its tile ends.  The warp leaves when a ballot finds no lane with a ray.
// Same arithmetic per ray as march_ray.
template <class Shade>
__device__ __forceinline__ void march_refill(const FrameArgs& f, const float4* tf, const Shade& sh, unsigned* work,
                                             const RayOrder& o) {
  unsigned n_all = 0, shaded = 0, aux = 0;
  bool have = false, done = false;
  int px = 0, py = 0;
  float3 dir = f3(0.0f, 0.0f, 1.0f), tex0 = f3(0.0f, 0.0f, 0.0f);
  float D = 0.0f, s = 0.0f;
  float4 dst = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  unsigned n = 0, max_iter = 0;
  typename Shade::Ray ray;
  auto finish = [&]() {
    const size_t off = (size_t)py * f.W + px;
    f.out[off] = dst;
    if (f.counts) f.counts[off] = n;
    n_all += n;
    have = false;
  };
  for (;;) {
    // lanes without a ray take new ones; rays that miss the box are written at once
    while (!have && !done) {
      const unsigned idx = take_ray(work);
      if (idx >= o.total) { done = true; break; }
      int dx, dy;
      spiral_tile(idx >> 5, dx, dy);
      const int tx = o.cx + dx, ty = o.cy + dy;
      if (tx < 0 || ty < 0 || tx >= o.tiles_x || ty >= o.tiles_y) continue;
      px = tx * 8 + (int)(idx & 7u);
      py = ty * 4 + (int)((idx >> 3) & 3u);
      if (px >= f.W || py >= f.H) continue;
      dir = primary_dir(f.cam, px, py, f.W, f.H);
      dst = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      n = 0;
      float tnear, tfar;
      if (!ray_aabb(f.cam.eye, dir, f.vol.grid, tnear, tfar)) {
        finish();
        continue;
      }
      sh.begin(ray, dir);
      D = fabsf(tfar - tnear);
      tex0 = f.cam.eye + dir * tnear + f.vol.grid * 0.5f;
      s = 0.0f;
      max_iter = (unsigned)fminf(D / f.step, 1.0e9f) + 4u;
      have = true;
    }
    if (__ballot_sync(0xffffffffu, have) == 0u) break;
    bool pending = false;
    float4 src = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float3 p = f3(0.0f, 0.0f, 0.0f);
    float h = 0.0f;
    if (have) {
      while (s < D && n < max_iter) {
        h = fminf(f.step, D - s);
        p = tex0 + dir * (s + h * 0.5f);
        src = tf_lookup(tf, f.tf_n, sample_volume(f.vol, p));
        ++n;
        if (src.w > 0.0f) { pending = true; break; }
        s = s + h;
      }
      if (!pending) finish();
    }
    if (pending) {
      ++shaded;
      src = sh.shade(src, p, ray, f, aux);
      composite(dst, src, h);
      s = s + h;
      if (dst.w > 0.99f) finish();
    }
  }
  add_stats(f, n_all, shaded, aux);
}

// The spiral order of a frame: centred on the pixel where the volume centre
// projects (the frame centre when it projects behind or far off the camera).
inline RayOrder ray_order(const FrameArgs& f) {
  const float3 d = f3(0.0f, 0.0f, 0.0f) - f.cam.eye;
  const float zf = dot3(d, f.cam.f);
  int px = f.W / 2, py = f.H / 2;
  if (zf > 1e-6f) {
    const float xn = dot3(d, f.cam.s) / (zf * f.cam.tan_half_fovy * f.cam.aspect);
    const float yn = dot3(d, f.cam.u) / (zf * f.cam.tan_half_fovy);
    if (xn == xn && yn == yn && fabsf(xn) < 4.0f && fabsf(yn) < 4.0f) {
      px = (int)((xn * 0.5f + 0.5f) * (float)f.W);
      py = (int)((yn * 0.5f + 0.5f) * (float)f.H);
    }
  }
  RayOrder o;
  o.tiles_x = (f.W + 7) / 8;
  o.tiles_y = (f.H + 3) / 4;
  o.cx = px / 8 < 0 ? 0 : (px / 8 >= o.tiles_x ? o.tiles_x - 1 : px / 8);
  o.cy = py / 4 < 0 ? 0 : (py / 4 >= o.tiles_y ? o.tiles_y - 1 : py / 4);
  const int R = std::max(std::max(o.cx, o.tiles_x - 1 - o.cx), std::max(o.cy, o.tiles_y - 1 - o.cy));
  o.total = (unsigned)(2 * R + 1) * (unsigned)(2 * R + 1) * 32u;  // frames <= 32768^2: below 2^32
  return o;
}

// Kernel vectors of the ground truth, staged after its extinction table.
struct GtStage {
  float2* alpha;
  float3 *occ, *sdw;
  __device__ __forceinline__ GtStage(const FrameArgs& f, const GtArgs& g, void* smem)
      : alpha(static_cast<float2*>(smem)), occ(reinterpret_cast<float3*>(alpha + f.tf_n + 1)), sdw(occ + g.n_occ) {
    stage_tf_alpha(f.tf, f.tf_n, alpha);
    for (int i = threadIdx.x; i < g.n_occ; i += blockDim.x) occ[i] = g.occ_vec[i];
    for (int i = threadIdx.x; i < g.n_sdw; i += blockDim.x) sdw[i] = g.sdw_vec[i];
  }
  static size_t bytes(int tf_n, const GtArgs& g) {
    return sizeof(float2) * ((size_t)tf_n + 1) + sizeof(float3) * ((size_t)g.n_occ + g.n_sdw);
  }
};

// Loads the RGBt table into shared memory (n <= tf_smem_cap) and returns it.
__device__ __forceinline__ const float4* stage_tf(const FrameArgs& f, float4* smem) {
  for (int i = threadIdx.x; i < f.tf_n; i += blockDim.x) smem[i] = f.tf[i];
  return smem;
}

}  // namespace cvr
