// light_dos.cu — the cone method's light terms of a frame's collected samples
// (deferred.cuh).
#include "../../include/cvr.h"
#include "deferred.cuh"
#include "march_ext.cuh"

namespace cvr {

// A cone's taps walk the same sections for every sample, so the sections and
// the levels they read are kernel parameters: a tap's extents, pitches and
// weights come from the constant bank by the (warp-uniform) section number.
// From shared memory they were a third of the L1 data pipe, which bounds the
// kernel (each 128-bit broadcast is four wavefronts of it).
constexpr int kDosSections = 2 * CVR_MAX_CONE_SECTIONS;
struct DosLevel {
  float2 dx, dy, dz;         // extents, twice each (packed operands)
  unsigned cell;             // first quad cell, less the cells' bias
  unsigned row, plane;       // pitches
  float falloff;             // 1 / (2 * 4^level): exact
};
struct DosConst {
  const float4* quads;
  float3 inv_grid;
  DosLevel level[CVR_MAX_LEVELS];  // by lod
  float4 section[kDosSections];  // occlusion, then shadow: distance, (unused), integral, amplitude
  // consecutive sections of one stage and level from this one on, and the level
  unsigned short run[kDosSections];
  unsigned char section_level[kDosSections];
};
static_assert(sizeof(DosConst) + sizeof(DosArgs) + sizeof(FrameArgs) + sizeof(Deferred) <= 32000,
              "kernel parameters are limited to 32764 bytes");

// DosShadeT's cones over whole-numbered lods of the quad copy (the tables the
// sampler builds), run by run of one level: two taps at a time, their
// coordinates in packed pairs, no clamp inside the volume (the copy's border).
struct DosConstShade {
  const DosArgs& d;
  const DosConst& c;
  struct Ray { float3 v_up, v_right; };
  __device__ __forceinline__ void begin(Ray& r, float3 dir) const {
    r.v_right = normalize3(cross3(dir, f3(0.0f, 1.0f, 0.0f)));
    r.v_up = normalize3(cross3(-dir, r.v_right));
  }

  // The level a run reads, in registers.
  struct Level {
    f2 dx, dy, dz;
    unsigned cell, row, plane;
    float falloff;
  };
  __device__ __forceinline__ Level level(int l) const {
    const DosLevel& v = c.level[l];
    return Level{mk2(v.dx.x, v.dx.y), mk2(v.dy.x, v.dy.y), mk2(v.dz.x, v.dz.y), v.cell, v.row, v.plane, v.falloff};
  }
  static __device__ __forceinline__ uint2 cells(f2 p, float inv_grid, f2 n, f2& t) {
    const f2 u = fma2(mul2(p, dup2(inv_grid)), n, dup2(-0.5f)), magic = dup2(12582912.0f);
    const f2 r = add_rd2(u, magic);
    t = sub2(u, sub2(r, magic));
    const float2 b = un2(r);
    return make_uint2(__float_as_uint(b.x), __float_as_uint(b.y));
  }
  // Outside the box, compared as unsigned bits: negative coordinates are
  // above every extent (so is -0, whose falloff is 1).
  static __device__ __forceinline__ bool outside(float x, float y, float z, float3 S) {
    return __float_as_uint(x) > __float_as_uint(S.x) || __float_as_uint(y) > __float_as_uint(S.y) ||
           __float_as_uint(z) > __float_as_uint(S.z);
  }
  // GetGaussianExtinction with CONSIDER_BORDERS (ray_bbox_marching.comp:92-112)
  // at two positions of one level: outside, the value at the nearest point of
  // the box (what clamp-to-edge reads) times the falloff of the distance to it.
  __device__ __forceinline__ float2 taps(pos2 p, const Level& L, const FrameArgs& f) const {
    const float3 S = f.vol.grid;
    const float2 x = un2(p.x), y = un2(p.y), z = un2(p.z);
    const bool out0 = outside(x.x, y.x, z.x, S), out1 = outside(x.y, y.y, z.y, S);
    float w0 = 1.0f, w1 = 1.0f;
    if (out0 || out1) {
      const float3 z3 = f3(0.0f, 0.0f, 0.0f);
      const float3 p0 = f3(x.x, y.x, z.x), p1 = f3(x.y, y.y, z.y);
      const float3 c0 = clamp3(p0, z3, S), c1 = clamp3(p1, z3, S);
      const float3 k0 = c0 - p0, k1 = c1 - p1;
      if (out0) w0 = expf(-(k0.x * k0.x + k0.y * k0.y + k0.z * k0.z) * L.falloff);
      if (out1) w1 = expf(-(k1.x * k1.x + k1.y * k1.y + k1.z * k1.z) * L.falloff);
      p = pos2{mk2(c0.x, c1.x), mk2(c0.y, c1.y), mk2(c0.z, c1.z)};
    }
    f2 tx, ty, tz;
    const uint2 cx = cells(p.x, c.inv_grid.x, L.dx, tx), cy = cells(p.y, c.inv_grid.y, L.dy, ty),
                cz = cells(p.z, c.inv_grid.z, L.dz, tz);
    const float4* q = c.quads + (L.cell + cx.x + L.row * cy.x + L.plane * cz.x);
    const float4* r = c.quads + (L.cell + cx.y + L.row * cy.y + L.plane * cz.y);
    const float4 q0 = __ldg(q), q1 = __ldg(q + L.plane), r0 = __ldg(r), r1 = __ldg(r + L.plane);
    const float2 fx = un2(tx), fy = un2(ty), fz = un2(tz);
    return make_float2(TapsQuads::level(q0, q1, fx.x, fy.x, fz.x) * w0, TapsQuads::level(r0, r1, fx.y, fy.y, fz.y) * w1);
  }

  // A stage of R > 1 rays over n sections from s0: rays two by two.
  template <int R>
  __device__ __forceinline__ void stage(const float3 (&vk)[R], float (&rays)[7], float (&last)[7], float& track, int s0,
                                        int n, float3 pos, float ui, const FrameArgs& f) const {
    for (int i = s0; i < s0 + n;) {
      const Level L = level(c.section_level[i]);
      const int end = i + c.run[i];
      for (; i < end; ++i) {
        const float4 s = c.section[i];
        const f2 t = dup2(track);
#pragma unroll
        for (int r = 0; r < R; r += 2) {
          const int k = r + 1 < R ? r + 1 : r;  // an odd last ray is looked up twice
          const pos2 p{fma2(mk2(vk[r].x, vk[k].x), t, dup2(pos.x)), fma2(mk2(vk[r].y, vk[k].y), t, dup2(pos.y)),
                       fma2(mk2(vk[r].z, vk[k].z), t, dup2(pos.z))};
          const float2 tau = taps(p, L, f);
          const float a = tau.x * s.w;
          rays[r] += (last[r] + a) * s.z * ui;
          last[r] = a;
          if (k != r) {
            const float b = tau.y * s.w;
            rays[k] += (last[k] + b) * s.z * ui;
            last[k] = b;
          }
        }
        track += s.x;
      }
    }
  }

  // DosShadeT::cone; s0: the table's first section.
  __device__ float cone(int s0, const ConeTableDev& T, float3 pos, float3 k, float3 u, float3 v, const FrameArgs& f,
                        unsigned& aux) const {
    aux += T.n1 + 3 * T.n3 + 7 * T.n7;
    float rays[7], last[7];
    float track = T.initial_step;
    rays[0] = 0.0f; last[0] = 0.0f;
    // Cone1Ray*: one sample per section, two sections at a time (an odd last
    // one of a run is looked up twice).
    for (int i = s0; i < s0 + T.n1;) {
      const Level L = level(c.section_level[i]);
      const int end = i + c.run[i];
      for (; i < end; i += 2) {
        const bool two = i + 1 < end;
        const float4 s = c.section[i], e = c.section[two ? i + 1 : i];
        const float next = track + s.x;
        const float2 tau = taps(along2(pos, k, mk2(track, next)), L, f);
        const float a = tau.x * s.w;
        rays[0] += (last[0] + a) * s.z * T.ui_weight;
        last[0] = a;
        track = next;
        if (two) {
          const float b = tau.y * e.w;
          rays[0] += (last[0] + b) * e.z * T.ui_weight;
          last[0] = b;
          track += e.x;
        }
      }
      i = end;
    }
    if (T.n3 + T.n7 == 0) return expf(-rays[0]);
    // Cone3Ray*: transform 1 -> 3.
    rays[2] = rays[0]; rays[1] = rays[0];
    last[2] = last[0]; last[1] = last[0];
    {
      float3 vk[3];
#pragma unroll
      for (int r = 0; r < 3; ++r) vk[r] = k * T.axes[r].z + u * T.axes[r].y + v * T.axes[r].x;
      stage<3>(vk, rays, last, track, s0 + T.n1, T.n3, pos, T.ui_weight, f);
    }
    if (T.n7 == 0) return (expf(-rays[0]) + expf(-rays[1]) + expf(-rays[2])) / 3.0f;
    // Cone7Ray*: transform 3 -> 7.
    rays[6] = rays[5] = rays[2];
    rays[4] = rays[3] = rays[1];
    const float avg = (rays[2] + rays[1] + rays[0]) / 3.0f;
    rays[2] = rays[1] = rays[0];
    rays[0] = avg;
    last[6] = last[5] = last[2];
    last[4] = last[3] = last[1];
    const float avgt = (last[2] + last[1] + last[0]) / 3.0f;
    last[2] = last[1] = last[0];
    last[0] = avgt;
    float3 vk[7];
#pragma unroll
    for (int r = 0; r < 7; ++r) vk[r] = k * T.axes[3 + r].z + u * T.axes[3 + r].y + v * T.axes[3 + r].x;
    stage<7>(vk, rays, last, track, s0 + T.n1 + T.n3, T.n7, pos, T.ui_weight, f);
    return (expf(-rays[0]) + (expf(-rays[1]) + expf(-rays[2]) + expf(-rays[3]) + expf(-rays[4]) +
                              expf(-rays[5]) + expf(-rays[6])) * T.w7) / (1.0f + T.w7 * 6.0f);
  }

  __device__ __forceinline__ float2 light(float3 tx, const Ray& r, const FrameArgs& f, unsigned& aux) const {
    float io = 0.0f, is = 0.0f;
    if (d.apply_occ) {
      const float3 k = normalize3(f.cam.eye - (tx - f.vol.grid * 0.5f));
      io = cone(0, d.occ, tx, k, r.v_up, r.v_right, f, aux);
    }
    if (d.apply_sdw) is = shadow(tx, f, aux);
    return make_float2(io, is);
  }
  // DosShadeT::shadow.
  __device__ __forceinline__ float shadow(float3 tx, const FrameArgs& f, unsigned& aux) const {
    float3 k, u, v;
    if (d.shadow_type == 0 || d.shadow_type == 1) {
      k = normalize3(d.light_pos - (tx - f.vol.grid * 0.5f));
      u = normalize3(cross3(k, d.light_right));
      v = normalize3(cross3(k, u));
      if (d.shadow_type == 1 && dot3(k, d.light_fwd) < d.spot_cos_max) return 0.0f;
    } else {
      k = d.light_fwd; v = d.light_up; u = d.light_right;
    }
    return cone(d.occ.n_sections, d.sdw, tx, k, v, u, f, aux);
  }
};

// 256^3, base 128^3, 156 taps a sample -> 512^2: 13.2 ms a frame, 37.1 with the
// taps along each ray (20.4 with the taps' constants in shared memory where this
// took 14.6).  Bound by instruction issue (78 %; 74 instructions a tap, 107
// without the runs) beside the L1 data pipe; 8 CTAs a SM (64 registers) 13.2 ms,
// 7 13.5, 6 14.2, 5 15.0.
__global__ void __launch_bounds__(128, 8) k_light_dos(const __grid_constant__ DosArgs a,
                                                                 const __grid_constant__ FrameArgs f,
                                                                 const __grid_constant__ Deferred d,
                                                                 const __grid_constant__ DosConst c) {
  light_samples(f, d, DosConstShade{a, c});
}

// Fractional lods, the texture unit, or pyramids without a quad copy.
template <class Taps>
__global__ void __launch_bounds__(128, 6) k_light_dos_general(const __grid_constant__ DosArgs a,
                                                              const __grid_constant__ FrameArgs f,
                                                              const __grid_constant__ Deferred d) {
  extern __shared__ float4 sm[];
  const int no = a.occ.n_sections, ns = a.sdw.n_sections;
  float4* occ = sm;
  float4* sdw = occ + no;
  for (int i = threadIdx.x; i < no; i += blockDim.x) occ[i] = a.occ_sections[i];
  for (int i = threadIdx.x; i < ns; i += blockDim.x) sdw[i] = a.sdw_sections[i];
  if constexpr (std::is_same<Taps, TapsQuads>::value) {
    QuadSection* q = reinterpret_cast<QuadSection*>(sdw + ns);
    for (int i = threadIdx.x; i < no + ns; i += blockDim.x)
      q[i] = quad_section(a.pyr, i < no ? a.occ_sections[i].y : a.sdw_sections[i - no].y);
    __syncthreads();
    light_samples(f, d, DosShadeT<Taps>{&a, occ, sdw, TapsQuads{a.pyr.quads, occ, q, a.pyr.inv_grid}});
  } else {
    __syncthreads();
    light_samples(f, d, DosShadeT<Taps>{&a, occ, sdw, Taps{&a}});
  }
}

// The constant form of two section tables (host copies); false: some lod is
// fractional or beyond any pyramid.
static bool dos_const(const DosArgs& a, const float4* occ, const float4* sdw, DosConst* c) {
  const PyramidView& P = a.pyr;
  c->quads = P.quads;
  c->inv_grid = P.inv_grid;
  // one entry per lod a table may name: past the pyramid's last level the
  // lookup stays there, the falloff follows the lod
  for (int lod = 0; lod < CVR_MAX_LEVELS; ++lod) {
    const int l = std::min(lod, P.n_levels - 1);
    const float x = (float)P.dims[l][0], y = (float)P.dims[l][1], z = (float)P.dims[l][2];
    const unsigned row = P.quad_row(l), plane = P.quad_plane(l);
    // cells arrive as 0x4B400000 + coordinate (cells()), the stored ones start at -1
    const unsigned bias = (1u - 0x4B400000u) * (1u + row + plane);
    c->level[lod] = DosLevel{make_float2(x, x), make_float2(y, y), make_float2(z, z), P.qoff[l] + bias, row, plane,
                           std::ldexp(0.5f, -2 * lod)};
  }
  const int no = a.occ.n_sections, n = no + a.sdw.n_sections;
  // the stages a run may not cross
  const int stops[6] = {a.occ.n1, a.occ.n1 + a.occ.n3, no, no + a.sdw.n1, no + a.sdw.n1 + a.sdw.n3, n};
  for (int i = n - 1; i >= 0; --i) {
    const float4 s = i < no ? occ[i] : sdw[i - no];
    if (!(s.y >= 0.0f && s.y < (float)CVR_MAX_LEVELS && s.y == std::floor(s.y))) return false;
    c->section[i] = s;
    c->section_level[i] = (unsigned char)s.y;
    const bool stop = std::find(stops, stops + 6, i + 1) != stops + 6;
    c->run[i] = (unsigned short)(stop || c->section_level[i] != c->section_level[i + 1] ? 1 : c->run[i + 1] + 1);
  }
  return true;
}

cudaError_t launch_light_dos(const FrameArgs& f, const DosArgs& a, const float4* occ, const float4* sdw, bool tex,
                             const Deferred& d, cudaStream_t st) {
  const size_t n = (size_t)a.occ.n_sections + a.sdw.n_sections;
  if (tex) return launch_persistent(k_light_dos_general<TapsTex>, sizeof(float4) * n, st, a, f, d);
  if (!a.pyr.quads) return launch_persistent(k_light_dos_general<TapsFp32>, sizeof(float4) * n, st, a, f, d);
  DosConst c;
  if (dos_const(a, occ, sdw, &c)) return launch_persistent(k_light_dos, 0, st, a, f, d, c);
  return launch_persistent(k_light_dos_general<TapsQuads>, (sizeof(float4) + sizeof(QuadSection)) * n, st, a, f, d);
}

}  // namespace cvr
