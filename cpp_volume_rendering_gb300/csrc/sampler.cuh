// sampler.cuh — the volume and transfer-function lookups of the marching
// loops, with the volume's storage a compile-time choice.
//
// sample_volume (cvr_device.cuh) decides layout and voxel type at every
// sample and numbers voxels with 64-bit brick arithmetic; the marchers spend
// most of a step there.  Here a frame's storage picks the kernel (with_sampler)
// and the loop keeps 32-bit cell numbers, floors on the FP32 adders (cell_of)
// and the fewest clamps that stay in bounds for any position.  Same values,
// bit for bit.  Instructions of one 256^3 -> 1024^2 step: see march_plain.cu.
#pragma once

#include "march.cuh"
#include "pack2.cuh"

namespace cvr {

// Any storage: bricks, volumes of 2^31 voxels and more, axes of 2^21 and more.
struct SampleAny {
  const VolumeView& v;
  __device__ __forceinline__ explicit SampleAny(const VolumeView& view) : v(view) {}
  __device__ __forceinline__ float operator()(float3 p) const { return sample_volume(v, p); }
  __device__ __forceinline__ f2 two(const pos2& p) const { return mk2((*this)(pos_lo(p)), (*this)(pos_hi(p))); }
  __device__ __forceinline__ f2 two_inside(const pos2& p) const { return two(p); }
  static constexpr bool kInside = false;
};

// The texture unit's copy.
struct SampleTex {
  const VolumeView& v;
  __device__ __forceinline__ explicit SampleTex(const VolumeView& view) : v(view) {}
  __device__ __forceinline__ float operator()(float3 p) const {
    return tex3D<float>(v.tex, p.x * v.inv_grid.x, p.y * v.inv_grid.y, p.z * v.inv_grid.z);
  }
  __device__ __forceinline__ f2 two(const pos2& p) const { return mk2((*this)(pos_lo(p)), (*this)(pos_hi(p))); }
  __device__ __forceinline__ f2 two_inside(const pos2& p) const { return two(p); }
  static constexpr bool kInside = false;
};

// Texel coordinate of one axis raised to 0: below the first texel centre both
// taps are voxel 0, so the value is the same.  NaN becomes 0.
__device__ __forceinline__ float texel_of(float p, float inv_spacing) { return fmaxf(fmaf(p, inv_spacing, -0.5f), 0.0f); }

__device__ __forceinline__ float trilinear(float c000, float c100, float c010, float c110, float c001, float c101,
                                           float c011, float c111, float tx, float ty, float tz) {
  const float c00 = fmaf(tx, c100 - c000, c000), c10 = fmaf(tx, c110 - c010, c010);
  const float c01 = fmaf(tx, c101 - c001, c001), c11 = fmaf(tx, c111 - c011, c011);
  const float c0 = fmaf(ty, c10 - c00, c00), c1 = fmaf(ty, c11 - c01, c01);
  return fmaf(tz, c1 - c0, c0);
}

// Cells and fractions of two positions along one axis (raised to 0, at most n - 1).
__device__ __forceinline__ int2 texel_cells2(f2 p, float inv_spacing, int n, f2& t) {
  const float2 u = un2(fma2(p, dup2(inv_spacing), dup2(-0.5f)));
  const int2 c = cell_of2(mk2(fmaxf(u.x, 0.0f), fmaxf(u.y, 0.0f)), t);
  return make_int2(min(c.x, n - 1), min(c.y, n - 1));
}
__device__ __forceinline__ f2 trilinear2(f2 c000, f2 c100, f2 c010, f2 c110, f2 c001, f2 c101, f2 c011, f2 c111,
                                         f2 tx, f2 ty, f2 tz) {
  const f2 c0 = lerp2(ty, lerp2(tx, c000, c100), lerp2(tx, c010, c110));
  const f2 c1 = lerp2(ty, lerp2(tx, c001, c101), lerp2(tx, c011, c111));
  return lerp2(tz, c0, c1);
}

// The part [ta, tb] of the line o + d t whose positions are at least 0.51
// voxels inside the box on every axis: there a sample's cell needs no clamp
// and both its planes exist (0.01 voxels are far more than the roundings of
// t and of the position, for axes of up to 8192 voxels; larger ones, axes of
// one voxel, which have no second plane, and lines with a NaN get an empty part).
__device__ __forceinline__ void inside_part(const VolumeView& v, float3 o, float3 d, float& ta, float& tb) {
  const float3 m = v.spacing * 0.51f;
  const float3 inv = f3(1.0f / d.x, 1.0f / d.y, 1.0f / d.z);
  const float3 t0 = (m - o) * inv, t1 = (v.grid - m - o) * inv;
  const float3 lo = fmin3(t0, t1), hi = fmax3(t0, t1);
  ta = fmaxf(fmaxf(lo.x, lo.y), lo.z);
  tb = fminf(fminf(hi.x, hi.y), hi.z);
  const float sum = d.x + d.y + d.z + o.x + o.y + o.z;
  if (!(sum - sum == 0.0f) || min(min(v.nx, v.ny), v.nz) < 2 || max(max(v.nx, v.ny), v.nz) > 8192) tb = -1.0f, ta = 0.0f;
}

// Voxel values as FP32 plus 2^23: the integer below 2^16 placed in the
// mantissa of 8388608.0f by one byte permute.  Differences of two such values
// are exact, so a lerp subtracts them as they are and unbiases one end.
struct biased8 {
  unsigned w;
  template <int K>
  __device__ __forceinline__ float at() const { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650u + K)); }
};
struct biased16 {
  uint2 w;
  template <int K>
  __device__ __forceinline__ float at() const {
    return __uint_as_float(__byte_perm(K < 2 ? w.x : w.y, 0x4B000000u, (K & 1) ? 0x7632u : 0x7610u));
  }
};
// lerp of biased ends: fmaf(t, b - a, a - 2^23).
__device__ __forceinline__ f2 lerp_biased2(f2 t, f2 a, f2 b) { return fma2(t, sub2(b, a), sub2(a, dup2(8388608.0f))); }

// Cells (plus 0x4B400000) and fractions of two positions inside the box along one axis.
__device__ __forceinline__ uint2 inside_cells2(f2 p, float inv_spacing, f2& t) {
  const f2 u = fma2(p, dup2(inv_spacing), dup2(-0.5f)), magic = dup2(12582912.0f);
  const f2 r = add_rd2(u, magic);
  t = sub2(u, sub2(r, magic));
  const float2 b = un2(r);
  return make_uint2(__float_as_uint(b.x), __float_as_uint(b.y));
}

// The x-y quad copy (VolumeView::quad): two loads, planes z0 and z0 + 1.
template <class Q>
struct SampleQuads {
  const VolumeView& v;
  __device__ __forceinline__ explicit SampleQuads(const VolumeView& view) : v(view) {}
  __device__ __forceinline__ float operator()(float3 p) const {
    float tx, ty, tz;
    const int x = min(cell_of(texel_of(p.x, v.inv_spacing.x), tx), v.nx - 1);
    const int y = min(cell_of(texel_of(p.y, v.inv_spacing.y), ty), v.ny - 1);
    const int z = min(cell_of(texel_of(p.z, v.inv_spacing.z), tz), v.nz - 1);
    const Q* q = static_cast<const Q*>(v.voxels) + ((unsigned)x + v.qrow * (unsigned)y + v.qplane * (unsigned)z);
    const Q a = __ldg(q), b = __ldg(q + (z < v.nz - 1 ? v.qplane : 0u));
    return trilinear(a.x, a.y, a.z, a.w, b.x, b.y, b.z, b.w, tx, ty, tz) * v.norm;
  }
  __device__ __forceinline__ f2 two(const pos2& p) const {
    f2 tx, ty, tz;
    const int2 x = texel_cells2(p.x, v.inv_spacing.x, v.nx, tx), y = texel_cells2(p.y, v.inv_spacing.y, v.ny, ty),
               z = texel_cells2(p.z, v.inv_spacing.z, v.nz, tz);
    const Q* base = static_cast<const Q*>(v.voxels);
    const Q* q = base + ((unsigned)x.x + v.qrow * (unsigned)y.x + v.qplane * (unsigned)z.x);
    const Q* r = base + ((unsigned)x.y + v.qrow * (unsigned)y.y + v.qplane * (unsigned)z.y);
    const Q a = __ldg(q), b = __ldg(q + (z.x < v.nz - 1 ? v.qplane : 0u));
    const Q c = __ldg(r), d = __ldg(r + (z.y < v.nz - 1 ? v.qplane : 0u));
    return mul2(trilinear2(mk2(a.x, c.x), mk2(a.y, c.y), mk2(a.z, c.z), mk2(a.w, c.w), mk2(b.x, d.x), mk2(b.y, d.y),
                           mk2(b.z, d.z), mk2(b.w, d.w), tx, ty, tz), dup2(v.norm));
  }
  // two() for positions inside_part holds: no raise, no clamp, no last plane.
  static constexpr bool kInside = true;
  __device__ __forceinline__ f2 two_inside(const pos2& p) const {
    using B = typename std::conditional<sizeof(Q) == 4, biased8, biased16>::type;
    f2 tx, ty, tz;
    const uint2 x = inside_cells2(p.x, v.inv_spacing.x, tx), y = inside_cells2(p.y, v.inv_spacing.y, ty),
                z = inside_cells2(p.z, v.inv_spacing.z, tz);
    // cells carry the bias: 32-bit arithmetic takes it off the sum
    const unsigned bias = 0u - 0x4B400000u * (1u + v.qrow + v.qplane);
    const B* base = static_cast<const B*>(v.voxels);
    const B* q = base + (x.x + bias + v.qrow * y.x + v.qplane * z.x);
    const B* r = base + (x.y + bias + v.qrow * y.y + v.qplane * z.y);
    const B a = load(q), b = load(q + v.qplane), c = load(r), d = load(r + v.qplane);
    const f2 c00 = lerp_biased2(tx, mk2(a.template at<0>(), c.template at<0>()), mk2(a.template at<1>(), c.template at<1>()));
    const f2 c10 = lerp_biased2(tx, mk2(a.template at<2>(), c.template at<2>()), mk2(a.template at<3>(), c.template at<3>()));
    const f2 c01 = lerp_biased2(tx, mk2(b.template at<0>(), d.template at<0>()), mk2(b.template at<1>(), d.template at<1>()));
    const f2 c11 = lerp_biased2(tx, mk2(b.template at<2>(), d.template at<2>()), mk2(b.template at<3>(), d.template at<3>()));
    return mul2(lerp2(tz, lerp2(ty, c00, c10), lerp2(ty, c01, c11)), dup2(v.norm));
  }
  static __device__ __forceinline__ biased8 load(const biased8* p) { return biased8{__ldg(&p->w)}; }
  static __device__ __forceinline__ biased16 load(const biased16* p) { return biased16{__ldg(&p->w)}; }
};

// The plain x-fastest array: eight loads.
template <class T>
struct SamplePlain {
  const VolumeView& v;
  __device__ __forceinline__ explicit SamplePlain(const VolumeView& view) : v(view) {}
  __device__ __forceinline__ float operator()(float3 p) const {
    float tx, ty, tz;
    const int x = min(cell_of(texel_of(p.x, v.inv_spacing.x), tx), v.nx - 1);
    const int y = min(cell_of(texel_of(p.y, v.inv_spacing.y), ty), v.ny - 1);
    const int z = min(cell_of(texel_of(p.z, v.inv_spacing.z), tz), v.nz - 1);
    const unsigned nx = (unsigned)v.nx, plane = nx * (unsigned)v.ny;
    const T* q = static_cast<const T*>(v.voxels) + ((unsigned)x + nx * (unsigned)y + plane * (unsigned)z);
    const unsigned dx = x < v.nx - 1 ? 1u : 0u, dy = y < v.ny - 1 ? nx : 0u, dz = z < v.nz - 1 ? plane : 0u;
    const T* r = q + dy;
    const T* s = q + dz;
    const T* t = r + dz;
    return trilinear(__ldg(q), __ldg(q + dx), __ldg(r), __ldg(r + dx), __ldg(s), __ldg(s + dx), __ldg(t), __ldg(t + dx),
                     tx, ty, tz) * v.norm;
  }
  __device__ __forceinline__ f2 two(const pos2& p) const {
    f2 tx, ty, tz;
    const int2 x = texel_cells2(p.x, v.inv_spacing.x, v.nx, tx), y = texel_cells2(p.y, v.inv_spacing.y, v.ny, ty),
               z = texel_cells2(p.z, v.inv_spacing.z, v.nz, tz);
    const unsigned nx = (unsigned)v.nx, plane = nx * (unsigned)v.ny;
    const T* base = static_cast<const T*>(v.voxels);
    T g[2][8];
    auto gather = [&](int X, int Y, int Z, T* o) {
      const T* q = base + ((unsigned)X + nx * (unsigned)Y + plane * (unsigned)Z);
      const unsigned dx = X < v.nx - 1 ? 1u : 0u, dy = Y < v.ny - 1 ? nx : 0u, dz = Z < v.nz - 1 ? plane : 0u;
      const T* r = q + dy;
      const T* s = q + dz;
      const T* t = r + dz;
      o[0] = __ldg(q); o[1] = __ldg(q + dx); o[2] = __ldg(r); o[3] = __ldg(r + dx);
      o[4] = __ldg(s); o[5] = __ldg(s + dx); o[6] = __ldg(t); o[7] = __ldg(t + dx);
    };
    gather(x.x, y.x, z.x, g[0]);
    gather(x.y, y.y, z.y, g[1]);
    f2 c[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) c[k] = mk2(g[0][k], g[1][k]);
    return mul2(trilinear2(c[0], c[1], c[2], c[3], c[4], c[5], c[6], c[7], tx, ty, tz), dup2(v.norm));
  }
  static constexpr bool kInside = true;
  __device__ __forceinline__ f2 two_inside(const pos2& p) const {
    f2 tx, ty, tz;
    const uint2 x = inside_cells2(p.x, v.inv_spacing.x, tx), y = inside_cells2(p.y, v.inv_spacing.y, ty),
                z = inside_cells2(p.z, v.inv_spacing.z, tz);
    const unsigned nx = (unsigned)v.nx, plane = nx * (unsigned)v.ny;
    const unsigned bias = 0u - 0x4B400000u * (1u + nx + plane);
    const T* base = static_cast<const T*>(v.voxels);
    const T* q = base + (x.x + bias + nx * y.x + plane * z.x);
    const T* r = base + (x.y + bias + nx * y.y + plane * z.y);
    auto pair = [&](unsigned o) { return mk2((float)__ldg(q + o), (float)__ldg(r + o)); };
    return mul2(trilinear2(pair(0u), pair(1u), pair(nx), pair(nx + 1u), pair(plane), pair(plane + 1u), pair(plane + nx),
                           pair(plane + nx + 1u), tx, ty, tz), dup2(v.norm));
  }
};

// Calls fn with the sampler type of a volume view.
template <class F>
cudaError_t with_sampler(const VolumeView& v, F fn) {
  const bool small = (size_t)v.nx * v.ny * v.nz < ((size_t)1 << 31) && v.nx < (1 << 21) && v.ny < (1 << 21) &&
                     v.nz < (1 << 21);
  if (v.tex) return fn(static_cast<SampleTex*>(nullptr));
  if (!small || v.bs > 0) return fn(static_cast<SampleAny*>(nullptr));
  if (v.quad)
    return v.dtype == 1 ? fn(static_cast<SampleQuads<uchar4>*>(nullptr)) : fn(static_cast<SampleQuads<ushort4>*>(nullptr));
  return v.dtype == 1 ? fn(static_cast<SamplePlain<uint8_t>*>(nullptr)) : fn(static_cast<SamplePlain<uint16_t>*>(nullptr));
}

// ---------------------------------------------------------------- transfer function
// Entry and fraction of two densities.
__device__ __forceinline__ uint2 tf_cells2(f2 density, int n, f2& t) {
  const int2 c = cell_of2(fma2(density, dup2((float)n), dup2(-0.5f)), t);
  return make_uint2(min((unsigned)(c.x + 1), (unsigned)n), min((unsigned)(c.y + 1), (unsigned)n));
}
// texture(TexTransferFunc, density) from a table of entries and differences:
// entry k holds tf[k - 1] and tf[k] - tf[k - 1] (0 past either end, where
// both taps are the edge entry), so a lookup is one index, one clamp and one
// FMA per channel, and gives tf_lookup's bits.  tf_n + 1 entries.
struct TfTable {
  const float4* e;  // 2 per entry: value, difference
  int n;
  __device__ __forceinline__ float4 operator()(float density) const {
    float t;
    const unsigned i = min((unsigned)(cell_of(fmaf(density, (float)n, -0.5f), t) + 1), (unsigned)n);
    const float4 a = e[2 * i], d = e[2 * i + 1];
    return make_float4(fmaf(t, d.x, a.x), fmaf(t, d.y, a.y), fmaf(t, d.z, a.z), fmaf(t, d.w, a.w));
  }
  __device__ __forceinline__ void two(f2 density, float4& s0, float4& s1) const {
    f2 t;
    const uint2 i = tf_cells2(density, n, t);
    const float2 f = un2(t);
    s0 = mix(i.x, f.x);
    s1 = mix(i.y, f.y);
  }
  __device__ __forceinline__ float4 mix(unsigned i, float t) const {
    const float4 a = e[2 * i], d = e[2 * i + 1];
    const float2 lo = un2(fma2(dup2(t), mk2(d.x, d.y), mk2(a.x, a.y))), hi = un2(fma2(dup2(t), mk2(d.z, d.w), mk2(a.z, a.w)));
    return make_float4(lo.x, lo.y, hi.x, hi.y);
  }
};
// The extinction channel alone: 8 bytes per entry.
struct TfAlpha {
  const float2* e;
  int n;
  __device__ __forceinline__ float operator()(float density) const {
    float t;
    const unsigned i = min((unsigned)(cell_of(fmaf(density, (float)n, -0.5f), t) + 1), (unsigned)n);
    const float2 a = e[i];
    return fmaf(t, a.y, a.x);
  }
  __device__ __forceinline__ f2 two(f2 density) const {
    f2 t;
    const uint2 i = tf_cells2(density, n, t);
    const float2 a = e[i.x], b = e[i.y];
    return fma2(t, mk2(a.y, b.y), mk2(a.x, b.x));
  }
};
// Filled by the whole CTA (a barrier before the first lookup is the caller's).
__device__ __forceinline__ void stage_tf_table(const float4* __restrict__ tf, int n, float4* out) {
  for (int i = threadIdx.x; i <= n; i += blockDim.x) {
    const float4 a = tf[max(i - 1, 0)], b = tf[min(i, n - 1)];
    out[2 * i] = a;
    out[2 * i + 1] = make_float4(b.x - a.x, b.y - a.y, b.z - a.z, b.w - a.w);
  }
}
__device__ __forceinline__ void stage_tf_alpha(const float4* __restrict__ tf, int n, float2* out) {
  for (int i = threadIdx.x; i <= n; i += blockDim.x) {
    const float a = tf[max(i - 1, 0)].w, b = tf[min(i, n - 1)].w;
    out[i] = make_float2(a, b - a);
  }
}
inline size_t tf_table_bytes(int n) { return sizeof(float4) * 2 * ((size_t)n + 1); }

}  // namespace cvr
