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

namespace cvr {

// Any storage: bricks, volumes of 2^31 voxels and more, axes of 2^21 and more.
struct SampleAny {
  const VolumeView& v;
  __device__ __forceinline__ explicit SampleAny(const VolumeView& view) : v(view) {}
  __device__ __forceinline__ float operator()(float3 p) const { return sample_volume(v, p); }
};

// The texture unit's copy.
struct SampleTex {
  const VolumeView& v;
  __device__ __forceinline__ explicit SampleTex(const VolumeView& view) : v(view) {}
  __device__ __forceinline__ float operator()(float3 p) const {
    return tex3D<float>(v.tex, p.x * v.inv_grid.x, p.y * v.inv_grid.y, p.z * v.inv_grid.z);
  }
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
