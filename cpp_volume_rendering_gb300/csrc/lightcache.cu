// lightcache.cu — object-space light cache (PreIlluminationStructuredVolume,
// cppvolrend/utils/preillumination.h:15-47): the occlusion and shadow terms
// evaluated once per frame at the centres of a coarse grid
// (rc1pextbsd/lightcachecomputation.comp:443-468,
// rc1pdosct/lightcachecomputation.comp:523-547), then the object-space
// marcher (_common_shaders/obj_ray_marching.comp:264-333) shades every sample
// from a trilinear lookup of that grid.
#include "shade.cuh"

namespace cvr {

// tex_pos = (cell + 0.5) * (VolumeScales * (VolumeDimensions / LightCacheDimensions))
__device__ __forceinline__ float3 cache_cell_pos(const FrameArgs& f, const int* dims, int x, int y, int z) {
  const float3 sc = f.vol.spacing;
  return f3((float(x) + 0.5f) * (sc.x * (float(f.vol.nx) / float(dims[0]))),
            (float(y) + 0.5f) * (sc.y * (float(f.vol.ny) / float(dims[1]))),
            (float(z) + 0.5f) * (sc.z * (float(f.vol.nz) / float(dims[2]))));
}

struct CacheDims { int d[3]; };

// Extinction cache: ExtinctionAmbientOcclusion and ExtinctionDirectionalShadows
// at the cell centre (1 where a term is off), the same functions as per sample.
__global__ void __launch_bounds__(128) k_cache_extinction(FrameArgs f, ExtArgs e, CacheDims cd, int table_n,
                                                          const __grid_constant__ ShadowBoxTable t,
                                                          float2* __restrict__ out) {
  extern __shared__ float4 sm_lc[];
  for (int i = threadIdx.x; i < table_n; i += blockDim.x) {
    sm_lc[i] = t.lo[i];
    sm_lc[table_n + i] = t.hi[i];
  }
  __syncthreads();
  const long long n = (long long)cd.d[0] * cd.d[1] * cd.d[2];
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int x = (int)(i % cd.d[0]), y = (int)((i / cd.d[0]) % cd.d[1]), z = (int)(i / ((long long)cd.d[0] * cd.d[1]));
  const float3 tx = cache_cell_pos(f, cd.d, x, y, z);
  ExtShade sh{&e};
  if (table_n > 0) {
    sh.tlo = sm_lc; sh.thi = sm_lc + table_n; sh.tn = table_n; sh.tax = t.axis;
    sh.tiw = t.interval; sh.tvmin = t.vmin; sh.tvmax = t.vmax;
  }
  unsigned aux = 0;
  const float ao = e.apply_occ ? sh.ambient_occlusion(tx, f) : 1.0f;
  const float sd = e.apply_sdw ? (table_n > 0 ? sh.shadow_table(tx, f, aux) : sh.shadow(tx, f, aux)) : 1.0f;
  out[i] = make_float2(ao, sd);
}

// Cone cache: OcclusionEvaluationKernel with the occlusion cone's frame from
// the camera's up vector (EyeCamUp, rc1pdosct/lightcachecomputation.comp:280-292)
// and ShadowEvaluationKernel, the same cone integration as per sample.
// One thread per cell and term (blockIdx.y), 64 to a CTA: a cache is few cells
// with long chains of taps, bound by their latency.  32^3 cells over a 128^3
// base 84 -> 63 us (both terms in one thread before).
__global__ void __launch_bounds__(128) k_cache_dos(FrameArgs f, DosArgs d, CacheDims cd, float2* __restrict__ out) {
  extern __shared__ float4 sm_lcd[];
  float4* occ = sm_lcd;
  float4* sdw = occ + d.occ.n_sections;
  for (int i = threadIdx.x; i < d.occ.n_sections; i += blockDim.x) occ[i] = d.occ_sections[i];
  for (int i = threadIdx.x; i < d.sdw.n_sections; i += blockDim.x) sdw[i] = d.sdw_sections[i];
  __syncthreads();
  const long long n = (long long)cd.d[0] * cd.d[1] * cd.d[2];
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= n) return;
  const int x = (int)(i % cd.d[0]), y = (int)((i / cd.d[0]) % cd.d[1]), z = (int)(i / ((long long)cd.d[0] * cd.d[1]));
  const float3 tx = cache_cell_pos(f, cd.d, x, y, z);
  DosShade ds{&d, occ, sdw, TapsFp32{&d}};
  unsigned aux = 0;
  if (blockIdx.y) {
    out[i].y = d.apply_sdw ? ds.shadow(tx, f, aux) : 1.0f;
    return;
  }
  float io = 1.0f;
  if (d.apply_occ) {
    const float3 realpos = tx - f.vol.grid * 0.5f;
    const float3 k = normalize3(f.cam.eye - realpos);
    const float3 v_right = normalize3(cross3(-k, f.cam.u));
    const float3 v_up = normalize3(cross3(k, v_right));
    io = ds.cone(occ, d.occ, tx, k, v_up, v_right, f, aux);
  }
  out[i].x = io;
}

// texture(TexVolumeLightCache, tx_pos / VolumeScaledSizes).rg: trilinear,
// texel centres, clamp-to-edge.  At most 2^30 cells: 32-bit cell numbers.
__device__ __forceinline__ float2 cache_lookup(const float2* __restrict__ c, const CacheDims& cd, float3 tx,
                                               float3 inv_grid) {
  // a coordinate clamped to [0, n - 1]: beyond it both taps are the edge cell
  auto cell = [](float p, int n, float& t, unsigned& step) {
    const int i = min(cell_of(fmaxf(fmaf(p, float(n), -0.5f), 0.0f), t), n - 1);
    step = i < n - 1 ? 1u : 0u;
    return (unsigned)i;
  };
  float a, b, g;
  unsigned dx, dy, dz;
  const unsigned x = cell(tx.x * inv_grid.x, cd.d[0], a, dx), y = cell(tx.y * inv_grid.y, cd.d[1], b, dy),
                 z = cell(tx.z * inv_grid.z, cd.d[2], g, dz);
  const unsigned row = (unsigned)cd.d[0], plane = row * (unsigned)cd.d[1];
  dy *= row;
  dz *= plane;
  const float2* q = c + (x + row * y + plane * z);
  const float2 *r = q + dy, *s = q + dz, *u = r + dz;
  auto pair = [](const float2* p) { const float2 v = __ldg(p); return mk2(v.x, v.y); };
  const f2 ta = dup2(a), tb = dup2(b);
  const f2 c0 = lerp2(tb, lerp2(ta, pair(q), pair(q + dx)), lerp2(ta, pair(r), pair(r + dx)));
  const f2 c1 = lerp2(tb, lerp2(ta, pair(s), pair(s + dx)), lerp2(ta, pair(u), pair(u + dx)));
  return un2(lerp2(dup2(g), c0, c1));
}

// obj_ray_marching.comp main() + ShadeSample (both branches): the a5
// loop, but a sample is composited only when occlusion or shadow is on (the
// reference's `src.a > 0.0 && Shade`), its light terms read from the cache.
// The two samples of a step of the loop are fetched together, as are their
// cache lookups' volume cells (march_ray_pairs).
struct CachedShade {
  CacheDims cd;
  const float2* cache;
  int apply_occ, apply_sdw;
  LightTerms terms;
  float3 inv_grid;
  struct Ray {};
  __device__ __forceinline__ void begin(Ray&, float3) const {}
  // the reference's `src.a > 0.0 && Shade`: nothing is composited with both terms off
  __device__ __forceinline__ bool shades() const { return apply_occ || apply_sdw; }
  __device__ __forceinline__ float4 shade(float4 src, float3 p, const Ray&, const FrameArgs& f, unsigned& aux) const {
    const float2 l = cache_lookup(cache, cd, p, inv_grid);
    ++aux;
    return terms.apply<true>(f, src, p, make_float2(apply_occ ? l.x : 0.0f, apply_sdw ? l.y : 0.0f));
  }
};

template <class S>
__global__ void __launch_bounds__(128) k_march_cached(const __grid_constant__ FrameArgs f, CacheDims cd,
                                                      const float2* __restrict__ cache, int apply_occ, int apply_sdw,
                                                      float ka, float kd) {
  extern __shared__ float4 sm_mc[];
  stage_tf_table(f.tf, f.tf_n, sm_mc);
  __syncthreads();
  int px, py;
  pixel_of(f, px, py);
  const float3 inv_grid = f3(1.0f / f.vol.grid.x, 1.0f / f.vol.grid.y, 1.0f / f.vol.grid.z);
  const CachedShade sh{cd, cache, apply_occ, apply_sdw, light_terms(apply_occ, apply_sdw, ka, kd), inv_grid};
  march_ray_pairs(f, S(f.vol), TfTable{sm_mc, f.tf_n}, sh, px, py);
}

cudaError_t launch_cache_extinction(const FrameArgs& f, const ExtArgs& e, const ShadowBoxTable* t,
                                    const ShadowBoxTable& storage, const int dims[3], float2* out, cudaStream_t st) {
  CacheDims cd{{dims[0], dims[1], dims[2]}};
  const long long n = (long long)dims[0] * dims[1] * dims[2];
  const int tn = t ? t->n : 0;
  k_cache_extinction<<<(unsigned)((n + 127) / 128), 128, sizeof(float4) * 2 * tn, st>>>(f, e, cd, tn, t ? *t : storage,
                                                                                        out);
  return cudaGetLastError();
}

cudaError_t launch_cache_dos(const FrameArgs& f, const DosArgs& d, const int dims[3], float2* out, cudaStream_t st) {
  CacheDims cd{{dims[0], dims[1], dims[2]}};
  const long long n = (long long)dims[0] * dims[1] * dims[2];
  const size_t sm = sizeof(float4) * (d.occ.n_sections + d.sdw.n_sections);
  if (sm > 48 * 1024) {
    cudaError_t e = cudaFuncSetAttribute(k_cache_dos, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
  }
  k_cache_dos<<<dim3((unsigned)((n + 63) / 64), 2), 64, sm, st>>>(f, d, cd, out);
  return cudaGetLastError();
}

cudaError_t launch_march_cached(const FrameArgs& f, const float2* cache, const int dims[3], int apply_occ,
                                int apply_sdw, float ka, float kd, cudaStream_t st) {
  CacheDims cd{{dims[0], dims[1], dims[2]}};
  FrameArgs g = f;
  g.tile_w = 16;  // 128-thread CTAs of 8x4-pixel warps
  g.tile_h = 8;
  const dim3 grid((f.W + 15) / 16, (f.H + 7) / 8, 1);
  return with_sampler(f.vol, [&](auto* s) {
    using S = std::remove_pointer_t<decltype(s)>;
    const size_t sm = tf_table_bytes(f.tf_n);
    auto kern = k_march_cached<S>;
    cudaError_t e = cudaSuccess;
    if (sm > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    kern<<<grid, 128, sm, st>>>(g, cd, cache, apply_occ, apply_sdw, ka, kd);
    return cudaGetLastError();
  });
}

}  // namespace cvr
