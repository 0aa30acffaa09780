// deferred.cu — the two marching passes of deferred shading.
#include "deferred.cuh"
#include "march_ext.cuh"

namespace cvr {

namespace {

constexpr size_t kDeferredRecords = (size_t)192 << 20;  // 24 bytes each: at most 4.5 GiB per context
constexpr unsigned kMaxBands = 512;

__device__ __forceinline__ void band_pixel(const FrameArgs& f, const Deferred& d, int& px, int& py, unsigned& warp) {
  pixel_of(f, px, py);
  py += (int)d.y0 * f.tile_h;
  warp = (blockIdx.y * gridDim.x + blockIdx.x) * (blockDim.x >> 5) + (threadIdx.x >> 5);
}

// The primary ray of a pixel; false: it misses the box or lies outside the image.
struct Primary {
  float3 dir, tex0;
  float D;
  unsigned max_iter;
};
__device__ __forceinline__ bool primary_ray(const FrameArgs& f, int px, int py, Primary& r) {
  r = Primary{f3(0.0f, 0.0f, 0.0f), f3(0.0f, 0.0f, 0.0f), 0.0f, 0u};
  if (px >= f.W || py >= f.H) return false;
  r.dir = primary_dir(f.cam, px, py, f.W, f.H);
  float tnear, tfar;
  if (!ray_aabb(f.cam.eye, r.dir, f.vol.grid, tnear, tfar)) return false;
  r.D = fabsf(tfar - tnear);
  r.tex0 = f.cam.eye + r.dir * tnear + f.vol.grid * 0.5f;
  r.max_iter = (unsigned)fminf(r.D / f.step, 1.0e9f) + 4u;
  return true;
}

// The next kAhead steps of a ray: lengths, positions and densities, fetched
// together (a small frame is one chain of loads per ray: with one sample in
// flight the two passes of a 256^2 frame took 0.9 ms).  A ray at its end gets
// steps past it, which the passes do not take.
constexpr int kAhead = 4;
struct Steps {
  float h[kAhead], end[kAhead];  // length, ray parameter after the step
  pos2 p[kAhead / 2];
  float density[kAhead];
  __device__ __forceinline__ float3 at(int j) const { return j & 1 ? pos_hi(p[j / 2]) : pos_lo(p[j / 2]); }
};
template <class S>
__device__ __forceinline__ void fetch_steps(const S& sample, const Primary& r, float step, float s, Steps& o) {
#pragma unroll
  for (int j = 0; j < kAhead; j += 2) {
    o.h[j] = fminf(step, r.D - s);
    o.end[j] = s + o.h[j];
    o.h[j + 1] = fminf(step, r.D - o.end[j]);
    o.end[j + 1] = o.end[j] + o.h[j + 1];
    o.p[j / 2] = along2(r.tex0, r.dir, mk2(s + o.h[j] * 0.5f, o.end[j] + o.h[j + 1] * 0.5f));
    const float2 d = un2(sample.two(o.p[j / 2]));
    o.density[j] = d.x;
    o.density[j + 1] = d.y;
    s = o.end[j + 1];
  }
}

template <int NT, class S>
__global__ void __launch_bounds__(NT) k_collect(const __grid_constant__ FrameArgs f, const __grid_constant__ Deferred d) {
  extern __shared__ float2 sm_alpha[];
  stage_tf_alpha(f.tf, f.tf_n, sm_alpha);
  __syncthreads();
  const TfAlpha tf{sm_alpha, f.tf_n};
  const S sample(f.vol);
  int px, py;
  unsigned warp;
  band_pixel(f, d, px, py, warp);
  const int lane = threadIdx.x & 31;
  unsigned* chunk = d.chunk + (size_t)warp * d.chunks;
  Primary r;
  bool live = primary_ray(f, px, py, r) && r.D > 0.0f;
  const int pixel = py * f.W + px;
  float s = 0.0f, opacity = 0.0f;
  unsigned n = 0;
  unsigned filled = 0, base = 0, next = 0;  // records of the warp; first slot of its current and of its next chunk
  bool room = true;  // deferred_plan's bound holds; never past the lists
  while (room && __any_sync(0xffffffffu, live)) {
    Steps st;
    fetch_steps(sample, r, f.step, s, st);
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      bool shaded = false;
      if (live) {
        const float a = tf(st.density[j]);
        ++n;
        if (a > 0.0f) {
          shaded = true;
          opacity = over(opacity, __fsub_rn(1.0f, opacity), step_opacity(a, st.h[j]));
          if (opacity > 0.99f) live = false;
        }
        s = st.end[j];
        live = live && s < r.D && n < r.max_iter;
      }
      const unsigned m = __ballot_sync(0xffffffffu, shaded);
      const unsigned take = (unsigned)__popc(m), slot = filled % kRecChunk;
      if (m == 0 || !room) continue;
      room = filled + take <= d.chunks * kRecChunk;
      if (!room) continue;
      // a step may end one chunk and begin the next
      const bool first = slot == 0, over = slot != 0 && slot + take > kRecChunk;
      if (first || over) {
        if (lane == 0) next = atomicAdd(d.counter, kRecChunk);
        next = __shfl_sync(0xffffffffu, next, 0);
        if (lane == 0) chunk[(filled + take - 1) / kRecChunk] = next;
        if (first) base = next;
      }
      if (shaded) {
        const unsigned i = slot + (unsigned)__popc(m & ((1u << lane) - 1u));
        const float3 p = st.at(j);
        d.rec[i < kRecChunk ? base + i : next + (i - kRecChunk)] = make_float4(p.x, p.y, p.z, __int_as_float(pixel));
      }
      if (over) base = next;
      filled += take;
    }
  }
  // the unused slots of the last chunk
  if (filled % kRecChunk)
    for (unsigned i = filled % kRecChunk + lane; i < kRecChunk; i += 32) d.rec[base + i].w = __int_as_float(-1);
}

template <int NT, class S>
__global__ void __launch_bounds__(NT) k_resolve(const __grid_constant__ FrameArgs f, const __grid_constant__ Deferred d,
                                                LightTerms t, int ext, unsigned taps) {
  extern __shared__ float4 sm_tf[];
  stage_tf_table(f.tf, f.tf_n, sm_tf);
  __syncthreads();
  const TfTable tf{sm_tf, f.tf_n};
  const S sample(f.vol);
  int px, py;
  unsigned warp;
  band_pixel(f, d, px, py, warp);
  const int lane = threadIdx.x & 31;
  const unsigned* chunk = d.chunk + (size_t)warp * d.chunks;
  Primary r;
  bool live = primary_ray(f, px, py, r) && r.D > 0.0f;
  float4 dst = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
  float s = 0.0f;
  unsigned n = 0, n_shaded = 0, filled = 0;
  bool room = true;  // as collect
  while (room && __any_sync(0xffffffffu, live)) {
    Steps st;
    fetch_steps(sample, r, f.step, s, st);
#pragma unroll
    for (int j = 0; j < kAhead; ++j) {
      float4 src = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
      if (live) {
        src = tf(st.density[j]);
        ++n;
      }
      const bool shaded = src.w > 0.0f;
      const unsigned m = __ballot_sync(0xffffffffu, shaded);
      room = room && filled + (unsigned)__popc(m) <= d.chunks * kRecChunk;
      if (shaded && room) {
        ++n_shaded;
        const unsigned i = filled + (unsigned)__popc(m & ((1u << lane) - 1u));
        const float2 l = d.light[chunk[i / kRecChunk] + i % kRecChunk];
        src = ext ? t.apply<true>(f, src, st.at(j), l) : t.apply<false>(f, src, st.at(j), l);
        composite(dst, src, st.h[j]);
        if (dst.w > 0.99f) live = false;
      }
      filled += (unsigned)__popc(m);
      if (live) {
        s = st.end[j];
        live = s < r.D && n < r.max_iter;
      }
    }
  }
  if (px < f.W && py < f.H) {
    const size_t o = (size_t)py * f.W + px;
    f.out[o] = dst;
    if (f.counts) f.counts[o] = n;
  }
  add_stats(f, n, n_shaded, n_shaded * taps);
}

dim3 band_grid(const FrameArgs& f, const Deferred& d, unsigned rows) {
  const unsigned all = (unsigned)((f.H + f.tile_h - 1) / f.tile_h);
  return dim3((unsigned)((f.W + f.tile_w - 1) / f.tile_w), std::min(rows, all - d.y0));
}

template <class F>
cudaError_t with_threads(const FrameArgs& f, F fn) {
  switch (threads_of(f)) {
    case 64: return fn(std::integral_constant<int, 64>());
    case 256: return fn(std::integral_constant<int, 256>());
    default: return fn(std::integral_constant<int, 128>());
  }
}

}  // namespace

bool deferred_plan(const FrameArgs& f, size_t limit, DeferredPlan* p) {
  // steps of the longest ray of any camera: the diagonal, and the four the
  // marchers' own bound allows past it
  const double diag = std::sqrt((double)dot3(f.vol.grid, f.vol.grid));
  const double steps = diag * 1.0001 / (double)f.step + 8.0;
  const double chunks = std::ceil(steps * 32.0 / kRecChunk) + 1.0;
  const size_t row_warps = (size_t)((f.W + f.tile_w - 1) / f.tile_w) * (size_t)(threads_of(f) / 32);
  const size_t all = (size_t)((f.H + f.tile_h - 1) / f.tile_h);
  if (!(chunks * kRecChunk * (double)row_warps <= (double)kDeferredRecords)) return false;
  if ((size_t)f.W * f.H > 0x7fffffff) return false;
  p->chunks = (unsigned)chunks;
  const size_t row = row_warps * p->chunks * kRecChunk;
  // a row's records (24 bytes each) and its warps' chunk numbers
  const size_t row_bytes = row * (sizeof(float4) + sizeof(float2)) + row_warps * p->chunks * sizeof(unsigned);
  const size_t fit = limit > 512 ? (limit - 512) / row_bytes : 0;
  if (fit == 0) return false;
  p->rows = (unsigned)std::min(std::min(all, kDeferredRecords / row), fit);
  p->bands = (unsigned)((all + p->rows - 1) / p->rows);
  p->records = row * p->rows;
  p->bytes = 256 + (p->rows * row_warps * p->chunks * sizeof(unsigned) + 255) / 256 * 256 +
             p->records * (sizeof(float4) + sizeof(float2));
  return p->bands <= kMaxBands;
}

cudaError_t launch_collect(const FrameArgs& f, const Deferred& d, unsigned rows, cudaStream_t st) {
  return with_sampler(f.vol, [&](auto* s) {
    using S = std::remove_pointer_t<decltype(s)>;
    return with_threads(f, [&](auto nt) {
      constexpr int NT = decltype(nt)::value;
      k_collect<NT, S><<<band_grid(f, d, rows), NT, sizeof(float2) * ((size_t)f.tf_n + 1), st>>>(f, d);
      return cudaGetLastError();
    });
  });
}

cudaError_t launch_resolve(const FrameArgs& f, const Deferred& d, unsigned rows, const LightTerms& t, bool ext,
                           unsigned taps, cudaStream_t st) {
  return with_sampler(f.vol, [&](auto* s) {
    using S = std::remove_pointer_t<decltype(s)>;
    return with_threads(f, [&](auto nt) {
      constexpr int NT = decltype(nt)::value;
      const size_t sm = tf_table_bytes(f.tf_n);
      auto kern = k_resolve<NT, S>;
      cudaError_t e = cudaSuccess;
      if (sm > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      if (e != cudaSuccess) return e;
      kern<<<band_grid(f, d, rows), NT, sm, st>>>(f, d, t, ext ? 1 : 0, taps);
      return cudaGetLastError();
    });
  });
}

cudaError_t load_deferred(const FrameArgs& f) {
  return with_sampler(f.vol, [&](auto* s) {
    using S = std::remove_pointer_t<decltype(s)>;
    return with_threads(f, [&](auto nt) {
      constexpr int NT = decltype(nt)::value;
      cudaFuncAttributes a;
      const cudaError_t e = cudaFuncGetAttributes(&a, k_collect<NT, S>);
      return e != cudaSuccess ? e : cudaFuncGetAttributes(&a, k_resolve<NT, S>);
    });
  });
}

}  // namespace cvr
