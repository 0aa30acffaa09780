// light_ext.cu — the extinction renderer's light terms of a frame's collected
// samples (deferred.cuh).
#include "deferred.cuh"
#include "march_ext.cuh"

namespace cvr {

// Directional lights on box tables (200x180x222 -> 512^2: 1.0 ms against 1.7 in
// the direct marcher, whose last rays it waits for).
__global__ void __launch_bounds__(128, 6) k_light_box(const __grid_constant__ FrameArgs f,
                                                      const __grid_constant__ ExtArgs e,
                                                      const __grid_constant__ BoxWalk w,
                                                      const __grid_constant__ Deferred d) {
  extern __shared__ float4 sm_lb[];
  float* scut = reinterpret_cast<float*>(sm_lb + w.n);
  stage_walk(sm_lb, scut, w.o, w.cut, w.n);
  __syncthreads();
  light_samples(f, d, ExtBoxShade{&e, sm_lb, scut, w.n, w.axis, w.pad_a, w.pad_b, w.pad_w, w.first, w.vmin, w.vmax, w.per});
}

// Queries on the SAT.  640x360, 2.3 M samples of a point light, 15 occlusion
// shells and 46 shadow boxes each: 2.6 ms, from 20 with the general 27-sub-box
// query along each ray (12.8 with the equal-fraction query, 3.8 deferred, 2.6
// with the occlusion shells on box tables).  128 registers: 3.7 ms where 96
// took 3.8 and 80 4.0.  C, A as k_march_extinction_dir; n: the table's boxes (0: per-sample cones).
template <bool C, bool A>
__global__ void __launch_bounds__(128, 4) k_light_ext(const __grid_constant__ FrameArgs f,
                                                      const __grid_constant__ ExtArgs e,
                                                      const __grid_constant__ ShadowBoxTable t, int n,
                                                      const __grid_constant__ Deferred d) {
  extern __shared__ float4 sm_le[];
  float4* lo = sm_le;
  float4* hi = lo + n;
  float4* tx = hi + n;
  for (int i = threadIdx.x; i < n; i += blockDim.x) {
    lo[i] = t.lo[i];
    hi[i] = t.hi[i];
    if (A) tx[i] = t.tx[i];
  }
  __syncthreads();
  ExtShadeT<C, A> sh{&e};
  if (n > 0) {
    sh.tlo = lo; sh.thi = hi; sh.tn = n; sh.tax = t.axis;
    sh.tiw = t.interval; sh.tvmin = t.vmin; sh.tvmax = t.vmax;
    if (A) sh.ttx = tx;
  }
  light_samples(f, d, sh);
}

cudaError_t launch_light_box(const FrameArgs& f, const ExtArgs& e, const BoxWalk& w, const Deferred& d,
                             cudaStream_t st) {
  return launch_persistent(k_light_box, (sizeof(float4) + sizeof(float)) * w.n, st, f, e, w, d);
}

cudaError_t launch_light_ext(const FrameArgs& f, const ExtArgs& e, const ShadowBoxTable* table,
                             const ShadowBoxTable& storage, const Deferred& d, cudaStream_t st) {
  const bool c = e.sat.sat32 != nullptr;
  const bool a = table && table->n > 0 && table->aligned && (e.ao_aligned || !e.apply_occ);
  const ShadowBoxTable& t = table ? *table : storage;
  const int n = table ? table->n : 0;
  const size_t sm = sizeof(float4) * 3 * n;
  if (a) return c ? launch_persistent(k_light_ext<true, true>, sm, st, f, e, t, n, d)
                  : launch_persistent(k_light_ext<false, true>, sm, st, f, e, t, n, d);
  return c ? launch_persistent(k_light_ext<true, false>, sm, st, f, e, t, n, d)
           : launch_persistent(k_light_ext<false, false>, sm, st, f, e, t, n, d);
}

}  // namespace cvr
