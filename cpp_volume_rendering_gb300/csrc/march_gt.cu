// march_gt.cu — the ground-truth marcher (gt_ray_marching.comp), one thread
// per pixel, specialised on the volume's storage.
#include "deferred.cuh"
#include "march_ext.cuh"

namespace cvr {

template <int NT, class S>
__global__ void __launch_bounds__(NT) k_march_gt(const __grid_constant__ GtArgs g, const __grid_constant__ FrameArgs f) {
  extern __shared__ float4 sm[];
  float4* tf = sm;
  for (int i = threadIdx.x; i < f.tf_n; i += blockDim.x) tf[i] = f.tf[i];
  const GtStage gs(f, g, sm + f.tf_n);
  __syncthreads();
  const S sample(f.vol);
  GtShadeT<S> sh{&g, sample, TfAlpha{gs.alpha, f.tf_n}, gs.occ, gs.sdw};
  int px, py;
  pixel_of(f, px, py);
  march_ray_with(f, sample, TfStaged{tf, f.tf_n}, sh, px, py);
}

template <int NT>
static cudaError_t launch_gt_nt(const FrameArgs& f, const GtArgs& g, cudaStream_t st) {
  return with_sampler(f.vol, [&](auto* s) {
    using S = std::remove_pointer_t<decltype(s)>;
    const size_t sm = sizeof(float4) * f.tf_n + GtStage::bytes(f.tf_n, g);
    auto kern = k_march_gt<NT, S>;
    cudaError_t e = cudaSuccess;
    if (sm > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e == cudaSuccess) e = carve_l1(kern, NT, sm);
    if (e != cudaSuccess) return e;
    kern<<<grid_of(f), NT, sm, st>>>(g, f);
    return cudaGetLastError();
  });
}

// The light terms of a frame's collected samples (deferred.cuh): the frame's
// whole time (256^3 quads -> 512^2, 14.8 G light steps: 37.3 ms of 37.7; with
// an exponential a step 45.4 of 45.8, the direct marcher then 72.6, 148.7 with
// one clamped sample in flight).  Bound by instruction issue; 6 CTAs a SM (80
// registers) 37.7 ms, 5 37.8, 7 37.5, 8 38.4.
template <class S>
__global__ void __launch_bounds__(128, 6) k_light_gt(const __grid_constant__ GtArgs g,
                                                        const __grid_constant__ FrameArgs f,
                                                        const __grid_constant__ Deferred d) {
  extern __shared__ float4 sm[];
  const GtStage gs(f, g, sm);
  __syncthreads();
  light_samples(f, d, GtShadeT<S>{&g, S(f.vol), TfAlpha{gs.alpha, f.tf_n}, gs.occ, gs.sdw});
}

cudaError_t launch_light_gt(const FrameArgs& f, const GtArgs& g, const Deferred& d, cudaStream_t st) {
  return with_sampler(f.vol, [&](auto* s) {
    using S = std::remove_pointer_t<decltype(s)>;
    return launch_persistent(k_light_gt<S>, GtStage::bytes(f.tf_n, g), st, g, f, d);
  });
}

cudaError_t load_light_gt(const FrameArgs& f) {
  return with_sampler(f.vol, [&](auto* s) {
    using S = std::remove_pointer_t<decltype(s)>;
    cudaFuncAttributes a;
    return cudaFuncGetAttributes(&a, k_light_gt<S>);
  });
}

cudaError_t launch_gt_tiles(const FrameArgs& f, const GtArgs& g, cudaStream_t st) {
  switch (threads_of(f)) {
    case 64: return launch_gt_nt<64>(f, g, st);
    case 256: return launch_gt_nt<256>(f, g, st);
    default: return launch_gt_nt<128>(f, g, st);
  }
}

}  // namespace cvr
