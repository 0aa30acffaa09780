// march_gt.cu — the ground-truth marcher (gt_ray_marching.comp), one thread
// per pixel, specialised on the volume's storage.
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

cudaError_t launch_gt_tiles(const FrameArgs& f, const GtArgs& g, cudaStream_t st) {
  switch (threads_of(f)) {
    case 64: return launch_gt_nt<64>(f, g, st);
    case 256: return launch_gt_nt<256>(f, g, st);
    default: return launch_gt_nt<128>(f, g, st);
  }
}

}  // namespace cvr
