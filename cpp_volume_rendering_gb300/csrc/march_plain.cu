// march_plain.cu — the plain marcher (ray_marching_1p.comp), one thread per
// pixel, specialised on the volume's storage.
#include "march_ext.cuh"

namespace cvr {

template <int NT, class S>
__global__ void __launch_bounds__(NT) k_march_plain(const __grid_constant__ FrameArgs f) {
  extern __shared__ float4 sm_tf[];
  stage_tf_table(f.tf, f.tf_n, sm_tf);
  __syncthreads();
  int px, py;
  pixel_of(f, px, py);
  march_ray_pairs(f, S(f.vol), TfTable{sm_tf, f.tf_n}, PlainShade{}, px, py);
}

template <int NT>
static cudaError_t launch_plain_nt(const FrameArgs& f, cudaStream_t st) {
  return with_sampler(f.vol, [&](auto* s) {
    using S = std::remove_pointer_t<decltype(s)>;
    const size_t sm = tf_table_bytes(f.tf_n);
    auto kern = k_march_plain<NT, S>;
    cudaError_t e = cudaSuccess;
    if (sm > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    kern<<<grid_of(f), NT, sm, st>>>(f);
    return cudaGetLastError();
  });
}

cudaError_t launch_plain_tiles(const FrameArgs& f, cudaStream_t st) {
  switch (threads_of(f)) {
    case 64: return launch_plain_nt<64>(f, st);
    case 256: return launch_plain_nt<256>(f, st);
    default: return launch_plain_nt<128>(f, st);
  }
}

}  // namespace cvr
