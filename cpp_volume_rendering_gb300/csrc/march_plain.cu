// march_plain.cu — the plain marcher (ray_marching_1p.comp), one thread per
// pixel, specialised on the volume's storage.
#include "march_ext.cuh"

namespace cvr {

// Bound by instruction issue (70 % issue active; data from L1): 148 thread
// instructions a step with the storage decided at run time, 104 with it
// compiled in, fewer with two samples' arithmetic packed (512^3 u16 quads ->
// 2048^2: 7.47, 5.75, 4.99 ms).  MINB: with more pixels than the GPU holds
// threads the kernel is cut to 64 registers (8 CTAs of 128 a SM: 4.99 ms
// against 6.27 ms with the compiler's choice); a smaller frame fills no SM
// and keeps them (64^3 -> 256^2: 26.4 against 28.3 us).
template <int NT, int MINB, class S>
__global__ void __launch_bounds__(NT, MINB) k_march_plain(const __grid_constant__ FrameArgs f) {
  extern __shared__ float4 sm_tf[];
  stage_tf_table(f.tf, f.tf_n, sm_tf);
  __syncthreads();
  int px, py;
  pixel_of(f, px, py);
  march_ray_pairs(f, S(f.vol), TfTable{sm_tf, f.tf_n}, PlainShade{}, px, py);
}

template <int NT, int MINB>
static cudaError_t launch_plain_nt(const FrameArgs& f, cudaStream_t st) {
  return with_sampler(f.vol, [&](auto* s) {
    using S = std::remove_pointer_t<decltype(s)>;
    const size_t sm = tf_table_bytes(f.tf_n);
    auto kern = k_march_plain<NT, MINB, S>;
    cudaError_t e = cudaSuccess;
    if (sm > 48 * 1024) e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    kern<<<grid_of(f), NT, sm, st>>>(f);
    return cudaGetLastError();
  });
}

template <int NT>
static cudaError_t launch_plain_size(const FrameArgs& f, cudaStream_t st) {
  const size_t full = (size_t)kSms * 1024;  // threads at 64 registers
  return (size_t)f.W * f.H > full ? launch_plain_nt<NT, 1024 / NT>(f, st) : launch_plain_nt<NT, 1>(f, st);
}

cudaError_t launch_plain_tiles(const FrameArgs& f, cudaStream_t st) {
  switch (threads_of(f)) {
    case 64: return launch_plain_size<64>(f, st);
    case 256: return launch_plain_size<256>(f, st);
    default: return launch_plain_size<128>(f, st);
  }
}

}  // namespace cvr
