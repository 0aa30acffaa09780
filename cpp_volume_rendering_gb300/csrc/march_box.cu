// march_box.cu — the extinction marcher on box tables (ExtBoxShade), single
// frames and batches.
#include "march_ext.cuh"

namespace cvr {

static size_t box_smem(int tf_n, int n) { return sizeof(float4) * tf_n + (sizeof(float4) + sizeof(float)) * n; }

template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_march_extinction_box(const __grid_constant__ FrameArgs f,
                                                                    const __grid_constant__ ExtArgs e,
                                                                    const __grid_constant__ BoxWalk w) {
  extern __shared__ float4 sm_tf[];
  const float4* tf = stage_tf(f, sm_tf);
  float4* so = sm_tf + f.tf_n;
  float* scut = reinterpret_cast<float*>(so + w.n);
  stage_walk(so, scut, w.o, w.cut, w.n);
  __syncthreads();
  ExtBoxShade sh{&e, so, scut, w.n, w.axis, w.pad_a, w.pad_b, w.pad_w, w.first, w.vmin, w.vmax, w.per};
  march_pixel(f, tf, sh);
}

template <int NT, int MINB>
static cudaError_t launch_box_t(const FrameArgs& f, const ExtArgs& e, const BoxWalk& w, cudaStream_t st) {
  const size_t sm = box_smem(f.tf_n, w.n);
  auto kern = k_march_extinction_box<NT, MINB>;
  cudaError_t err = cudaSuccess;
  if (sm > 48 * 1024) err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
  if (err == cudaSuccess) err = carve_l1(kern, NT, sm);
  if (err != cudaSuccess) return err;
  kern<<<grid_of(f), NT, sm, st>>>(f, e, w);
  return cudaGetLastError();
}

template <int NT>
static cudaError_t launch_box_nt(const FrameArgs& f, const ExtArgs& e, const BoxWalk& w, cudaStream_t st) {
  switch (f.variant) {
    case 1: return launch_box_t<NT, minb_of<NT>(1)>(f, e, w, st);
    case 2: return launch_box_t<NT, minb_of<NT>(2)>(f, e, w, st);
    case 3: return launch_box_t<NT, minb_of<NT>(3)>(f, e, w, st);
    default: return launch_box_t<NT, 1>(f, e, w, st);
  }
}

cudaError_t launch_extinction_box(const FrameArgs& f, const ExtArgs& e, const BoxWalk& w, cudaStream_t st) {
  switch (threads_of(f)) {
    case 64: return launch_box_nt<64>(f, e, w, st);
    case 256: return launch_box_nt<256>(f, e, w, st);
    default: return launch_box_nt<128>(f, e, w, st);
  }
}

// Batched frames: tiles of all jobs from one counter, as k_batch_extinction.
template <int NT, int MINB>
__global__ void __launch_bounds__(NT, MINB) k_batch_box(const BatchExtJob* __restrict__ jobs, int n_jobs,
                                                         unsigned total, unsigned* counter) {
  __shared__ BatchExtJob J;
  __shared__ unsigned s_blk;
  __shared__ int s_job;
  extern __shared__ float4 sm_bt[];
  int cur = -1;
  while (true) {
    if (threadIdx.x == 0) {
      const unsigned b = atomicAdd(counter, 1u);
      s_blk = b;
      s_job = b < total ? batch_job_of(jobs, n_jobs, b) : 0;
    }
    __syncthreads();
    const unsigned b = s_blk;
    if (b >= total) break;
    const int j = s_job;
    float4* so = sm_bt + jobs[j].f.tf_n;
    float* scut = reinterpret_cast<float*>(so + jobs[j].tn);
    if (j != cur) {
      copy_job(&J, jobs + j);
      __syncthreads();
      for (int i = threadIdx.x; i < J.f.tf_n; i += blockDim.x) sm_bt[i] = J.f.tf[i];
      stage_walk(so, scut, J.bo, J.bcut, J.tn);
      cur = j;
      __syncthreads();
    }
    int px, py;
    batch_pixel(J, b, px, py);
    ExtBoxShade sh{&J.e, so, scut, J.tn, J.tax, J.bpad_a, J.bpad_b, J.bpad_w, J.bfirst, J.tvmin, J.tvmax, J.bper};
    march_ray(J.f, sm_bt, sh, px, py);
    __syncthreads();  // J and the staged tables are reused by the next tile
  }
}

template <int NT, int MINB>
static cudaError_t launch_batch_box_t(const BatchExtJob* jobs, int n_jobs, unsigned total_blocks, unsigned* counter,
                                      size_t smem, cudaStream_t st) {
  return launch_batch_kernel(k_batch_box<NT, MINB>, NT, jobs, n_jobs, total_blocks, counter, smem, st);
}

template <int NT>
static cudaError_t launch_batch_box_nt(const BatchExtJob* jobs, int n_jobs, unsigned total_blocks, unsigned* counter,
                                       size_t smem, int variant, cudaStream_t st) {
  switch (variant) {
    case 1: return launch_batch_box_t<NT, minb_of<NT>(1)>(jobs, n_jobs, total_blocks, counter, smem, st);
    case 2: return launch_batch_box_t<NT, minb_of<NT>(2)>(jobs, n_jobs, total_blocks, counter, smem, st);
    case 3: return launch_batch_box_t<NT, minb_of<NT>(3)>(jobs, n_jobs, total_blocks, counter, smem, st);
    default: return launch_batch_box_t<NT, 1>(jobs, n_jobs, total_blocks, counter, smem, st);
  }
}

cudaError_t launch_batch_box(const BatchExtJob* jobs, int n_jobs, unsigned total_blocks, unsigned* counter, int tf_n,
                             int max_table, int tile_threads, int variant, cudaStream_t st) {
  const size_t smem = box_smem(tf_n, max_table);
  switch (tile_threads) {
    case 64: return launch_batch_box_nt<64>(jobs, n_jobs, total_blocks, counter, smem, variant, st);
    case 256: return launch_batch_box_nt<256>(jobs, n_jobs, total_blocks, counter, smem, variant, st);
    default: return launch_batch_box_nt<128>(jobs, n_jobs, total_blocks, counter, smem, variant, st);
  }
}

}  // namespace cvr
