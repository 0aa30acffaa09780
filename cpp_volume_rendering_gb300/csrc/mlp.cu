// mlp.cu — tensor-core (tcgen05) kernels of the surrogate network: weight
// packing, batch inference, fused forward + backward of training tiles, and
// the Adam update.  All GEMMs are M = 128 (one row per point of a tile),
// BF16 operands from shared memory, FP32 accumulators in tensor memory.
#include "mlp_tile.cuh"

namespace cvr {


// ---------------------------------------------------------------- pack
__global__ void k_mlp_pack(const float* __restrict__ p, uint8_t* __restrict__ pk) {
  int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < 64 * 64) {
    int o = i / 64, k = i % 64;
    uint16_t w1 = k < 48 ? to_bf16(p[kOffW1 + o * 48 + k]) : (uint16_t)0;
    *reinterpret_cast<uint16_t*>(pk + kPkW1 + tile_off(o, k, 128, kRowSbo)) = w1;
    uint16_t w2 = to_bf16(p[kOffW2 + o * 64 + k]);
    *reinterpret_cast<uint16_t*>(pk + kPkW2 + tile_off(o, k, 128, kRowSbo)) = w2;
    *reinterpret_cast<uint16_t*>(pk + kPkW2T + tile_off(k, o, 128, kRowSbo)) = w2;  // W2^T[in][out]
  }
  if (i < 16 * 64) {
    int o = i / 64, k = i % 64;
    uint16_t w3 = o < 2 ? to_bf16(p[kOffW3 + o * 64 + k]) : (uint16_t)0;
    *reinterpret_cast<uint16_t*>(pk + kPkW3 + tile_off(o, k, 128, kRowSbo)) = w3;
    *reinterpret_cast<uint16_t*>(pk + kPkW3T + tile_off(k, o, 128, kRow16Sbo)) = w3;  // W3^T[hidden][out]
  }
  if (i < 130) {
    float* b = reinterpret_cast<float*>(pk + kPkBias);
    b[i] = i < 64 ? p[kOffB1 + i] : (i < 128 ? p[kOffB2 + i - 64] : p[kOffB3 + i - 128]);
  }
}

cudaError_t launch_mlp_pack(const float* params, uint8_t* packed, cudaStream_t st) {
  k_mlp_pack<<<16, 256, 0, st>>>(params, packed);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- inference
__global__ void __launch_bounds__(128, 1) k_mlp_infer(const uint8_t* __restrict__ packed, const float* __restrict__ x,
                                                      int n, float* __restrict__ y, int* err) {
  extern __shared__ __align__(1024) uint8_t sm[];
  uint8_t* w = sm;
  uint8_t* xt = sm + kPkBytes;
  uint8_t* ht = xt + kRowTile;
  uint64_t* bar = reinterpret_cast<uint64_t*>(ht + kRowTile);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
  mlp_cta_begin(w, packed, bar, tslot);
  const int m = blockIdx.x * 128 + threadIdx.x;
  float v[48];
#pragma unroll
  for (int k = 0; k < 48; ++k) v[k] = m < n ? __ldg(x + (size_t)m * 48 + k) : 0.0f;
  store_row64(xt, threadIdx.x, v, 48);
  fence_async_smem();
  __syncthreads();
  MlpSmem s{w, xt, ht, bar, *tslot, 0u};
  float out[2];
  if (!mlp_forward_tile(s, out)) atomicExch(err, 1);
  if (m < n) {
    y[2 * (size_t)m] = out[0];
    y[2 * (size_t)m + 1] = out[1];
  }
  mlp_cta_end(s.tmem);
}

cudaError_t launch_mlp_infer(const uint8_t* packed, const float* x, int n, float* y, int* err, cudaStream_t st) {
  const size_t smem = kPkBytes + 2 * kRowTile + 16;
  cudaError_t e = cudaFuncSetAttribute(k_mlp_infer, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  if (n <= 0) return cudaSuccess;
  k_mlp_infer<<<(n + 127) / 128, 128, smem, st>>>(packed, x, n, y, err);
  return cudaGetLastError();
}

// ---------------------------------------------------------------- training
// An Adam step is a chain: six MMAs of a tile, each between an epilogue that
// needs the one before it, then the sum over tiles, the update, and the
// weights that the next step's first MMA reads.  A step of 32 tiles is 1/5 of
// the SMs and bound by the latency of that chain, so the kernels here spend
// threads to shorten it: two threads per point (32 of its 64 hidden units
// each), and four more warps that reduce dW3 and the biases beside the chain.
// The two kernels of a step are launched with programmatic serialization: a
// step's tiles have gathered their points, allocated tensor memory and
// initialised the barrier before the update in front of them has finished.
// Measured: a step of 32 tiles 30 -> 9 us (one thread per point, five launches
// a step, before); 131072 points, 3 epochs of 32 steps 3.84 -> 1.89 ms, of
// which 1.1 ms is the host's shuffling of the points.
constexpr int kChain = 256;         // threads of the chain
constexpr int kTrain = kChain + 128;
constexpr uint32_t kHLbo = 144, kHSbo = 8 * 144;  // the H2 tile: its columns are read along points (dW3) without conflicts
constexpr uint32_t kHTile = 16 * kHSbo;
constexpr uint32_t kTrainSmem =
    kPkBytes + 3 * kRowTile + kHTile + kRow16Tile + 2 * kTTile + (256 + 4) * (uint32_t)sizeof(float) + 16;

// Everything of the launch in front of this one is complete and visible after
// the wait; the launch behind may start once every CTA has signalled.
__device__ __forceinline__ void grid_wait() { asm volatile("griddepcontrol.wait;" ::: "memory"); }
__device__ __forceinline__ void grid_signal() { asm volatile("griddepcontrol.launch_dependents;" ::: "memory"); }
__device__ __forceinline__ void bar_sync(int id, int n) { asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(n) : "memory"); }
__device__ __forceinline__ void bar_arrive(int id, int n) {
  __threadfence_block();
  asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(n) : "memory");
}
// The chain's barriers: its tiles written (1), and on to the reducing warps
// (2: H2 and dY, 3: dZ2, 4: dZ1).
__device__ __forceinline__ void chain_sync() {
  fence_before_sync();
  fence_async_smem();
  bar_sync(1, kChain);
}

// Half a row of a K = 64 row tile (units 32 half .. 32 half + 31), 16 B stores.
__device__ __forceinline__ void store_half(uint8_t* tile, int r, int half, const uint32_t* w, uint32_t lbo,
                                           uint32_t sbo) {
  uint8_t* p = tile + (uint32_t)(r >> 3) * sbo + (uint32_t)half * 4u * lbo + (uint32_t)(r & 7) * 16u;
#pragma unroll
  for (int c = 0; c < 4; ++c)
    *reinterpret_cast<uint4*>(p + c * lbo) = make_uint4(w[4 * c], w[4 * c + 1], w[4 * c + 2], w[4 * c + 3]);
}

// Rows r0 .. r0 + 2n - 1 of column m of a transposed K = 128 tile from n BF16
// pairs: neighbouring lanes swap, so that each stores one row of two columns.
template <int N>
__device__ __forceinline__ void store_cols(uint8_t* tile, int m, int r0, const uint32_t* w) {
  const bool odd = m & 1;
  uint8_t* p = tile + tile_off(r0 + (odd ? 1 : 0), m & ~1, kTLbo, kTSbo);
#pragma unroll
  for (int i = 0; i < N; ++i) {
    const uint32_t other = __shfl_xor_sync(0xffffffffu, w[i], 1);
    const uint32_t v = odd ? __byte_perm(other, w[i], 0x7632) : __byte_perm(w[i], other, 0x5410);
    *reinterpret_cast<uint32_t*>(p + (uint32_t)((2 * i) >> 3) * kTSbo + (uint32_t)((2 * i) & 7) * 16u) = v;
  }
}

// One tile of 128 points: forward, MSE loss gradient, backward; writes this
// CTA's gradient of every parameter (and its loss) to partials[blockIdx.x].
//   L = 1/(2 count) * sum_points sum_o (y_o - t_o)^2
// Weight gradients of layers 1 and 2 come from one M=128 N=128 K=128 MMA of
//   A = [dZ2^T ; dZ1^T]  (128 x points)  and  B = [H1^T ; X^T ; 0]  (128 x points),
// whose diagonal 64x64 blocks are dW2 and dW1 (the off-diagonal blocks are
// discarded).  dW3 and the biases are reduced on the CUDA cores, in the order
// of the points.  step (if given) counts the update that follows this launch.
__global__ void __launch_bounds__(kTrain, 1) k_mlp_train(const uint8_t* __restrict__ packed,
                                                         const float* __restrict__ x, const float* __restrict__ t,
                                                         const int* __restrict__ idx, int n, float inv_count,
                                                         float* __restrict__ partials, int* step, int* err) {
  extern __shared__ __align__(1024) uint8_t sm[];
  uint8_t* w = sm;
  uint8_t* xt = w + kPkBytes;
  uint8_t* h1 = xt + kRowTile;
  uint8_t* dz2 = h1 + kRowTile;
  uint8_t* h2 = dz2 + kRowTile;
  uint8_t* dyt = h2 + kHTile;
  uint8_t* at = dyt + kRow16Tile;
  uint8_t* bt = at + kTTile;
  float* dyf = reinterpret_cast<float*>(bt + kTTile);  // dY in FP32, 128 x 2
  float* lossw = dyf + 256;                            // loss of each warp of points
  uint64_t* bar = reinterpret_cast<uint64_t*>(lossw + 4);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bar + 1);
  const int tid = threadIdx.x;
  const int r = tid & 127, half = tid >> 7;  // chain: point of the tile, half of its units
  const int slot = blockIdx.x * 128 + r;
  const bool valid = slot < n;

  // ---- what no earlier launch of the epoch writes
  if (tid < 32) tmem_alloc(tslot, 128);
  if (tid == 0) {
    mbar_init(bar, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  float tgt0 = 0.0f, tgt1 = 0.0f;
  if (tid < kChain) {
    const int p = valid ? idx[slot] : 0;
    float v[24];
    const float* xp = x + (size_t)p * 48 + 24 * half;
    if (!valid) {
#pragma unroll
      for (int k = 0; k < 24; ++k) v[k] = 0.0f;
    } else if ((reinterpret_cast<uintptr_t>(x) & 15u) == 0) {  // a caller's own features may lie at any float
#pragma unroll
      for (int k = 0; k < 6; ++k) reinterpret_cast<float4*>(v)[k] = __ldg(reinterpret_cast<const float4*>(xp) + k);
    } else {
#pragma unroll
      for (int k = 0; k < 24; ++k) v[k] = __ldg(xp + k);
    }
    if (valid && half == 0) {
      tgt0 = __ldg(t + 2 * (size_t)p);
      tgt1 = __ldg(t + 2 * (size_t)p + 1);
    }
    uint32_t q[12];
#pragma unroll
    for (int k = 0; k < 12; ++k) q[k] = pack_bf16(v[2 * k], v[2 * k + 1]);
    uint8_t* row = xt + (uint32_t)(r >> 3) * kRowSbo + (uint32_t)(r & 7) * 16u;
#pragma unroll
    for (int c = 0; c < 3; ++c)
      *reinterpret_cast<uint4*>(row + (3 * half + c) * 128) =
          make_uint4(q[4 * c], q[4 * c + 1], q[4 * c + 2], q[4 * c + 3]);
    *reinterpret_cast<uint4*>(row + (6 + half) * 128) = make_uint4(0, 0, 0, 0);  // features 48..63
    store_cols<12>(bt, r, 64 + 24 * half, q);
  } else {
    // rows 112..127 of B (past the 48 input features) are zero
    for (int i = r; i < (int)(2 * kTSbo / 16); i += 128)
      reinterpret_cast<uint4*>(bt + 14 * kTSbo)[i] = make_uint4(0, 0, 0, 0);
  }

  // ---- the weights
  grid_wait();
  for (int i = tid; i < (int)(kPkBytes / 16); i += kTrain)
    reinterpret_cast<uint4*>(w)[i] = __ldcg(reinterpret_cast<const uint4*>(packed) + i);
  if (step && blockIdx.x == 0 && tid == 0) *step += 1;  // read by the update, which waits for this launch
  grid_signal();
  fence_before_sync();
  fence_async_smem();
  __syncthreads();
  const uint32_t tmem = *tslot;
  const float* bias = reinterpret_cast<const float*>(w + kPkBias);
  float* part = partials + (size_t)blockIdx.x * kMlpPitch;
  bool ok = true;

  if (tid < kChain) {
    uint32_t phase = 0u;
    const uint32_t lane = (uint32_t)(r & ~31), col = 32u * (uint32_t)half;
    const float* b1 = bias + 32 * half;
    const float* b2 = bias + 64 + 32 * half;
    float v[32];
    uint32_t q[16], mask1 = 0u, mask2 = 0u;
    // ---- layer 1
    if (tid == 0) {
      fence_after_sync();
      issue_k64(tmem, xt, w + kPkW1, idesc_bf16(128, 64));
    }
    ok &= complete(bar, phase);
    tmem_ld32(taddr(tmem, lane, col), v);
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      v[j] += b1[j];
      if (v[j] > 0.0f) mask1 |= 1u << j;
      v[j] = fmaxf(v[j], 0.0f);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) q[j] = pack_bf16(v[2 * j], v[2 * j + 1]);
    store_half(h1, r, half, q, 128u, kRowSbo);
    chain_sync();
    // ---- layer 2 (H1^T, an operand of the weight gradients, is stored while it runs)
    if (tid == 0) {
      fence_after_sync();
      issue_k64(tmem + 64, h1, w + kPkW2, idesc_bf16(128, 64));
      commit(bar);
    }
    store_cols<16>(bt, r, 32 * half, q);
    ok &= complete(bar, phase, false);
    tmem_ld32(taddr(tmem, lane, 64u + col), v);
#pragma unroll
    for (int j = 0; j < 32; ++j) {
      v[j] += b2[j];
      if (v[j] > 0.0f) mask2 |= 1u << j;
      v[j] = fmaxf(v[j], 0.0f);
    }
#pragma unroll
    for (int j = 0; j < 16; ++j) q[j] = pack_bf16(v[2 * j], v[2 * j + 1]);
    store_half(h2, r, half, q, kHLbo, kHSbo);
    chain_sync();
    // ---- layer 3 + loss
    if (tid == 0) {
      fence_after_sync();
#pragma unroll
      for (int kb = 0; kb < 4; ++kb)
        mma_bf16(tmem, sdesc(smem_u32(h2) + kb * 2u * kHLbo, kHLbo, kHSbo),
                 sdesc(smem_u32(w + kPkW3) + kb * 256u, 128u, kRowSbo), idesc_bf16(128, 16), kb > 0);
    }
    ok &= complete(bar, phase);
    if (half == 0) {
      float o[16];
      tmem_ld16(taddr(tmem, lane, 0), o);
      float y0 = o[0] + bias[128], y1 = o[1] + bias[129];
      float e0 = valid ? (y0 - tgt0) : 0.0f, e1 = valid ? (y1 - tgt1) : 0.0f;
      float dy0 = e0 * inv_count, dy1 = e1 * inv_count;
      dyf[2 * r] = dy0;
      dyf[2 * r + 1] = dy1;
      // dY row (K = 16: two values and zero padding)
      uint32_t w0 = (uint32_t)to_bf16(dy0) | ((uint32_t)to_bf16(dy1) << 16);
      uint8_t* rowp = dyt + (uint32_t)(r >> 3) * kRow16Sbo + (uint32_t)(r & 7) * 16u;
      *reinterpret_cast<uint4*>(rowp) = make_uint4(w0, 0, 0, 0);
      *reinterpret_cast<uint4*>(rowp + 128) = make_uint4(0, 0, 0, 0);
      float loss = 0.5f * (e0 * e0 + e1 * e1) * inv_count;
      for (int off = 16; off > 0; off >>= 1) loss += __shfl_down_sync(0xffffffffu, loss, off);
      if ((r & 31) == 0) lossw[r >> 5] = loss;
    }
    chain_sync();
    bar_arrive(2, kTrain);
    // ---- dH2 = dY W3  (K = 16)
    if (tid == 0) {
      fence_after_sync();
      mma_bf16(tmem, sdesc(smem_u32(dyt), 128u, kRow16Sbo), sdesc(smem_u32(w + kPkW3T), 128u, kRow16Sbo),
               idesc_bf16(128, 64), 0u);
    }
    ok &= complete(bar, phase);
    tmem_ld32(taddr(tmem, lane, col), v);
#pragma unroll
    for (int j = 0; j < 16; ++j)
      q[j] = pack_bf16((mask2 >> (2 * j)) & 1u ? v[2 * j] : 0.0f, (mask2 >> (2 * j + 1)) & 1u ? v[2 * j + 1] : 0.0f);
    store_half(dz2, r, half, q, 128u, kRowSbo);
    chain_sync();
    // ---- dH1 = dZ2 W2
    if (tid == 0) {
      fence_after_sync();
      issue_k64(tmem + 64, dz2, w + kPkW2T, idesc_bf16(128, 64));
      commit(bar);
    }
    store_cols<16>(at, r, 32 * half, q);
    bar_arrive(3, kTrain);
    ok &= complete(bar, phase, false);
    tmem_ld32(taddr(tmem, lane, 64u + col), v);
#pragma unroll
    for (int j = 0; j < 16; ++j)
      q[j] = pack_bf16((mask1 >> (2 * j)) & 1u ? v[2 * j] : 0.0f, (mask1 >> (2 * j + 1)) & 1u ? v[2 * j + 1] : 0.0f);
    store_cols<16>(at, r, 64 + 32 * half, q);
    chain_sync();
    bar_arrive(4, kTrain);
    // ---- [dW2 | dW1] = A B^T over the 128 points (K = 128)
    if (tid == 0) {
      fence_after_sync();
#pragma unroll
      for (int kb = 0; kb < 8; ++kb)
        mma_bf16(tmem, sdesc(smem_u32(at) + kb * 2u * kTLbo, kTLbo, kTSbo),
                 sdesc(smem_u32(bt) + kb * 2u * kTLbo, kTLbo, kTSbo), idesc_bf16(128, 128), kb > 0);
    }
    ok &= complete(bar, phase);
    if (r < 64) {  // row j = r: dW2[j][0..63]
      tmem_ld32(taddr(tmem, lane, col), v);
      float4* d = reinterpret_cast<float4*>(part + kOffW2 + r * 64 + 32 * half);
#pragma unroll
      for (int i = 0; i < 8; ++i) d[i] = reinterpret_cast<const float4*>(v)[i];
    } else {  // row 64 + j: dW1[j][0..47]
      tmem_ld32(taddr(tmem, lane, 64u + col), v);
      float4* d = reinterpret_cast<float4*>(part + kOffW1 + (r - 64) * 48 + 32 * half);
#pragma unroll
      for (int i = 0; i < 8; ++i)
        if (i < 4 || half == 0) d[i] = reinterpret_cast<const float4*>(v)[i];
    }
  } else {
    // ---- reductions over the 128 points: dW3, db3, db2, db1
    const int oo = r >> 6, j = r & 63;
    bar_sync(2, kTrain);
    float acc = 0.0f;
#pragma unroll 16
    for (int m = 0; m < 128; ++m)
      acc = fmaf(dyf[2 * m + oo], from_bf16(*reinterpret_cast<const uint16_t*>(h2 + tile_off(m, j, kHLbo, kHSbo))),
                 acc);
    part[kOffW3 + oo * 64 + j] = acc;
    if (r < 2) {
      float sy = 0.0f;
      for (int m = 0; m < 128; ++m) sy += dyf[2 * m + r];
      part[kOffB3 + r] = sy;
    }
    if (r == 0) part[kMlpParams] = lossw[0] + lossw[1] + lossw[2] + lossw[3];
    // db2 from dZ2^T (rows 0..63), db1 from dZ1^T (rows 64..127)
    bar_sync(3, kTrain);
    if (r >= 64) bar_sync(4, kTrain);
    float sb = 0.0f;
#pragma unroll
    for (int c = 0; c < 16; ++c) {
      const uint4 u = *reinterpret_cast<const uint4*>(at + tile_off(r, 8 * c, kTLbo, kTSbo));
      const uint32_t a[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
      for (int i = 0; i < 4; ++i) {
        sb += __uint_as_float(a[i] << 16);
        sb += __uint_as_float(a[i] & 0xffff0000u);
      }
    }
    if (r < 64) bar_sync(4, kTrain);
    part[(r < 64 ? kOffB2 : kOffB1 - 64) + r] = sb;
  }
  if (!ok) atomicExch(err, 1);
  mlp_cta_end(tmem);
}

// A launch of an epoch that may start while the one in front of it runs.
template <class... K, class... A>
static cudaError_t launch_behind(void (*k)(K...), unsigned grid, unsigned block, size_t smem, bool behind,
                                 cudaStream_t st, A... a) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3(grid);
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute at = {};
  at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
  at.val.programmaticStreamSerializationAllowed = 1;
  cfg.attrs = &at;
  cfg.numAttrs = behind ? 1 : 0;
  return cudaLaunchKernelEx(&cfg, k, static_cast<K>(a)...);
}

cudaError_t launch_mlp_train_tiles(const uint8_t* packed, const float* x, const float* t, const int* idx, int n,
                                   float inv_count, float* partials, int* step, int* err, bool behind,
                                   cudaStream_t st) {
  cudaError_t e = cudaFuncSetAttribute(k_mlp_train, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrainSmem);
  if (e != cudaSuccess) return e;
  if (n <= 0) return cudaSuccess;
  return launch_behind(k_mlp_train, (unsigned)((n + 127) / 128), kTrain, kTrainSmem, behind, st, packed, x, t, idx, n,
                       inv_count, partials, step, err);
}

// ---------------------------------------------------------------- Adam
// The packed values of parameter p (k_mlp_pack's layout; the padding is never written).
__device__ __forceinline__ void pack_param(int p, float v, uint8_t* pk) {
  const uint16_t h = to_bf16(v);
  auto put = [&](uint32_t off) { *reinterpret_cast<uint16_t*>(pk + off) = h; };
  if (p < kOffB1) {
    put(kPkW1 + tile_off(p / 48, p % 48, 128, kRowSbo));
  } else if (p >= kOffW2 && p < kOffB2) {
    const int o = (p - kOffW2) / 64, k = (p - kOffW2) % 64;
    put(kPkW2 + tile_off(o, k, 128, kRowSbo));
    put(kPkW2T + tile_off(k, o, 128, kRowSbo));
  } else if (p >= kOffW3 && p < kOffB3) {
    const int o = (p - kOffW3) / 64, k = (p - kOffW3) % 64;
    put(kPkW3 + tile_off(o, k, 128, kRowSbo));
    put(kPkW3T + tile_off(k, o, 128, kRow16Sbo));
  } else {
    const int b = p < kOffW2 ? p - kOffB1 : (p < kOffW3 ? 64 + p - kOffB2 : 128 + p - kOffB3);
    reinterpret_cast<float*>(pk + kPkBias)[b] = v;
  }
}

// Thread p sums the per-CTA partials of parameter p in their order (slot
// kMlpParams is the loss), applies one Adam step and writes the parameter's
// packed values; lr <= 0 only reduces (gradient check).  Bound by the latency
// of its loads: 16 partials are in flight per thread, small CTAs spread the
// 7427 threads over the chip.
constexpr int kAdamThreads = 64;
__global__ void __launch_bounds__(kAdamThreads) k_mlp_adam(float* __restrict__ params, float* __restrict__ m,
                                                           float* __restrict__ v, uint8_t* __restrict__ packed,
                                                           float* __restrict__ loss_acc,
                                                           const float* __restrict__ partials, int n_parts, float lr,
                                                           float b1, float b2, float eps, const int* step_dev,
                                                           float* __restrict__ grad_out) {
  grid_signal();
  grid_wait();
  int p = blockIdx.x * blockDim.x + threadIdx.x;
  if (p > kMlpParams) return;
  const int step = step_dev ? __ldcg(step_dev) : 1;  // 1-based step of this update
  const bool update = p < kMlpParams && lr > 0.0f;
  const float p0 = update ? __ldcg(params + p) : 0.0f;
  const float m0 = update ? __ldcg(m + p) : 0.0f, v0 = update ? __ldcg(v + p) : 0.0f;
  const float* q = partials + p;
  float g = 0.0f;
  int c = 0;
  for (; c + 16 <= n_parts; c += 16) {
    float a[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) a[i] = __ldcg(q + (size_t)(c + i) * kMlpPitch);
#pragma unroll
    for (int i = 0; i < 16; ++i) g += a[i];
  }
  for (; c < n_parts; ++c) g += __ldcg(q + (size_t)c * kMlpPitch);
  if (grad_out) grad_out[p] = g;
  if (p == kMlpParams && loss_acc) *loss_acc += g;
  if (!update) return;
  // the roundings are spelled out: which product of each sum is fused shows in
  // the weights after a few steps
  const float mm = fmaf(1.0f - b1, g, __fmul_rn(b1, m0));
  const float vv = fmaf(__fmul_rn(1.0f - b2, g), g, __fmul_rn(b2, v0));
  m[p] = mm;
  v[p] = vv;
  float mh = mm / (1.0f - powf(b1, (float)step));
  float vh = vv / (1.0f - powf(b2, (float)step));
  const float pn = p0 - lr * mh / (sqrtf(vh) + eps);
  params[p] = pn;
  if (packed) pack_param(p, pn, packed);
}

cudaError_t launch_mlp_adam(float* params, float* m, float* v, uint8_t* packed, float* loss_acc, const float* partials,
                            int n_parts, float lr, float beta1, float beta2, float eps, const int* step_dev,
                            float* grad_out, bool behind, cudaStream_t st) {
  return launch_behind(k_mlp_adam, (unsigned)(kMlpParams + kAdamThreads) / kAdamThreads, kAdamThreads, 0, behind, st,
                       params, m, v, packed, loss_acc, partials, n_parts, lr, beta1, beta2, eps, step_dev, grad_out);
}

}  // namespace cvr
