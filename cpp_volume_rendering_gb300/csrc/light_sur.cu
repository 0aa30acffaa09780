// light_sur.cu — the surrogate's light terms of a frame's collected samples
// (deferred.cuh): the network's inputs and its three layers on the tensor
// cores, 128 records to a tile.
#include "deferred.cuh"
#include "march_ext.cuh"
#include "surrogate.cuh"
#include "tile_sink.cuh"

namespace cvr {

// One CTA a SM of NG groups of 128 threads, each with its own tile, TMEM
// columns, mbarrier and named barrier: a group's texture fetches run while
// another's layers do.  The groups share one copy of the weights (19 KB), so
// the SM keeps more L1 for the pyramid's texels than with a CTA per tile.
// Bound by the texture pipe (67 trilinear 3D fetches a sample).  8 groups (64
// registers, all 512 TMEM columns): 320^3 -> 720^2 10.1 ms through the texture
// unit, 17.1 with FP32 taps; 6 groups 10.5 and 19.7, 4 groups 11.8 and 27.3;
// the direct marcher 14.0 and 35.2 (128^3 -> 256^2: 0.68 against 1.60 ms).
constexpr int kSurGroups = 8;
template <bool TEX, int NG>
__global__ void __launch_bounds__(128 * NG, 1) k_light_sur(const __grid_constant__ FrameArgs f,
                                                           const __grid_constant__ SurArgs a,
                                                           const __grid_constant__ Deferred d, int* err) {
  constexpr uint32_t kCols = NG > 4 ? 512 : (NG > 2 ? 256 : 128);
  extern __shared__ __align__(1024) uint8_t sm_sur[];
  uint8_t* w = sm_sur;
  uint8_t* tiles = w + kPkFwdBytes;
  uint64_t* bars = reinterpret_cast<uint64_t*>(tiles + NG * kRowTile);
  uint32_t* tslot = reinterpret_cast<uint32_t*>(bars + NG);
  volatile unsigned* grab = tslot + 1;     // first record of each group's tile
  volatile unsigned* gave_up = grab + NG;  // a group whose tensor-core wait ran out
  mlp_cta_begin(w, a.packed, bars, tslot, kCols, kPkFwdBytes, NG);
  if (threadIdx.x < NG) gave_up[threadIdx.x] = 0;
  fence_async_smem();
  __syncthreads();
  const int g = threadIdx.x >> 7;
  const TileGroup tile{1 + g};
  const int tid = tile.tid();
  uint8_t* xt = tiles + g * kRowTile;
  MlpSmem ms{w, xt, xt, bars + g, *tslot + 64u * (uint32_t)g, 0u};
  const unsigned total = *d.counter;
  for (;;) {
    if (tid == 0) grab[g] = atomicAdd(d.counter + 1, 128u);
    tile.sync();
    const unsigned at = grab[g];
    if (at >= total || gave_up[g]) break;
    const unsigned i = at + (unsigned)tid;
    const float4 r = d.rec[i];
    const int pixel = __float_as_int(r.w);
    const bool used = pixel >= 0;
    // rows of unused slots keep whatever the tile holds: a row's outputs
    // depend on that row alone
    if (used) {
      TileSink out{xt, tid};
      sur_features<TEX>(a, f.vol, nullptr, 0, f3(r.x, r.y, r.z), primary_dir(f.cam, pixel % f.W, pixel / f.W, f.W, f.H),
                        out);
    }
    store_chunk(xt, tid, 6, 0u, 0u, 0u, 0u);
    store_chunk(xt, tid, 7, 0u, 0u, 0u, 0u);
    sync_tiles(tile);
    float y[2];
    if (!mlp_forward_tile(ms, y, tile)) {
      gave_up[g] = 1;
      atomicExch(err, 1);
    }
    // sur_shade's light terms
    if (used)
      d.light[i] = make_float2(fminf(fmaxf(y[0], 0.0f), 1.0f),
                               a.shadow_type == 1 ? 0.0f : fminf(fmaxf(y[1], 0.0f), 1.0f));
  }
  mlp_cta_end(*tslot, kCols);
}

template <bool TEX>
static cudaError_t launch_light_sur_t(const FrameArgs& f, const SurArgs& a, const Deferred& d, int* err,
                                      cudaStream_t st) {
  constexpr int NG = kSurGroups;
  const size_t smem = kPkFwdBytes + NG * kRowTile + NG * sizeof(uint64_t) + (1 + 2 * NG) * sizeof(unsigned);
  auto kern = k_light_sur<TEX, NG>;
  cudaError_t e = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess) e = carve_l1(kern, 128 * NG, smem);
  int dev = 0, sms = 0;
  if (e == cudaSuccess) e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) return e;
  kern<<<sms, 128 * NG, smem, st>>>(f, a, d, err);
  return cudaGetLastError();
}

cudaError_t launch_light_sur(const FrameArgs& f, const SurArgs& a, bool tex, const Deferred& d, int* err,
                             cudaStream_t st) {
  return tex ? launch_light_sur_t<true>(f, a, d, err, st) : launch_light_sur_t<false>(f, a, d, err, st);
}

cudaError_t load_light_sur(bool tex) {
  cudaFuncAttributes a;
  return cudaFuncGetAttributes(&a, tex ? k_light_sur<true, kSurGroups> : k_light_sur<false, kSurGroups>);
}

}  // namespace cvr
