// deferred.cuh — deferred shading of a frame: its samples' light terms
// evaluated by one thread per sample instead of one thread per ray.
//
// Shading changes a sample's colour, never its opacity, so which samples a
// ray shades and where it stops is known without the light integrals.  A
// direct marcher runs them one after another along each ray: a ray through
// the whole volume is a chain of hundreds of samples times hundreds of light
// steps, and the frame lasts as long as its longest rays (ground truth, 256^3:
// 47 ms at 256^2, 73 ms at 512^2, for a quarter of the work).  Here
//   collect  marches the opacity alone and appends every shaded sample
//            (position, pixel) to a list;
//   light    takes the list, 32 samples of one ray tile and step to a warp,
//            from a cursor: full warps, no chain longer than one sample;
//   resolve  marches again with the colours and composites each sample with
//            its light terms, in ray order.
// The arithmetic of a sample and the order of a ray's composites are the
// direct marcher's, so the image is too, bit for bit.
//
// A warp's records are numbered in the order of its steps (ranks of a ballot
// within a step) and stored in chunks of kRecChunk, taken from one counter when a
// chunk fills; chunk[w][i] is where the i-th chunk of warp w lies.
#pragma once

#include "shade.cuh"

namespace cvr {

struct Deferred {
  float4* rec;        // position, pixel (as int bits; -1: an unused slot)
  float2* light;      // (occlusion, shadow) of record i
  unsigned* chunk;    // [warps of the band][chunks]: first record
  unsigned* counter;  // [0] records handed out, [1] light's cursor (zeroed before collect)
  unsigned chunks;    // chunks a warp may need
  unsigned y0;        // first tile row of the band
};
constexpr unsigned kRecChunk = 256;
constexpr unsigned kBoxBands = 4;    // most bands of a deferred box-table frame
constexpr unsigned kLightGrab = 64;  // records a warp takes at a time

// The light terms of every record, by persistent warps.
template <class Shade>
__device__ __forceinline__ void light_samples(const FrameArgs& f, const Deferred& d, const Shade& sh) {
  const unsigned total = *d.counter;
  const int lane = threadIdx.x & 31;
  unsigned long long aux = 0;
  for (;;) {
    unsigned at = 0;
    if (lane == 0) at = atomicAdd(d.counter + 1, kLightGrab);
    at = __shfl_sync(0xffffffffu, at, 0);
    if (at >= total) break;
    for (unsigned i = at + lane; i < at + kLightGrab; i += 32) {
      // an unused slot takes the pixel and the place of a neutral sample, so
      // that the warp stays whole through the light terms
      const float4 r = d.rec[i];
      const int pixel = __float_as_int(r.w);
      const bool used = pixel >= 0;
      const int at_pixel = used ? pixel : 0;
      const float3 p = used ? f3(r.x, r.y, r.z) : f.vol.grid * 0.5f;
      typename Shade::Ray ray;
      sh.begin(ray, primary_dir(f.cam, at_pixel % f.W, at_pixel / f.W, f.W, f.H));
      unsigned a = 0;
      const float2 l = sh.light(p, ray, f, a);
      if (used) {
        d.light[i] = l;
        aux += a;
      }
    }
  }
  if (f.stats) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) aux += __shfl_down_sync(0xffffffffu, aux, o);
    if (lane == 0) atomicAdd(f.stats + 2, aux);
  }
}

// A frame's bands (of 'rows' tile rows), the chunks a warp may need, and the
// lists of a band: 'bytes' of memory, at most limit, its records at the end.
// false: not one row fits (its rays have too many steps).
struct DeferredPlan {
  unsigned chunks, rows, bands;
  size_t records, bytes;
};
bool deferred_plan(const FrameArgs& f, size_t limit, DeferredPlan* p);
cudaError_t launch_collect(const FrameArgs& f, const Deferred& d, unsigned rows, cudaStream_t st);
// A kernel's code is loaded at its first use (0.1 to 0.4 ms each): loaded ahead
// of a frame that is timed.
cudaError_t load_deferred(const FrameArgs& f);
cudaError_t load_light_gt(const FrameArgs& f);
// ext: the extinction renderer's gradient branch; taps: secondary lookups per
// shaded sample to count (0: the light pass counts its own).
cudaError_t launch_resolve(const FrameArgs& f, const Deferred& d, unsigned rows, const LightTerms& t, bool ext,
                           unsigned taps, cudaStream_t st);

// occ, sdw: host copies of the section tables.
cudaError_t launch_light_dos(const FrameArgs& f, const DosArgs& a, const float4* occ, const float4* sdw, bool tex,
                             const Deferred& d, cudaStream_t st);
// table, storage as launch_extinction.
cudaError_t launch_light_ext(const FrameArgs& f, const ExtArgs& e, const ShadowBoxTable* table,
                             const ShadowBoxTable& storage, const Deferred& d, cudaStream_t st);
cudaError_t launch_light_box(const FrameArgs& f, const ExtArgs& e, const BoxWalk& w, const Deferred& d, cudaStream_t st);
cudaError_t launch_light_gt(const FrameArgs& f, const GtArgs& g, const Deferred& d, cudaStream_t st);

}  // namespace cvr
