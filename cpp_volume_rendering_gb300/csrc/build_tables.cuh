// build_tables.cuh — launchers of the SAT / pyramid builders and utilities.
#pragma once

#include "cvr_device.cuh"

namespace cvr {

// Builds the (nx+2)(ny+2)(nz+2) int64 SAT of lut[voxel] with a zero border.
cudaError_t launch_sat_build(const void* vox, int dtype, int nx, int ny, int nz, const long long* lut,
                             long long* sat, cudaStream_t st);
// The compact table: the same prefix sums of a 32-bit lut, wrapping modulo
// 2^32, in the x-y predecessor-quad layout (SatView::sat32) in out;
// scratch holds (nx+2)(ny+2)(nz+2) 32-bit values (the plane prefixes).
cudaError_t launch_sat_build_quads(const void* vox, int dtype, int nx, int ny, int nz, const unsigned* lut,
                                   unsigned* scratch, uint4* out, cudaStream_t st);
// The walk table of a directional shadow cone (WalkView: 32 bytes per cell)
// along axis, box depth w, from the compact predecessor-quad table.
cudaError_t launch_sat_walk(const uint4* quads, uint4* out, int sx, int sy, int sz, int axis, int w,
                            cudaStream_t st);
// The x-y predecessor-quad layout of a finished plain (sx, sy, sz) table.
cudaError_t launch_sat_quads(const unsigned* sat, uint4* out, int sx, int sy, int sz, cudaStream_t st);

// The plain 32-bit table (prefix sums of a 32-bit lut modulo 2^32, x fastest)
// in out: the source of a compact frame's box tables.
cudaError_t launch_sat_build32(const void* vox, int dtype, int nx, int ny, int nz, const unsigned* lut, unsigned* out,
                               cudaStream_t st);

// One box table (BoxView): its grid and first cell; per table axis (fastest,
// middle, slowest) the SAT axis it runs along, the box width and the pad.
struct BoxTableDesc {
  BoxGrid g;
  unsigned cell;
  int axis[3], w[3], pad[3];
};
constexpr int kMaxBoxTables = 96;
struct BoxTableSet {
  int n;
  BoxTableDesc t[kMaxBoxTables];
};
// The prefix sums the tables are differences of: the int64 table (s64), or a
// 32-bit one, element i at s32[i * stride + first] (the plain table: 1, 0; the
// predecessor quads: 4, 3).  scale: 2^-F of its fixed point.
struct BoxSource {
  const long long* s64;
  const unsigned* s32;
  int stride, first;
  float scale;
  int n[3];  // SAT extents
};
// Whether a table of this grid fits the build's launches.
bool box_table_builds(const BoxGrid& g);
cudaError_t launch_box_tables(const BoxSource& src, const BoxTableSet& set, float* out, cudaStream_t st);

// Builds every level of P (dims/offsets/grid filled by the caller) into data,
// their opacities into opacity (as many floats; nullptr: none to spare, and the
// extinctions are converted in place at the end).  vol: the marchers' storage
// of the volume, plain: the x-fastest array.  lattice: room for
// pyramid_lattice_floats, or nullptr (the levels that would use it take slower
// forms).
cudaError_t launch_pyramid_build(const VolumeView& vol, const VolumeView& plain, const float4* tf_rgba, int tf_n,
                                 float s0, PyramidView& P, float* data, float* opacity, float* lattice,
                                 cudaStream_t st);
long long pyramid_lattice_floats(const VolumeView& plain, const PyramidView& P, float s0);

// Grid-stride fill of a device buffer (used to flush L2 between timed frames).
cudaError_t launch_fill(void* p, size_t bytes, unsigned int v, cudaStream_t st);
// The x-y quad copy of every pyramid level (float4 per value, at P.qoff with
// pitches quad_row, quad_plane).
cudaError_t launch_pyramid_quads(const PyramidView& P, const float* data, float4* dst, cudaStream_t st);
// The x-y quad copy of a plain volume (uchar4 / ushort4 per voxel), rows of
// qrow and planes of qplane cells.
cudaError_t launch_quad_volume(const void* src, void* dst, int dtype, int nx, int ny, int nz, unsigned qrow,
                               unsigned qplane, cudaStream_t st);
// Bricked copy of a plain volume (bricks of 2^bs voxels per edge); the copy
// holds brick_elements(...) elements.
long long brick_elements(int nx, int ny, int nz, int bs);
cudaError_t launch_brick_volume(const void* src, void* dst, int dtype, int nx, int ny, int nz, int bs,
                                cudaStream_t st);

}  // namespace cvr
