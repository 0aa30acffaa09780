// build_tables.cu — device builders for the two illumination tables:
//  * the extinction summed-area table of RC1PExtinctionBasedShading
//    (GenerateExtinctionSAT3DTex, ebsrenderer.cpp:624-723, and
//    SummedAreaTable3D<double>::BuildSAT, libs/vis_utils/summedareatable.h:218-280),
//  * the Gaussian extinction mip pyramid of RC1PConeTracingDirOcclusionShading
//    (ExtinctionCoefficientVolume::GenerateExtinctionCoefficientVolumeAnySize,
//    extcoefvolumegenerator.cpp:230-408, gen_extcoefvol_anysize*.comp, backtotau.comp).
#include "build_tables.cuh"
#include "sampler.cuh"

#include <algorithm>
#include <cmath>

namespace cvr {

// ------------------------------------------------------------------ SAT
// Pass 1: fill + x-scan.  One warp per SAT row (y, z).  Interior cells take
// lut[voxel(x-1, y-1, z-1)] (the extinction of that voxel value in fixed
// point); the one-cell border is zero (ebsrenderer.cpp:651-659).
// W: long long (exact int64 prefix sums) or unsigned (sums modulo 2^32).
template <class W>
__global__ void k_sat_fill_xscan(const void* vox, int dtype, int nx, int ny, int nz,
                                 const W* __restrict__ lut, W* __restrict__ sat) {
  const int sx = nx + 2, sy = ny + 2, sz = nz + 2;
  int warp = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  int lane = threadIdx.x & 31;
  if (warp >= sy * sz) return;
  int y = warp % sy, z = warp / sy;
  W* row = sat + ((size_t)z * sy + y) * (size_t)sx;
  bool border_row = (y == 0 || z == 0 || y == sy - 1 || z == sz - 1);
  size_t vrow = border_row ? 0 : ((size_t)(z - 1) * ny + (y - 1)) * (size_t)nx;
  W carry = 0;
  for (int base = 0; base < sx; base += 32) {
    int x = base + lane;
    W v = 0;
    if (!border_row && x > 0 && x < sx - 1) {
      unsigned int q = (dtype == 1) ? (unsigned int)__ldg(static_cast<const uint8_t*>(vox) + vrow + (x - 1))
                                    : (unsigned int)__ldg(static_cast<const uint16_t*>(vox) + vrow + (x - 1));
      v = __ldg(lut + q);
    }
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
      W n = __shfl_up_sync(0xffffffffu, v, o);
      if (lane >= o) v += n;
    }
    v += carry;
    if (x < sx) row[x] = v;
    carry = __shfl_sync(0xffffffffu, v, 31);
  }
}

// Pass 2 / 3: inclusive scan along y (stride sx) or z (stride sx*sy).  One
// thread per line; consecutive threads own consecutive x, so every step is a
// coalesced 256-byte warp access.
template <class W>
__global__ void k_sat_scan_lines(W* __restrict__ sat, int sx, int n_lines_inner, int n_lines_outer,
                                 size_t line_stride_inner, size_t line_stride_outer, size_t step, int len) {
  int t = blockIdx.x * blockDim.x + threadIdx.x;
  int total = sx * n_lines_inner * n_lines_outer;
  if (t >= total) return;
  int x = t % sx;
  int r = t / sx;
  int a = r % n_lines_inner, b = r / n_lines_inner;
  W* p = sat + (size_t)x + (size_t)a * line_stride_inner + (size_t)b * line_stride_outer;
  W acc = 0;
  int i = 0;
  for (; i + 4 <= len; i += 4) {
    W v0 = p[(size_t)(i + 0) * step], v1 = p[(size_t)(i + 1) * step];
    W v2 = p[(size_t)(i + 2) * step], v3 = p[(size_t)(i + 3) * step];
    acc += v0; p[(size_t)(i + 0) * step] = acc;
    acc += v1; p[(size_t)(i + 1) * step] = acc;
    acc += v2; p[(size_t)(i + 2) * step] = acc;
    acc += v3; p[(size_t)(i + 3) * step] = acc;
  }
  for (; i < len; ++i) {
    acc += p[(size_t)i * step];
    p[(size_t)i * step] = acc;
  }
}

// ---- blocked builder: x-y prefix of every plane in shared memory, then a
// z-scan (in place for the int64 table; fused with the quad layout for the
// compact one).  Two passes over the table instead of three.

// Pass 1: one CTA per z plane, in chunks of R <= kSatChunkRows rows.  Phase A: a
// thread per column (or per few columns) carries the column's running
// y-prefix from chunk to chunk (in shared memory); the voxel loads and table
// lookups of the chunk's rows are issued before the adds, and each row's
// prefix goes to shared memory.  Phase B: a warp per row
// scans it along x (shuffles, carried across 32-cell segments) and writes
// the plane's row out (coalesced).  The y-then-x order gives the same 2D
// prefix sums (integer adds).  Interior cells take lut[voxel(x-1, y-1, z-1)];
// the one-cell border is zero.
constexpr int kSatPlaneThreads = 512;
constexpr int kSatChunkRows = 16;
template <class W>
__global__ void __launch_bounds__(kSatPlaneThreads, 2) k_sat_planes(const void* vox, int dtype, int nx, int ny,
                                                                     int nz, const W* __restrict__ lut,
                                                                     W* __restrict__ out, int R) {
  extern __shared__ __align__(16) unsigned char sm_sat[];
  const int sx = nx + 2, sy = ny + 2, sz = nz + 2;
  W* chunk = reinterpret_cast<W*>(sm_sat);  // R x sx
  W* carry = chunk + (size_t)R * sx;        // sx running column sums
  const int z = blockIdx.x;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, warps = blockDim.x >> 5;
  const bool border_plane = z == 0 || z == sz - 1;
  W* plane = out + (size_t)z * sx * sy;
  for (int x = threadIdx.x; x < sx; x += blockDim.x) carry[x] = 0;
  for (int y0 = 0; y0 < sy; y0 += R) {
    const int rows = min(R, sy - y0);
#pragma unroll 1
    for (int x = threadIdx.x; x < sx; x += blockDim.x) {
      const bool col = !border_plane && x > 0 && x < sx - 1;
      unsigned q[kSatChunkRows];
#pragma unroll
      for (int r = 0; r < kSatChunkRows; ++r) {
        const int y = y0 + r;
        q[r] = 0xffffffffu;
        if (col && r < rows && y > 0 && y < sy - 1) {
          const size_t i = ((size_t)(z - 1) * ny + (y - 1)) * (size_t)nx + (x - 1);
          q[r] = dtype == 1 ? (unsigned)__ldg(static_cast<const uint8_t*>(vox) + i)
                            : (unsigned)__ldg(static_cast<const uint16_t*>(vox) + i);
        }
      }
      W v[kSatChunkRows];
#pragma unroll
      for (int r = 0; r < kSatChunkRows; ++r) v[r] = q[r] != 0xffffffffu ? __ldg(lut + q[r]) : W(0);
      W run = carry[x];
#pragma unroll
      for (int r = 0; r < kSatChunkRows; ++r) {
        if (r >= rows) break;
        run += v[r];
        chunk[(size_t)r * sx + x] = run;
      }
      carry[x] = run;
    }
    __syncthreads();
    for (int r = warp; r < rows; r += warps) {
      W run = 0;
      W* dst = plane + (size_t)(y0 + r) * sx;
      const W* src = chunk + (size_t)r * sx;
      for (int base = 0; base < sx; base += 32) {
        const int x = base + lane;
        W t = x < sx ? src[x] : W(0);
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
          const W n = __shfl_up_sync(0xffffffffu, t, o);
          if (lane >= o) t += n;
        }
        t += run;
        if (x < sx) dst[x] = t;
        run = __shfl_sync(0xffffffffu, t, 31);
      }
    }
    __syncthreads();  // the chunk is read before the next one is written
  }
}

// Pass 2 (int64 table): in-place running sum along z of every (x, y) column,
// a thread per column (coalesced along x), 16 planes loaded before they are
// summed so that enough loads are in flight to stream at HBM rate.
template <class W>
__global__ void __launch_bounds__(256) k_sat_zscan(W* __restrict__ sat, long long columns, int sz) {
  const long long c = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (c >= columns) return;
  W* p = sat + c;
  W run = 0;
  constexpr int B = 16;
  for (int z0 = 0; z0 < sz; z0 += B) {
    W v[B];
#pragma unroll
    for (int k = 0; k < B; ++k) v[k] = z0 + k < sz ? p[(size_t)(z0 + k) * columns] : W(0);
#pragma unroll
    for (int k = 0; k < B; ++k) {
      run += v[k];
      if (z0 + k < sz) p[(size_t)(z0 + k) * columns] = run;
    }
  }
}

// Pass 2 (compact table): the z-scan of 32 x 8 columns and of their low halo
// (x0 - 1, y0 - 1) per CTA, writing the predecessor quads of each plane
// (S at (x-1, y-1), (x, y-1), (x-1, y), (x, y), coordinates clamped to the
// table) from shared-memory tiles of the planes' running sums.  Two groups of
// kQuadGroup tiles alternate, so one barrier serves kQuadGroup planes: a
// group is rewritten only after the barrier that follows the reads of its
// previous planes.
constexpr int kQuadTileX = 32, kQuadTileY = 8, kQuadHaloCols = (kQuadTileX + 1) * (kQuadTileY + 1);
constexpr int kQuadThreads = ((kQuadHaloCols + 31) / 32) * 32;
constexpr int kQuadGroup = 4;
__global__ void __launch_bounds__(kQuadThreads) k_sat_zscan_quads(const unsigned* __restrict__ P, uint4* __restrict__ out,
                                                                  int sx, int sy, int sz) {
  __shared__ unsigned tile[2][kQuadGroup][kQuadTileY + 1][kQuadTileX + 1];
  const int x0 = blockIdx.x * kQuadTileX, y0 = blockIdx.y * kQuadTileY;
  const int t = threadIdx.x;
  const bool owner = t < kQuadHaloCols;
  const int hx = t % (kQuadTileX + 1), hy = t / (kQuadTileX + 1);
  const int gx = min(max(x0 - 1 + hx, 0), sx - 1), gy = min(max(y0 - 1 + hy, 0), sy - 1);
  const size_t sxy = (size_t)sx * sy;
  const unsigned* col = P + (size_t)gy * sx + gx;
  const int lx = t % kQuadTileX, ly = t / kQuadTileX;
  const int ox = x0 + lx, oy = y0 + ly;
  const bool writer = t < kQuadTileX * kQuadTileY && ox < sx && oy < sy;
  uint4* dst = out + (size_t)oy * sx + ox;
  unsigned run = 0;
  constexpr int B = 16;  // planes loaded per round (a multiple of kQuadGroup)
  int grp = 0;
  for (int z0 = 0; z0 < sz; z0 += B) {
    unsigned v[B];
#pragma unroll
    for (int k = 0; k < B; ++k) v[k] = (owner && z0 + k < sz) ? __ldg(col + (size_t)(z0 + k) * sxy) : 0u;
#pragma unroll
    for (int k0 = 0; k0 < B; k0 += kQuadGroup) {
      if (z0 + k0 >= sz) break;
#pragma unroll
      for (int j = 0; j < kQuadGroup; ++j) {
        run += v[k0 + j];
        if (owner) tile[grp][j][hy][hx] = run;
      }
      __syncthreads();
      if (writer) {
#pragma unroll
        for (int j = 0; j < kQuadGroup; ++j) {
          const int z = z0 + k0 + j;
          if (z < sz)
            dst[(size_t)z * sxy] = make_uint4(tile[grp][j][ly][lx], tile[grp][j][ly][lx + 1], tile[grp][j][ly + 1][lx],
                                              tile[grp][j][ly + 1][lx + 1]);
        }
      }
      grp ^= 1;
    }
  }
}

// Rows per chunk of k_sat_planes for rows of sx cells of type W: the chunk
// and the column sums within 200 KB of shared memory (0: fewer than 4 rows
// fit; the line-scan builder below is used).
template <class W>
static int sat_plane_rows(int sx) {
  const long long r = (long long)(200 * 1024 / sizeof(W)) / sx - 1;
  return r >= 4 ? (int)std::min<long long>(r, kSatChunkRows) : 0;
}

template <class W>
static cudaError_t sat_planes(const void* vox, int dtype, int nx, int ny, int nz, const W* lut, W* out, int R,
                              cudaStream_t st) {
  const int sx = nx + 2, sz = nz + 2;
  const size_t smem = sizeof(W) * (size_t)(R + 1) * sx;
  cudaError_t e = cudaFuncSetAttribute(k_sat_planes<W>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  k_sat_planes<W><<<sz, kSatPlaneThreads, smem, st>>>(vox, dtype, nx, ny, nz, lut, out, R);
  return cudaGetLastError();
}

// The previous builder (three passes: fill + x-scan, y-scan, z-scan), kept
// for planes too wide for shared memory.
template <class W>
static cudaError_t sat_build_lines(const void* vox, int dtype, int nx, int ny, int nz, const W* lut, W* sat,
                                   cudaStream_t st) {
  const int sx = nx + 2, sy = ny + 2, sz = nz + 2;
  {
    long long rows = (long long)sy * sz;
    int threads = 256;
    long long blocks = (rows * 32 + threads - 1) / threads;
    k_sat_fill_xscan<W><<<(unsigned)blocks, threads, 0, st>>>(vox, dtype, nx, ny, nz, lut, sat);
  }
  {
    // y-scan: lines indexed by (x, z); stride along y = sx.
    int total = sx * sz;
    k_sat_scan_lines<W><<<(total + 255) / 256, 256, 0, st>>>(sat, sx, 1, sz, 0, (size_t)sx * sy, (size_t)sx, sy);
  }
  {
    // z-scan: lines indexed by (x, y); stride along z = sx*sy.
    int total = sx * sy;
    k_sat_scan_lines<W><<<(total + 255) / 256, 256, 0, st>>>(sat, sx, sy, 1, (size_t)sx, 0, (size_t)sx * sy, sz);
  }
  return cudaGetLastError();
}

cudaError_t launch_sat_build(const void* vox, int dtype, int nx, int ny, int nz, const long long* lut,
                             long long* sat, cudaStream_t st) {
  const int sx = nx + 2, sy = ny + 2, sz = nz + 2;
  const int R = sat_plane_rows<long long>(sx);
  if (R == 0) return sat_build_lines(vox, dtype, nx, ny, nz, lut, sat, st);
  cudaError_t e = sat_planes(vox, dtype, nx, ny, nz, lut, sat, R, st);
  if (e != cudaSuccess) return e;
  const long long columns = (long long)sx * sy;
  k_sat_zscan<long long><<<(unsigned)((columns + 255) / 256), 256, 0, st>>>(sat, columns, sz);
  return cudaGetLastError();
}

cudaError_t launch_sat_build32(const void* vox, int dtype, int nx, int ny, int nz, const unsigned* lut, unsigned* out,
                               cudaStream_t st) {
  const int R = sat_plane_rows<unsigned>(nx + 2);
  if (R == 0) return sat_build_lines(vox, dtype, nx, ny, nz, lut, out, st);
  cudaError_t e = sat_planes(vox, dtype, nx, ny, nz, lut, out, R, st);
  if (e != cudaSuccess) return e;
  const long long columns = (long long)(nx + 2) * (ny + 2);
  k_sat_zscan<unsigned><<<(unsigned)((columns + 255) / 256), 256, 0, st>>>(out, columns, nz + 2);
  return cudaGetLastError();
}

cudaError_t launch_sat_build_quads(const void* vox, int dtype, int nx, int ny, int nz, const unsigned* lut,
                                   unsigned* scratch, uint4* out, cudaStream_t st) {
  const int sx = nx + 2, sy = ny + 2, sz = nz + 2;
  const int R = sat_plane_rows<unsigned>(sx);
  cudaError_t e = R == 0 ? sat_build_lines(vox, dtype, nx, ny, nz, lut, scratch, st) : cudaSuccess;
  if (e != cudaSuccess) return e;
  if (R > 0) {
    // x-y plane prefixes only: the quad pass below adds them up along z
    e = sat_planes(vox, dtype, nx, ny, nz, lut, scratch, R, st);
    if (e != cudaSuccess) return e;
    dim3 grid((sx + kQuadTileX - 1) / kQuadTileX, (sy + kQuadTileY - 1) / kQuadTileY);
    k_sat_zscan_quads<<<grid, kQuadThreads, 0, st>>>(scratch, out, sx, sy, sz);
    return cudaGetLastError();
  }
  return launch_sat_quads(scratch, out, sx, sy, sz, st);  // the line builder made the whole table
}

// x-y quads of the volume: cell (x, y, z) = the voxels at (x, y), (x', y),
// (x, y'), (x', y') of plane z, with the successors clamped to the volume.  A
// warp takes a row, four cells of a lane in flight: 301 x 257 x 190 16-bit
// voxels 77 -> 33 us, 512^3 531 -> 308 (one cell per thread, CTAs of 128 along
// a row, before).
template <class T, class Q>
__global__ void __launch_bounds__(256) k_quad_volume(const T* __restrict__ v, Q* __restrict__ out, int nx, int ny,
                                                     int nz, unsigned qrow, unsigned qplane) {
  const int y = blockIdx.x * 8 + (threadIdx.x >> 5);
  if (y >= ny) return;
  const int up = y + 1 < ny ? nx : 0;
  for (int z = blockIdx.y; z < nz; z += gridDim.y) {  // planes beyond the grid's limit are strided over
    const T* p = v + ((size_t)z * ny + y) * (size_t)nx;
    Q* o = out + ((size_t)z * qplane + (size_t)y * qrow);
#pragma unroll 4
    for (int x = threadIdx.x & 31; x < nx; x += 32) {
      const int x1 = min(x + 1, nx - 1);
      Q q;
      q.x = __ldg(p + x); q.y = __ldg(p + x1); q.z = __ldg(p + up + x); q.w = __ldg(p + up + x1);
      o[x] = q;
    }
  }
}

template <class T, class Q>
static cudaError_t launch_quads(const T* v, Q* out, int nx, int ny, int nz, unsigned qrow, unsigned qplane,
                                cudaStream_t st) {
  const dim3 grid((ny + 7) / 8, std::min(nz, 65535));
  k_quad_volume<T, Q><<<grid, 256, 0, st>>>(v, out, nx, ny, nz, qrow, qplane);
  return cudaGetLastError();
}

cudaError_t launch_quad_volume(const void* src, void* dst, int dtype, int nx, int ny, int nz, unsigned qrow,
                               unsigned qplane, cudaStream_t st) {
  if (dtype == 1)
    return launch_quads(static_cast<const uint8_t*>(src), static_cast<uchar4*>(dst), nx, ny, nz, qrow, qplane, st);
  return launch_quads(static_cast<const uint16_t*>(src), static_cast<ushort4*>(dst), nx, ny, nz, qrow, qplane, st);
}

// The bordered x-y quads of every pyramid level (PyramidView::quads) in one
// launch: blockIdx.y runs over the planes of all levels, a warp takes a row.
// Bound by its 16-byte stores: 128^3 and its levels 36 -> 11 us (CTAs of 128
// cells left the last of 129 to a CTA of its own).
__global__ void __launch_bounds__(256) k_quad_pyramid(const __grid_constant__ PyramidView P, const float* __restrict__ v,
                                                      float4* __restrict__ out) {
  int l = 0, z = blockIdx.y;
  while (z >= P.dims[l][2] + 2) z -= P.dims[l++][2] + 2;
  const int nx = P.dims[l][0], ny = P.dims[l][1], nz = P.dims[l][2];
  const float* p = v + P.offset[l] + (size_t)min(max(z - 1, 0), nz - 1) * nx * ny;
  float4* o = out + (size_t)P.qoff[l] + (size_t)z * P.quad_plane(l);
  for (int y = blockIdx.x * 8 + (threadIdx.x >> 5); y <= ny; y += gridDim.x * 8) {
    const float *lo = p + max(y - 1, 0) * nx, *hi = p + min(y, ny - 1) * nx;
    float4* row = o + (size_t)y * P.quad_row(l);
#pragma unroll 4
    for (int x = threadIdx.x & 31; x <= nx; x += 32) {
      const int x0 = max(x - 1, 0), x1 = min(x, nx - 1);
      row[x] = make_float4(__ldg(lo + x0), __ldg(hi + x0), __ldg(lo + x1), __ldg(hi + x1));
    }
  }
}

cudaError_t launch_pyramid_quads(const PyramidView& P, const float* data, float4* dst, cudaStream_t st) {
  int planes = 0;
  for (int l = 0; l < P.n_levels; ++l) planes += P.dims[l][2] + 2;
  k_quad_pyramid<<<dim3((P.dims[0][1] + 8) / 8, planes), 256, 0, st>>>(P, data, dst);
  return cudaGetLastError();
}

// x-y predecessor quads of a table: out[(x, y, z)] = s at (x-1, y-1),
// (x, y-1), (x-1, y), (x, y) of plane z, the predecessors clamped to 0.
__global__ void k_sat_quads(const unsigned* __restrict__ s, uint4* __restrict__ out, int sx, int sy,
                            long long cells) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cells) return;
  const int x = (int)(i % sx), y = (int)((i / sx) % sy);
  const long long dx = x > 0 ? 1 : 0, dy = y > 0 ? sx : 0;
  out[i] = make_uint4(s[i - dy - dx], s[i - dy], s[i - dx], s[i]);
}

// Walk table (WalkView) from the predecessor-quad table: the oct of cell
// (x, y, z) is D = S(shifted) - S at the clamped coordinates (x-1..x, y-1..y,
// z-1..z), read as four quads: planes z-1 and z of the cell (S at the x-y
// pairs) and the same two shifted by w along the walk axis (clamped to the
// table).  Along the walk axis this uses the predecessor of the shifted
// coordinate, which equals the shift of the clamped predecessor except at
// walk coordinate 0, a cell no query reads (a box reaching below the table
// on the walk axis takes the quad query); past the high face S repeats.
__global__ void k_sat_walk(const uint4* __restrict__ q, uint4* __restrict__ out, int sx, int sy, int sz, int axis,
                           int w, long long cells) {
  const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= cells) return;
  const int x = (int)(i % sx), y = (int)((i / sx) % sy), z = (int)(i / ((long long)sx * sy));
  const size_t sxy = (size_t)sx * sy;
  auto Q = [&](int X, int Y, int Z) {
    X = min(max(X, 0), sx - 1); Y = min(max(Y, 0), sy - 1); Z = min(max(Z, 0), sz - 1);
    return __ldg(&q[(size_t)X + (size_t)sx * Y + sxy * Z]);
  };
  const int z0 = max(z - 1, 0);
  const uint4 lo0 = Q(x, y, z0), lo1 = Q(x, y, z);
  const int dx = axis == 0 ? w : 0, dy = axis == 1 ? w : 0;
  const uint4 up0 = Q(x + dx, y + dy, axis == 2 ? z0 + w : z0), up1 = Q(x + dx, y + dy, axis == 2 ? z + w : z);
  out[2 * i] = make_uint4(up0.x - lo0.x, up0.y - lo0.y, up0.z - lo0.z, up0.w - lo0.w);
  out[2 * i + 1] = make_uint4(up1.x - lo1.x, up1.y - lo1.y, up1.z - lo1.z, up1.w - lo1.w);
}

cudaError_t launch_sat_walk(const uint4* quads, uint4* out, int sx, int sy, int sz, int axis, int w,
                            cudaStream_t st) {
  const long long cells = (long long)sx * sy * sz;
  k_sat_walk<<<(unsigned)((cells + 255) / 256), 256, 0, st>>>(quads, out, sx, sy, sz, axis, w, cells);
  return cudaGetLastError();
}

cudaError_t launch_sat_quads(const unsigned* sat, uint4* out, int sx, int sy, int sz, cudaStream_t st) {
  const long long cells = (long long)sx * sy * sz;
  k_sat_quads<<<(unsigned)((cells + 255) / 256), 256, 0, st>>>(sat, out, sx, sy, cells);
  return cudaGetLastError();
}

// ------------------------------------------------------------- box tables
// All tables of a set in one launch (as many as its grid holds): a warp per row segment of 31 cells (lane
// 31 only supplies the last cell's successor), 8 rows per CTA, kBoxPlanes
// planes per thread, the sums of the box's rectangle in the planes at its two
// ends.  Along a walk of interval 2 (the default) a plane's rectangle is the
// low end of one cell and the high end of the cell two planes before: a ring
// of two keeps it, four loads a cell instead of eight.
constexpr int kBoxRow = 31, kBoxRows = 8, kBoxPlanes = 16;
// I: the type of an element's number, 32-bit where the sums have fewer than
// 2^32 elements: a cell is then 4 loads and some 30 instructions, and the tables
// are bound by their stores (200 x 180 x 222, shadow tables of 1.4 GB: 393 us,
// 546 with 64-bit numbers, bound by issue).
template <class W, class I>
__global__ void __launch_bounds__(32 * kBoxRows) k_box_tables(BoxSource src, const __grid_constant__ BoxTableSet set,
                                                               int first, int count, float* __restrict__ out) {
  const int ti = first + blockIdx.z % count, c0 = (blockIdx.z / count) * kBoxPlanes;
  const BoxTableDesc& d = set.t[ti];
  const int lane = threadIdx.x & 31;
  const int a = blockIdx.x * kBoxRow + lane, b = blockIdx.y * kBoxRows + (threadIdx.x >> 5);
  if ((int)(blockIdx.x * kBoxRow) >= d.g.na || b >= d.g.nb || c0 >= d.g.nc) return;  // whole warps
  const I each = sizeof(W) == 8 ? (I)1 : (I)src.stride;
  const I strides[3] = {each, each * (I)src.n[0], each * (I)src.n[0] * (I)src.n[1]};
  I lo[2], hi[2];  // element numbers of the box's low and high corner along the fastest and middle axis
  const int at[2] = {a, b};
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int ax = d.axis[i], n = src.n[ax], p = at[i] - d.pad[i];
    lo[i] = strides[ax] * (I)min(max(p, 0), n - 1);
    hi[i] = strides[ax] * (I)min(max(p + d.w[i], 0), n - 1);
  }
  const I i00 = lo[0] + lo[1], i10 = hi[0] + lo[1], i01 = lo[0] + hi[1], i11 = hi[0] + hi[1];
  const int nc = src.n[d.axis[2]];
  const I sc = strides[d.axis[2]];
  const W* base;
  if constexpr (sizeof(W) == 8) base = reinterpret_cast<const W*>(src.s64);
  else base = src.s32 + src.first;
  auto rect = [&](int c) -> W {
    const I o = sc * (I)min(max(c, 0), nc - 1);
    return __ldg(base + (o + i11)) - __ldg(base + (o + i01)) - __ldg(base + (o + i10)) + __ldg(base + (o + i00));
  };
  auto value = [&](W v) {
    if constexpr (sizeof(W) == 8) return ll_to_float((long long)v) * src.scale;
    else return (float)(int)v * src.scale;
  };
  const bool store = lane < kBoxRow && a < d.g.na;
  const size_t plane = d.g.nab;
  float2* dst = reinterpret_cast<float2*>(out) + d.cell + (size_t)b * d.g.row + a + (size_t)c0 * plane;
  auto put = [&](float v) {
    const float next = __shfl_down_sync(0xffffffffu, v, 1);
    if (store) *dst = make_float2(v, next);
    dst += plane;
  };
  const int end = min(c0 + kBoxPlanes, d.g.nc) - d.pad[2];
  int c = c0 - d.pad[2];
  if (d.w[2] == 2) {
    W r0 = rect(c), r1 = rect(c + 1);
#pragma unroll 4
    for (; c < end; ++c) {
      const W r2 = rect(c + 2);
      put(value(r2 - r0));
      r0 = r1;
      r1 = r2;
    }
  } else {
    const int w = d.w[2];
#pragma unroll 2
    for (; c < end; ++c) put(value(rect(c + w) - rect(c)));
  }
}

cudaError_t launch_box_tables(const BoxSource& src, const BoxTableSet& set, float* out, cudaStream_t st) {
  if (set.n == 0) return cudaSuccess;
  int na = 0, nb = 0, nc = 0;
  for (int i = 0; i < set.n; ++i) {
    na = std::max(na, set.t[i].g.na); nb = std::max(nb, set.t[i].g.nb); nc = std::max(nc, set.t[i].g.nc);
  }
  const int chunks = (nc + kBoxPlanes - 1) / kBoxPlanes;
  const size_t cells = (size_t)src.n[0] * src.n[1] * src.n[2];
  const bool small = cells * (src.s32 ? src.stride : 1) < ((size_t)1 << 32);
  auto kern = src.s32 ? (small ? k_box_tables<unsigned, unsigned> : k_box_tables<unsigned, size_t>)
                      : (small ? k_box_tables<unsigned long long, unsigned> : k_box_tables<unsigned long long, size_t>);
  const int most = std::max(65535 / chunks, 1);  // tables a launch: a grid has at most 65535 along z
  for (int first = 0; first < set.n; first += most) {
    const int count = std::min(most, set.n - first);
    const dim3 grid((na + kBoxRow - 1) / kBoxRow, (nb + kBoxRows - 1) / kBoxRows, chunks * count);
    kern<<<grid, 32 * kBoxRows, 0, st>>>(src, set, first, count, out);
    const cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
  }
  return cudaSuccess;
}

bool box_table_builds(const BoxGrid& g) {
  return (g.nb + kBoxRows - 1) / kBoxRows <= 65535 && (g.nc + kBoxPlanes - 1) / kBoxPlanes <= 65535;
}

// --------------------------------------------------------------- pyramid
// gen_extcoefvol_anysize.comp: base level voxel (i,j,k) holds the normalised
// 7x7x7 Gaussian average (sigma S0, taps at integer multiples of S0) of the
// TF opacity of the trilinearly sampled volume; samples outside the grid
// count as 0 opacity but keep their weight.
// The 7^3 Gaussian weights s^3 exp(-|f|^2 / (2 s^2)) of the tap offsets f =
// (ptx, pty, ptz) * s, in the loops' order, and their sum in the same order:
// the same values for every output voxel, computed once per CTA.
__device__ __forceinline__ float stage_gauss(float s, float* w) {
  for (int k = threadIdx.x; k < 343; k += blockDim.x) {
    const int ptx = k / 49 - 3, pty = (k / 7) % 7 - 3, ptz = k % 7 - 3;
    const float fx = float(ptx) * s, fy = float(pty) * s, fz = float(ptz) * s;
    w[k] = (s * s * s) * expf(-(fx * fx + fy * fy + fz * fz) / (2.0f * s * s));
  }
  __syncthreads();
  float sum_w = 0.0f;
  for (int k = 0; k < 343; ++k) sum_w += w[k];
  return sum_w;
}

// Inside the grid: t = p / S in [0, 1] on every axis, which for a correctly
// rounded division is p in [0, S].
__device__ __forceinline__ bool in_grid(float3 p, float3 g) {
  return !(p.x < 0.0f || p.y < 0.0f || p.z < 0.0f || p.x > g.x || p.y > g.y || p.z > g.z);
}

// A level's cell: its opacity (what the next level reads) and its extinction
// (backtotau.comp: -log(1 - opacity)).  tau == nullptr: op is converted later.
struct PyrOut {
  float *op, *tau;
  __device__ __forceinline__ void put(size_t i, float o) const {
    op[i] = o;
    if (tau) tau[i] = -1.0f * logf(1.0f - o);
  }
};

__global__ void k_pyr_base(VolumeView vol, const float4* __restrict__ tf_rgba, int tf_n, int bx, int by, int bz,
                           float s0, PyrOut out) {
  __shared__ float sm_w[343];
  extern __shared__ float4 sm_tf[];
  for (int i = threadIdx.x; i < tf_n; i += blockDim.x) sm_tf[i] = tf_rgba[i];
  const float sum_w = stage_gauss(s0, sm_w);
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)bx * by * bz;
  if (idx >= total) return;
  int x = int(idx % bx), y = int((idx / bx) % by), z = int(idx / ((long long)bx * by));
  float3 vs = f3(vol.grid.x / float(bx), vol.grid.y / float(by), vol.grid.z / float(bz));
  float3 gp = f3((float(x) + 0.5f) * vs.x, (float(y) + 0.5f) * vs.y, (float(z) + 0.5f) * vs.z);
  float sum_wc = 0.0f;
  int k = 0;
  for (int ptx = -3; ptx < 4; ++ptx) {
    for (int pty = -3; pty < 4; ++pty) {
      for (int ptz = -3; ptz < 4; ++ptz, ++k) {
        const float3 p = gp + f3(float(ptx) * s0, float(pty) * s0, float(ptz) * s0);
        float ck = 0.0f;
        if (in_grid(p, vol.grid)) ck = tf_alpha(sm_tf, tf_n, sample_volume(vol, p));
        sum_wc += sm_w[k] * ck;
      }
    }
  }
  out.put(idx, sum_wc / sum_w);
}

// gen_extcoefvol_anysize_mmlevel.comp: level l from level l-1 with sigma
// Si = S0 * 2^l, sampling level l-1 trilinearly (textureLod at an integer lod).
__global__ void k_pyr_level(PyramidView P, int l, float si, PyrOut out) {
  __shared__ float sm_w[343];
  const float sum_w = stage_gauss(si, sm_w);
  const int* d = P.dims[l];
  long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  long long total = (long long)d[0] * d[1] * d[2];
  if (idx >= total) return;
  int x = int(idx % d[0]), y = int((idx / d[0]) % d[1]), z = int(idx / ((long long)d[0] * d[1]));
  float3 lvs = P.grid / f3(float(d[0]), float(d[1]), float(d[2]));
  float3 gp = f3((float(x) + 0.5f) * lvs.x, (float(y) + 0.5f) * lvs.y, (float(z) + 0.5f) * lvs.z);
  float sum_wc = 0.0f;
  int k = 0;
  for (int ptx = -3; ptx < 4; ++ptx) {
    for (int pty = -3; pty < 4; ++pty) {
      for (int ptz = -3; ptz < 4; ++ptz, ++k) {
        const float3 p = gp + f3(float(ptx) * si, float(pty) * si, float(ptz) * si);
        float ck = 0.0f;
        if (in_grid(p, P.grid)) ck = pyr_sample_level(P, l - 1, p);
        sum_wc += sm_w[k] * ck;
      }
    }
  }
  out.put(idx, sum_wc / sum_w);
}

// Opacity -> extinction of every level, in place: only where there was no room
// for the opacities beside the extinctions.
__global__ void k_pyr_backtotau(float* data, long long n) {
  long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) data[i] = -1.0f * logf(1.0f - data[i]);
}

// ---- the level builders without 343 samples per cell
// The Gaussian weights factor per axis (exp(-|k|^2 / 2) = product of
// exp(-k_a^2 / 2)) and so does the mask of the box (in_grid), so only what
// stands between the taps and the sum decides what can be shared:
//  - levels from the level below: trilinear sampling is linear and factors per
//    axis too, whatever the sizes, so a level is three passes of dense weights
//    (k_pyr_level_tile);
//  - the base: the transfer function stands between, so every tap's value is
//    needed.  With taps one voxel apart a cell's 343 taps have one fraction per
//    axis and lie in an 8^3 window of voxels, interpolated axis by axis
//    (k_pyr_base_window); with half as many cells as voxels on every axis (the
//    reference's 128^3 base of a 256^3 volume) the taps of all cells are one
//    lattice, whose points are taken once (k_pyr_base_half);
//  - where cells and taps are whole numbers of texels apart on every axis, a
//    lattice of any such ratio in memory and a 7-tap pass along each axis
//    (k_pyr_lattice_base, k_pyr_lattice_level, k_pyr_pass): other bases that
//    have few lattice points per cell (a base of the volume's own size, taps of
//    several voxels), and levels whose windows shared memory cannot hold.
// Everything else takes the direct kernels above.
struct PyrWeights { float w[7]; };

// The centre of cell i in texels of the input, exact before the one rounding
// of its fraction.  I: holds 2 n_out n_in.
template <class I>
__device__ __forceinline__ int cell_centre(int i, int n_in, int n_out, float& frac) {
  const I num = (I)(2 * i + 1) * n_in - n_out, den = (I)2 * n_out;
  I q = num / den, r = num - q * den;
  if (r < 0) r += den, --q;
  frac = (float)r / (float)den;
  return (int)q;
}
// Texel coordinate i + f in [-0.5, n - 0.5]: inside the box.
__device__ __forceinline__ bool in_axis(int i, float f, int n) {
  return (i >= 0 || (i == -1 && f >= 0.5f)) && (i <= n - 2 || (i == n - 1 && f <= 0.5f));
}

// The opacity of a mean of voxels v in [0, 2^bits): tf_alpha of v * norm, the
// scale folded into the table's (scale = norm * n).  v lies between its voxels
// to FP32 rounding, so the entry is in the table without a clamp.
__device__ __forceinline__ float alpha_of(const float2* e, float v, float scale) {
  float t;
  const float2 a = e[cell_of(fmaf(v, scale, -0.5f), t) + 1];
  return fmaf(t, a.y, a.x);
}

// Base of half the volume's size, S0 = one voxel.  A CTA takes 16 x 16 columns
// of kHalfZ cells and streams the lattice planes of its window along z: voxels
// of two planes added in registers, the 37 x 37 points of a plane (each the
// mean of 8 voxels, exact in FP32) through the transfer function once, 7-tap
// passes along x and y in shared memory, along z in four running sums per
// thread.  Bound by issue (the points of a tile overlap its neighbours' by a
// third) and shared memory.  256^3 -> 128^3: 78 us; 204 as one lattice in memory
// and three passes.
constexpr int kHalfT = 16, kHalfL = 2 * kHalfT + 5, kHalfV = kHalfL + 1, kHalfZ = 16;
template <class T>
__global__ void __launch_bounds__(256, 4) k_pyr_base_half(const T* __restrict__ vox, int nx, int ny, int nz, float norm,
                                                       const float4* __restrict__ tf_rgba, int tf_n, PyrWeights w,
                                                       int bx, int by, int bz, PyrOut out) {
  constexpr int kV = (kHalfV * kHalfV + 255) / 256, kL = (kHalfL * kHalfL + 255) / 256;
  constexpr int kX = (kHalfL * kHalfT + 255) / 256;
  __shared__ float V[kHalfV * kHalfV], A[kHalfL * kHalfL], X[kHalfL * kHalfT];
  extern __shared__ float2 sm_alpha[];
  stage_tf_alpha(tf_rgba, tf_n, sm_alpha);
  const int tid = threadIdx.x;
  // lattice point q of an axis is the middle of texels q - 3 and q - 2; inside the box: 2 <= q <= n + 2
  const int qx0 = blockIdx.x * 2 * kHalfT, qy0 = blockIdx.y * 2 * kHalfT, oz0 = blockIdx.z * kHalfZ;
  unsigned off[kV], inside = 0u;
#pragma unroll
  for (int s = 0; s < kV; ++s) {
    const int i = min(tid + 256 * s, kHalfV * kHalfV - 1);
    const int x = min(max(qx0 - 3 + i % kHalfV, 0), nx - 1), y = min(max(qy0 - 3 + i / kHalfV, 0), ny - 1);
    off[s] = (unsigned)x + (unsigned)nx * (unsigned)y;
  }
#pragma unroll
  for (int s = 0; s < kL; ++s) {
    const int i = tid + 256 * s, x = qx0 + i % kHalfL, y = qy0 + i / kHalfL;
    if (x >= 2 && x <= nx + 2 && y >= 2 && y <= ny + 2) inside |= 1u << s;
  }
  const float scale = 0.125f * norm * (float)tf_n;
  const size_t plane = (size_t)nx * ny;
  const int planes = 2 * min(kHalfZ, bz - oz0) + 5;
  const int ox = blockIdx.x * kHalfT + (tid & 15), oy = blockIdx.y * kHalfT + (tid >> 4);
  float prev[kV], r0 = 0.0f, r1 = 0.0f, r2 = 0.0f, r3 = 0.0f;
  const T* pl = vox + plane * (size_t)min(max(2 * oz0 - 3, 0), nz - 1);
#pragma unroll
  for (int s = 0; s < kV; ++s) prev[s] = (float)__ldg(pl + off[s]);
  __syncthreads();
  for (int p = 0; p < planes; ++p) {
    const int qz = 2 * oz0 + p;
    pl = vox + plane * (size_t)min(max(qz - 2, 0), nz - 1);
#pragma unroll
    for (int s = 0; s < kV; ++s) {
      const float cur = (float)__ldg(pl + off[s]);
      if (tid + 256 * s < kHalfV * kHalfV) V[tid + 256 * s] = prev[s] + cur;
      prev[s] = cur;
    }
    float g = 0.0f;
    __syncthreads();
    if (qz >= 2 && qz <= nz + 2) {  // the same for the whole CTA
#pragma unroll
      for (int s = 0; s < kL; ++s) {
        const int i = tid + 256 * s;
        if (i < kHalfL * kHalfL) {
          const float* v = V + (i + i / kHalfL);
          A[i] = (inside >> s) & 1u ? alpha_of(sm_alpha, (v[0] + v[1]) + (v[kHalfV] + v[kHalfV + 1]), scale) : 0.0f;
        }
      }
      __syncthreads();
#pragma unroll
      for (int s = 0; s < kX; ++s) {
        const int i = tid + 256 * s;
        if (i < kHalfL * kHalfT) {
          const float* a = A + (i >> 4) * kHalfL + 2 * (i & 15);
          float acc = 0.0f;
#pragma unroll
          for (int k = 0; k < 7; ++k) acc = fmaf(w.w[k], a[k], acc);
          X[i] = acc;
        }
      }
      __syncthreads();
      const float* c = X + 2 * (tid >> 4) * kHalfT + (tid & 15);
#pragma unroll
      for (int k = 0; k < 7; ++k) g = fmaf(w.w[k], c[k * kHalfT], g);
    }
    if (p & 1) {
      r0 = fmaf(w.w[1], g, r0);
      r1 = fmaf(w.w[3], g, r1);
      r2 = fmaf(w.w[5], g, r2);
    } else {
      r3 = fmaf(w.w[6], g, r2);
      r2 = fmaf(w.w[4], g, r1);
      r1 = fmaf(w.w[2], g, r0);
      r0 = w.w[0] * g;
      if (p >= 6 && ox < bx && oy < by) out.put(((size_t)(oz0 + p / 2 - 3) * by + oy) * bx + ox, r3);
    }
  }
}

// Base of any size with taps one voxel apart: one thread per cell walks the
// eight voxel planes of its window, holding the 7 x 7 in-plane interpolations
// of the plane before.  Bound by issue: 343 transfer-function lookups and 1183
// lerps per cell instead of 343 trilinear samples of eight voxels; three CTAs
// per SM hold the 7 x 7 values in registers (two: 595 us, four: 470).
// 203 x 171 x 230 -> 101 x 85 x 115: 450 us; 1130 with the direct kernel.
template <class T>
__global__ void __launch_bounds__(128, 3) k_pyr_base_window(const T* __restrict__ vox, int nx, int ny, int nz, float norm,
                                                         const float4* __restrict__ tf_rgba, int tf_n, PyrWeights w,
                                                         int bx, int by, int bz, PyrOut out) {
  extern __shared__ float2 sm_alpha[];
  stage_tf_alpha(tf_rgba, tf_n, sm_alpha);
  __syncthreads();
  const float scale = norm * (float)tf_n;
  const long long idx = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (long long)bx * by * bz) return;
  const unsigned row = (unsigned)(idx / bx);
  const int x = (int)(idx - (long long)row * bx), y = (int)(row % (unsigned)by), z = (int)(row / (unsigned)by);
  float fx, fy, fz;
  const int cx = cell_centre<long long>(x, nx, bx, fx), cy = cell_centre<long long>(y, ny, by, fy),
            cz = cell_centre<long long>(z, nz, bz, fz);
  float wx[7], wy[7];
  unsigned xo[8], yo[8];
#pragma unroll
  for (int k = 0; k < 8; ++k) {
    if (k < 7) {
      wx[k] = in_axis(cx + k - 3, fx, nx) ? w.w[k] : 0.0f;
      wy[k] = in_axis(cy + k - 3, fy, ny) ? w.w[k] : 0.0f;
    }
    xo[k] = (unsigned)min(max(cx + k - 3, 0), nx - 1);
    yo[k] = (unsigned)min(max(cy + k - 3, 0), ny - 1) * (unsigned)nx;
  }
  float prev[7][7], sum = 0.0f;
  for (int kz = 0; kz < 8; ++kz) {
    const T* pl = vox + (size_t)nx * ny * (size_t)min(max(cz + kz - 3, 0), nz - 1);
    const float wz = kz > 0 && in_axis(cz + kz - 4, fz, nz) ? w.w[max(kz - 1, 0)] : 0.0f;
    float before[7], acc = 0.0f;
#pragma unroll
    for (int ky = 0; ky < 8; ++ky) {
      float t[8], line = 0.0f;
#pragma unroll
      for (int k = 0; k < 8; ++k) t[k] = (float)__ldg(pl + (yo[ky] + xo[k]));
#pragma unroll
      for (int k = 0; k < 7; ++k) {
        const float r = fmaf(fx, t[k + 1] - t[k], t[k]);
        if (ky > 0) {
          const float q = fmaf(fy, r - before[k], before[k]);
          if (kz > 0) line = fmaf(wx[k], alpha_of(sm_alpha, fmaf(fz, q - prev[ky - 1][k], prev[ky - 1][k]), scale), line);
          prev[ky - 1][k] = q;
        }
        before[k] = r;
      }
      if (ky > 0) acc = fmaf(wy[ky - 1], line, acc);
    }
    sum = fmaf(wz, acc, sum);
  }
  out.put(idx, sum);
}

// ---- lattices: cell i, tap k of a level reads lattice point i m + (k + 3) t, at
// texel coordinate j0 + q + f.  One pass takes every lattice point once (0
// outside the box, as in_grid), three more apply the 7 weights of each axis.
// Bound by the traffic of the points (9 ps each with their passes).
struct PyrAxis {
  int m, t;   // texels per cell, per tap step
  int j0, g;  // lattice start (integer part) and size
  int n_out;  // cells
  float f;    // the constant fraction
};
struct PyrAxes { PyrAxis a[3]; };

// Lattice point (qx, qy, qz) in texels; whether it lies inside the box: texel
// coordinates in [-0.5, n - 0.5].
__device__ __forceinline__ bool pyr_lattice_point(const PyrAxis* A, const int* n_in, int qx, int qy, int qz, float3& u) {
  u = f3((float)(A[0].j0 + qx) + A[0].f, (float)(A[1].j0 + qy) + A[1].f, (float)(A[2].j0 + qz) + A[2].f);
  return u.x >= -0.5f && u.y >= -0.5f && u.z >= -0.5f && u.x <= (float)n_in[0] - 0.5f &&
         u.y <= (float)n_in[1] - 0.5f && u.z <= (float)n_in[2] - 0.5f;
}

// Grids of (x blocks, y, z): no division of a flat index per point.
template <class S>
__global__ void k_pyr_lattice_base(const __grid_constant__ VolumeView vol, const float4* __restrict__ tf_rgba, int tf_n,
                                   PyrAxes A, float* __restrict__ G) {
  extern __shared__ float2 sm_alpha[];
  stage_tf_alpha(tf_rgba, tf_n, sm_alpha);
  __syncthreads();
  const int qx = blockIdx.x * blockDim.x + threadIdx.x, qy = blockIdx.y, qz = blockIdx.z;
  if (qx >= A.a[0].g) return;
  const int n_in[3] = {vol.nx, vol.ny, vol.nz};
  float3 u;
  const bool inside = pyr_lattice_point(A.a, n_in, qx, qy, qz, u);
  const float3 p = f3((u.x + 0.5f) * vol.spacing.x, (u.y + 0.5f) * vol.spacing.y, (u.z + 0.5f) * vol.spacing.z);
  G[((size_t)qz * A.a[1].g + qy) * A.a[0].g + qx] = inside ? TfAlpha{sm_alpha, tf_n}(S(vol)(p)) : 0.0f;
}

__global__ void k_pyr_lattice_level(PyramidView P, int l_in, PyrAxes A, float* __restrict__ G) {
  const int qx = blockIdx.x * blockDim.x + threadIdx.x, qy = blockIdx.y, qz = blockIdx.z;
  if (qx >= A.a[0].g) return;
  const int* n_in = P.dims[l_in];
  float3 u;
  const bool inside = pyr_lattice_point(A.a, n_in, qx, qy, qz, u);
  const float3 p = f3((u.x + 0.5f) * (P.grid.x / (float)n_in[0]), (u.y + 0.5f) * (P.grid.y / (float)n_in[1]),
                      (u.z + 0.5f) * (P.grid.z / (float)n_in[2]));
  G[((size_t)qz * A.a[1].g + qy) * A.a[0].g + qx] = inside ? pyr_sample_level(P, l_in, p) : 0.0f;
}

// One 7-tap pass along axis ax of an (nx, ny, nz) array: out has n_out cells
// along that axis, out[i] = sum_k w[k] in[i m + (k + 3) t]; the last pass is
// the level.
template <class Out>
__global__ void k_pyr_pass(const float* __restrict__ in, int nx, int ny, int nz, int ax, PyrAxis a, PyrWeights w,
                           Out out) {
  const int ox = ax == 0 ? a.n_out : nx, oy = ax == 1 ? a.n_out : ny;
  const int x = blockIdx.x * blockDim.x + threadIdx.x, y = blockIdx.y, z = blockIdx.z;
  if (x >= ox) return;
  const size_t idx = ((size_t)z * oy + y) * ox + x;
  const int i = ax == 0 ? x : (ax == 1 ? y : z);
  const long long stride = ax == 0 ? 1 : (ax == 1 ? (long long)nx : (long long)nx * ny);
  const long long base = (ax == 0 ? 0 : x) + (ax == 1 ? 0 : (long long)y * nx) + (ax == 2 ? 0 : (long long)z * nx * ny);
  float acc = 0.0f;
#pragma unroll
  for (int k = 0; k < 7; ++k) acc = fmaf(w.w[k], __ldg(in + base + (long long)(i * a.m + k * a.t) * stride), acc);
  out.put(idx, acc);
}
struct PassOut {
  float* p;
  __device__ __forceinline__ void put(size_t i, float v) const { p[i] = v; }
};

// A level from the one below, all three passes in one CTA of T^3 cells: the
// window of the input in shared memory, then along each axis a dense dot
// product per cell, whose weights (7 taps of two texels each, folded to the
// span they cover) the CTA works out first.  Latency-bound at these sizes
// (64^3 cells are 512 CTAs, 8^3 one), so what counts is one launch per level
// instead of four (lattices) or 343 samples in a row per thread (other sizes):
// levels 1-4 of a 256^3 volume 112 -> 76 us, of a 203 x 171 x 230 one 416 -> 54
// (cold caches, serialised).
struct LevelAxis {
  int n_in, n_out, span, win;  // span: texels of a cell's taps; win: of a tile's (upper bound)
  float t;                     // texels per tap step
};
struct LevelAxes { LevelAxis a[3]; };

template <int kLevelT>
__global__ void __launch_bounds__(kLevelT * 64) k_pyr_level_tile(const float* __restrict__ in, LevelAxes L,
                                                                 PyrWeights w, PyrOut out) {
  constexpr int kThreads = kLevelT * 64, kLanes = 4 * kLevelT;  // lanes per row of the window's load
  extern __shared__ float sm_level[];
  __shared__ int start[3][kLevelT], first[3], extent[3];
  const int tid = threadIdx.x;
  const int cell0[3] = {(int)blockIdx.x * kLevelT, (int)blockIdx.y * kLevelT, (int)blockIdx.z * kLevelT};
  const int pitch = L.a[0].win | 1;
  float* win = sm_level;                                                // [z][y][pitch]
  float* X = win + (size_t)L.a[2].win * L.a[1].win * pitch;             // [z][y][T]
  float* Y = X + (size_t)L.a[2].win * L.a[1].win * kLevelT;             // [z][T][T]
  float* wt = Y + (size_t)L.a[2].win * kLevelT * kLevelT;               // axis: [T][span]
  if (tid < 3 * kLevelT) {
    const int ax = tid / kLevelT, c = tid % kLevelT;
    const LevelAxis A = ax == 0 ? L.a[0] : (ax == 1 ? L.a[1] : L.a[2]);
    float* d = wt + kLevelT * ((ax > 0 ? L.a[0].span : 0) + (ax > 1 ? L.a[1].span : 0)) + c * A.span;
    const int last = min(kLevelT, A.n_out - cell0[ax]) - 1;  // cells past the level repeat the last one
    float f, f0, f1;
    const int i = cell_centre<int>(cell0[ax] + min(c, last), A.n_in, A.n_out, f);
    const int lo = i + (int)floorf(fmaf(-3.0f, A.t, f));
    const int i0 = cell_centre<int>(cell0[ax], A.n_in, A.n_out, f0) + (int)floorf(fmaf(-3.0f, A.t, f0));
    const int i1 = cell_centre<int>(cell0[ax] + last, A.n_in, A.n_out, f1) + (int)floorf(fmaf(-3.0f, A.t, f1));
    for (int j = 0; j < A.span; ++j) d[j] = 0.0f;
    for (int k = 0; k < 7; ++k) {
      const float u = fmaf((float)(k - 3), A.t, f), fl = floorf(u);
      float g = u - fl;
      int j = i + (int)fl - lo;
      if (!in_axis(i + (int)fl, g, A.n_in)) continue;
      if (j > A.span - 2) g += (float)(j - (A.span - 2)), j = A.span - 2;  // a coordinate rounded up to a whole texel
      d[j] += w.w[k] * (1.0f - g);
      d[j + 1] += w.w[k] * g;
    }
    start[ax][c] = min(lo - i0, A.win - A.span);
    if (c == 0) first[ax] = i0, extent[ax] = min(i1 - i0 + A.span, A.win);
  }
  __syncthreads();
  const int ex = extent[0], ey = extent[1], ez = extent[2];
  {
    const int nx = L.a[0].n_in, ny = L.a[1].n_in, nz = L.a[2].n_in;
#pragma unroll 8
    for (int r = tid / kLanes; r < ey * ez; r += kThreads / kLanes) {
      const int y = r % ey, z = r / ey;
      const float* src = in + ((size_t)min(max(first[2] + z, 0), nz - 1) * ny + min(max(first[1] + y, 0), ny - 1)) * nx;
      float* dst = win + ((size_t)z * ey + y) * pitch;
      const int x = tid % kLanes;
      if (x < ex) dst[x] = __ldg(src + min(max(first[0] + x, 0), nx - 1));
      for (int u = x + kLanes; u < ex; u += kLanes) dst[u] = __ldg(src + min(max(first[0] + u, 0), nx - 1));
    }
  }
  __syncthreads();
  const int cx = tid % kLevelT, cy = tid / kLevelT % kLevelT;
  {
    const float* d = wt + cx * L.a[0].span;
#pragma unroll 4
    for (int r = tid / kLevelT; r < ey * ez; r += kThreads / kLevelT) {
      const float* v = win + (size_t)r * pitch + start[0][cx];
      float acc = 0.0f;
      for (int j = 0; j < L.a[0].span; ++j) acc = fmaf(d[j], v[j], acc);
      X[r * kLevelT + cx] = acc;
    }
  }
  __syncthreads();
  {
    const float* d = wt + kLevelT * L.a[0].span + cy * L.a[1].span;
    for (int z = tid / (kLevelT * kLevelT); z < ez; z += kThreads / (kLevelT * kLevelT)) {
      const float* v = X + (size_t)(z * ey + start[1][cy]) * kLevelT + cx;
      float acc = 0.0f;
      for (int j = 0; j < L.a[1].span; ++j) acc = fmaf(d[j], v[j * kLevelT], acc);
      Y[(z * kLevelT + cy) * kLevelT + cx] = acc;
    }
  }
  __syncthreads();
  const int cz = tid / (kLevelT * kLevelT), x = cell0[0] + cx, y = cell0[1] + cy, z = cell0[2] + cz;
  if (cz >= kLevelT || x >= L.a[0].n_out || y >= L.a[1].n_out || z >= L.a[2].n_out) return;
  const float* d = wt + kLevelT * (L.a[0].span + L.a[1].span) + cz * L.a[2].span;
  const float* v = Y + (start[2][cz] * kLevelT + cy) * kLevelT + cx;
  float acc = 0.0f;
  for (int j = 0; j < L.a[2].span; ++j) acc = fmaf(d[j], v[j * kLevelT * kLevelT], acc);
  out.put(((size_t)z * L.a[1].n_out + y) * L.a[0].n_out + x, acc);
}

// Texels per tap step of level l (0: from the volume) along axis a.
static double pyr_tap_step(const VolumeView& vol, const PyramidView& P, int l, float s0, int a) {
  const int in[3] = {l == 0 ? vol.nx : P.dims[l - 1][0], l == 0 ? vol.ny : P.dims[l - 1][1],
                     l == 0 ? vol.nz : P.dims[l - 1][2]};
  const double grid[3] = {P.grid.x, P.grid.y, P.grid.z};
  return (double)s0 * std::ldexp(1.0, l) * in[a] / grid[a];
}

// The tile plan of level l >= 1; returns its shared memory, 0 if a tap span is
// out of proportion (such a window never fits).
static size_t pyr_level_plan(const VolumeView& vol, const PyramidView& P, int l, float s0, int tile, LevelAxes* L) {
  for (int a = 0; a < 3; ++a) {
    LevelAxis& A = L->a[a];
    const double t = pyr_tap_step(vol, P, l, s0, a);
    if (!(t < 64.0)) return 0;
    A.n_in = P.dims[l - 1][a];
    A.n_out = P.dims[l][a];
    A.t = (float)t;
    A.span = (int)std::ceil(6.0 * t - 1e-6) + 2;
    A.win = (int)std::ceil((double)(std::min(tile, A.n_out) - 1) * A.n_in / A.n_out) + 1 + A.span;
  }
  const size_t yz = (size_t)L->a[1].win * L->a[2].win;
  return sizeof(float) * (yz * (L->a[0].win | 1) + yz * tile + (size_t)L->a[2].win * tile * tile +
                          (size_t)tile * (L->a[0].span + L->a[1].span + L->a[2].span));
}

// The lattice of level l (0: from the volume): false when cells or taps are not
// whole numbers of texels apart.
static bool pyr_lattice(const VolumeView& vol, const PyramidView& P, int l, float s0, PyrAxes* L) {
  const int in[3] = {l == 0 ? vol.nx : P.dims[l - 1][0], l == 0 ? vol.ny : P.dims[l - 1][1],
                     l == 0 ? vol.nz : P.dims[l - 1][2]};
  for (int a = 0; a < 3; ++a) {
    PyrAxis& A = L->a[a];
    const double step = pyr_tap_step(vol, P, l, s0, a), t = std::nearbyint(step);
    A.n_out = P.dims[l][a];
    if (in[a] % A.n_out || !(t >= 1.0 && t < 65536.0) || std::fabs(step - t) > 1e-9 * t) return false;
    A.m = in[a] / A.n_out;
    A.t = (int)t;
    const double c0 = 0.5 * A.m - 0.5;  // texel coordinate of cell 0, tap 0
    A.f = (float)(c0 - std::floor(c0));
    A.j0 = (int)std::floor(c0) - 3 * A.t;
    const long long g = (long long)(A.n_out - 1) * A.m + 6LL * A.t + 1;
    if (g > 65535) return false;  // a grid dimension of the launches
    A.g = (int)g;
  }
  return true;
}
static long long pyr_lattice_points(const PyrAxes& L) { return (long long)L.a[0].g * L.a[1].g * L.a[2].g; }
// Floats of the lattice and of the first two passes' results.
static long long pyr_lattice_floats(const PyrAxes& L) {
  return pyr_lattice_points(L) + (long long)L.a[0].n_out * L.a[1].g * L.a[2].g +
         (long long)L.a[0].n_out * L.a[1].n_out * L.a[2].g;
}

// Which form the base takes (see above).  A window costs as much as 55 lattice
// points a cell (384^3 -> 128^3, 28 points a cell, 1.09 ms; as a lattice 0.61;
// 128^3 -> 128^3, 1.2 points, 1.09 against 0.17), a direct cell as much as 200
// (256^3 -> 128^3 with taps of two voxels, 9 points, 3.67 ms against 0.33).
enum class PyrBase { kHalf, kWindow, kLattice, kDirect };
static PyrBase pyr_base_form(const VolumeView& plain, const PyramidView& P, float s0, bool lattices, PyrAxes* L) {
  const int* d = P.dims[0];
  // a step of one voxel to FP32 accuracy: the taps of a cell share their fractions
  bool window = (size_t)plain.nx * plain.ny < ((size_t)1 << 31);
  for (int a = 0; a < 3; ++a) window = window && std::fabs(pyr_tap_step(plain, P, 0, s0, a) - 1.0) <= 1e-6;
  if (window && plain.nx == 2 * d[0] && plain.ny == 2 * d[1] && plain.nz == 2 * d[2]) return PyrBase::kHalf;
  if (lattices && pyr_lattice(plain, P, 0, s0, L) &&
      pyr_lattice_points(*L) <= (window ? 55LL : 200LL) * d[0] * d[1] * d[2])
    return PyrBase::kLattice;
  return window ? PyrBase::kWindow : PyrBase::kDirect;
}

// Cells per edge of level l's tiles.  8^3 cells read 2.6 times their texels,
// 4^3 cells 5.4 times: the smaller tile where the larger leaves SMs idle
// (32^3: 21 -> 12 us as 512 CTAs; 64^3 would take 52 instead of 41).
static int pyr_level_tile(const PyramidView& P, int l) {
  auto tiles = [&](int a) { return (long long)(P.dims[l][a] + 7) / 8; };
  return tiles(0) * tiles(1) * tiles(2) < kSms ? 4 : 8;
}
// windows of up to 160 KB: taps of up to three texels apart
constexpr size_t kLevelSmem = 160 * 1024;

// Which form level l >= 1 takes.  Tiles read windows that grow with the cube of
// the tap step: with steps beyond a texel (2 with a base of the volume's own
// size) levels from 30^3 cells on are lattices where they can be (the pyramid of
// 256^3 -> 256^3: 751 us, 1298 with tiles; 128^3 178 against 218, 100 x 90 x 80
// 118 against 136; levels of 32^3 and below the same).
constexpr long long kLatticeLevel = 27000;
enum class PyrLevel { kTile, kLattice, kDirect };
static PyrLevel pyr_level_form(const VolumeView& vol, const PyramidView& P, int l, float s0, bool lattices, int* tile,
                               size_t* smem, LevelAxes* L, PyrAxes* A) {
  *tile = pyr_level_tile(P, l);
  *smem = pyr_level_plan(vol, P, l, s0, *tile, L);
  const int* d = P.dims[l];
  const bool fits = *smem > 0 && *smem <= kLevelSmem;
  const bool wide = std::max(L->a[0].t, std::max(L->a[1].t, L->a[2].t)) > 1.5f &&
                    (long long)d[0] * d[1] * d[2] >= kLatticeLevel;
  if (fits && !wide) return PyrLevel::kTile;
  if (lattices && pyr_lattice(vol, P, l, s0, A)) return PyrLevel::kLattice;
  return fits ? PyrLevel::kTile : PyrLevel::kDirect;
}

long long pyramid_lattice_floats(const VolumeView& plain, const PyramidView& P, float s0) {
  PyrAxes A;
  long long need = pyr_base_form(plain, P, s0, true, &A) == PyrBase::kLattice ? pyr_lattice_floats(A) : 0;
  for (int l = 1; l < P.n_levels; ++l) {
    LevelAxes L;
    int tile;
    size_t sm;
    if (pyr_level_form(plain, P, l, s0, true, &tile, &sm, &L, &A) == PyrLevel::kLattice)
      need = std::max(need, pyr_lattice_floats(A));
  }
  return need;
}

// The three passes of a lattice G (followed by room for two of their results).
static cudaError_t launch_pyr_passes(const PyrAxes& L, float* G, const PyrWeights& w, const PyrOut& out, cudaStream_t st) {
  const PyrAxis* A = L.a;
  float* T1 = G + pyr_lattice_points(L);
  float* T2 = T1 + (long long)A[0].n_out * A[1].g * A[2].g;
  const unsigned bx = (unsigned)(A[0].n_out + 127) / 128;  // every pass's output has n_out along x
  k_pyr_pass<<<dim3(bx, A[1].g, A[2].g), 128, 0, st>>>(G, A[0].g, A[1].g, A[2].g, 0, A[0], w, PassOut{T1});
  k_pyr_pass<<<dim3(bx, A[1].n_out, A[2].g), 128, 0, st>>>(T1, A[0].n_out, A[1].g, A[2].g, 1, A[1], w, PassOut{T2});
  k_pyr_pass<<<dim3(bx, A[1].n_out, A[2].n_out), 128, 0, st>>>(T2, A[0].n_out, A[1].n_out, A[2].g, 2, A[2], w, out);
  return cudaGetLastError();
}

template <class T>
static cudaError_t launch_pyr_base(const VolumeView& v, const float4* tf_rgba, int tf_n, const int* d, bool half,
                                   const PyrWeights& w, const PyrOut& out, cudaStream_t st) {
  const T* vox = static_cast<const T*>(v.voxels);
  const size_t sm = sizeof(float2) * ((size_t)tf_n + 1);
  auto raise = [&](auto kern) {
    return sm > 30 * 1024 ? cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm) : cudaSuccess;
  };
  if (half) {
    cudaError_t e = raise(k_pyr_base_half<T>);
    if (e != cudaSuccess) return e;
    const dim3 grid((d[0] + kHalfT - 1) / kHalfT, (d[1] + kHalfT - 1) / kHalfT, (d[2] + kHalfZ - 1) / kHalfZ);
    k_pyr_base_half<T><<<grid, 256, sm, st>>>(vox, v.nx, v.ny, v.nz, v.norm, tf_rgba, tf_n, w, d[0], d[1], d[2], out);
  } else {
    cudaError_t e = raise(k_pyr_base_window<T>);
    if (e != cudaSuccess) return e;
    const long long n = (long long)d[0] * d[1] * d[2];
    k_pyr_base_window<T><<<(unsigned)((n + 127) / 128), 128, sm, st>>>(vox, v.nx, v.ny, v.nz, v.norm, tf_rgba, tf_n, w,
                                                                      d[0], d[1], d[2], out);
  }
  return cudaGetLastError();
}

cudaError_t launch_pyramid_build(const VolumeView& vol, const VolumeView& plain, const float4* tf_rgba, int tf_n,
                                 float s0, PyramidView& P, float* data, float* opacity, float* lattice,
                                 cudaStream_t st) {
  const int threads = 128;
  const int* d0 = P.dims[0];
  float* op = opacity ? opacity : data;
  auto out = [&](int l) { return PyrOut{op + P.offset[l], opacity ? data + P.offset[l] : nullptr}; };
  PyrWeights w;
  double sum = 0.0;
  for (int k = -3; k <= 3; ++k) sum += std::exp(-0.5 * k * k);
  for (int k = -3; k <= 3; ++k) w.w[k + 3] = (float)(std::exp(-0.5 * k * k) / sum);

  cudaError_t e = cudaSuccess;
  PyrAxes A;
  const PyrBase form = pyr_base_form(plain, P, s0, lattice != nullptr, &A);
  if (form == PyrBase::kHalf || form == PyrBase::kWindow) {
    const bool half = form == PyrBase::kHalf;
    e = plain.dtype == 1 ? launch_pyr_base<uint8_t>(plain, tf_rgba, tf_n, d0, half, w, out(0), st)
                         : launch_pyr_base<uint16_t>(plain, tf_rgba, tf_n, d0, half, w, out(0), st);
  } else if (form == PyrBase::kLattice) {
    const size_t sm = sizeof(float2) * ((size_t)tf_n + 1);
    e = with_sampler(vol, [&](auto* smp) {
      auto kern = k_pyr_lattice_base<std::remove_pointer_t<decltype(smp)>>;
      cudaError_t err = cudaSuccess;
      if (sm > 48 * 1024) err = cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
      if (err != cudaSuccess) return err;
      kern<<<dim3((A.a[0].g + 127) / 128, A.a[1].g, A.a[2].g), 128, sm, st>>>(vol, tf_rgba, tf_n, A, lattice);
      return cudaGetLastError();
    });
    if (e == cudaSuccess) e = launch_pyr_passes(A, lattice, w, out(0), st);
  } else {
    const size_t sm = sizeof(float4) * tf_n;
    if (sm > 48 * 1024) e = cudaFuncSetAttribute(k_pyr_base, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sm);
    if (e != cudaSuccess) return e;
    const long long n0 = (long long)d0[0] * d0[1] * d0[2];
    k_pyr_base<<<(unsigned)((n0 + threads - 1) / threads), threads, sm, st>>>(vol, tf_rgba, tf_n, d0[0], d0[1], d0[2],
                                                                              s0, out(0));
    e = cudaGetLastError();
  }
  if (e != cudaSuccess) return e;
  P.data = op;
  e = cudaFuncSetAttribute(k_pyr_level_tile<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLevelSmem);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(k_pyr_level_tile<4>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kLevelSmem);
  if (e != cudaSuccess) return e;
  for (int l = 1; l < P.n_levels; ++l) {
    LevelAxes L;
    const int* d = P.dims[l];
    int tile;
    size_t sm;
    const PyrLevel form = pyr_level_form(plain, P, l, s0, lattice != nullptr, &tile, &sm, &L, &A);
    if (form == PyrLevel::kTile) {
      const float* below = op + P.offset[l - 1];
      const dim3 grid((d[0] + tile - 1) / tile, (d[1] + tile - 1) / tile, (d[2] + tile - 1) / tile);
      if (tile == 8) k_pyr_level_tile<8><<<grid, 512, sm, st>>>(below, L, w, out(l));
      else k_pyr_level_tile<4><<<grid, 256, sm, st>>>(below, L, w, out(l));
    } else if (form == PyrLevel::kLattice) {
      k_pyr_lattice_level<<<dim3((A.a[0].g + 127) / 128, A.a[1].g, A.a[2].g), 128, 0, st>>>(P, l - 1, A, lattice);
      if ((e = launch_pyr_passes(A, lattice, w, out(l), st)) != cudaSuccess) return e;
    } else {
      const long long nl = (long long)d[0] * d[1] * d[2];
      const float si = s0 * powf(2.0f, float(l));
      k_pyr_level<<<(unsigned)((nl + threads - 1) / threads), threads, 0, st>>>(P, l, si, out(l));
    }
    if ((e = cudaGetLastError()) != cudaSuccess) return e;
  }
  P.data = data;
  if (!opacity) {
    const int top = P.n_levels - 1;
    const long long total = P.offset[top] + (long long)P.dims[top][0] * P.dims[top][1] * P.dims[top][2];
    k_pyr_backtotau<<<(unsigned)((total + 255) / 256), 256, 0, st>>>(data, total);
  }
  return cudaGetLastError();
}

// ----------------------------------------------------------- L2 flush
// ---------------------------------------------------------------- bricks
// Copies a plain x-fastest volume into bricks of 2^bs voxels per edge
// (brick-local x fastest, bricks x fastest); voxels past the volume's edge
// inside the last bricks are zero and never read.
template <class T>
__global__ void k_brick(const T* __restrict__ src, T* __restrict__ dst, int nx, int ny, int nz, int bs,
                        long long total) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= total) return;
  const int m = (1 << bs) - 1;
  const int local = (int)(e & ((1ll << (3 * bs)) - 1));
  const long long brick = e >> (3 * bs);
  const int bx = (nx + m) >> bs, by = (ny + m) >> bs;
  const int x = (int)(brick % bx) * (m + 1) + (local & m);
  const int y = (int)((brick / bx) % by) * (m + 1) + ((local >> bs) & m);
  const int z = (int)(brick / ((long long)bx * by)) * (m + 1) + (local >> (2 * bs));
  dst[e] = (x < nx && y < ny && z < nz) ? src[(size_t)x + (size_t)nx * ((size_t)y + (size_t)ny * z)] : T(0);
}

long long brick_elements(int nx, int ny, int nz, int bs) {
  const int m = (1 << bs) - 1;
  return (long long)((nx + m) >> bs) * ((ny + m) >> bs) * ((nz + m) >> bs) << (3 * bs);
}

cudaError_t launch_brick_volume(const void* src, void* dst, int dtype, int nx, int ny, int nz, int bs,
                                cudaStream_t st) {
  const long long total = brick_elements(nx, ny, nz, bs);
  const unsigned blocks = (unsigned)((total + 255) / 256);
  if (dtype == 1)
    k_brick<<<blocks, 256, 0, st>>>(static_cast<const uint8_t*>(src), static_cast<uint8_t*>(dst), nx, ny, nz, bs, total);
  else
    k_brick<<<blocks, 256, 0, st>>>(static_cast<const uint16_t*>(src), static_cast<uint16_t*>(dst), nx, ny, nz, bs,
                                    total);
  return cudaGetLastError();
}

__global__ void k_fill(uint4* p, size_t n, unsigned int v) {
  size_t i = (size_t)blockIdx.x * blockDim.x + threadIdx.x;
  size_t stride = (size_t)gridDim.x * blockDim.x;
  for (; i < n; i += stride) p[i] = make_uint4(v, v, v, v);
}
cudaError_t launch_fill(void* p, size_t bytes, unsigned int v, cudaStream_t st) {
  size_t n = bytes / sizeof(uint4);
  k_fill<<<152 * 8, 256, 0, st>>>(static_cast<uint4*>(p), n, v);
  return cudaGetLastError();
}

}  // namespace cvr
