// box_host.cu — box tables of the extinction marcher: which a frame needs,
// when they pay, and their pools.
#include <algorithm>
#include <cmath>
#include <cstring>

#include "ctx.cuh"

namespace cvr {
namespace ctxutil {

namespace {

// Pixels a frame (or the frames so far that went without) must have per cell
// to build.  Building costs 2 to 3.5 ps a cell (shadow tables of a 200 x 180 x
// 222 volume, 190 M cells: 0.39 ms, and their source); the tables save 9 ns a pixel against the
// compact table and its walk table (1024^2 frame 13.7 -> 4.3 ms) and 53 ns
// against the int64 table (61 -> 5.5 ms).  At 4e-4 pixels a cell the frame
// itself repays the build; smaller frames add up, and the tables are built
// once the pixels rendered without them would have paid for them.
constexpr double kPixelsPerCell = 4.0e-4;

constexpr size_t kCellBytes = sizeof(float) * kBoxCellFloats;

int texel_width(const ShadowBoxTable& t, int k, int axis) {
  int packed;
  std::memcpy(&packed, &t.tx[k].w, sizeof packed);
  return (packed >> (10 * axis)) & 1023;
}

// Grid of a table along SAT axes ax (fastest first) with pads; one cell per
// low corner -pad ... n-1, and one plane more, the successor of the last.
// False: beyond 32-bit plane pitches or the build's launches.
bool table_desc(const int n[3], const int ax[3], const int w[3], const int pad[3], BoxTableDesc* out) {
  BoxTableDesc d{};
  for (int i = 0; i < 3; ++i) {
    d.axis[i] = ax[i];
    d.w[i] = w[i];
    d.pad[i] = pad[i];
  }
  d.g.na = n[ax[0]] + pad[0];
  d.g.nb = n[ax[1]] + pad[1] + 1;
  d.g.nc = n[ax[2]] + pad[2] + 1;
  d.g.row = (int)padded_row((unsigned)d.g.na, (int)kCellBytes);
  if ((size_t)d.g.row * (size_t)d.g.nb > kBoxPoolBytes / kCellBytes || !box_table_builds(d.g)) return false;
  d.g.nab = padded_plane((unsigned)d.g.row * (unsigned)d.g.nb, (int)kCellBytes);
  *out = d;
  return true;
}
size_t cells_of(const BoxGrid& g) { return (size_t)g.nab * (size_t)g.nc; }
// The grid a lookup clamps to: without the successor row and plane.
BoxGrid lookup_grid(BoxGrid g) {
  --g.nb;
  --g.nc;
  return g;
}

// The shadow tables of box_plan, and the frame's walk over them.
bool shadow_plan(BoxTables& B, unsigned long long gen, const int n[3], const ShadowBoxTable& t, BoxWalk* W, ExtArgs* e,
                 BoxPlan* P) {
  const BoxPool& pool = B.sdw;
  // shadow: one table per pair of lateral widths, the walk axis slowest
  const int axis = t.axis;
  const int ax[3] = {axis == 0 ? 1 : 0, axis == 2 ? 1 : 2, axis};
  const int ww = texel_width(t, 0, axis);
  int pad[3] = {0, 0, ww + 1};
  std::vector<int> need, pair(t.n);
  for (int k = 0; k < t.n; ++k) {
    const int wa = texel_width(t, k, ax[0]), wb = texel_width(t, k, ax[1]);
    if (texel_width(t, k, axis) != ww) return false;
    pad[0] = std::max(pad[0], wa);
    pad[1] = std::max(pad[1], wb);
    pair[k] = wa | (wb << 10);
    if (std::find(need.begin(), need.end(), pair[k]) == need.end()) need.push_back(pair[k]);
  }
  // pads in steps of eight: a light that moves a little keeps the pool's grid
  for (int i = 0; i < 2; ++i) pad[i] = (pad[i] + 7) / 8 * 8 + 1;
  const bool kin = pool.data && pool.gen == gen && pool.key.size() == 4 && pool.key[0] == axis && pool.key[1] == ww;
  if (kin) {
    pad[0] = std::max(pad[0], pool.key[2]);
    pad[1] = std::max(pad[1], pool.key[3]);
  }
  const bool same = kin && pool.key[2] == pad[0] && pool.key[3] == pad[1];
  const int none[3] = {0, 0, 0};
  BoxTableDesc grid;
  if (!table_desc(n, ax, none, pad, &grid)) return false;
  const size_t cells = cells_of(grid.g);
  P->shadow = true;
  P->sdw_key = {axis, ww, pad[0], pad[1]};
  if (kin) P->have = pool.have;
  const size_t had = P->have.size();
  for (int p : need)
    if (std::find(P->have.begin(), P->have.end(), p) == P->have.end()) P->have.push_back(p);
  auto fits = [&]() { return P->have.size() <= (size_t)kMaxBoxTables && P->have.size() * cells * kCellBytes <= B.limit; };
  P->sdw_new = !same;
  if (!fits() || P->have.size() * cells * kCellBytes > pool.cap) {
    P->sdw_new = true;          // the pool grows: its tables are built again
    if (!fits()) P->have = need;  // without the widths of earlier lights
    if (!fits()) return false;
  }
  // room for a few more widths (a moving light's), as far as the bound goes
  const size_t room = std::min((P->have.size() + 3) / 4 * 4, B.limit / (cells * kCellBytes));
  P->sdw_bytes = P->sdw_new ? std::max(room, P->have.size()) * cells * kCellBytes : pool.cap;
  for (size_t i = P->sdw_new ? 0 : had; i < P->have.size(); ++i) {
    const int w[3] = {P->have[i] & 1023, P->have[i] >> 10, ww};
    BoxTableDesc d;
    if (!table_desc(n, ax, w, pad, &d)) return false;
    d.cell = (unsigned)(i * cells);
    P->sdw.t[P->sdw.n++] = d;
    P->missing += cells;
  }
  // the walk
  e->box.sdw_grid = lookup_grid(grid.g);
  W->n = t.n;
  W->axis = axis;
  W->pad_w = pad[2];
  W->vmin = t.vmin;
  W->vmax = t.vmax;
  W->per = 1.0f / t.interval;
  auto comp = [](const float4& v, int i) { return i == 0 ? v.x : (i == 1 ? v.y : v.z); };
  W->first = comp(t.tx[0], axis);
  const int step = t.interval < 0.0f ? -ww : ww;
  for (int k = 0; k < t.n; ++k) {
    const size_t i = std::find(P->have.begin(), P->have.end(), pair[k]) - P->have.begin();
    // 32-bit cell arithmetic wraps: a walk towards the low face steps down
    const unsigned cell = (unsigned)(i * cells) + (unsigned)(k * step) * grid.g.nab;
    float cb;
    std::memcpy(&cb, &cell, sizeof cb);
    W->o[k] = make_float4(comp(t.tx[k], ax[0]), comp(t.tx[k], ax[1]), t.hi[k].w, cb);
    W->cut[k] = t.lo[k].w + t.interval;
  }
  W->pad_a = pad[0];
  W->pad_b = pad[1];
  return true;
}

}  // namespace

bool box_plan(BoxTables& B, unsigned long long gen, const int n[3], const ShadowBoxTable* table, double pixels,
              ExtArgs* e, BoxWalk* W, BoxPlan* P) {
  // ambient occlusion: one table per shell, each with its own pad
  if (e->apply_occ) {
    const int xyz[3] = {0, 1, 2};
    size_t cell = 0;
    for (int i = 0; i < e->n_shells; ++i) {
      const int w = (int)std::nearbyint(2.0f * e->radii[i]);
      const int ww[3] = {w, w, w}, pad[3] = {w + 1, w + 1, w + 1};
      BoxTableDesc d;
      if (!table_desc(n, xyz, ww, pad, &d)) return false;
      d.cell = (unsigned)cell;
      cell += cells_of(d.g);
      if (cell * kCellBytes > B.limit) return false;
      e->box.ao_cell[i] = d.cell;
      e->box.ao_grid[i] = lookup_grid(d.g);
      P->ao.t[P->ao.n++] = d;
      P->ao_key.push_back(w);
    }
    P->ao_bytes = cell * kCellBytes;
    P->ao_new = !(B.ao.data && B.ao.gen == gen && B.ao.key == P->ao_key);
    if (P->ao_new) P->missing += cell;
    else P->ao.n = 0;
  }
  if (table && !shadow_plan(B, gen, n, *table, W, e, P)) return false;
  if (P->missing > 0 && pixels >= 0.0) {
    if (B.seen_gen != gen) {
      B.seen_gen = gen;
      B.seen = 0.0;
    }
    B.seen += pixels;
    if ((double)P->missing * kPixelsPerCell > B.seen) return false;
    B.seen = 0.0;
  }
  return true;
}

cvr_status box_build(cvr_ctx* c, BoxTables& B, const BoxSource& src, unsigned long long gen, const BoxPlan& P,
                     ExtArgs* e, bool* used) {
  *used = false;
  auto build = [&](BoxPool& pool, bool fresh, size_t bytes, const BoxTableSet& set) -> cudaError_t {
    if (fresh) {
      pool.gen = 0;
      cudaError_t err = ensure_spare(c, pool.data, pool.cap, bytes);
      if (err != cudaSuccess) return err;
    }
    return launch_box_tables(src, set, pool.data, c->stream);
  };
  cudaError_t err = cudaSuccess;
  if (e->apply_occ) {
    err = build(B.ao, P.ao_new, P.ao_bytes, P.ao);
    if (err == cudaSuccess) {
      B.ao.gen = gen;
      B.ao.key = P.ao_key;
    }
  }
  if (err == cudaSuccess && P.shadow) {
    err = build(B.sdw, P.sdw_new, P.sdw_bytes, P.sdw);
    if (err == cudaSuccess) {
      B.sdw.gen = gen;
      B.sdw.key = P.sdw_key;
      B.sdw.have = P.have;
    }
  }
  if (err == cudaErrorMemoryAllocation) {
    cudaGetLastError();
    return CVR_OK;
  }
  if (err != cudaSuccess) return cuda_fail(c, err, "box tables");
  e->box.ao = e->apply_occ ? B.ao.data : nullptr;
  e->box.sdw = P.shadow ? B.sdw.data : nullptr;
  *used = true;
  return CVR_OK;
}

}  // namespace ctxutil
}  // namespace cvr
