// batch_host.cu — resident volume slots and batched rendering: a fixed list
// of frames over the resident volumes, captured in one CUDA graph: the
// extinction jobs in persistent launches, the surrogate jobs as deferred
// frames on lanes beside them.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <numeric>
#include <vector>

#include "ctx.cuh"

using namespace cvr::ctxutil;

// Lanes of the surrogate jobs in a batch's graph: a frame's collect and resolve
// passes leave most of the GPU idle, so they run beside another lane's.
constexpr int kSurLanes = 3;

struct cvr_batch {
  cvr_ctx* ctx = nullptr;
  int n_jobs = 0;
  BatchExtJob* d_ext = nullptr;           // the jobs on SATs, then those on box tables
  int n_ext = 0, n_box = 0;
  unsigned ext_blocks = 0, box_blocks = 0;
  int ext_max_table = 0;                  // longest shadow table of either
  int ext_variant = 0;
  int ext_threads = 128;
  float4* d_tables = nullptr;
  float* d_cuts = nullptr;
  void* lists[kSurLanes] = {};            // deferred shading's lists, one set per lane
  unsigned int* d_counters = nullptr;  // [0] extinction tiles, [1] box-table tiles, [2 + k] rays of surrogate job k (direct marcher)
  unsigned long long* d_stats = nullptr;  // 3 per job, in the caller's job order
  bool ext_compact = false;
  bool ext_aligned = false;  // every job: an aligned shadow table and aligned AO boxes (or AO off)
  std::vector<std::shared_ptr<DevCopy>> copies;  // the volume and pyramid copies its jobs read
  std::vector<uint4*> sat32;              // the batch's own compact SATs, one per volume slot used
  std::vector<uint4*> walks;              // their walk tables, one per (slot, walk axis, depth) in use
  std::vector<long long> walk_keys;
  std::vector<std::unique_ptr<BoxTables>> boxes;  // box tables, one set per (slot, walk axis, interval) in use
  std::vector<long long> box_keys;
  cudaGraphExec_t graph = nullptr;
  ~cvr_batch() {
    if (graph) cudaGraphExecDestroy(graph);
    void* bufs[] = {d_ext, d_tables, d_cuts, d_counters, d_stats};
    for (void* p : bufs)
      if (p) cudaFree(p);
    for (void* p : lists)
      if (p) cudaFree(p);
    for (uint4* p : sat32)
      if (p) cudaFree(p);
    for (uint4* p : walks)
      if (p) cudaFree(p);
  }
};

namespace {

// Makes slot s current; returns the slot that was.
int select_slot(cvr_ctx* c, int s) {
  int prev = c->cur_slot;
  if (s != prev) {
    swap_volume(c, c->slots[prev]);
    swap_volume(c, c->slots[s]);
    c->cur_slot = s;
  }
  return prev;
}

// Dominant axis of a job's directional light (the walk axis of its shadow
// table), 3 for other lights: jobs that share a volume and this axis read
// the same walk table.
int job_walk_axis(const cvr_job& j) {
  if (j.light.type != CVR_LIGHT_DIRECTIONAL) return 3;
  const float a[3] = {std::fabs(j.light.forward[0]), std::fabs(j.light.forward[1]), std::fabs(j.light.forward[2])};
  return (a[2] > a[0] && a[2] > a[1]) ? 2 : (a[1] > a[0] ? 1 : 0);
}

double job_cost(const cvr_job& j, const cvr_ctx* c) {
  const VolSlot& v = c->slots[j.volume];
  int nx = j.volume == c->cur_slot ? c->nx : v.nx, ny = j.volume == c->cur_slot ? c->ny : v.ny,
      nz = j.volume == c->cur_slot ? c->nz : v.nz;
  return (double)j.width * j.height * std::sqrt((double)nx * nx + (double)ny * ny + (double)nz * nz);
}

}  // namespace

extern "C" {

cvr_status cvr_select_volume(cvr_ctx* c, int slot) {
  if (!c) return CVR_ERR_INVALID_ARG;
  if (slot < 0 || slot >= CVR_MAX_VOLUMES) return fail(c, CVR_ERR_INVALID_ARG, "cvr_select_volume: slot out of range");
  select_slot(c, slot);
  return CVR_OK;
}

int cvr_current_volume(cvr_ctx* c) { return c ? c->cur_slot : -1; }

cvr_status cvr_batch_create(cvr_ctx* c, const cvr_job* jobs, int n_jobs, cvr_batch** out) {
  if (!c || !jobs || n_jobs <= 0 || !out) return fail(c, CVR_ERR_INVALID_ARG, "cvr_batch_create: bad arguments");
  *out = nullptr;
  for (int i = 0; i < n_jobs; ++i) {
    const cvr_job& j = jobs[i];
    if (j.volume < 0 || j.volume >= CVR_MAX_VOLUMES || !j.params)
      return fail(c, CVR_ERR_INVALID_ARG, "cvr_batch_create: bad job (volume slot or params)");
    if (j.method == CVR_METHOD_EXTINCTION ? j.params_size != sizeof(cvr_ext_params)
                                          : (j.method == CVR_METHOD_SURROGATE ? j.params_size != sizeof(cvr_gt_params)
                                                                              : true))
      return fail(c, CVR_ERR_INVALID_ARG, "cvr_batch_create: jobs must be extinction or surrogate with their params");
  }
  if (c->lc_dims[0] > 0)
    return fail(c, CVR_ERR_UNSUPPORTED, "cvr_batch_create: the light cache is per frame, not batched (turn it off)");
  if (c->ms_mode != CVR_MULTISCALE_SINGLE)
    return fail(c, CVR_ERR_UNSUPPORTED, "cvr_batch_create: multiscaling is per frame, not batched (turn it off)");
  CK(c, cudaSetDevice(c->device));
  CK(c, cudaStreamSynchronize(c->stream));
  std::unique_ptr<cvr_batch> b(new cvr_batch());
  b->ctx = c;
  b->n_jobs = n_jobs;
  // longest jobs first within each method group
  std::vector<int> order(n_jobs);
  std::iota(order.begin(), order.end(), 0);
  // longest jobs first; among equal costs, jobs of one volume, method and
  // walk axis together, so that consecutive jobs share their tables in L2
  std::stable_sort(order.begin(), order.end(), [&](int x, int y) {
    const double cx = job_cost(jobs[x], c), cy = job_cost(jobs[y], c);
    if (cx != cy) return cx > cy;
    if (jobs[x].volume != jobs[y].volume) return jobs[x].volume < jobs[y].volume;
    if (jobs[x].method != jobs[y].method) return jobs[x].method < jobs[y].method;
    return job_walk_axis(jobs[x]) < job_walk_axis(jobs[y]);
  });
  NEED(c, cudaMalloc((void**)&b->d_stats, sizeof(unsigned long long) * 3 * n_jobs));
  std::vector<BatchExtJob> ext;
  std::vector<int> ext_slot;
  double slot_vmax[CVR_MAX_VOLUMES] = {};
  bool all_compact = c->compact_sat;
  std::vector<std::vector<float4>> tables;
  std::vector<std::unique_ptr<ShadowBoxTable>> aligned;  // of the jobs box tables can serve, else null
  struct SurFrameJob {
    FrameArgs f;
    SurArgs a;
    DeferredPlan plan;
    size_t bytes;  // of its lists; 0: the direct marcher
    bool tex;
  };
  std::vector<SurFrameJob> sur;
  const int keep = c->cur_slot;
  cvr_status st = CVR_OK;
  for (int oi = 0; oi < n_jobs && st == CVR_OK; ++oi) {
    const int i = order[oi];
    const cvr_job& j = jobs[i];
    select_slot(c, j.volume);
    FrameArgs f;
    st = frame_args(c, &j.camera, j.params, j.out_rgba_dev, j.width, j.height, &f);
    if (st != CVR_OK) break;
    auto hold = [&](const std::shared_ptr<DevCopy>& p) {
      if (std::find(b->copies.begin(), b->copies.end(), p) == b->copies.end()) b->copies.push_back(p);
    };
    if (f.vol.voxels != c->d_vol) hold(c->vcopy);
    st = grad_args(c, j.method, &j.light, &f);
    if (st != CVR_OK) break;
    f.stats = b->d_stats + 3 * (size_t)i;
    if (j.method == CVR_METHOD_EXTINCTION) {
      BatchExtJob J{};
      const ShadowBoxTable* table = nullptr;
      double vmax = 0.0;
      st = ext_args(c, static_cast<const cvr_ext_params*>(j.params), &j.light, f, &J.e, &table, &vmax);
      if (st != CVR_OK) break;
      if (vmax > 0.0) slot_vmax[j.volume] = std::max(slot_vmax[j.volume], vmax);
      else all_compact = false;
      ext_slot.push_back(j.volume);
      J.f = f;
      J.blocks_x = (unsigned)((j.width + f.tile_w - 1) / f.tile_w);
      std::vector<float4> t;
      if (table) {
        J.tn = table->n; J.tax = table->axis; J.tiw = table->interval; J.tvmin = table->vmin; J.tvmax = table->vmax;
        t.assign(table->lo, table->lo + table->n);
        t.insert(t.end(), table->hi, table->hi + table->n);
        if (table->aligned) t.insert(t.end(), table->tx, table->tx + table->n);
        b->ext_max_table = std::max(b->ext_max_table, table->n);
      }
      tables.push_back(std::move(t));
      aligned.emplace_back(table && table->aligned && table->n > 0 && (J.e.ao_aligned || !J.e.apply_occ)
                               ? new ShadowBoxTable(*table) : nullptr);
      ext.push_back(J);
    } else {
      SurFrameJob J{};
      st = sur_job_args(c, static_cast<const cvr_gt_params*>(j.params), &j.light, &J.a, &J.tex);
      if (st != CVR_OK) break;
      J.f = f;
      if (J.a.pyr.quads) hold(c->pyrq);
      J.bytes = deferred_bytes(c, f, &J.plan);
      sur.push_back(J);
    }
  }
  // Compact SATs owned by the batch (a later frame may rebuild the context's
  // own at another fixed point): one per slot, at the largest region of its jobs
  if (st == CVR_OK && all_compact && !ext.empty()) {
    float inv[CVR_MAX_VOLUMES] = {};
    uint4* tab[CVR_MAX_VOLUMES] = {};
    for (int v = 0; v < CVR_MAX_VOLUMES && st == CVR_OK && all_compact; ++v) {
      if (slot_vmax[v] <= 0.0) continue;
      select_slot(c, v);
      int F;
      std::vector<unsigned> q;
      if (!compact_plan(c->sat_ext, slot_vmax[v], &F, &q)) { all_compact = false; break; }
      const size_t cells = (size_t)(c->nx + 2) * (c->ny + 2) * (c->nz + 2);
      if (cells >= kCompactMaxCells) { all_compact = false; break; }
      uint4* d = nullptr;
      cudaError_t e = need(c, [&] { return cudaMalloc((void**)&d, cells * sizeof(uint4)); });
      if (e == cudaErrorMemoryAllocation) { cudaGetLastError(); all_compact = false; break; }  // int64 tables
      if (e != cudaSuccess) { st = cuda_fail(c, e, "cvr_batch_create: compact SAT"); break; }
      b->sat32.push_back(d);
      st = build_compact_sat(c, q, d);
      if (st == CVR_ERR_OUT_OF_MEMORY) { st = CVR_OK; all_compact = false; break; }
      tab[v] = d;
      inv[v] = (float)std::ldexp(1.0, -F);
    }
    if (st == CVR_OK && all_compact) {
      for (size_t k = 0; k < ext.size(); ++k) {
        ext[k].e.sat.sat32 = tab[ext_slot[k]];
        ext[k].e.sat.inv_scale32 = inv[ext_slot[k]];
      }
      b->ext_compact = true;
    }
  }
  // Box tables for the jobs whose boxes all have integer widths: a batch is
  // run many times, so they are built whenever they fit (all sets together
  // within a quarter of the GPU).  The first pass collects every job's widths
  // in its set, the second takes the jobs whose tables are all there.
  std::vector<std::unique_ptr<BoxWalk>> walks(ext.size());
  size_t box_budget = 0, mem_free = 0;
  if (st == CVR_OK && !ext.empty()) {
    const cudaError_t e = cudaMemGetInfo(&mem_free, &box_budget);
    if (e != cudaSuccess) st = cuda_fail(c, e, "cvr_batch_create: free memory");  // the current volume is set back below
    box_budget /= 4;
  }
  for (int pass = 0; pass < 2 && st == CVR_OK; ++pass) {
    for (size_t k = 0; k < ext.size() && st == CVR_OK; ++k) {
      if (!aligned[k]) continue;
      BatchExtJob& J = ext[k];
      const ShadowBoxTable& t = *aligned[k];
      int widths;
      std::memcpy(&widths, &t.tx[0].w, sizeof widths);
      const long long key = ((long long)ext_slot[k] * 3 + t.axis) * 1024 + ((widths >> (10 * t.axis)) & 1023);
      size_t at = std::find(b->box_keys.begin(), b->box_keys.end(), key) - b->box_keys.begin();
      if (at == b->box_keys.size()) {
        b->box_keys.push_back(key);
        b->boxes.emplace_back(new BoxTables());
        b->boxes.back()->limit = std::min(kBoxPoolBytes, c->cache_limit);
      }
      select_slot(c, ext_slot[k]);
      const int n[3] = {c->nx + 2, c->ny + 2, c->nz + 2};
      const bool cm = b->ext_compact;
      const BoxSource src{cm ? nullptr : c->d_sat, cm ? reinterpret_cast<const unsigned*>(J.e.sat.sat32) : nullptr, 4, 3,
                          cm ? J.e.sat.inv_scale32 : J.e.sat.inv_scale, {n[0], n[1], n[2]}};
      std::unique_ptr<BoxWalk> w(new BoxWalk());
      BoxPlan plan;
      ExtArgs e = J.e;
      const unsigned long long gen = 1;  // one source per slot
      if (!box_plan(*b->boxes[at], gen, n, &t, -1.0, &e, w.get(), &plan)) continue;
      if (pass == 1 && plan.missing > 0) continue;
      size_t held = 0;
      for (size_t i = 0; i < b->boxes.size(); ++i)
        if (i != at) held += b->boxes[i]->ao.cap + b->boxes[i]->sdw.cap;
      if (held + plan.ao_bytes + plan.sdw_bytes > box_budget) continue;
      bool used = false;
      st = box_build(c, *b->boxes[at], src, gen, plan, &e, &used);
      if (st == CVR_OK && used && pass == 1) {
        J.e = e;
        walks[k] = std::move(w);
      }
    }
  }
  if (st == CVR_OK && b->ext_compact) {
    {
      // walk tables of these compact tables, one per (slot, walk axis, box
      // depth) that the jobs with an aligned directional table use (a job's
      // table holds its texel offsets after lo and hi when it is aligned)
      for (size_t k = 0; k < ext.size() && st == CVR_OK && c->walk_tables; ++k) {
        BatchExtJob& J = ext[k];
        if (walks[k] || J.tn <= 0 || tables[k].size() != 3 * (size_t)J.tn) continue;
        const int slot = ext_slot[k], axis = J.tax, w = (int)std::nearbyint(J.e.interval);
        if (w < 1 || w > 1023) continue;
        const long long key = ((long long)slot * 3 + axis) * 1024 + w;
        uint4* d = nullptr;
        for (size_t i = 0; i < b->walk_keys.size(); ++i)
          if (b->walk_keys[i] == key) d = b->walks[i];
        if (!d) {
          select_slot(c, slot);
          const int sx = c->nx + 2, sy = c->ny + 2, sz = c->nz + 2;
          cudaError_t e = need(c, [&] { return cudaMalloc((void**)&d, (size_t)sx * sy * sz * 2 * sizeof(uint4)); });
          if (e == cudaErrorMemoryAllocation) { cudaGetLastError(); continue; }  // this job reads the quads
          if (e != cudaSuccess) { st = cuda_fail(c, e, "cvr_batch_create: walk table"); break; }
          b->walks.push_back(d);
          b->walk_keys.push_back(key);
          e = launch_sat_walk(J.e.sat.sat32, d, sx, sy, sz, axis, w, c->stream);
          if (e != cudaSuccess) { st = cuda_fail(c, e, "cvr_batch_create: walk table"); break; }
        }
        J.e.walk = WalkView{d, axis, w};
      }
    }
  }
  select_slot(c, keep);
  if (st != CVR_OK) return st;
  if (!sur.empty() && (!c->mlp || !c->mlp->err)) return fail(c, CVR_ERR_NOT_READY, "cvr_batch_create: no network");
  b->ext_variant = c->variant;
  b->ext_threads = (c->tile_w / 8) * (c->tile_h / 4) * 32;
  if (!ext.empty()) {
    // jobs on SATs first, then those on box tables, each group's tiles numbered from 0
    std::vector<BatchExtJob> jobs_dev;
    std::vector<float4> table_dev;
    std::vector<float> cuts;
    std::vector<size_t> table_at, cut_at;
    b->ext_aligned = true;
    for (int group = 0; group < 2; ++group) {
      unsigned blocks = 0;
      for (size_t k = 0; k < ext.size(); ++k) {
        if ((walks[k] != nullptr) != (group == 1)) continue;
        BatchExtJob J = ext[k];
        J.first_block = blocks;
        blocks += J.blocks_x * (unsigned)((J.f.H + J.f.tile_h - 1) / J.f.tile_h);
        table_at.push_back(table_dev.size());
        cut_at.push_back(cuts.size());
        if (group == 1) {
          const BoxWalk& w = *walks[k];
          table_dev.insert(table_dev.end(), w.o, w.o + w.n);
          cuts.insert(cuts.end(), w.cut, w.cut + w.n);
          J.bpad_a = w.pad_a; J.bpad_b = w.pad_b; J.bpad_w = w.pad_w; J.bfirst = w.first; J.bper = w.per;
        } else {
          if (!J.e.sat.sat32 && !J.e.sat.sat) return fail(c, CVR_ERR_NOT_READY, "cvr_batch_create: a job without a SAT");
          if (!aligned[k]) b->ext_aligned = false;
          table_dev.insert(table_dev.end(), tables[k].begin(), tables[k].end());
        }
        (group ? b->n_box : b->n_ext) += 1;
        jobs_dev.push_back(J);
      }
      (group ? b->box_blocks : b->ext_blocks) = blocks;
    }
    if (!table_dev.empty()) {
      NEED(c, cudaMalloc((void**)&b->d_tables, sizeof(float4) * table_dev.size()));
      CK(c, cudaMemcpy(b->d_tables, table_dev.data(), sizeof(float4) * table_dev.size(), cudaMemcpyHostToDevice));
    }
    if (!cuts.empty()) {
      NEED(c, cudaMalloc((void**)&b->d_cuts, sizeof(float) * cuts.size()));
      CK(c, cudaMemcpy(b->d_cuts, cuts.data(), sizeof(float) * cuts.size(), cudaMemcpyHostToDevice));
    }
    for (size_t k = 0; k < jobs_dev.size(); ++k) {
      BatchExtJob& J = jobs_dev[k];
      const float4* base = b->d_tables + table_at[k];
      if ((int)k >= b->n_ext) {
        J.bo = base;
        J.bcut = b->d_cuts + cut_at[k];
      } else if (J.tn > 0) {
        J.tlo = base;
        J.thi = base + J.tn;
        const size_t next = k + 1 < jobs_dev.size() ? table_at[k + 1] : table_dev.size();
        J.ttx = next - table_at[k] == 3 * (size_t)J.tn ? base + 2 * J.tn : nullptr;
      }
    }
    NEED(c, cudaMalloc((void**)&b->d_ext, sizeof(BatchExtJob) * jobs_dev.size()));
    CK(c, cudaMemcpy(b->d_ext, jobs_dev.data(), sizeof(BatchExtJob) * jobs_dev.size(), cudaMemcpyHostToDevice));
    // the compact SATs were the box tables' source: they go when no job reads them
    if (b->n_ext == 0) {
      CK(c, cudaStreamSynchronize(c->stream));
      for (uint4* p : b->sat32) cudaFree(p);
      b->sat32.clear();
    }
  }
  const size_t n_counters = 2 + sur.size();
  NEED(c, cudaMalloc((void**)&b->d_counters, sizeof(unsigned int) * n_counters));
  // the lanes' lists, each as large as its largest job needs (a lane without
  // room leaves its jobs to the direct marcher)
  const int lanes = (int)std::min<size_t>(sur.size(), kSurLanes);
  for (int l = 0; l < lanes; ++l) {
    size_t bytes = 0;
    for (size_t k = l; k < sur.size(); k += lanes) bytes = std::max(bytes, sur[k].bytes);
    if (bytes == 0) continue;
    cudaError_t me = spare_room(c, bytes, 0);
    if (me == cudaSuccess) me = cudaMalloc(&b->lists[l], bytes);
    if (me == cudaErrorMemoryAllocation) {
      cudaGetLastError();
      for (size_t k = l; k < sur.size(); k += lanes) sur[k].bytes = 0;
    } else if (me != cudaSuccess) {
      return cuda_fail(c, me, "cvr_batch_create: sample lists");
    }
  }
  // capture: counter and statistics resets, then the extinction launches
  // beside the lanes of surrogate frames
  struct Lanes {
    cudaStream_t s[kSurLanes] = {};
    cudaEvent_t fork = nullptr, join[kSurLanes] = {};
    ~Lanes() {
      for (cudaStream_t x : s)
        if (x) cudaStreamDestroy(x);
      for (cudaEvent_t x : join)
        if (x) cudaEventDestroy(x);
      if (fork) cudaEventDestroy(fork);
    }
  } lane;
  if (lanes > 0) CK(c, cudaEventCreateWithFlags(&lane.fork, cudaEventDisableTiming));
  for (int l = 0; l < lanes; ++l) {
    CK(c, cudaStreamCreateWithFlags(&lane.s[l], cudaStreamNonBlocking));
    CK(c, cudaEventCreateWithFlags(&lane.join[l], cudaEventDisableTiming));
  }
  cudaGraph_t g = nullptr;
  CK(c, cudaStreamBeginCapture(c->stream, cudaStreamCaptureModeRelaxed));
  cudaError_t e = cudaMemsetAsync(b->d_counters, 0, sizeof(unsigned int) * n_counters, c->stream);
  if (e == cudaSuccess) e = cudaMemsetAsync(b->d_stats, 0, sizeof(unsigned long long) * 3 * n_jobs, c->stream);
  if (e == cudaSuccess && lanes > 0) e = cudaEventRecord(lane.fork, c->stream);
  for (int l = 0; l < lanes && e == cudaSuccess; ++l) {
    cudaStream_t ls = lane.s[l];
    e = cudaStreamWaitEvent(ls, lane.fork, 0);
    for (size_t k = l; k < sur.size() && e == cudaSuccess; k += lanes) {
      const SurFrameJob& J = sur[k];
      if (J.bytes > 0)
        e = launch_deferred(b->lists[l], J.plan, J.f, light_terms(J.a.apply_occ, J.a.apply_sdw, J.a.ka, J.a.kd), false,
                            (unsigned)kSurPyramidTaps,
                            [&](const Deferred& d) { return launch_light_sur(J.f, J.a, J.tex, d, c->mlp->err, ls); },
                            ls);
      else
        e = launch_surrogate(J.f, J.a, J.tex, sur_spiral(J.f), b->d_counters + 2 + k, c->mlp->err, ls);
    }
    if (e == cudaSuccess) e = cudaEventRecord(lane.join[l], ls);
  }
  if (e == cudaSuccess && b->n_ext)
    e = launch_batch_extinction(b->d_ext, b->n_ext, b->ext_blocks, b->d_counters, c->tf_n, b->ext_max_table,
                                b->ext_threads, b->ext_variant, b->ext_compact, b->ext_aligned, c->stream);
  if (e == cudaSuccess && b->n_box)
    e = launch_batch_box(b->d_ext + b->n_ext, b->n_box, b->box_blocks, b->d_counters + 1, c->tf_n, b->ext_max_table,
                         b->ext_threads, b->ext_variant, c->stream);
  for (int l = 0; l < lanes && e == cudaSuccess; ++l) e = cudaStreamWaitEvent(c->stream, lane.join[l], 0);
  cudaError_t e2 = cudaStreamEndCapture(c->stream, &g);
  if (e != cudaSuccess || e2 != cudaSuccess) {
    if (g) cudaGraphDestroy(g);
    return cuda_fail(c, e != cudaSuccess ? e : e2, "cvr_batch_create: capture");
  }
  e = cudaGraphInstantiate(&b->graph, g, 0);
  cudaGraphDestroy(g);
  if (e != cudaSuccess) return cuda_fail(c, e, "cvr_batch_create: graph instantiate");
  *out = b.release();
  return CVR_OK;
}

cvr_status cvr_batch_run(cvr_batch* b) {
  if (!b || !b->ctx) return CVR_ERR_INVALID_ARG;
  cvr_ctx* c = b->ctx;
  CK(c, cudaSetDevice(c->device));
  CK(c, cudaGraphLaunch(b->graph, c->stream));
  return CVR_OK;
}

cvr_status cvr_batch_job_stats(cvr_batch* b, int job, cvr_frame_stats* out) {
  if (!b || !b->ctx || !out || job < 0 || job >= b->n_jobs) return CVR_ERR_INVALID_ARG;
  cvr_ctx* c = b->ctx;
  CK(c, cudaSetDevice(c->device));
  unsigned long long h[3];
  CK(c, cudaMemcpyAsync(h, b->d_stats + 3 * (size_t)job, sizeof h, cudaMemcpyDeviceToHost, c->stream));
  CK(c, cudaStreamSynchronize(c->stream));
  out->samples = h[0];
  out->shaded_samples = h[1];
  out->aux_fetches = h[2];
  out->kernel_ms = 0.0f;
  return mlp_check_err(c);
}

void cvr_batch_destroy(cvr_batch* b) {
  if (!b) return;
  if (b->ctx) {
    cudaSetDevice(b->ctx->device);
    cudaStreamSynchronize(b->ctx->stream);
  }
  delete b;
}

}  // extern "C"
