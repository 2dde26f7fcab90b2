// solver.cu - host side of the GB300 Frank-Wolfe solver: builds the device
// graph, demand and per-scenario state, enqueues FW iterations (captured into
// CUDA graphs), and implements the tapgpu_* handle API of include/tap_gpu.h.
#include "solver.cuh"

#include <signal.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cmath>
#include <cstdio>
#include <cstring>
#include <functional>
#include <future>
#include <limits>
#include <memory>
#include <numeric>
#include <system_error>
#include <thread>

namespace tapgpu {

namespace {
thread_local std::string g_message;
}

void set_message(const std::string& m) { g_message = m; }

#define TG_CUDA(call)                                                                   \
  do {                                                                                  \
    cudaError_t e_ = (call);                                                            \
    if (e_ != cudaSuccess) {                                                            \
      ::tapgpu::set_message(std::string(#call) + ": " + cudaGetErrorString(e_));       \
      return TAPGPU_ERR_CUDA;                                                           \
    }                                                                                   \
  } while (0)

#define TG_TRY(call)        \
  do {                      \
    int r_ = (call);        \
    if (r_ != TAPGPU_OK) {  \
      return r_;            \
    }                       \
  } while (0)

Ctx::~Ctx() {
  builder.reset();  // (its thread reads the context)
  if (gexec) cudaGraphExecDestroy(gexec);
  for (cudaEvent_t e : ev_pool) cudaEventDestroy(e);
  if (stream) cudaStreamDestroy(stream);
  for (auto& m : owned) cudaFree(m.p);
}

int Ctx::alloc(void** p, size_t bytes) {
  if (bytes == 0) bytes = 16;
  void* q = nullptr;
  cudaError_t e = cudaMalloc(&q, bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    set_message(std::string("cudaMalloc of ") + std::to_string(bytes) + " bytes: " +
                cudaGetErrorString(e));
    return TAPGPU_ERR_ALLOC;
  }
  owned.push_back({q, bytes});
  *p = q;
  return TAPGPU_OK;
}

cudaEvent_t Ctx::next_event() {
  if (ev_used == ev_pool.size()) {
    cudaEvent_t e = nullptr;
    if (cudaEventCreate(&e) != cudaSuccess) return nullptr;
    ev_pool.push_back(e);
  }
  return ev_pool[ev_used++];
}

// Record a timing event before (begin) or after a launch; inside a stream
// capture the record becomes an event node of the graph.
int Ctx::mark(int kind, bool begin) {
  if (!timing) return TAPGPU_OK;
  cudaEvent_t e = next_event();
  if (!e) return TAPGPU_ERR_CUDA;
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  TG_CUDA(cudaStreamIsCapturing(stream, &cs));
  if (cs == cudaStreamCaptureStatusActive)
    TG_CUDA(cudaEventRecordWithFlags(e, stream, cudaEventRecordExternal));
  else
    TG_CUDA(cudaEventRecord(e, stream));
  if (begin)
    timed.push_back({kind, e, nullptr});
  else if (!timed.empty())
    timed.back().b = e;
  return TAPGPU_OK;
}

// Accumulate the durations of the marked launches (stream already synchronised).
int Ctx::collect_timing() {
  for (const Timed& t : timed) {
    float ms = 0.f;
    if (t.a && t.b && cudaEventElapsedTime(&ms, t.a, t.b) == cudaSuccess) {
      kt_ms[t.kind] += ms;
      kt_n[t.kind] += 1;
    }
  }
  cudaGetLastError();
  return TAPGPU_OK;
}

static void free_owned(Ctx* c, void* p) {
  if (!p) return;
  for (size_t i = 0; i < c->owned.size(); ++i) {
    if (c->owned[i].p == p) {
      cudaFree(p);
      c->owned.erase(c->owned.begin() + static_cast<long>(i));
      return;
    }
  }
}

Graph Ctx::graph() const {
  Graph g;
  g.n1 = n1;
  g.m = M;
  g.first_thru = F;
  g.row_ptr = row_ptr;
  g.head = head;
  g.tail = tail;
  g.in_ptr = in_ptr;
  g.in_link = in_link;
  g.in_head = in_head;
  g.out_deg = out_deg;
  return g;
}

LinkParams Ctx::link_params() const {
  LinkParams lp;
  if (use_link_scen && sc_fft) {
    lp.fft = sc_fft;
    lp.alpha = sc_alpha;
    lp.beta = sc_beta;
    lp.ipow = sc_ipow;
    lp.stride = M;
    return lp;
  }
  lp.fft = fft;
  lp.alpha = alpha;
  lp.beta = beta;
  lp.ipow = ipow;
  lp.stride = 0;
  return lp;
}

LinkParams Ctx::link_params_of(int scen) const {
  LinkParams lp = link_params();
  const size_t off = static_cast<size_t>(scen) * static_cast<size_t>(lp.stride);
  lp.fft += off;
  lp.alpha += off;
  lp.beta += off;
  lp.ipow += off;
  lp.stride = 0;
  return lp;
}

Demand Ctx::demand() const {
  Demand dm;
  dm.od_ptr = od_ptr;
  dm.od_dest = od_dest;
  dm.od_q = use_dem_scen ? sc_od_q : od_q;
  dm.q_stride = use_dem_scen ? nnz : 0;
  dm.od_dem = od_dem;
  dm.inv_scale = inv_scale;
  dm.total = total_demand;
  return dm;
}

PathArgs Ctx::path_args(int nscen_slots) const {
  PathArgs a;
  std::memset(&a, 0, sizeof(a));
  a.g = graph();
  a.sources = sources;
  a.num_sources = Z;
  a.scen_list = scen_list;
  a.state = state;
  a.task_begin = 0;
  a.task_end = nscen_slots * Z;
  a.dist = dist;
  a.counter = counters;
  a.err = err;
  a.err_info = err_info;
  a.max_rounds = n1 + 2;
  a.dem = demand();
  a.y_fx = yfx;
  a.do_load = 1;
  a.scratch = path_scratch;
  a.scratch_stride = 0;
  a.all_global = opt.global_scratch == 2;
  a.stats = timing ? path_stats : nullptr;
  a.nf_delta = nf_delta;
  a.e4 = (!fp64 && e4 && (sssp_variant == kSsspNearFarQueue || sssp_variant == kSsspNearFarQueueWide))
             ? e4
             : nullptr;
  a.r4 = rev4 ? r4 : nullptr;
  a.r4d = fp64 ? r4d : nullptr;
  a.aon_c64 = aon_c64 ? 1 : 0;
  a.r4_more = r4_more;
  return a;
}

LinkArgs Ctx::link_args(int nscen, bool records) const {
  LinkArgs a;
  std::memset(&a, 0, sizeof(a));
  a.m = M;
  a.num_scen = nscen;
  a.scen_list = scen_list;
  a.lp = link_params();
  a.cap = cap;
  a.x = x;
  a.t = t;
  a.d = d;
  a.y_fx = yfx;
  // the label-correction kernels' records (with the hierarchy only where
  // those kernels take over)
  records |= !hier_on;
  if (records && !fp64) {
    a.e32 = e32;
    a.r32 = r32;
    a.e4 = e4;
    a.r4 = rev4 ? r4 : nullptr;
  }
  if (records && fp64) {
    a.r4d = r4d;
    a.w64 = w64;
  }
  a.ell_pos = ell_pos;
  a.e4x = e4x;
  a.r4_pos = r4_pos;
  a.r4x = r4x;
  a.n1 = n1;
  a.head = head;
  a.tail = tail;
  a.rpos = rpos;
  a.dtdx = dtdx;
  a.partials = partials;
  a.arrive = arrive;
  a.state = state;
  a.trace = trace;
  a.trace_cap = trace_cap;
  a.inv_scale = inv_scale;
  a.total_demand = total_demand;
  a.total_demand_s = use_dem_scen ? sc_total : nullptr;
  a.err = err;
  a.x_hist = x_hist;
  a.d_hist = d_hist;
  a.lam_hist = lam_hist;
  a.hist_cap = hist_cap;
  a.ckpt_every = ckpt_every;
  a.ls_mode = ls_mode;
  a.ls_ratio = fp64 ? 0 : 1;
  a.absent = use_link_scen ? sc_absent : nullptr;
  a.absent_words = absent_words;
  return a;
}

int Ctx::ensure_scenarios(int S) {
  if (S <= S_cap) return TAPGPU_OK;
  release_scenarios();
  const int rc = alloc_scenarios(S);
  if (rc != TAPGPU_OK) {
    release_scenarios();
    return rc;
  }
  S_cap = S;  // (last: a call after one that found no memory allocates again)
  return TAPGPU_OK;
}

// The per-scenario arrays, and the captured launches that hold their addresses.
void Ctx::release_scenarios() {
  S_cap = 0;
  if (gexec) {
    cudaGraphExecDestroy(gexec);
    gexec = nullptr;
  }
  g_nscen = -1;
  h_scen_list.clear();
  release_records();
  void* olds[] = {cap, x, t, d, dtdx, yfx, state, partials, arrive, trace, scen_list, x_hist, d_hist,
                  lam_hist};
  for (void* p : olds) free_owned(this, p);
  cap = x = t = d = dtdx = nullptr;
  yfx = nullptr;
  state = nullptr;
  partials = nullptr;
  arrive = nullptr;
  trace = nullptr;
  scen_list = nullptr;
  x_hist = d_hist = lam_hist = nullptr;
}

int Ctx::alloc_scenarios(int S) {
  const size_t sm = static_cast<size_t>(S) * M;
  TG_TRY(alloc_n(&cap, sm));
  TG_TRY(alloc_n(&x, sm));
  TG_TRY(alloc_n(&t, sm));
  TG_TRY(alloc_n(&d, sm));
  TG_TRY(alloc_n(&yfx, sm));
  if (opt.record_tape) TG_TRY(alloc_n(&dtdx, sm));
  TG_TRY(alloc_n(&state, static_cast<size_t>(S)));
  TG_TRY(alloc_n(&partials, static_cast<size_t>(S) * std::max(link_grid, ls_link_grid) * kNumSums));
  TG_TRY(alloc_n(&arrive, static_cast<size_t>(S)));
  TG_CUDA(cudaMemset(arrive, 0, sizeof(unsigned) * S));
  trace_cap = S == 1 ? 100000 : 4096;
  TG_TRY(alloc_n(&trace, static_cast<size_t>(S) * trace_cap * kTraceCols));
  TG_TRY(alloc_n(&scen_list, static_cast<size_t>(S)));
  if (opt.record_tape && opt.tape_capacity > 0) {
    hist_cap = opt.tape_capacity;
    ckpt_every = opt.tape_checkpoint > 0
                     ? opt.tape_checkpoint
                     : std::max(1, static_cast<int>(std::ceil(std::sqrt(double(hist_cap)))));
    TG_TRY(alloc_n(&x_hist, sm * (hist_cap / ckpt_every + 1)));
    TG_TRY(alloc_n(&d_hist, sm * hist_cap));
    TG_TRY(alloc_n(&lam_hist, static_cast<size_t>(S) * hist_cap));
  }
  return TAPGPU_OK;
}

// Whether an iteration of nscen scenarios takes less time on the hierarchy than
// on the label-correction kernels.  Both times (us) from fits to measurements
// on synthetic city networks of 1,200 to 40,000 nodes, 40 to 1,000 origins and 1
// to 64 scenarios, FP64:
//   label correction: one task 100 + 27 n/1000 or 250 + 15.5 n/1000 (80 n/1000
//     with its labels in global memory); among many, 0.05 + 0.132 n/1000 each
//     (0.17 where one of them fills an SM)
//   hierarchy: its levels one after the other, 140 + 25 each, however little
//     there is to do; 3.5 per 10^6 relaxations of an elimination per
//     scenario; 1.2 per 10^6 arcs and origin
// Measured, hierarchy : label correction in ms: 10,000 nodes, 1,000 origins, 1
// scenario 1.33 : 1.67, 4 scenarios 2.30 : 5.70, 16 scenarios 5.99 : 21.9; 40
// origins, 64 scenarios 5.42 : 3.63; 3,569 nodes, 101 origins, 16 scenarios
// 0.87 : 0.92, 64 scenarios 1.76 : 3.10; 22,500 nodes, 400 origins, 1 scenario
// 1.83 : 1.83, 2 scenarios 2.06 : 3.47; 40,000 nodes, 1,000 origins, 1 scenario
// 3.41 : 8.27, 4 scenarios 7.38 : 25.0.  Above the fitted sizes the line lies on
// the safe side: 60,000 nodes, 500 origins, 1 scenario 4.45 : 6.86, 4 scenarios
// 7.78 : 20.4; 100,000 nodes, 1,000 origins, 1 scenario 7.39 : 21.7, 4 scenarios
// 21.3 : 69.2, where the fits give 10.3 : 19.2 and 31.9 : 58.9.
bool Ctx::hier_pays(int nscen, int levels, double relaxations, int arcs) const {
  const double kn = n1 * 1e-3, tasks = static_cast<double>(nscen) * Z;
  const double one = sssp_smem ? std::min(100.0 + 27.0 * kn, 250.0 + 15.5 * kn) : 80.0 * kn;
  const double each = 0.05 + (sssp_smem && sssp_grid <= num_sms ? 0.17 : 0.132) * kn;
  const double corrected = std::max(one, 0.75 * one + each * tasks);
  const double swept = 140.0 + 25.0 * levels + 3.5e-6 * relaxations * nscen + 1.2e-6 * arcs * tasks;
  return corrected > 1.05 * swept;
}

// The path kernels of the next iterations of nscen scenarios, and their buffers.
int Ctx::choose_paths(int nscen) {
  TG_TRY(take_plan());
  bool on = false;  // (no room: the label-correction kernels)
  if (hier && hier_pays(nscen)) TG_TRY(have_hier(nscen, use_dem_scen, &on));
  if (!on) {
    const int rc = ensure_legacy(S_cap);
    if (rc != TAPGPU_OK) {  // (the next call starts from its own number of scenarios)
      release_scenarios();
      return rc;
    }
  }
  if (on != hier_on && gexec) {
    cudaGraphExecDestroy(gexec);
    gexec = nullptr;
  }
  hier_on = on;
  return TAPGPU_OK;
}

// The hierarchy's buffers and demand table for nscen scenarios; *there stays false
// where there is no room for them.
int Ctx::have_hier(int nscen, bool own_demand, bool* there) {
  // (the scenarios share the base demand: one row)
  unsigned long long** dem = own_demand ? &h_sc_dem : &h_dem;
  const long long* q = own_demand ? sc_od_q : od_q;
  const int rows = own_demand ? nscen : 1;
  if (hier_cap < nscen || !*dem) {
    if (gexec) cudaGraphExecDestroy(gexec);
    gexec = nullptr;
    int rc = *dem ? TAPGPU_OK : hier_demand(q, rows, dem);
    if (rc == TAPGPU_OK && hier_cap < nscen) rc = ensure_hier(nscen);
    if (rc != TAPGPU_OK) {
      release_hier();
      if (own_demand) {
        free_owned(this, h_sc_dem);
        h_sc_dem = nullptr;
      }
      return rc == TAPGPU_ERR_ALLOC ? TAPGPU_OK : rc;
    }
  }
  *there = true;
  return TAPGPU_OK;
}

// The weight records and the label buffer of the label-correction kernels.
int Ctx::ensure_legacy(int S) {
  if (records_ready) return TAPGPU_OK;
  const int rc = alloc_records(S);
  if (rc != TAPGPU_OK) {
    release_records();
    return rc;
  }
  // Unless the caller fixed the chunk, the label buffer grows to hold a whole
  // batch's tasks (up to 16 GiB), so that an iteration runs one shortest-path
  // and one loading launch instead of one per chunk, each with its tail.
  const int64_t tb = static_cast<int64_t>(n1) * (fp64 ? 8 : 4);
  if (opt.chunk_tasks <= 0) {
    const int64_t want = std::min<int64_t>(std::max<int64_t>(1, (int64_t(16) << 30) / tb),
                                           static_cast<int64_t>(S) * std::max(Z, 1));
    if (want > dist_tasks) {
      free_owned(this, dist);
      dist = nullptr;
      if (alloc(&dist, static_cast<size_t>(tb) * static_cast<size_t>(want)) == TAPGPU_OK)
        dist_tasks = want;
    }
  }
  const int held = ensure_labels();  // (no room for the larger one: by chunks of the first size)
  if (held != TAPGPU_OK) {
    release_records();
    return held;
  }
  records_ready = true;  // (last: a call after one that found no memory allocates again)
  return TAPGPU_OK;
}

// The label buffer of dist_tasks tasks.
int Ctx::ensure_labels() {
  if (dist) return TAPGPU_OK;
  return alloc(&dist, static_cast<size_t>(n1) * (fp64 ? 8 : 4) * static_cast<size_t>(dist_tasks));
}

void Ctx::release_records() {
  records_ready = false;
  void* olds[] = {e32, r32, e4, r4, r4d, w64};
  for (void* p : olds) free_owned(this, p);
  e32 = r32 = e4 = r4 = nullptr;
  r4d = nullptr;
  w64 = nullptr;
}

int Ctx::alloc_records(int S) {
  const size_t sm = static_cast<size_t>(S) * M, s4 = static_cast<size_t>(S) * n1 * 4;
  if (fp64) {
    TG_TRY(alloc_n(&w64, sm));
    // slots beyond a node's in-links keep an infinite weight: never tight
    TG_TRY(alloc_n(&r4d, s4));
    TG_CUDA(launch_fill_records4(r4d, s4, make_uint4(0u, 0u, 0u, 0x7ff00000u), 2 * num_sms, stream));
    return TAPGPU_OK;
  }
  TG_TRY(alloc_n(&e32, sm));
  TG_TRY(alloc_n(&r32, sm));
  TG_TRY(alloc_n(&e4, s4));
  TG_CUDA(cudaMemsetAsync(e4, 0, sizeof(uint2) * s4, stream));
  if (rev4) {
    // slots beyond a node's in-links keep an infinite weight: never tight
    TG_TRY(alloc_n(&r4, s4));
    TG_CUDA(launch_fill_records(r4, s4, make_uint2(0u, 0x7f800000u), 2 * num_sms, stream));
  }
  return TAPGPU_OK;
}

// ---------------------------------------------------------------------------
// elimination hierarchy
// ---------------------------------------------------------------------------

// The host plan and its image for the device, made by a thread of its own from
// the context's setup on; the first solve or loading waits for it (trees alone
// never do, and without demand it is not started).  Setup, and setup with a first
// solve of two iterations, ms: 10,000 nodes 9.3 and 17.0, 100,000 nodes 20 and
// 144; with the setup waiting for the plan 14.8 and 19.4, 120 and 144; without a
// plan 9.4 and 14.7, 20 and 89.
class HierBuilder {
 public:
  // (c has its network; dem is the caller's, see wait_read)
  HierBuilder(Ctx& c, const tapgpu_demand& dem) : dests_(c.n1, 0) {
    auto work = [this, &c, &dem] {
      each_pair(c, dem, [this](int64_t d) {
        dests_[d] = 1;
        return false;
      });
      read_.set_value();
      try {
        make(c);
      } catch (const std::bad_alloc&) {
        made_ = false;
      }
    };
    // (outlives the call: the caller's signals are not for it)
    sigset_t all, mask;
    sigfillset(&all);
    pthread_sigmask(SIG_SETMASK, &all, &mask);
    bool started = true;
    try {
      thread_ = std::thread(work);
    } catch (const std::system_error&) {
      started = false;
    }
    pthread_sigmask(SIG_SETMASK, &mask, nullptr);
    if (!started) work();
  }
  ~HierBuilder() {
    stop_ = true;
    if (thread_.joinable()) thread_.join();
  }
  // FP64 paths (integer labels break near-ties as exact sums do, which FP64
  // sums do too; the FP32 sums' ties fall otherwise) with demand between two
  // nodes.  A caller's choice of a label-correction kernel or of its shape
  // stands; networks small enough for the edge-list sweeps keep them.
  static bool wanted(const Ctx& c, const tapgpu_demand* dem) {
    const tapgpu_options& o = c.opt;
    return c.fp64 && dem && (c.n1 > kSmallNet || c.M > kSmallNet) &&
           !(o.sssp_variant || o.sssp_block || o.aon_block || o.nf_delta > 0 || o.global_scratch ||
             o.chunk_tasks || o.sssp_ctas_per_sm || o.aon_ctas_per_sm) &&
           each_pair(c, *dem, [](int64_t) { return true; });
  }
  // the caller's demand has been read
  void wait_read() { read_.get_future().wait(); }
  int finish(Ctx& c);

 private:
  // fn(destination) of the pairs of two nodes with demand, until it returns true
  template <class Fn>
  static bool each_pair(const Ctx& c, const tapgpu_demand& dem, Fn fn) {
    for (int64_t o = 1; o <= c.Z; ++o)
      for (int64_t i = dem.od_ptr[o]; i < dem.od_ptr[o + 1]; ++i)
        if (dem.od_demand[i] > 0 && dem.od_dest[i] != o && fn(dem.od_dest[i])) return true;
    return false;
  }
  void make(Ctx& c);

  HierPlan plan_;
  std::vector<char> dests_;
  std::promise<void> read_;
  std::atomic<bool> stop_{false};
  bool made_ = false;
  std::thread thread_;
  // one allocation and one copy for all of the plan's arrays
  std::vector<unsigned char> blob_;
  std::vector<std::function<void(unsigned char*)>> at_;
  HierPlan::Node* nodes_ = nullptr;
  int* chunk_of_ = nullptr;
  int u_exp0_ = 0, width_ = 0;
};

// (reads the context's network, notes where its pointers to the device go)
void HierBuilder::make(Ctx& c) {
  HierPlan& p = plan_;
  const int n1 = c.n1, Z = c.Z, M = c.M;
  if (!hier_build(n1, M, c.h_tail.data(), c.h_head.data(), c.F, dests_, 80.0 * n1, 1e11, p, &stop_))
    return;
  if (hier_climb_smem(p.climb) > kHierMaxClimb || p.climb > 0xffff) return;
  std::vector<int> dest_of(n1, -1);
  for (size_t i = 0; i < p.dest_node.size(); ++i) dest_of[p.dest_node[i]] = static_cast<int>(i);
  std::vector<unsigned short> iclimb(p.idx.size()), aclimb(static_cast<size_t>(p.arcs), 0);
  for (size_t i = 0; i < p.idx.size(); ++i) {
    const HierChunk& k = p.chunks[p.chunk_of[p.idx[i]]];
    iclimb[i] = static_cast<unsigned short>(k.coff + p.idx[i] - k.first);
  }
  for (const auto& k : p.chunks)
    for (int i = 0; i < k.k; ++i)
      std::fill_n(aclimb.begin() + k.woff + i * k.ld, k.ld, static_cast<unsigned short>(k.coff + i));
  auto put = [&](auto** dst, const auto& v) {
    at_.push_back([dst, off = blob_.size()](unsigned char* base) {
      *dst = reinterpret_cast<typename std::remove_reference<decltype(*dst)>::type>(base + off);
    });
    const auto* q = reinterpret_cast<const unsigned char*>(v.data());
    blob_.insert(blob_.end(), q, q + v.size() * sizeof(v[0]));
    blob_.resize((blob_.size() + 255) / 256 * 256);
  };
  blob_.reserve(sizeof(int) * (8 * static_cast<size_t>(p.arcs) + 8 * p.idx.size() + p.rel.size() +
                               64 * static_cast<size_t>(n1)));
  put(&c.hg.chunks, p.chunks);
  put(&c.hg.shut, p.shut);
  put(&c.hg.idx, p.idx);
  put(&c.hg.idx_climb, iclimb);
  put(&c.hg.arc_climb, aclimb);
  put(&c.hg.tgt_base, p.tgt_base);
  put(&c.hg.tgt_rel, p.tgt_rel);
  put(&c.hg.rel, p.rel);
  put(&c.hg.arc_link, p.arc_link);
  put(&c.hg.link_arc, p.link_arc);
  put(&c.hg.link_next, p.link_next);
  put(&c.hg.elims, p.elims);
  put(&c.hg.elim_pair, p.elim_pair);
  put(&c.hg.elim_close, p.elim_close);
  put(&nodes_, p.nodes);
  put(&chunk_of_, p.chunk_of);
  put(&c.hg.tiles, p.tiles);
  put(&c.hg.marks, p.marks);
  put(&c.hg.tops, p.tops);
  put(&c.hg.top_uidx, p.top_uidx);
  put(&c.hg.top_dest, p.top_dest);
  put(&c.hg.job_ptr, p.job_ptr);
  put(&c.hg.jobs, p.jobs);
  put(&c.hg.subs, p.subs);
  put(&c.hg.sub_ext, p.sub_ext);
  put(&c.hg.sub_rows, p.sub_rows);
  put(&c.hg.sub_slot, p.sub_slot);
  put(&c.hg.sub_ids, p.sub_ids);
  put(&c.h_dest_of, dest_of);
  // origins in position order: neighbours in the network share a group
  std::vector<int> opos(Z), by_pos(Z), column(Z), chain_ptr(Z + 1, 0), chain;
  for (int o = 0; o < Z; ++o) opos[o] = p.pos[o + 1];
  std::iota(by_pos.begin(), by_pos.end(), 0);
  std::sort(by_pos.begin(), by_pos.end(), [&](int a, int b) { return opos[a] < opos[b]; });
  for (int i = 0; i < Z; ++i) column[by_pos[i]] = i;
  for (int o = 0; o < Z; ++o) {
    for (int k = p.chunk_of[opos[o]]; k >= 0; k = p.chunks[k].parent) chain.push_back(k);
    chain_ptr[o + 1] = static_cast<int>(chain.size());
  }
  while (by_pos.size() % kHierWidth) by_pos.push_back(-1);
  put(&c.h_opos, opos);
  put(&c.h_group, by_pos);
  put(&c.h_column, column);
  put(&c.h_chain_ptr, chain_ptr);
  put(&c.h_chain, chain);
  width_ = static_cast<int>(by_pos.size());
  // first exponent: twice the largest cost of a path with the fewest links
  // from the first origin at free flow just fits
  std::vector<int> rp(n1 + 1, 0), queue{1};
  for (int k = 0; k < M; ++k) ++rp[c.h_tail[k] + 1];
  for (int v = 0; v < n1; ++v) rp[v + 1] += rp[v];
  std::vector<double> far(n1, -1.0);
  far[1] = 0.0;
  double most = 0.0;
  for (size_t i = 0; i < queue.size(); ++i) {
    const int v = queue[i];
    most = std::max(most, far[v]);
    for (int k = rp[v]; k < rp[v + 1]; ++k)
      if (far[c.h_head[k]] < 0) {
        far[c.h_head[k]] = far[v] + c.h_fft[k];
        queue.push_back(c.h_head[k]);
      }
  }
  int e = 0;
  if (most > 0) e = 59 - static_cast<int>(std::ceil(std::log2(most))) - 1;
  u_exp0_ = std::max(-900, std::min(900, e));
  made_ = true;
}

// The plan on the device, where the hierarchy can pay and there is room for it.
int HierBuilder::finish(Ctx& c) {
  if (thread_.joinable()) thread_.join();
  const HierPlan& p = plan_;
  if (!made_ || !c.hier_pays(4096, p.num_levels, p.relaxations, p.arcs)) return TAPGPU_OK;
  unsigned char* dev = nullptr;
  HierPlan::Pair* pairs = nullptr;
  if (c.alloc_n(&dev, blob_.size()) != TAPGPU_OK ||
      c.alloc_n(&pairs, static_cast<size_t>(p.num_pairs)) != TAPGPU_OK) {
    free_owned(&c, dev);
    return TAPGPU_OK;
  }
  TG_CUDA(cudaMemcpyAsync(dev, blob_.data(), blob_.size(), cudaMemcpyHostToDevice, c.stream));
  for (const auto& f : at_) f(dev);
  HierGraph& hg = c.hg;
  hg.n = p.n;
  hg.arcs = p.arcs;
  hg.climb = p.climb;
  hg.num_elims = static_cast<int>(p.elims.size());
  hg.num_marks = static_cast<int>(p.marks.size());
  hg.top_rows = p.top_rows;
  hg.top_levels = p.top_levels;
  hg.num_subs = static_cast<int>(p.subs.size());
  hg.pairs = pairs;
  TG_CUDA(launch_hier_pairs(hg, nodes_, static_cast<int>(p.nodes.size()), chunk_of_, pairs, c.stream));
  TG_CUDA(cudaStreamSynchronize(c.stream));  // (the copy reads blob_)
  c.hier_relaxations = p.relaxations;
  c.h_tile_ptr = p.tile_ptr;
  c.h_dests = static_cast<int>(p.dest_node.size());
  c.h_width = width_;
  c.u_exp0 = u_exp0_;
  c.hier = true;
  return TAPGPU_OK;
}

// Waits for a plan under way.
int Ctx::take_plan() {
  if (!builder) return TAPGPU_OK;
  const std::shared_ptr<HierBuilder> b = std::move(builder);
  return b->finish(*this);
}

// Demand by destination from the OD entries dev_q [nscen][nnz] (device).  A table of
// destinations x origins however few pairs there are (1,000 zones: 8 MB a
// scenario, 5,000: 200 MB), so it is made once a solve or loading takes the
// hierarchy and no larger than kHierBytes.
int Ctx::hier_demand(const long long* dev_q, int nscen, unsigned long long** dem) {
  const size_t row = static_cast<size_t>(h_dests) * h_width;
  if (!*dem) {
    if (row * nscen > kHierBytes / sizeof(unsigned long long)) return TAPGPU_ERR_ALLOC;
    TG_TRY(alloc_n(dem, row * nscen));
  }
  TG_CUDA(cudaMemsetAsync(*dem, 0, sizeof(unsigned long long) * row * nscen, stream));
  TG_CUDA(launch_hier_demand(od_ptr, od_dest, od_dem, h_dest_of, dev_q, nnz, nscen, Z, h_column, *dem, h_width,
                             static_cast<long long>(row), dem != &h_dem, stream));
  TG_CUDA(cudaStreamSynchronize(stream));
  return TAPGPU_OK;
}

void Ctx::release_hier() {
  void* olds[] = {h_w, h_mid, h_flow, h_d0, h_from, h_via, h_fup, h_dlab, h_vol, h_arr, h_list, h_list_n};
  for (void* p : olds) free_owned(this, p);
  h_w = h_mid = h_flow = h_d0 = h_fup = h_dlab = h_vol = nullptr;
  h_from = h_list = h_list_n = nullptr;
  h_arr = nullptr;
  h_via = nullptr;
  hier_cap = 0;
}

int Ctx::ensure_hier(int S) {
  release_hier();
  const size_t arcs3 = 3 * static_cast<size_t>(hg.arcs);
  const size_t climb = static_cast<size_t>(Z) * hg.climb;
  // labels of the top rows for every origin (padded to whole groups)
  const size_t top = static_cast<size_t>(h_width) * hg.top_rows;
  // per-scenario buffers within hier_bytes; more scenarios take turns in them
  const size_t per = arcs3 * 32 + climb * 21 + top * 18;
  hier_slots = static_cast<int>(std::max<size_t>(1, std::min<size_t>(S, hier_bytes / per)));
  const size_t ns = static_cast<size_t>(hier_slots), nc = ns * top;
  TG_TRY(alloc_n(&h_w, ns * arcs3));
  TG_TRY(alloc_n(&h_mid, ns * arcs3));
  TG_TRY(alloc_n(&h_flow, ns * arcs3));
  TG_TRY(alloc_n(&h_d0, ns * climb));
  TG_TRY(alloc_n(&h_from, ns * climb));
  TG_TRY(alloc_n(&h_via, ns * climb));
  TG_TRY(alloc_n(&h_fup, ns * climb));
  TG_TRY(alloc_n(&h_dlab, nc));
  TG_TRY(alloc_n(&h_vol, nc));
  TG_TRY(alloc_n(&h_arr, nc));
  TG_TRY(alloc_n(&h_list, ns * 2 * arcs3));
  TG_TRY(alloc_n(&h_list_n, ns * 4));
  // volumes are zero between tasks and iterations; padding reads labels of
  // other rows, which only have to be in range
  TG_CUDA(cudaMemsetAsync(h_flow, 0, ns * arcs3 * sizeof(unsigned long long), stream));
  TG_CUDA(cudaMemsetAsync(h_list_n, 0, ns * 4 * sizeof(int), stream));
  TG_CUDA(cudaMemsetAsync(h_vol, 0, nc * sizeof(*h_vol), stream));
  TG_CUDA(cudaMemsetAsync(h_dlab, 0, nc * sizeof(*h_dlab), stream));
  hier_cap = S;
  return TAPGPU_OK;
}

// Shortest paths and loading of the first nscen entries of scen_list at link
// costs cost[scenario * stride + link], into yfx.
int Ctx::enqueue_hier(int nscen, const double* cost, long long stride, cudaEvent_t between) {
  HierArgs a = hier_args(cost, stride);
  for (int s0 = 0; s0 < nscen; s0 += hier_slots) {
    a.slot0 = s0;
    a.nslots = std::min(hier_slots, nscen - s0);
    if (measuring) TG_TRY(mark(0, true));
    const int levels = static_cast<int>(h_tile_ptr.size()) - 1;
    TG_CUDA(launch_hier_eliminate(a, levels, h_tile_ptr.data(), stream));
    TG_CUDA(launch_hier_climb(a, stream));
    TG_CUDA(launch_hier_sweep(a, num_sms, stream));
    if (measuring) TG_TRY(mark(0, false));
    if (between) TG_CUDA(cudaEventRecord(between, stream));
    if (measuring) TG_TRY(mark(1, true));
    TG_CUDA(launch_hier_load(a, num_sms, stream));
    if (measuring) TG_TRY(mark(1, false));
    count_launches(hier_launches(hg, levels));
  }
  return TAPGPU_OK;
}

HierArgs Ctx::hier_args(const double* cost, long long stride) const {
  HierArgs a;
  std::memset(&a, 0, sizeof(a));
  a.h = hg;
  a.m = M;
  a.num_sources = Z;
  a.scen_list = scen_list;
  a.state = state;
  a.cost = cost;
  a.cost_stride = stride;
  a.absent = use_link_scen ? sc_absent : nullptr;
  a.absent_words = absent_words;
  a.w = h_w;
  a.mid = h_mid;
  a.flow = h_flow;
  a.d0 = h_d0;
  a.from = h_from;
  a.via = h_via;
  a.fup = h_fup;
  a.opos = h_opos;
  a.chain_ptr = h_chain_ptr;
  a.chain = h_chain;
  a.dest_dem = use_dem_scen ? h_sc_dem : h_dem;
  a.dest_stride = use_dem_scen ? static_cast<long long>(h_dests) * h_width : 0;
  a.dest_width = h_width;
  a.dlab = h_dlab;
  a.vol = h_vol;
  a.arr = h_arr;
  a.group = h_group;
  a.groups = h_width / kHierWidth;
  a.list = h_list;
  a.list_n = h_list_n;
  a.y_fx = yfx;
  return a;
}

constexpr int kHierRetries = 4;
constexpr int kHierRetryBits = 5;

// A paused scenario's state for its next try; false where the label-correction
// kernels take over.
static bool next_try(ScenState& st, int tries) {
  const int why = st.done;
  st.done = 0;
  st.maxlab = 0;
  st.minlab = ~0ull;
  if (why == kSpread || tries >= kHierRetries) return false;
  if (why == kPaused) st.u_exp -= kHierRetryBits;  // (of a coarse one the device set it)
  return true;
}

// One loading of the base demand at the costs of an API call (api_w64) into
// api_yfx, with a state of its own.  *loaded stays false where the labels do
// not fit after kHierRetries exponents: the label-correction kernels' case.
int Ctx::hier_load_api(bool* loaded) {
  HierArgs a = hier_args(api_w64, 0);
  a.scen_list = nullptr;
  a.absent = nullptr;
  a.dest_dem = h_dem;
  a.dest_stride = 0;
  a.y_fx = api_yfx;
  a.nslots = 1;
  if (!api_state) TG_TRY(alloc_n(&api_state, 1));
  a.state = api_state;
  ScenState st;
  std::memset(&st, 0, sizeof(st));
  st.u_exp = u_exp0;
  st.minlab = ~0ull;
  for (int tries = 0;; ++tries) {
    TG_CUDA(cudaMemcpyAsync(api_state, &st, sizeof(st), cudaMemcpyHostToDevice, stream));
    const int levels = static_cast<int>(h_tile_ptr.size()) - 1;
    TG_CUDA(launch_hier_eliminate(a, levels, h_tile_ptr.data(), stream));
    TG_CUDA(launch_hier_climb(a, stream));
    TG_CUDA(launch_hier_sweep(a, num_sms, stream));
    TG_CUDA(launch_hier_load(a, num_sms, stream));
    count_launches(hier_launches(hg, levels));
    TG_CUDA(cudaStreamSynchronize(stream));
    TG_CUDA(cudaMemcpy(&st, api_state, sizeof(st), cudaMemcpyDeviceToHost));
    if (!st.done) {
      *loaded = true;
      return TAPGPU_OK;
    }
    if (!next_try(st, tries)) return TAPGPU_OK;
  }
}

// Scenarios that left the integers' range repeat their iteration at a smaller
// exponent (those that used too little of it have their new one); one that
// does so repeatedly, or whose labels are spread too far, takes this iteration
// with the label-correction kernels, which also report a missing path.
int Ctx::resume_paused(int S, std::vector<ScenState>& st) {
  if (!hier_on) return TAPGPU_OK;
  std::vector<int> corrected;
  bool any = false;
  hier_course.resize(S);
  for (int s = 0; s < S; ++s) {
    if (st[s].done <= 1) continue;
    any = true;
    auto& c = hier_course[s];
    if (c.iter != st[s].iter) {
      c.iter = st[s].iter;
      c.pauses = 0;
    }
    if (st[s].done == kSpread) ++c.spread;
    if (!next_try(st[s], c.pauses++)) corrected.push_back(s);
    TG_CUDA(cudaMemcpyAsync(state + s, &st[s], sizeof(ScenState), cudaMemcpyHostToDevice, stream));
  }
  if (!any) return TAPGPU_OK;
  TG_CUDA(cudaStreamSynchronize(stream));
  if (corrected.empty()) return TAPGPU_OK;
  TG_TRY(run_corrected(corrected, 1));
  TG_TRY(sync_check());
  return read_states(S, st);
}

// Iterations of the listed scenarios with the label-correction kernels while
// the others are on the hierarchy.
int Ctx::run_corrected(const std::vector<int>& list, int iters) {
  TG_TRY(ensure_legacy(S_cap));
  TG_TRY(set_active(list));
  const int n = static_cast<int>(list.size());
  // (the hierarchy's loading writes volumes, that of these kernels adds to them)
  TG_CUDA(cudaMemsetAsync(yfx, 0, sizeof(unsigned long long) * static_cast<size_t>(S_cap) * M, stream));
  TG_CUDA(launch_records(link_args(n, true), link_grid, stream));
  for (int i = 0; i < iters; ++i) {
    TG_TRY(enqueue_paths(n, true, e32, r32, w64, yfx, true));
    TG_TRY(enqueue_tail(n, true));
  }
  return TAPGPU_OK;
}

// Iterations of the active scenarios.  One whose labels were spread too far in
// kSpreadIters iterations keeps the label-correction kernels for the rest of
// the solve: trying the hierarchy first costs an iteration more every time.
int Ctx::run_active(const std::vector<int>& active, int iters) {
  std::vector<int> swept, corrected;
  for (int s : active) (on_hierarchy(s) || !hier_on ? swept : corrected).push_back(s);
  if (!swept.empty()) {
    TG_TRY(set_active(swept));
    TG_TRY(run_graph(iters, static_cast<int>(swept.size())));
  }
  return corrected.empty() ? TAPGPU_OK : run_corrected(corrected, iters);
}

int Ctx::set_active(const std::vector<int>& active) {
  if (active == h_scen_list) return TAPGPU_OK;
  h_scen_list = active;
  TG_CUDA(cudaMemcpyAsync(scen_list, h_scen_list.data(), sizeof(int) * active.size(),
                          cudaMemcpyHostToDevice, stream));
  return TAPGPU_OK;
}

int Ctx::plan_launches() {
  cudaDeviceProp prop;
  TG_CUDA(cudaGetDeviceProperties(&prop, device));
  num_sms = prop.multiProcessorCount;
  const int optin = max_smem_optin(device);
  ls_mode = opt.line_search == kLsExact ? kLsExact : kLsReference;
  // default: the edge-list sweeps for small networks (tasks too small to
  // keep a queue busy), else the queue kernel
  const bool small = n1 <= kSmallNet && M <= kSmallNet;
  sssp_variant = (opt.sssp_variant >= kSsspRounds && opt.sssp_variant <= kSsspNearFarQueue) ||
                         opt.sssp_variant == kSsspSmall
                     ? opt.sssp_variant
                     : (small ? kSsspSmall : kSsspNearFarQueue);
  // the ring of the queue variant holds 16-bit node ids, and its padded
  // records 16-bit heads and degrees
  if (sssp_variant == kSsspNearFarQueue && !deg16) sssp_variant = kSsspNearFarQueueWide;
  const bool nf = sssp_variant == kSsspNearFar || sssp_variant == kSsspNearFarQueue ||
                  sssp_variant == kSsspNearFarQueueWide;
  sssp_block = opt.sssp_block > 0 ? opt.sssp_block : (nf ? 256 : 512);
  // the ring keeps one free slot per thread
  if ((sssp_variant == kSsspNearFarQueue || sssp_variant == kSsspNearFarQueueWide) &&
      sssp_block >= kQueueSlots)
    sssp_block = 256;
  // FP64 loading in the compact layout (10 bytes per node, two 512-thread
  // CTAs per SM) up to 65535 nodes
  aon_c64 = fp64 && n1 <= 0xffff && !opt.global_scratch;
  aon_block = opt.aon_block > 0 ? opt.aon_block : (aon_c64 ? 512 : 1024);
  // leave room for the kernels' static shared memory (a few words)
  const size_t room = optin > 1024 ? static_cast<size_t>(optin - 1024) : 0;
  sssp_smem = sssp_smem_bytes(n1, fp64, sssp_variant, M) <= room && !opt.global_scratch;
  aon_smem = aon_smem_bytes(n1, fp64, aon_c64) <= room && !opt.global_scratch;
  // near-far kernels whose shared memory leaves at most four 256-thread CTAs
  // per SM (FP64 labels of a 10k-node network: two) take 512 threads, so
  // that each task has more warps in flight (10k nodes, FP64: 77.0 -> 67.5 ms
  // per 64-scenario iteration)
  if (opt.sssp_block <= 0 && nf && sssp_smem &&
      sssp_occupancy(fp64, 256, true, n1, sssp_variant, M) * 256 <= 1024)
    sssp_block = 512;
  int so = sssp_occupancy(fp64, sssp_block, sssp_smem, n1, sssp_variant, M, opt.global_scratch == 2);
  int ao = aon_occupancy(fp64, aon_block, aon_smem, n1, aon_c64);
  if (so <= 0 || ao <= 0) {
    set_message("no resident CTA fits for the shortest-path kernels");
    return TAPGPU_ERR_UNSUPPORTED;
  }
  if (opt.sssp_ctas_per_sm > 0) so = std::min(so, opt.sssp_ctas_per_sm);
  if (opt.aon_ctas_per_sm > 0) ao = std::min(ao, opt.aon_ctas_per_sm);
  sssp_grid = so * num_sms;
  aon_grid = ao * num_sms;
  size_t scratch = 0;
  if (!sssp_smem) scratch = std::max(scratch, sssp_smem_bytes(n1, fp64, sssp_variant, M) * sssp_grid);
  if (!aon_smem) scratch = std::max(scratch, aon_smem_bytes(n1, fp64, aon_c64) * aon_grid);
  if (scratch) {
    TG_TRY(alloc(&path_scratch, scratch));
    path_scratch_bytes = scratch;
  }
  link_grid = std::max(1, std::min((M + 255) / 256, 2 * num_sms));
  // small networks: 64-thread blocks spread the line search's FP64 work
  // over more SMs
  ls_block = M <= kSmallNet ? kSmallLinkBlock : 256;
  ls_link_grid = std::max(1, std::min((M + ls_block - 1) / ls_block, 2 * num_sms * (256 / ls_block)));
  return TAPGPU_OK;
}

int Ctx::enqueue_paths(int nscen, bool load, const uint2* e32p, const uint2* r32p, const double* w64p,
                       unsigned long long* ydst, bool use_state) {
  const int64_t tasks = static_cast<int64_t>(nscen) * Z;
  for (int64_t t0 = 0; t0 < tasks; t0 += dist_tasks) {
    const int64_t t1 = std::min(tasks, t0 + dist_tasks);
    PathArgs a = path_args(nscen);
    if (!fp64 && (sssp_variant == kSsspNearFarQueue || sssp_variant == kSsspNearFarQueueWide))
      a.e4 = e32p == api_e32 ? api_e4 : e4;
    a.e32 = e32p;
    a.r32 = r32p;
    if (r32p != r32) a.r4 = nullptr;  // (the padded reverse records follow the context's own)
    if (w64p != w64) a.r4d = nullptr;
    a.w64 = w64p;
    a.y_fx = ydst;
    a.do_load = load ? 1 : 0;
    a.task_begin = static_cast<int>(t0);
    a.task_end = static_cast<int>(t1);
    if (!use_state) {
      a.state = nullptr;
      a.scen_list = nullptr;
      a.dem.od_q = od_q;
      a.dem.q_stride = 0;
    }
    const int ntask = static_cast<int>(t1 - t0);
    a.scratch_stride = static_cast<long long>(sssp_smem_bytes(n1, fp64, sssp_variant, M));
    // a block per task where the grids hold all of them
    const bool own = sssp_own_tasks(M, sssp_variant, sssp_block, sssp_smem) && ntask <= sssp_grid;
    const bool own_aon = ntask <= aon_grid;
    if (!own || !own_aon) TG_CUDA(cudaMemsetAsync(counters, 0, 2 * sizeof(int), stream));
    a.counter = own ? nullptr : counters;
    if (measuring) TG_TRY(mark(0, true));
    TG_CUDA(launch_sssp(a, fp64, std::min(sssp_grid, ntask), sssp_block, sssp_smem, sssp_variant,
                        stream));
    if (measuring) TG_TRY(mark(0, false));
    a.counter = own_aon ? nullptr : counters + 1;
    a.scratch_stride = static_cast<long long>(aon_smem_bytes(n1, fp64, aon_c64));
    if (measuring) TG_TRY(mark(1, true));
    TG_CUDA(launch_aon(a, fp64, std::min(aon_grid, ntask), aon_block, aon_smem, stream));
    if (measuring) TG_TRY(mark(1, false));
    count_launches(2);
  }
  return TAPGPU_OK;
}

void Ctx::count_launches(long long n) {
  cudaStreamCaptureStatus cs = cudaStreamCaptureStatusNone;
  cudaStreamIsCapturing(stream, &cs);
  if (cs == cudaStreamCaptureStatusActive)
    g_kernels += n;
  else
    launches += n;
}

int Ctx::enqueue_iteration(int nscen) {
  measuring = true;
  const int rc = hier_on ? enqueue_hier(nscen, t, M)
                      : enqueue_paths(nscen, true, e32, r32, w64, yfx, true);
  measuring = false;
  TG_TRY(rc);
  return enqueue_tail(nscen);
}

// line search and step of an iteration
int Ctx::enqueue_tail(int nscen, bool records) {
  LinkArgs la = link_args(nscen, records);
  if (M <= kSmallTail) {  // small networks: the line search and the step in one launch
    TG_TRY(mark(2, true));
    TG_CUDA(launch_fw_tail_small(la, stream));
    TG_TRY(mark(2, false));
    count_launches(1);
    return TAPGPU_OK;
  }
  TG_TRY(mark(2, true));
  const int passes = grid_passes();
  for (la.pass = 0; la.pass < passes; ++la.pass)
    TG_CUDA(launch_ls_pass(la, ls_grid(nscen), ls_block, stream));
  TG_CUDA(launch_ls_rest(la, stream));
  TG_TRY(mark(2, false));
  TG_TRY(mark(3, true));
  TG_CUDA(launch_step(la, step_grid(nscen), ls_block, stream));
  TG_TRY(mark(3, false));
  count_launches(passes + 2);
  return TAPGPU_OK;
}

// State reset, first all-or-nothing at free-flow costs (or warm flows), costs.
int Ctx::enqueue_initial(int nscen, bool warm) {
  if (!warm) TG_TRY(begin_paths(nscen));
  LinkArgs la = link_args(nscen);
  la.pass = warm ? 1 : 0;
  TG_CUDA(launch_init_flows(la, link_grid, stream));
  count_launches(1);
  return TAPGPU_OK;
}

// All-or-nothing at free-flow costs of scenarios 0 .. nscen-1
int Ctx::begin_paths(int nscen) {
  std::vector<int> all(nscen);
  std::iota(all.begin(), all.end(), 0);
  std::vector<int> corrected;
  if (!hier_on) corrected = all;
  const LinkParams lp = link_params();
  std::vector<ScenState> st;
  std::vector<int> todo = hier_on ? all : std::vector<int>(), again;
  for (int tries = 0; !todo.empty(); ++tries, todo.swap(again)) {
    TG_TRY(set_active(todo));
    TG_TRY(enqueue_hier(static_cast<int>(todo.size()), lp.fft, lp.stride));
    TG_TRY(read_states(nscen, st));
    again.clear();
    for (int s : todo) {
      if (st[s].done <= 1) continue;
      (next_try(st[s], tries) ? again : corrected).push_back(s);
      TG_CUDA(cudaMemcpyAsync(state + s, &st[s], sizeof(ScenState), cudaMemcpyHostToDevice, stream));
    }
    TG_CUDA(cudaStreamSynchronize(stream));
  }
  if (!corrected.empty()) {  // (these kernels also report a missing path)
    const int n = static_cast<int>(corrected.size());
    TG_TRY(ensure_legacy(S_cap));
    TG_TRY(set_active(corrected));
    TG_CUDA(launch_set_costs(link_args(n, true), link_grid, stream));
    count_launches(1);
    TG_TRY(enqueue_paths(n, true, e32, r32, w64, yfx, true));
  }
  return set_active(all);
}

int Ctx::run_graph(int iters, int nscen) {
  if (!opt.use_graphs) {
    timed.clear();
    ev_used = 0;
    for (int i = 0; i < iters; ++i) TG_TRY(enqueue_iteration(nscen));
    if (timing) {
      TG_CUDA(cudaStreamSynchronize(stream));
      collect_timing();
    }
    return TAPGPU_OK;
  }
  if (!gexec || g_iters != iters || g_nscen != nscen || g_dem != use_dem_scen ||
      g_links != use_link_scen) {
    if (gexec) {
      cudaGraphExecDestroy(gexec);
      gexec = nullptr;
    }
    timed.clear();
    ev_used = 0;
    g_kernels = 0;
    cudaGraph_t graph = nullptr;
    TG_CUDA(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal));
    int rc = TAPGPU_OK;
    for (int i = 0; i < iters && rc == TAPGPU_OK; ++i) rc = enqueue_iteration(nscen);
    cudaError_t ec = cudaStreamEndCapture(stream, &graph);
    if (rc != TAPGPU_OK) {
      if (graph) cudaGraphDestroy(graph);
      return rc;
    }
    if (ec != cudaSuccess) {
      set_message(std::string("graph capture: ") + cudaGetErrorString(ec));
      return TAPGPU_ERR_CUDA;
    }
    cudaError_t ei = cudaGraphInstantiate(&gexec, graph, 0);
    cudaGraphDestroy(graph);
    if (ei != cudaSuccess) {
      set_message(std::string("graph instantiate: ") + cudaGetErrorString(ei));
      gexec = nullptr;
      return TAPGPU_ERR_CUDA;
    }
    g_iters = iters;
    g_nscen = nscen;
    g_dem = use_dem_scen;
    g_links = use_link_scen;
  }
  TG_CUDA(cudaGraphLaunch(gexec, stream));
  launches += g_kernels;
  if (timing) {
    // the graph's event nodes are re-recorded by every replay: read them now
    TG_CUDA(cudaStreamSynchronize(stream));
    collect_timing();
  }
  return TAPGPU_OK;
}

int Ctx::sync_check() {
  TG_CUDA(cudaStreamSynchronize(stream));
  int e = 0;
  TG_CUDA(cudaMemcpy(&e, err, sizeof(int), cudaMemcpyDeviceToHost));
  if (e & kErrNoPath) {
    int info[2] = {0, 0};
    cudaMemcpy(info, err_info, sizeof(info), cudaMemcpyDeviceToHost);
    set_message("ERROR: no path from " + std::to_string(info[0]) + " to " +
                std::to_string(info[1]));
    return TAPGPU_ERR_NO_PATH;
  }
  if (e & (kErrRounds | kErrWalk | kErrPending)) {
    set_message("device loop hit its bound (error bits " + std::to_string(e) + ")");
    return TAPGPU_ERR_NO_CONVERGENCE;
  }
  return TAPGPU_OK;
}

int Ctx::read_states(int S, std::vector<ScenState>& out) {
  out.resize(S);
  TG_CUDA(cudaMemcpyAsync(out.data(), state, sizeof(ScenState) * S, cudaMemcpyDeviceToHost,
                          stream));
  TG_CUDA(cudaStreamSynchronize(stream));
  return TAPGPU_OK;
}

// ---------------------------------------------------------------------------
// construction
// ---------------------------------------------------------------------------

static int validate(const tapgpu_network* net, const tapgpu_demand* dem) {
  if (!net || !net->init || !net->term || !net->capacity || !net->fft || !net->alpha ||
      !net->beta) {
    set_message("network arrays missing");
    return TAPGPU_ERR_ARG;
  }
  if (net->num_nodes < 1 || net->num_links < 1 || net->num_nodes > (1 << 30) ||
      net->num_links > (1ll << 31) - 2) {
    set_message("network size out of range");
    return TAPGPU_ERR_ARG;
  }
  if (net->num_zones < 0 || net->num_zones > net->num_nodes || net->first_thru_node < 0) {
    set_message("zone count or first thru node out of range");
    return TAPGPU_ERR_ARG;
  }
  for (int64_t k = 0; k < net->num_links; ++k) {
    const int64_t a = net->init[k], b = net->term[k];
    // node 0 is the reference's unused row; 0-based graphs (the Python
    // extension's) use it as an ordinary node
    if (a < 0 || a > net->num_nodes || b < 0 || b > net->num_nodes) {
      set_message("link " + std::to_string(k) + " has a node outside 0..N");
      return TAPGPU_ERR_ARG;
    }
    if (!(net->fft[k] >= 0) || !std::isfinite(net->fft[k]) || !(net->alpha[k] >= 0) ||
        !std::isfinite(net->alpha[k]) || !std::isfinite(net->beta[k]) ||
        std::isnan(net->capacity[k])) {
      set_message("link " + std::to_string(k) + " has an invalid cost parameter");
      return TAPGPU_ERR_ARG;
    }
  }
  if (dem) {
    if (dem->num_origins < 0 || dem->num_origins > net->num_nodes ||
        (dem->num_origins > 0 && (!dem->od_ptr || !dem->od_dest || !dem->od_demand))) {
      set_message("demand arrays missing or origin count out of range");
      return TAPGPU_ERR_ARG;
    }
    for (int64_t o = 1; o <= dem->num_origins; ++o)
      if (dem->od_ptr[o + 1] < dem->od_ptr[o]) {
        set_message("demand pointers not monotone");
        return TAPGPU_ERR_ARG;
      }
    const int64_t nnz = dem->num_origins > 0 ? dem->od_ptr[dem->num_origins + 1] : 0;
    for (int64_t i = 0; i < nnz; ++i)
      if (dem->od_dest[i] < 0 || dem->od_dest[i] > net->num_nodes ||
          std::isnan(dem->od_demand[i])) {
        set_message("demand entry " + std::to_string(i) + " invalid");
        return TAPGPU_ERR_ARG;
      }
  }
  return TAPGPU_OK;
}

static int create_impl(const tapgpu_network* net, const tapgpu_demand* dem,
                       const tapgpu_options* opt_in, Ctx** out) {
  TG_TRY(validate(net, dem));
  int ndev = 0;
  if (cudaGetDeviceCount(&ndev) != cudaSuccess || ndev == 0) {
    cudaGetLastError();
    set_message("no CUDA device");
    return TAPGPU_ERR_NO_DEVICE;
  }
  tapgpu_options opt;
  tapgpu_default_options(&opt);
  if (opt_in) opt = *opt_in;
  if (opt.device < 0 || opt.device >= ndev) {
    set_message("device ordinal out of range");
    return TAPGPU_ERR_ARG;
  }
  TG_CUDA(cudaSetDevice(opt.device));
  Ctx* c = new Ctx();
  std::unique_ptr<Ctx> guard(c);
  c->opt = opt;
  c->device = opt.device;
  c->fp64 = opt.precision == TAPGPU_FP64;
  c->N = static_cast<int>(net->num_nodes);
  c->n1 = c->N + 1;
  c->M = static_cast<int>(net->num_links);
  c->Z = static_cast<int>(dem ? dem->num_origins : net->num_zones);
  c->F = static_cast<int>(std::min<int64_t>(net->first_thru_node, c->n1 + 1));
  const int M = c->M, n1 = c->n1;

  // links sorted by (init, term) as tap/parsetapfiles.c:528-540 orders them
  c->perm.resize(M);
  std::iota(c->perm.begin(), c->perm.end(), 0);
  std::stable_sort(c->perm.begin(), c->perm.end(), [&](int64_t a, int64_t b) {
    if (net->init[a] != net->init[b]) return net->init[a] < net->init[b];
    return net->term[a] < net->term[b];
  });
  c->h_tail.resize(M);
  c->h_head.resize(M);
  c->h_cap.resize(M);
  c->h_fft.resize(M);
  c->h_alpha.resize(M);
  c->h_beta.resize(M);
  std::vector<unsigned char> ip(M);
  double min_cap = DBL_MAX;
  for (int k = 0; k < M; ++k) {
    const int64_t e = c->perm[k];
    c->h_tail[k] = static_cast<int>(net->init[e]);
    c->h_head[k] = static_cast<int>(net->term[e]);
    c->h_cap[k] = net->capacity[e];
    c->h_fft[k] = net->fft[e];
    c->h_alpha[k] = net->alpha[e];
    c->h_beta[k] = net->beta[e];
    const double b = net->beta[e];
    ip[k] = (b >= 0 && b <= 15 && std::floor(b) == b) ? static_cast<unsigned char>(b) : 255;
    if (c->h_cap[k] > 0.0 && c->h_cap[k] < min_cap) min_cap = c->h_cap[k];
  }
  // tap/tap_frankwolfe_pthread.c:654-669 zero capacity -> smallest nonzero capacity
  for (int k = 0; k < M; ++k)
    if (!(c->h_cap[k] > 0.0)) c->h_cap[k] = min_cap;
  {
    double s = 0.0;
    for (int k = 0; k < M; ++k) s += c->h_fft[k];
    const double mean = s / M;
    c->nf_delta = opt.nf_delta > 0 ? opt.nf_delta : (mean > 0 ? 16.0 * mean : 1.0);
  }

  if (HierBuilder::wanted(*c, dem)) c->builder = std::make_shared<HierBuilder>(*c, *dem);

  std::vector<int> rp(n1 + 1, 0), ip_in(n1 + 1, 0), inl(M);
  for (int k = 0; k < M; ++k) {
    rp[c->h_tail[k] + 1]++;
    ip_in[c->h_head[k] + 1]++;
  }
  for (int v = 0; v < n1; ++v) {
    rp[v + 1] += rp[v];
    ip_in[v + 1] += ip_in[v];
  }
  c->h_rpos.resize(M);
  {
    std::vector<int> fill(ip_in.begin(), ip_in.end() - 1);
    for (int k = 0; k < M; ++k) {
      c->h_rpos[k] = fill[c->h_head[k]];
      inl[fill[c->h_head[k]]++] = k;
    }
  }

  TG_TRY(c->alloc_n(&c->row_ptr, n1 + 1));
  TG_TRY(c->alloc_n(&c->head, M));
  TG_TRY(c->alloc_n(&c->tail, M));
  TG_TRY(c->alloc_n(&c->in_ptr, n1 + 1));
  TG_TRY(c->alloc_n(&c->in_link, M));
  TG_TRY(c->alloc_n(&c->in_head, M));
  TG_TRY(c->alloc_n(&c->out_deg, n1));
  TG_TRY(c->alloc_n(&c->ell_pos, M));
  TG_TRY(c->alloc_n(&c->e4x, M));
  TG_TRY(c->alloc_n(&c->rpos, M));
  TG_TRY(c->alloc_n(&c->fft, M));
  TG_TRY(c->alloc_n(&c->alpha, M));
  TG_TRY(c->alloc_n(&c->beta, M));
  TG_TRY(c->alloc_n(&c->ipow, M));
  TG_CUDA(cudaMemcpy(c->row_ptr, rp.data(), sizeof(int) * (n1 + 1), cudaMemcpyHostToDevice));
  TG_CUDA(cudaMemcpy(c->head, c->h_head.data(), sizeof(int) * M, cudaMemcpyHostToDevice));
  TG_CUDA(cudaMemcpy(c->tail, c->h_tail.data(), sizeof(int) * M, cudaMemcpyHostToDevice));
  TG_CUDA(cudaMemcpy(c->in_ptr, ip_in.data(), sizeof(int) * (n1 + 1), cudaMemcpyHostToDevice));
  TG_CUDA(cudaMemcpy(c->in_link, inl.data(), sizeof(int) * M, cudaMemcpyHostToDevice));
  {
    std::vector<int> ih(M);
    for (int i = 0; i < M; ++i) ih[i] = c->h_head[inl[i]];
    TG_CUDA(cudaMemcpy(c->in_head, ih.data(), sizeof(int) * M, cudaMemcpyHostToDevice));
    std::vector<int> deg(n1), pos(M);
    for (int v = 0; v < n1; ++v) deg[v] = rp[v + 1] - rp[v];
    for (int k = 0; k < M; ++k) {
      const int v = c->h_tail[k], j = k - rp[v];
      pos[k] = j < 4 ? v * 4 + j : -1;
    }
    c->h_ell_pos = pos;
    int maxdeg = 0;
    for (int v = 0; v < n1; ++v) maxdeg = std::max(maxdeg, deg[v]);
    c->deg16 = n1 <= 0xffff && maxdeg <= 0xffff;
    c->h_e4x.resize(M);
    for (int k = 0; k < M; ++k) {
      const unsigned h = static_cast<unsigned>(c->h_head[k]);
      c->h_e4x[k] = c->deg16 ? h | (static_cast<unsigned>(deg[c->h_tail[k]]) << 16) : h;
    }
    TG_CUDA(cudaMemcpy(c->out_deg, deg.data(), sizeof(int) * n1, cudaMemcpyHostToDevice));
    TG_CUDA(cudaMemcpy(c->ell_pos, pos.data(), sizeof(int) * M, cudaMemcpyHostToDevice));
    // padded reverse records: FP64 paths always ({link, tail, weight}),
    // FP32 paths when nodes and links fit 16 bits ({link << 16 | tail, weight})
    c->rev4 = !c->fp64 && n1 <= 0xffff && M <= 0xffff;
    if (c->rev4 || c->fp64) {
      std::vector<int> rpos4(M);
      for (int k = 0; k < M; ++k) {
        const int v = c->h_head[k], j = c->h_rpos[k] - ip_in[v];
        rpos4[k] = j < 4 ? v * 4 + j : -1;
      }
      std::vector<unsigned> more((n1 + 31) / 32, 0u);
      for (int v = 0; v < n1; ++v)
        if (ip_in[v + 1] - ip_in[v] > 4) more[v >> 5] |= 1u << (v & 31);
      TG_TRY(c->alloc_n(&c->r4_pos, M));
      TG_TRY(c->alloc_n(&c->r4_more, more.size()));
      TG_CUDA(cudaMemcpy(c->r4_pos, rpos4.data(), sizeof(int) * M, cudaMemcpyHostToDevice));
      TG_CUDA(cudaMemcpy(c->r4_more, more.data(), sizeof(unsigned) * more.size(),
                         cudaMemcpyHostToDevice));
    }
    if (c->rev4) {
      std::vector<unsigned> rx(M);
      for (int k = 0; k < M; ++k)
        rx[k] = (static_cast<unsigned>(k) << 16) | static_cast<unsigned>(c->h_tail[k]);
      TG_TRY(c->alloc_n(&c->r4x, M));
      TG_CUDA(cudaMemcpy(c->r4x, rx.data(), sizeof(unsigned) * M, cudaMemcpyHostToDevice));
    }
    TG_CUDA(cudaMemcpy(c->e4x, c->h_e4x.data(), sizeof(unsigned) * M, cudaMemcpyHostToDevice));
  }
  TG_CUDA(cudaMemcpy(c->rpos, c->h_rpos.data(), sizeof(int) * M, cudaMemcpyHostToDevice));
  TG_CUDA(cudaMemcpy(c->fft, c->h_fft.data(), sizeof(double) * M, cudaMemcpyHostToDevice));
  TG_CUDA(cudaMemcpy(c->alpha, c->h_alpha.data(), sizeof(double) * M, cudaMemcpyHostToDevice));
  TG_CUDA(cudaMemcpy(c->beta, c->h_beta.data(), sizeof(double) * M, cudaMemcpyHostToDevice));
  TG_CUDA(cudaMemcpy(c->ipow, ip.data(), M, cudaMemcpyHostToDevice));

  // demand as a CSR over origin slots 0..Z-1 (origin node = slot + 1)
  const int Z = c->Z;
  std::vector<int> optr(Z + 1, 0), odest;
  std::vector<long long> oq;
  std::vector<double> odem;
  double total = 0.0, pos = 0.0;
  if (dem && Z > 0) {
    for (int o = 1; o <= Z; ++o)
      for (int64_t i = dem->od_ptr[o]; i < dem->od_ptr[o + 1]; ++i) {
        total += dem->od_demand[i];  // tap/tap_functions.c:377-386 sums every entry
        if (dem->od_demand[i] > 0) pos += dem->od_demand[i];
      }
    // fixed point with headroom: every node/link total stays below 2^61
    int bits = 40;
    if (pos > 1.0) bits = std::min(40, 61 - static_cast<int>(std::ceil(std::log2(pos))) - 1);
    c->scale_bits = bits;
    const double scale = std::ldexp(1.0, bits);
    for (int o = 1; o <= Z; ++o) {
      for (int64_t i = dem->od_ptr[o]; i < dem->od_ptr[o + 1]; ++i) {
        const double v = dem->od_demand[i];
        odest.push_back(static_cast<int>(dem->od_dest[i]));
        odem.push_back(v);
        oq.push_back(v > 0 ? std::llrint(v * scale) : 0);
      }
      optr[o] = static_cast<int>(odest.size());
    }
  }
  c->inv_scale = std::ldexp(1.0, -c->scale_bits);
  c->total_demand = total;
  c->h_od_dem = odem;
  c->nnz = static_cast<long long>(odem.size());
  std::vector<int> src(std::max(Z, 1));
  for (int i = 0; i < Z; ++i) src[i] = i + 1;
  TG_TRY(c->alloc_n(&c->od_ptr, Z + 1));
  TG_TRY(c->alloc_n(&c->od_dest, std::max<size_t>(odest.size(), 1)));
  TG_TRY(c->alloc_n(&c->od_q, std::max<size_t>(oq.size(), 1)));
  TG_TRY(c->alloc_n(&c->od_dem, std::max<size_t>(odem.size(), 1)));
  TG_TRY(c->alloc_n(&c->sources, std::max(Z, 1)));
  TG_CUDA(cudaMemcpy(c->od_ptr, optr.data(), sizeof(int) * (Z + 1), cudaMemcpyHostToDevice));
  if (!odest.empty()) {
    TG_CUDA(cudaMemcpy(c->od_dest, odest.data(), sizeof(int) * odest.size(),
                       cudaMemcpyHostToDevice));
    TG_CUDA(cudaMemcpy(c->od_q, oq.data(), sizeof(long long) * oq.size(), cudaMemcpyHostToDevice));
    TG_CUDA(cudaMemcpy(c->od_dem, odem.data(), sizeof(double) * odem.size(),
                       cudaMemcpyHostToDevice));
  }
  TG_CUDA(cudaMemcpy(c->sources, src.data(), sizeof(int) * src.size(), cudaMemcpyHostToDevice));

  TG_CUDA(cudaStreamCreateWithFlags(&c->stream, cudaStreamNonBlocking));
  TG_TRY(c->plan_launches());
  TG_TRY(c->alloc_n(&c->counters, 2));
  TG_TRY(c->alloc_n(&c->err, 1));
  TG_TRY(c->alloc_n(&c->err_info, 2));
  TG_TRY(c->alloc_n(&c->path_stats, 8));
  TG_CUDA(cudaMemset(c->err, 0, sizeof(int)));
  TG_CUDA(cudaMemset(c->path_stats, 0, 8 * sizeof(unsigned long long)));

  // shortest-path label scratch between the two path kernels
  const size_t tb = static_cast<size_t>(n1) * (c->fp64 ? 8 : 4);
  int64_t chunk = opt.chunk_tasks > 0 ? opt.chunk_tasks
                                      : std::max<int64_t>(1, (int64_t(2) << 30) / static_cast<int64_t>(tb));
  chunk = std::max<int64_t>(1, std::min<int64_t>(chunk, 1 << 30));
  c->dist_tasks = std::min<int64_t>(chunk, std::max<int64_t>(Z, 1) * 4096);
  TG_TRY(c->ensure_labels());
  TG_TRY(c->alloc_n(&c->api_e32, M));
  TG_TRY(c->alloc_n(&c->api_e4, static_cast<size_t>(n1) * 4));
  TG_CUDA(cudaMemset(c->api_e4, 0, sizeof(uint2) * static_cast<size_t>(n1) * 4));
  TG_TRY(c->alloc_n(&c->api_r32, M));
  TG_TRY(c->alloc_n(&c->api_w64, M));
  TG_TRY(c->alloc_n(&c->api_yfx, M));
  TG_TRY(c->ensure_scenarios(1));
  TG_CUDA(cudaMemcpy(c->cap, c->h_cap.data(), sizeof(double) * M, cudaMemcpyHostToDevice));
  if (c->builder)
    c->builder->wait_read();
  else
    TG_TRY(c->choose_paths(1));
  *out = guard.release();
  return TAPGPU_OK;
}

static int upload_states(Ctx* c, int S, int max_iters, double target) {
  std::vector<ScenState> st(S);
  for (auto& s : st) {
    std::memset(&s, 0, sizeof(s));
    s.max_iters = max_iters;
    s.target_relgap = target;
    s.relgap = DBL_MAX;
    s.best_lb = -DBL_MAX;
    s.u_exp = c->u_exp0;
    s.minlab = ~0ull;
  }
  c->hier_course.clear();
  TG_CUDA(cudaMemcpyAsync(c->state, st.data(), sizeof(ScenState) * S, cudaMemcpyHostToDevice,
                          c->stream));
  TG_CUDA(cudaMemsetAsync(c->err, 0, sizeof(int), c->stream));
  return TAPGPU_OK;
}

// Iterations per launch, at most cap, such that launches of one size (one
// captured graph) make up the total: a divisor of it over cap / 2, else equal
// parts, the last of which finds the scenario done for what it has too much.
// (10 iterations as 8 and 2 made two graphs in every call: 1 of 18 ms with the
// hierarchy's 60 nodes an iteration.)
static int equal_parts(int total, int cap) {
  if (total <= 0) return cap;
  if (total <= cap) return total;
  for (int n = cap; 2 * n > cap; --n)
    if (total % n == 0) return n;
  const int launches = (total + cap - 1) / cap;
  return (total + launches - 1) / launches;
}

static int iterate_until_done(Ctx* c, int S, int max_iters, std::vector<ScenState>& st) {
  // iterations per graph launch: enough to hide launch gaps, few enough that
  // finished scenarios do not linger
  // (small networks: the wait and the state's copy after a launch cost 30 us)
  const bool small = c->n1 <= kSmallNet && c->M <= kSmallNet;
  const int cap = c->opt.iters_per_launch > 0 ? c->opt.iters_per_launch
                                              : (S == 1 ? (small ? 16 : 8) : 4);
  const int per = equal_parts(max_iters, cap);
  std::vector<int> active;
  for (;;) {
    TG_TRY(c->read_states(S, st));
    TG_TRY(c->sync_check());
    TG_TRY(c->resume_paused(S, st));
    active.clear();
    for (int s = 0; s < S; ++s)
      if (!st[s].done) active.push_back(s);
    if (active.empty()) break;
    TG_TRY(c->run_active(active, per));
  }
  return TAPGPU_OK;
}

static void fill_result(const ScenState& s, int err_bits, tapgpu_result* r) {
  r->iterations = s.iter;
  r->error_bits = err_bits;
  r->objective = s.obj;
  r->relgap = s.relgap;
  r->total_cost = s.vht_end;
  r->avg_excess = s.avg_excess;
  r->lambda_last = s.lambda;
}

}  // namespace tapgpu

using tapgpu::Ctx;

extern "C" {

void tapgpu_default_options(tapgpu_options* o) {
  std::memset(o, 0, sizeof(*o));
  o->precision = TAPGPU_FP64;
  o->device = 0;
  o->use_graphs = 1;
}

const char* tapgpu_status_string(int s) {
  switch (s) {
    case TAPGPU_OK: return "ok";
    case TAPGPU_ERR_ARG: return "invalid argument";
    case TAPGPU_ERR_CUDA: return "CUDA error";
    case TAPGPU_ERR_NO_PATH: return "no path for a positive demand";
    case TAPGPU_ERR_NO_CONVERGENCE: return "device loop hit its bound";
    case TAPGPU_ERR_ALLOC: return "allocation failed";
    case TAPGPU_ERR_UNSUPPORTED: return "unsupported size";
    case TAPGPU_ERR_NO_DEVICE: return "no CUDA device";
    default: return "unknown status";
  }
}

const char* tapgpu_last_message(void) { return tapgpu::g_message.c_str(); }

int tapgpu_create(const tapgpu_network* net, const tapgpu_demand* dem, const tapgpu_options* opt,
                  tapgpu_ctx** out) {
  if (!out) return TAPGPU_ERR_ARG;
  *out = nullptr;
  Ctx* c = nullptr;
  int rc = tapgpu::create_impl(net, dem, opt, &c);
  if (rc != TAPGPU_OK) return rc;
  *out = new tapgpu_ctx{c};
  return TAPGPU_OK;
}

void tapgpu_destroy(tapgpu_ctx* ctx) {
  if (!ctx) return;
  cudaSetDevice(ctx->c->device);
  delete ctx->c;
  delete ctx;
}

int tapgpu_set_capacity(tapgpu_ctx* ctx, const double* capacity) {
  if (!ctx || !capacity) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  double min_cap = DBL_MAX;
  for (int k = 0; k < c->M; ++k) {
    const double v = capacity[c->perm[k]];
    if (v > 0 && v < min_cap) min_cap = v;
  }
  for (int k = 0; k < c->M; ++k) {
    const double v = capacity[c->perm[k]];
    c->h_cap[k] = v > 0 ? v : min_cap;
  }
  c->base_dirty = true;
  if (!c->S_cap) return TAPGPU_OK;  // (no arrays after a failed allocation: the next solve copies it)
  TG_CUDA(cudaSetDevice(c->device));
  TG_CUDA(cudaMemcpy(c->cap, c->h_cap.data(), sizeof(double) * c->M, cudaMemcpyHostToDevice));
  return TAPGPU_OK;
}

int tapgpu_solve_begin(tapgpu_ctx* ctx, int max_iters, double target_relgap, const double* x0) {
  if (!ctx || (max_iters <= 0 && !(target_relgap > 0))) {
    tapgpu::set_message("need an iteration cap or a positive relative-gap target");
    return TAPGPU_ERR_ARG;
  }
  Ctx* c = ctx->c;
  TG_CUDA(cudaSetDevice(c->device));
  TG_TRY(c->ensure_scenarios(1));
  c->use_dem_scen = false;
  c->use_link_scen = false;
  TG_TRY(c->choose_paths(1));
  TG_CUDA(cudaMemcpy(c->cap, c->h_cap.data(), sizeof(double) * c->M, cudaMemcpyHostToDevice));
  std::vector<int> one{0};
  TG_CUDA(cudaMemcpyAsync(c->scen_list, one.data(), sizeof(int), cudaMemcpyHostToDevice, c->stream));
  c->h_scen_list = one;
  TG_TRY(tapgpu::upload_states(c, 1, max_iters, target_relgap));
  if (x0) {
    std::vector<double> xi(c->M);
    for (int k = 0; k < c->M; ++k) xi[k] = x0[c->perm[k]];
    TG_CUDA(cudaMemcpyAsync(c->x, xi.data(), sizeof(double) * c->M, cudaMemcpyHostToDevice,
                            c->stream));
    TG_CUDA(cudaStreamSynchronize(c->stream));
  }
  TG_TRY(c->enqueue_initial(1, x0 != nullptr));
  TG_TRY(c->sync_check());
  c->solve_max_iters = max_iters;
  c->last_nscen = 1;
  return TAPGPU_OK;
}

int tapgpu_solve_advance(tapgpu_ctx* ctx, int max_new_iters, int* done, tapgpu_result* res) {
  if (!ctx || max_new_iters < 1) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  if (!c->can_iterate()) {
    tapgpu::set_message("no solve to go on with");
    return TAPGPU_ERR_ARG;
  }
  TG_CUDA(cudaSetDevice(c->device));
  std::vector<tapgpu::ScenState> st;
  TG_TRY(c->read_states(1, st));
  int n = max_new_iters;
  if (c->solve_max_iters > 0) n = std::max(1, std::min(n, c->solve_max_iters - st[0].iter));
  const int goal = st[0].iter + n;
  while (!st[0].done && st[0].iter < goal) {  // (again after a pause)
    TG_TRY(c->run_active({0}, goal - st[0].iter));
    TG_TRY(c->read_states(1, st));
    TG_TRY(c->sync_check());
    TG_TRY(c->resume_paused(1, st));
  }
  TG_TRY(c->sync_check());
  int e = 0;
  TG_CUDA(cudaMemcpy(&e, c->err, sizeof(int), cudaMemcpyDeviceToHost));
  if (done) *done = st[0].done;
  if (res) tapgpu::fill_result(st[0], e, res);
  return TAPGPU_OK;
}

int tapgpu_solve(tapgpu_ctx* ctx, int max_iters, double target_relgap, const double* x0,
                 tapgpu_result* res) {
  int rc = tapgpu_solve_begin(ctx, max_iters, target_relgap, x0);
  if (rc != TAPGPU_OK) return rc;
  Ctx* c = ctx->c;
  std::vector<tapgpu::ScenState> st;
  TG_TRY(tapgpu::iterate_until_done(c, 1, max_iters, st));
  int e = 0;
  TG_CUDA(cudaMemcpy(&e, c->err, sizeof(int), cudaMemcpyDeviceToHost));
  if (res) tapgpu::fill_result(st[0], e, res);
  return TAPGPU_OK;
}

// Writes to each page of an output array before the device copies to it: a page
// that is not there yet costs the device's copy a fault (20 MB of fresh pages:
// 1 to 17 ms; written by the host first, 0.8 ms and a copy of 0.15 ms).
static void touch_pages(void* p, size_t bytes) {
  auto* b = static_cast<volatile unsigned char*>(p);
  for (size_t i = 0; i < bytes; i += 4096) b[i] = 0;
  if (bytes) b[bytes - 1] = 0;
}

int tapgpu_get_link_flows(tapgpu_ctx* ctx, int scenario, double* volume, double* cost) {
  if (!ctx) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  if (scenario < 0 || scenario >= c->S_cap) return TAPGPU_ERR_ARG;
  TG_CUDA(cudaSetDevice(c->device));
  TG_CUDA(cudaStreamSynchronize(c->stream));
  std::vector<double> tmp(c->M);
  const size_t off = static_cast<size_t>(scenario) * c->M;
  if (volume) {
    TG_CUDA(cudaMemcpy(tmp.data(), c->x + off, sizeof(double) * c->M, cudaMemcpyDeviceToHost));
    for (int k = 0; k < c->M; ++k) volume[c->perm[k]] = tmp[k];
  }
  if (cost) {
    TG_CUDA(cudaMemcpy(tmp.data(), c->t + off, sizeof(double) * c->M, cudaMemcpyDeviceToHost));
    for (int k = 0; k < c->M; ++k) cost[c->perm[k]] = tmp[k];
  }
  return TAPGPU_OK;
}

int tapgpu_get_link_flows_batch(tapgpu_ctx* ctx, int first, int count, double* volume,
                                double* cost) {
  if (!ctx || count < 1) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  if (first < 0 || static_cast<int64_t>(first) + count > c->S_cap) return TAPGPU_ERR_ARG;
  TG_CUDA(cudaSetDevice(c->device));
  TG_CUDA(cudaStreamSynchronize(c->stream));
  const int M = c->M;
  const size_t off = static_cast<size_t>(first) * M, n = static_cast<size_t>(count) * M;
  bool identity = true;
  for (int k = 0; k < M && identity; ++k) identity = c->perm[k] == k;
  double* outs[2] = {volume, cost};
  const double* srcs[2] = {c->x + off, c->t + off};
  std::vector<double> tmp;
  for (int a = 0; a < 2; ++a) {
    if (!outs[a]) continue;
    if (identity) {  // the caller's link order is the device's: one copy
      touch_pages(outs[a], sizeof(double) * n);
      TG_CUDA(cudaMemcpy(outs[a], srcs[a], sizeof(double) * n, cudaMemcpyDeviceToHost));
      continue;
    }
    tmp.resize(n);
    TG_CUDA(cudaMemcpy(tmp.data(), srcs[a], sizeof(double) * n, cudaMemcpyDeviceToHost));
    for (int s = 0; s < count; ++s) {
      const double* row = tmp.data() + static_cast<size_t>(s) * M;
      double* out = outs[a] + static_cast<size_t>(s) * M;
      for (int k = 0; k < M; ++k) out[c->perm[k]] = row[k];
    }
  }
  return TAPGPU_OK;
}

int tapgpu_get_trace(tapgpu_ctx* ctx, int scenario, double* rows, int max_rows, int* nrows) {
  if (!ctx || !rows || !nrows) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  if (scenario < 0 || scenario >= c->S_cap) return TAPGPU_ERR_ARG;
  TG_CUDA(cudaSetDevice(c->device));
  tapgpu::ScenState st;
  TG_CUDA(cudaStreamSynchronize(c->stream));
  TG_CUDA(cudaMemcpy(&st, c->state + scenario, sizeof(st), cudaMemcpyDeviceToHost));
  const int n = std::min(std::min(st.iter, c->trace_cap), max_rows);
  if (n > 0)
    TG_CUDA(cudaMemcpy(rows, c->trace + static_cast<size_t>(scenario) * c->trace_cap * tapgpu::kTraceCols,
                       sizeof(double) * n * tapgpu::kTraceCols, cudaMemcpyDeviceToHost));
  *nrows = n;
  return TAPGPU_OK;
}

int tapgpu_solve_scenarios(tapgpu_ctx* ctx, int num_scen, const int64_t* scen_ptr,
                           const int64_t* scen_links, const double* scen_cap, int max_iters,
                           double target_relgap, const double* x0, tapgpu_result* results) {
  if (!ctx || num_scen < 1 || !scen_ptr || (max_iters <= 0 && !(target_relgap > 0))) {
    tapgpu::set_message("bad scenario arguments");
    return TAPGPU_ERR_ARG;
  }
  Ctx* c = ctx->c;
  const int M = c->M;
  // every argument is checked before the context's state changes
  const int64_t nedit = scen_ptr[num_scen] - scen_ptr[0];
  if (nedit > std::numeric_limits<int>::max() - 1) {
    tapgpu::set_message("too many scenario edits in one call");
    return TAPGPU_ERR_ARG;
  }
  if (nedit > 0 && (!scen_links || !scen_cap)) {
    tapgpu::set_message("scenario edits without link or capacity arrays");
    return TAPGPU_ERR_ARG;
  }
  std::vector<int64_t> inv(M);
  for (int k = 0; k < M; ++k) inv[c->perm[k]] = k;
  for (int s = 0; s < num_scen; ++s) {
    if (scen_ptr[s + 1] < scen_ptr[s]) return TAPGPU_ERR_ARG;
    for (int64_t i = scen_ptr[s]; i < scen_ptr[s + 1]; ++i)
      if (scen_links[i] < 0 || scen_links[i] >= M || std::isnan(scen_cap[i])) {
        tapgpu::set_message("scenario link index out of range");
        return TAPGPU_ERR_ARG;
      }
  }
  if (c->dem_scen && c->dem_scen != num_scen) {
    tapgpu::set_message("demand scenarios were set for " + std::to_string(c->dem_scen) +
                        " scenarios, not " + std::to_string(num_scen));
    return TAPGPU_ERR_ARG;
  }
  if (c->link_scen && c->link_scen != num_scen) {
    tapgpu::set_message("link-record scenarios were set for " + std::to_string(c->link_scen) +
                        " scenarios, not " + std::to_string(num_scen));
    return TAPGPU_ERR_ARG;
  }
  TG_CUDA(cudaSetDevice(c->device));
  TG_TRY(c->ensure_scenarios(num_scen));
  c->use_dem_scen = c->dem_scen == num_scen;
  c->use_link_scen = c->link_scen == num_scen;
  TG_TRY(c->choose_paths(num_scen));
  c->last_nscen = num_scen;
  // capacities of every scenario, made on the device from the base row and
  // the edits; the host finds each scenario's smallest positive capacity
  // for the zero-capacity fix-up
  if (c->base_dirty) {
    if (!c->base_cap) TG_TRY(c->alloc_n(&c->base_cap, M));
    TG_CUDA(cudaMemcpy(c->base_cap, c->h_cap.data(), sizeof(double) * M, cudaMemcpyHostToDevice));
    c->h_cap_order.resize(M);
    std::iota(c->h_cap_order.begin(), c->h_cap_order.end(), 0);
    std::stable_sort(c->h_cap_order.begin(), c->h_cap_order.end(),
                     [c](int a, int b) { return c->h_cap[a] < c->h_cap[b]; });
    c->base_dirty = false;
  }
  std::vector<int> eptr(num_scen + 1), elink(static_cast<size_t>(std::max<int64_t>(nedit, 1)));
  std::vector<double> evalv(elink.size()), emin(num_scen);
  {
    std::vector<int> seen;  // links edited in this scenario (few)
    int64_t j = 0;
    for (int s = 0; s < num_scen; ++s) {
      eptr[s] = static_cast<int>(j);
      seen.clear();
      for (int64_t i = scen_ptr[s]; i < scen_ptr[s + 1]; ++i, ++j) {
        elink[j] = static_cast<int>(inv[scen_links[i]]);
        evalv[j] = scen_cap[i];
        seen.push_back(elink[j]);
      }
      // smallest positive capacity of the final row: edits (the last edit of
      // a link wins) and the smallest base capacity of a link not edited
      double mn = DBL_MAX;
      for (int64_t i = eptr[s]; i < j; ++i) {
        bool last = true;
        for (int64_t i2 = i + 1; i2 < j; ++i2) last = last && elink[i2] != elink[i];
        if (last && evalv[i] > 0 && evalv[i] < mn) mn = evalv[i];
      }
      for (int k : c->h_cap_order) {
        if (std::find(seen.begin(), seen.end(), k) != seen.end()) continue;
        if (c->absent_in(s, k)) continue;  // not part of this scenario's network
        if (c->h_cap[k] < mn) mn = c->h_cap[k];
        break;
      }
      emin[s] = mn;
    }
    eptr[num_scen] = static_cast<int>(j);
  }
  if (num_scen + 1 > c->ed_scen_cap) {
    if (c->ed_ptr) tapgpu::free_owned(c, c->ed_ptr);
    if (c->ed_min) tapgpu::free_owned(c, c->ed_min);
    c->ed_ptr = nullptr;
    c->ed_min = nullptr;
    TG_TRY(c->alloc_n(&c->ed_ptr, num_scen + 1));
    TG_TRY(c->alloc_n(&c->ed_min, num_scen + 1));
    c->ed_scen_cap = num_scen + 1;
  }
  if (static_cast<int64_t>(elink.size()) > c->ed_cap) {
    if (c->ed_link) tapgpu::free_owned(c, c->ed_link);
    if (c->ed_val) tapgpu::free_owned(c, c->ed_val);
    c->ed_link = nullptr;
    c->ed_val = nullptr;
    TG_TRY(c->alloc_n(&c->ed_link, elink.size()));
    TG_TRY(c->alloc_n(&c->ed_val, elink.size()));
    c->ed_cap = static_cast<int64_t>(elink.size());
  }
  TG_CUDA(cudaMemcpyAsync(c->ed_ptr, eptr.data(), sizeof(int) * eptr.size(),
                          cudaMemcpyHostToDevice, c->stream));
  TG_CUDA(cudaMemcpyAsync(c->ed_link, elink.data(), sizeof(int) * elink.size(),
                          cudaMemcpyHostToDevice, c->stream));
  TG_CUDA(cudaMemcpyAsync(c->ed_val, evalv.data(), sizeof(double) * evalv.size(),
                          cudaMemcpyHostToDevice, c->stream));
  TG_CUDA(cudaMemcpyAsync(c->ed_min, emin.data(), sizeof(double) * emin.size(),
                          cudaMemcpyHostToDevice, c->stream));
  TG_CUDA(tapgpu::launch_scenario_caps(c->cap, c->base_cap, M, num_scen, c->ed_ptr, c->ed_link,
                                       c->ed_val, c->ed_min, c->link_grid, c->stream));
  // the host vectors above must outlive the copies
  TG_CUDA(cudaStreamSynchronize(c->stream));
  std::vector<int> all(num_scen);
  std::iota(all.begin(), all.end(), 0);
  TG_CUDA(cudaMemcpyAsync(c->scen_list, all.data(), sizeof(int) * num_scen,
                          cudaMemcpyHostToDevice, c->stream));
  c->h_scen_list = all;
  TG_TRY(tapgpu::upload_states(c, num_scen, max_iters, target_relgap));
  if (x0) {
    // the warm start once, then copied to every scenario on the device
    std::vector<double> xi(M);
    for (int k = 0; k < M; ++k) xi[k] = x0[c->perm[k]];
    TG_CUDA(cudaMemcpyAsync(c->x, xi.data(), sizeof(double) * M, cudaMemcpyHostToDevice, c->stream));
    TG_CUDA(tapgpu::launch_replicate_rows(c->x, M, num_scen, c->link_grid, c->stream));
    TG_CUDA(cudaStreamSynchronize(c->stream));
    TG_TRY(c->enqueue_initial(num_scen, true));
  } else if (c->use_dem_scen || c->use_link_scen) {
    // every scenario has its own demand or links: load each at its own free flow
    TG_TRY(c->enqueue_initial(num_scen, false));
  } else {
    // free-flow all-or-nothing does not depend on capacity: load scenario 0
    // once and start every scenario from it
    TG_TRY(c->begin_paths(1));
    TG_TRY(c->set_active(all));
    if (c->hier_on && num_scen > 1) {  // its exponent too
      std::vector<tapgpu::ScenState> st0;
      TG_TRY(c->read_states(num_scen, st0));
      for (int s = 1; s < num_scen; ++s) st0[s].u_exp = st0[0].u_exp;
      TG_CUDA(cudaMemcpyAsync(c->state, st0.data(), sizeof(tapgpu::ScenState) * num_scen,
                              cudaMemcpyHostToDevice, c->stream));
      TG_CUDA(cudaStreamSynchronize(c->stream));
    }
    for (int s = 1; s < num_scen; ++s)
      TG_CUDA(cudaMemcpyAsync(c->yfx + static_cast<size_t>(s) * M, c->yfx,
                              sizeof(unsigned long long) * M, cudaMemcpyDeviceToDevice,
                              c->stream));
    tapgpu::LinkArgs la = c->link_args(num_scen);
    la.pass = 0;
    TG_CUDA(tapgpu::launch_init_flows(la, c->link_grid, c->stream));
  }
  TG_TRY(c->sync_check());
  std::vector<tapgpu::ScenState> st;
  TG_TRY(tapgpu::iterate_until_done(c, num_scen, max_iters, st));
  int e = 0;
  TG_CUDA(cudaMemcpy(&e, c->err, sizeof(int), cudaMemcpyDeviceToHost));
  if (results)
    for (int s = 0; s < num_scen; ++s) tapgpu::fill_result(st[s], e, &results[s]);
  return TAPGPU_OK;
}

int tapgpu_set_scenario_demand(tapgpu_ctx* ctx, int num_scen, const double* demand) {
  if (!ctx || num_scen < 0) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  TG_CUDA(cudaSetDevice(c->device));
  TG_CUDA(cudaStreamSynchronize(c->stream));
  if (c->sc_od_q) tapgpu::free_owned(c, c->sc_od_q);
  if (c->sc_total) tapgpu::free_owned(c, c->sc_total);
  if (c->h_sc_dem) tapgpu::free_owned(c, c->h_sc_dem);
  c->h_sc_dem = nullptr;
  c->sc_od_q = nullptr;
  c->sc_total = nullptr;
  c->dem_scen = 0;
  c->use_dem_scen = false;
  if (c->gexec) {  // captured launches hold the old demand pointers
    cudaGraphExecDestroy(c->gexec);
    c->gexec = nullptr;
  }
  c->g_nscen = -1;
  if (num_scen == 0 || !demand) return TAPGPU_OK;
  const long long nnz = c->nnz;
  if (nnz == 0) {
    tapgpu::set_message("the context has no demand to vary");
    return TAPGPU_ERR_ARG;
  }
  std::vector<double> totals(num_scen);
  double max_pos = 0.0;
  for (int s = 0; s < num_scen; ++s) {
    double tot = 0.0, pos = 0.0;
    for (long long i = 0; i < nnz; ++i) {
      const double v = demand[static_cast<size_t>(s) * nnz + i];
      if (std::isnan(v) || std::isinf(v)) {
        tapgpu::set_message("scenario demand must be finite");
        return TAPGPU_ERR_ARG;
      }
      if (v > 0 && !(c->h_od_dem[i] > 0)) {
        tapgpu::set_message("a demand scenario can only change OD pairs with positive base demand");
        return TAPGPU_ERR_ARG;
      }
      tot += v;  // tap/tap_functions.c:377-386 sums every entry
      if (v > 0) pos += v;
    }
    totals[s] = tot;
    max_pos = std::max(max_pos, pos);
  }
  // keep every node/link total below 2^61 in the shared fixed point
  int bits = 40;
  if (max_pos > 1.0) bits = std::min(40, 61 - static_cast<int>(std::ceil(std::log2(max_pos))) - 1);
  if (bits < c->scale_bits) {
    const double scale = std::ldexp(1.0, bits);
    std::vector<long long> oq(nnz);
    for (long long i = 0; i < nnz; ++i)
      oq[i] = c->h_od_dem[i] > 0 ? std::llrint(c->h_od_dem[i] * scale) : 0;
    TG_CUDA(cudaMemcpy(c->od_q, oq.data(), sizeof(long long) * nnz, cudaMemcpyHostToDevice));
    c->scale_bits = bits;
    c->inv_scale = std::ldexp(1.0, -bits);
    if (c->h_dem) TG_TRY(c->hier_demand(c->od_q, 1, &c->h_dem));
  }
  const double scale = std::ldexp(1.0, c->scale_bits);
  std::vector<long long> q(static_cast<size_t>(num_scen) * nnz);
  for (size_t i = 0; i < q.size(); ++i) q[i] = demand[i] > 0 ? std::llrint(demand[i] * scale) : 0;
  TG_TRY(c->alloc_n(&c->sc_od_q, q.size()));
  TG_TRY(c->alloc_n(&c->sc_total, static_cast<size_t>(num_scen)));
  TG_CUDA(cudaMemcpy(c->sc_od_q, q.data(), sizeof(long long) * q.size(), cudaMemcpyHostToDevice));
  TG_CUDA(cudaMemcpy(c->sc_total, totals.data(), sizeof(double) * num_scen, cudaMemcpyHostToDevice));
  c->dem_scen = num_scen;
  return TAPGPU_OK;
}

int tapgpu_set_scenario_links(tapgpu_ctx* ctx, int num_scen, const int64_t* edit_ptr,
                              const int64_t* edit_links, const double* edit_fft,
                              const double* edit_alpha, const double* edit_beta,
                              const int64_t* absent_ptr, const int64_t* absent_links) {
  if (!ctx || num_scen < 0) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  const int M = c->M;
  if (num_scen > 0) {  // every argument is checked before the context's state changes
    if (!edit_ptr || !absent_ptr) {
      tapgpu::set_message("link-record scenarios need edit and absent-link offsets");
      return TAPGPU_ERR_ARG;
    }
    const int64_t ne = edit_ptr[num_scen] - edit_ptr[0];
    const int64_t na = absent_ptr[num_scen] - absent_ptr[0];
    if (ne < 0 || na < 0 || ne > std::numeric_limits<int>::max() - 1 ||
        (ne > 0 && (!edit_links || !edit_fft || !edit_alpha || !edit_beta)) ||
        (na > 0 && !absent_links)) {
      tapgpu::set_message("bad link-record scenario arrays");
      return TAPGPU_ERR_ARG;
    }
    for (int s = 0; s < num_scen; ++s) {
      if (edit_ptr[s + 1] < edit_ptr[s] || absent_ptr[s + 1] < absent_ptr[s]) {
        tapgpu::set_message("link-record scenario offsets not monotone");
        return TAPGPU_ERR_ARG;
      }
      for (int64_t i = edit_ptr[s]; i < edit_ptr[s + 1]; ++i) {
        if (edit_links[i] < 0 || edit_links[i] >= M || !(edit_fft[i] >= 0) ||
            !std::isfinite(edit_fft[i]) || !(edit_alpha[i] >= 0) ||
            !std::isfinite(edit_alpha[i]) || !std::isfinite(edit_beta[i])) {
          tapgpu::set_message("link-record edit " + std::to_string(i) +
                              " has a link out of range or an invalid cost parameter");
          return TAPGPU_ERR_ARG;
        }
      }
      for (int64_t i = absent_ptr[s]; i < absent_ptr[s + 1]; ++i)
        if (absent_links[i] < 0 || absent_links[i] >= M) {
          tapgpu::set_message("absent link index out of range");
          return TAPGPU_ERR_ARG;
        }
    }
  }
  TG_CUDA(cudaSetDevice(c->device));
  TG_CUDA(cudaStreamSynchronize(c->stream));
  void* olds[] = {c->sc_fft, c->sc_alpha, c->sc_beta, c->sc_ipow, c->sc_absent};
  for (void* p : olds) tapgpu::free_owned(c, p);
  c->sc_fft = c->sc_alpha = c->sc_beta = nullptr;
  c->sc_ipow = nullptr;
  c->sc_absent = nullptr;
  c->h_absent.clear();
  c->link_scen = 0;
  c->use_link_scen = false;
  if (c->gexec) {  // captured launches hold the old parameter pointers
    cudaGraphExecDestroy(c->gexec);
    c->gexec = nullptr;
  }
  c->g_nscen = -1;
  if (num_scen == 0) return TAPGPU_OK;

  std::vector<int64_t> inv(M);
  for (int k = 0; k < M; ++k) inv[c->perm[k]] = k;
  const int64_t ne = edit_ptr[num_scen] - edit_ptr[0];
  std::vector<int> eptr(num_scen + 1), elink(static_cast<size_t>(std::max<int64_t>(ne, 1)));
  std::vector<double> efft(elink.size()), ealpha(elink.size()), ebeta(elink.size());
  std::vector<unsigned char> eip(elink.size());
  int64_t j = 0;
  for (int s = 0; s < num_scen; ++s) {
    eptr[s] = static_cast<int>(j);
    for (int64_t i = edit_ptr[s]; i < edit_ptr[s + 1]; ++i, ++j) {
      elink[j] = static_cast<int>(inv[edit_links[i]]);
      efft[j] = edit_fft[i];
      ealpha[j] = edit_alpha[i];
      const double b = edit_beta[i];
      ebeta[j] = b;
      eip[j] = (b >= 0 && b <= 15 && std::floor(b) == b) ? static_cast<unsigned char>(b) : 255;
    }
  }
  eptr[num_scen] = static_cast<int>(j);
  const int words = (M + 31) / 32;
  c->h_absent.assign(static_cast<size_t>(num_scen) * words, 0u);
  for (int s = 0; s < num_scen; ++s)
    for (int64_t i = absent_ptr[s]; i < absent_ptr[s + 1]; ++i) {
      const int k = static_cast<int>(inv[absent_links[i]]);
      c->h_absent[static_cast<size_t>(s) * words + (k >> 5)] |= 1u << (k & 31);
    }
  const size_t rows = static_cast<size_t>(num_scen) * M;
  TG_TRY(c->alloc_n(&c->sc_fft, rows));
  TG_TRY(c->alloc_n(&c->sc_alpha, rows));
  TG_TRY(c->alloc_n(&c->sc_beta, rows));
  TG_TRY(c->alloc_n(&c->sc_ipow, rows));
  TG_TRY(c->alloc_n(&c->sc_absent, c->h_absent.size()));
  int* d_ptr = nullptr;
  int* d_link = nullptr;
  double* d_val = nullptr;
  unsigned char* d_ip = nullptr;
  TG_TRY(c->alloc_n(&d_ptr, eptr.size()));
  TG_TRY(c->alloc_n(&d_link, elink.size()));
  TG_TRY(c->alloc_n(&d_val, 3 * elink.size()));
  TG_TRY(c->alloc_n(&d_ip, elink.size()));
  const size_t ns = elink.size();
  int rc = TAPGPU_OK;
  if (cudaMemcpy(d_ptr, eptr.data(), sizeof(int) * eptr.size(), cudaMemcpyHostToDevice) ||
      cudaMemcpy(d_link, elink.data(), sizeof(int) * ns, cudaMemcpyHostToDevice) ||
      cudaMemcpy(d_val, efft.data(), sizeof(double) * ns, cudaMemcpyHostToDevice) ||
      cudaMemcpy(d_val + ns, ealpha.data(), sizeof(double) * ns, cudaMemcpyHostToDevice) ||
      cudaMemcpy(d_val + 2 * ns, ebeta.data(), sizeof(double) * ns, cudaMemcpyHostToDevice) ||
      cudaMemcpy(d_ip, eip.data(), ns, cudaMemcpyHostToDevice) ||
      cudaMemcpy(c->sc_absent, c->h_absent.data(), sizeof(unsigned) * c->h_absent.size(),
                 cudaMemcpyHostToDevice) ||
      tapgpu::launch_param_rows(c->sc_fft, c->fft, M, num_scen, d_ptr, d_link, d_val,
                                c->link_grid, c->stream) ||
      tapgpu::launch_param_rows(c->sc_alpha, c->alpha, M, num_scen, d_ptr, d_link, d_val + ns,
                                c->link_grid, c->stream) ||
      tapgpu::launch_param_rows(c->sc_beta, c->beta, M, num_scen, d_ptr, d_link, d_val + 2 * ns,
                                c->link_grid, c->stream) ||
      tapgpu::launch_param_rows(c->sc_ipow, c->ipow, M, num_scen, d_ptr, d_link, d_ip,
                                c->link_grid, c->stream) ||
      cudaStreamSynchronize(c->stream)) {
    tapgpu::set_message(std::string("link-record scenario rows: ") +
                        cudaGetErrorString(cudaGetLastError()));
    rc = TAPGPU_ERR_CUDA;
  }
  void* tmp[] = {d_ptr, d_link, d_val, d_ip};
  for (void* p : tmp) tapgpu::free_owned(c, p);
  if (rc != TAPGPU_OK) return rc;
  c->absent_words = words;
  c->link_scen = num_scen;
  return TAPGPU_OK;
}

// The link costs of a call, in device order in api_w64, and the records of the
// FP32 kernels made from them.  w stays until the stream has been waited for.
static int to_device_weights(Ctx* c, const double* weights, std::vector<double>& w) {
  w.resize(c->M);
  double sum = 0.0;
  for (int k = 0; k < c->M; ++k) {
    const double v = weights[c->perm[k]];
    if (!(v >= 0) || std::isinf(v)) {
      tapgpu::set_message("link costs must be finite and non-negative");
      return TAPGPU_ERR_ARG;
    }
    w[k] = v;
    sum += v;
  }
  const double mean = sum / c->M;
  c->api_nf_delta = c->opt.nf_delta > 0 ? c->opt.nf_delta : (mean > 0 ? 16.0 * mean : 1.0);
  TG_CUDA(cudaMemcpyAsync(c->api_w64, w.data(), sizeof(double) * c->M, cudaMemcpyHostToDevice,
                          c->stream));
  if (!c->fp64) {
    tapgpu::LinkArgs la = c->link_args(1);
    la.scen_list = nullptr;
    la.absent = nullptr;
    la.t = c->api_w64;
    la.w64 = nullptr;
    la.e32 = c->api_e32;
    la.r32 = c->api_r32;
    la.e4 = c->api_e4;
    la.r4 = nullptr;
    la.r4d = nullptr;
    TG_CUDA(tapgpu::launch_records(la, c->link_grid, c->stream));
  }
  return TAPGPU_OK;
}

int tapgpu_sssp(tapgpu_ctx* ctx, const double* weights, const int64_t* srcs, int64_t num_sources,
                double* dist, int64_t* pred) {
  if (!ctx || !weights || (num_sources > 0 && !srcs)) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  for (int64_t i = 0; i < num_sources; ++i)
    if (srcs[i] < 0 || srcs[i] >= c->n1) {
      tapgpu::set_message("source node out of range");
      return TAPGPU_ERR_ARG;
    }
  TG_CUDA(cudaSetDevice(c->device));
  std::vector<double> w;
  TG_TRY(to_device_weights(c, weights, w));
  const int n1 = c->n1;
  TG_TRY(c->ensure_labels());
  // FP64 labels: a FP32 context's label buffer holds half as many sources
  const int64_t chunk = c->fp64 ? c->dist_tasks : std::max<int64_t>(1, c->dist_tasks / 2);
  const int64_t rows = std::max<int64_t>(1, std::min(chunk, num_sources));
  if (rows > c->api_rows) {  // sources, predecessors and their wide form
    void* olds[] = {c->api_src, c->pred_buf, c->api_pred};
    for (void* p : olds) tapgpu::free_owned(c, p);
    c->api_src = c->pred_buf = nullptr;
    c->api_pred = nullptr;
    c->api_rows = 0;
    c->api_pred_rows = tapgpu::rows_at_once(rows, n1);
    TG_TRY(c->alloc_n(&c->api_src, static_cast<size_t>(rows)));
    TG_TRY(c->alloc_n(&c->pred_buf, static_cast<size_t>(rows) * n1));
    TG_TRY(c->alloc_n(&c->api_pred, static_cast<size_t>(c->api_pred_rows) * n1));
    if (!c->api_perm) {
      TG_TRY(c->alloc_n(&c->api_perm, static_cast<size_t>(c->M)));
      TG_CUDA(cudaMemcpy(c->api_perm, c->perm.data(), sizeof(int64_t) * c->M, cudaMemcpyHostToDevice));
    }
    c->api_rows = rows;
  }
  std::vector<int> hs;
  int rc = TAPGPU_OK;
  // the API always computes FP64 labels: they equal the reference's bit for bit
  for (int64_t s0 = 0; s0 < num_sources && rc == TAPGPU_OK; s0 += chunk) {
    const int64_t s1 = std::min(num_sources, s0 + chunk);
    const int ns = static_cast<int>(s1 - s0);
    hs.resize(ns);
    for (int i = 0; i < ns; ++i) hs[i] = static_cast<int>(srcs[s0 + i]);
    if (cudaMemcpyAsync(c->api_src, hs.data(), sizeof(int) * ns, cudaMemcpyHostToDevice, c->stream) !=
        cudaSuccess) {
      rc = TAPGPU_ERR_CUDA;
      break;
    }
    tapgpu::PathArgs a = c->path_args(1);
    a.sources = c->api_src;
    a.num_sources = ns;
    a.scen_list = nullptr;
    a.state = nullptr;
    a.task_begin = 0;
    a.task_end = ns;
    a.w64 = c->api_w64;
    a.e32 = nullptr;
    a.r4 = nullptr;
    a.r4d = nullptr;
    a.aon_c64 = 0;
    a.do_load = 0;
    a.pred_out = c->pred_buf;
    a.y_fx = c->api_yfx;
    a.nf_delta = c->api_nf_delta;
    const int optin = tapgpu::max_smem_optin(c->device);
    const bool s_smem = tapgpu::sssp_smem_bytes(n1, true, c->sssp_variant, c->M) + 1024 <= static_cast<size_t>(optin);
    const int occ = tapgpu::sssp_occupancy(true, c->sssp_block, s_smem, n1, c->sssp_variant, c->M,
                                           c->opt.global_scratch == 2);
    int grid = std::max(1, std::min(occ * c->num_sms, ns));
    if (!s_smem) {
      const size_t need = tapgpu::sssp_smem_bytes(n1, true, c->sssp_variant, c->M) * static_cast<size_t>(grid);
      if (need > c->path_scratch_bytes) {
        grid = std::max<int>(1, static_cast<int>(c->path_scratch_bytes / tapgpu::sssp_smem_bytes(n1, true, c->sssp_variant, c->M)));
        if (c->path_scratch_bytes == 0) {
          rc = TAPGPU_ERR_UNSUPPORTED;
          break;
        }
      }
    }
    // FP64 labels: the 16-byte-per-node loading layout, whatever the context's
    const size_t abytes = tapgpu::aon_smem_bytes(n1, true);
    const bool a_smem = abytes + 1024 <= static_cast<size_t>(optin) && !c->opt.global_scratch;
    int agrid = std::max(1, std::min(tapgpu::aon_occupancy(true, c->aon_block, a_smem, n1) *
                                         c->num_sms, ns));
    if (!a_smem) {
      agrid = std::min<int>(agrid, static_cast<int>(c->path_scratch_bytes / abytes));
      if (agrid < 1) {
        rc = TAPGPU_ERR_UNSUPPORTED;
        break;
      }
    }
    const bool own = tapgpu::sssp_own_tasks(c->M, c->sssp_variant, c->sssp_block, s_smem) && grid == ns;
    if (!own || agrid < ns) cudaMemsetAsync(c->counters, 0, 2 * sizeof(int), c->stream);
    a.counter = own ? nullptr : c->counters;
    a.scratch_stride = static_cast<long long>(tapgpu::sssp_smem_bytes(n1, true, c->sssp_variant, c->M));
    if (tapgpu::launch_sssp(a, true, grid, c->sssp_block, s_smem, c->sssp_variant, c->stream) !=
        cudaSuccess) {
      rc = TAPGPU_ERR_CUDA;
      break;
    }
    a.counter = agrid == ns ? nullptr : c->counters + 1;
    a.scratch_stride = static_cast<long long>(abytes);
    if (tapgpu::launch_aon(a, true, agrid, c->aon_block, a_smem, c->stream) != cudaSuccess) {
      rc = TAPGPU_ERR_CUDA;
      break;
    }
    const size_t at = static_cast<size_t>(s0) * n1, count = static_cast<size_t>(ns) * n1;
    const size_t step = pred ? static_cast<size_t>(c->api_pred_rows) * n1 : count;
    if (tapgpu::launch_tree_rows(static_cast<double*>(c->dist), count, c->pred_buf, c->api_perm,
                                 c->api_pred, pred ? std::min(step, count) : 0, c->stream) != cudaSuccess) {
      rc = TAPGPU_ERR_CUDA;
      break;
    }
    // (while the kernels run)
    if (dist) touch_pages(dist + at, sizeof(double) * count);
    if (pred) touch_pages(pred + at, sizeof(int64_t) * count);
    rc = c->sync_check();
    if (rc != TAPGPU_OK) break;
    bool copied = !dist || cudaMemcpy(dist + at, c->dist, sizeof(double) * count,
                                      cudaMemcpyDeviceToHost) == cudaSuccess;
    for (size_t i = 0; pred && i < count && copied; i += step) {
      const size_t n = std::min(step, count - i);
      copied = (i == 0 || tapgpu::launch_tree_rows(nullptr, 0, c->pred_buf + i, c->api_perm, c->api_pred,
                                                   n, c->stream) == cudaSuccess) &&
               cudaStreamSynchronize(c->stream) == cudaSuccess &&
               cudaMemcpy(pred + at + i, c->api_pred, sizeof(int64_t) * n, cudaMemcpyDeviceToHost) ==
                   cudaSuccess;
    }
    if (!copied) rc = TAPGPU_ERR_CUDA;
  }
  if (rc == TAPGPU_ERR_CUDA && tapgpu::g_message.empty())
    tapgpu::set_message(cudaGetErrorString(cudaGetLastError()));
  return rc;
}

int tapgpu_aon(tapgpu_ctx* ctx, const double* weights, double* volume) {
  if (!ctx || !weights || !volume) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  TG_CUDA(cudaSetDevice(c->device));
  std::vector<double> w;
  TG_TRY(to_device_weights(c, weights, w));
  TG_CUDA(cudaMemsetAsync(c->api_yfx, 0, sizeof(unsigned long long) * c->M, c->stream));
  TG_CUDA(cudaMemsetAsync(c->err, 0, sizeof(int), c->stream));
  bool swept = false, loaded = false;
  TG_TRY(c->take_plan());
  if (c->hier && c->hier_pays(1)) TG_TRY(c->have_hier(1, false, &swept));
  if (swept) {
    TG_TRY(c->hier_load_api(&loaded));
    if (!loaded)
      TG_CUDA(cudaMemsetAsync(c->api_yfx, 0, sizeof(unsigned long long) * c->M, c->stream));
  }
  if (!loaded) TG_TRY(c->ensure_labels());
  const double solver_delta = c->nf_delta;
  c->nf_delta = c->api_nf_delta;
  const int rc = loaded ? TAPGPU_OK : c->enqueue_paths(1, true, c->fp64 ? nullptr : c->api_e32,
                                  c->fp64 ? nullptr : c->api_r32, c->fp64 ? c->api_w64 : nullptr,
                                  c->api_yfx, false);
  c->nf_delta = solver_delta;
  TG_TRY(rc);
  TG_TRY(c->sync_check());
  std::vector<unsigned long long> y(c->M);
  TG_CUDA(cudaMemcpy(y.data(), c->api_yfx, sizeof(unsigned long long) * c->M,
                     cudaMemcpyDeviceToHost));
  for (int k = 0; k < c->M; ++k)
    volume[c->perm[k]] = static_cast<double>(static_cast<long long>(y[k])) * c->inv_scale;
  return TAPGPU_OK;
}

void* tapgpu_stream(tapgpu_ctx* ctx) { return ctx ? ctx->c->stream : nullptr; }

int tapgpu_run_iterations(tapgpu_ctx* ctx, int iters) {
  if (!ctx || iters < 1) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  if (!c->can_iterate()) {
    tapgpu::set_message("no solve to go on with");
    return TAPGPU_ERR_ARG;
  }
  TG_CUDA(cudaSetDevice(c->device));
  const int S = c->last_nscen;
  std::vector<tapgpu::ScenState> st;
  TG_TRY(c->read_states(S, st));
  for (auto& s : st) {
    s.done = 0;
    s.max_iters = s.iter + iters;
    s.target_relgap = 0.0;
  }
  TG_CUDA(cudaMemcpyAsync(c->state, st.data(), sizeof(tapgpu::ScenState) * S,
                          cudaMemcpyHostToDevice, c->stream));
  std::vector<int> all(S);
  std::iota(all.begin(), all.end(), 0);
  const int per = tapgpu::equal_parts(iters, c->opt.iters_per_launch > 0 ? c->opt.iters_per_launch : 8);
  for (int done = 0; done < iters; done += per) TG_TRY(c->run_active(all, per));
  if (!c->hier_on) return TAPGPU_OK;
  for (;;) {  // scenarios that paused on the way take their remaining iterations
    TG_TRY(c->read_states(S, st));
    bool paused = false;
    for (auto& s : st) paused |= s.done > 1;
    if (!paused) return TAPGPU_OK;
    TG_TRY(c->resume_paused(S, st));
    std::vector<int> active;
    int left = 0;
    for (int s = 0; s < S; ++s)
      if (!st[s].done) {
        active.push_back(s);
        left = std::max(left, st[s].max_iters - st[s].iter);
      }
    if (active.empty()) return TAPGPU_OK;
    TG_TRY(c->run_active(active, std::max(1, std::min(per, left))));
  }
}

int tapgpu_set_hierarchy_limit(tapgpu_ctx* ctx, int64_t bytes) {
  if (!ctx) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  TG_CUDA(cudaSetDevice(c->device));
  TG_CUDA(cudaStreamSynchronize(c->stream));
  c->hier_bytes = bytes > 0 ? static_cast<size_t>(bytes) : tapgpu::kHierBytes;
  if (c->gexec) {  // captured launches hold the buffers' addresses
    cudaGraphExecDestroy(c->gexec);
    c->gexec = nullptr;
  }
  c->release_hier();
  return TAPGPU_OK;
}

int tapgpu_set_timing(tapgpu_ctx* ctx, int on) {
  if (!ctx) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  TG_CUDA(cudaSetDevice(c->device));
  TG_CUDA(cudaStreamSynchronize(c->stream));
  if (c->gexec) {
    cudaGraphExecDestroy(c->gexec);
    c->gexec = nullptr;
  }
  c->timing = on != 0;
  c->timed.clear();
  c->ev_used = 0;
  for (int i = 0; i < 4; ++i) {
    c->kt_ms[i] = 0.0;
    c->kt_n[i] = 0;
  }
  c->launches = 0;
  TG_CUDA(cudaMemset(c->path_stats, 0, 8 * sizeof(unsigned long long)));
  return TAPGPU_OK;
}

int tapgpu_get_path_stats(tapgpu_ctx* ctx, int64_t* out) {
  if (!ctx || !out) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  TG_CUDA(cudaSetDevice(c->device));
  TG_CUDA(cudaStreamSynchronize(c->stream));
  unsigned long long v[6];
  TG_CUDA(cudaMemcpy(v, c->path_stats, sizeof(v), cudaMemcpyDeviceToHost));
  for (int i = 0; i < 6; ++i) out[i] = static_cast<int64_t>(v[i]);
  return TAPGPU_OK;
}

int tapgpu_get_timing(tapgpu_ctx* ctx, double* ms, int64_t* counts, int64_t* kernel_launches) {
  if (!ctx) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  TG_CUDA(cudaSetDevice(c->device));
  TG_CUDA(cudaStreamSynchronize(c->stream));
  for (int i = 0; i < 4; ++i) {
    if (ms) ms[i] = c->kt_ms[i];
    if (counts) counts[i] = c->kt_n[i];
  }
  if (kernel_launches) *kernel_launches = c->launches;
  return TAPGPU_OK;
}

int tapgpu_profile_iteration(tapgpu_ctx* ctx, int reps, float* ms) {
  if (!ctx || !ms || reps < 1) return TAPGPU_ERR_ARG;
  Ctx* c = ctx->c;
  if (!c->can_iterate()) {
    tapgpu::set_message("no solve to go on with");
    return TAPGPU_ERR_ARG;
  }
  TG_CUDA(cudaSetDevice(c->device));
  std::vector<tapgpu::ScenState> st;
  TG_TRY(c->read_states(1, st));
  st[0].done = 0;
  st[0].max_iters = 0;
  st[0].target_relgap = 0.0;
  TG_CUDA(cudaMemcpyAsync(c->state, st.data(), sizeof(tapgpu::ScenState), cudaMemcpyHostToDevice,
                          c->stream));
  std::vector<int> one{0};
  TG_CUDA(cudaMemcpyAsync(c->scen_list, one.data(), sizeof(int), cudaMemcpyHostToDevice, c->stream));
  c->h_scen_list = one;
  cudaEvent_t ev[5];
  for (auto& e : ev) TG_CUDA(cudaEventCreate(&e));
  double acc[5] = {0, 0, 0, 0, 0};
  int rc = TAPGPU_OK;
  const int64_t tasks = c->Z;
  int pauses = 0;
  for (int r = 0; r < reps && rc == TAPGPU_OK;) {
    const bool swept = c->on_hierarchy(0);
    if (!swept && tasks > c->dist_tasks) {
      rc = TAPGPU_ERR_UNSUPPORTED;
      break;
    }
    if (!swept && c->hier_on) tapgpu::launch_records(c->link_args(1, true), c->link_grid, c->stream);
    cudaEventRecord(ev[0], c->stream);
    if (swept) {
      rc = c->enqueue_hier(1, c->t, c->M, ev[1]);
      if (rc != TAPGPU_OK) break;
      cudaEventRecord(ev[2], c->stream);
    } else {
      tapgpu::PathArgs a = c->path_args(1);
      a.task_end = static_cast<int>(tasks);
      cudaMemsetAsync(c->counters, 0, 2 * sizeof(int), c->stream);
      a.counter = c->counters;
      a.scratch_stride = static_cast<long long>(tapgpu::sssp_smem_bytes(c->n1, c->fp64, c->sssp_variant, c->M));
      a.e32 = c->fp64 ? nullptr : c->e32;
      a.r32 = c->fp64 ? nullptr : c->r32;
      a.w64 = c->fp64 ? c->w64 : nullptr;
      tapgpu::launch_sssp(a, c->fp64, std::min<int64_t>(c->sssp_grid, tasks), c->sssp_block,
                          c->sssp_smem, c->sssp_variant, c->stream);
      cudaEventRecord(ev[1], c->stream);
      a.counter = c->counters + 1;
      a.scratch_stride = static_cast<long long>(tapgpu::aon_smem_bytes(c->n1, c->fp64, c->aon_c64));
      tapgpu::launch_aon(a, c->fp64, std::min<int64_t>(c->aon_grid, tasks), c->aon_block,
                         c->aon_smem, c->stream);
      cudaEventRecord(ev[2], c->stream);
    }
    tapgpu::LinkArgs la = c->link_args(1);
    for (la.pass = 0; la.pass < c->grid_passes(); ++la.pass)
      tapgpu::launch_ls_pass(la, c->ls_grid(1), c->ls_block, c->stream);
    tapgpu::launch_ls_rest(la, c->stream);
    cudaEventRecord(ev[3], c->stream);
    tapgpu::launch_step(la, c->step_grid(1), c->ls_block, c->stream);
    cudaEventRecord(ev[4], c->stream);
    if (cudaEventSynchronize(ev[4]) != cudaSuccess) {
      rc = TAPGPU_ERR_CUDA;
      break;
    }
    if (swept) {  // an iteration that paused is repeated, not counted
      rc = c->read_states(1, st);
      if (rc != TAPGPU_OK) break;
      if (st[0].done > 1) {
        rc = ++pauses <= reps + 64 ? c->resume_paused(1, st) : TAPGPU_ERR_NO_CONVERGENCE;
        continue;  // (the list of active scenarios stays {0})
      }
    }
    float t;
    for (int i = 0; i < 4; ++i) {
      cudaEventElapsedTime(&t, ev[i], ev[i + 1]);
      acc[i] += t;
    }
    cudaEventElapsedTime(&t, ev[0], ev[4]);
    acc[4] += t;
    ++r;
  }
  for (auto& e : ev) cudaEventDestroy(e);
  if (rc != TAPGPU_OK) return rc;
  TG_TRY(c->sync_check());
  for (int i = 0; i < 5; ++i) ms[i] = static_cast<float>(acc[i] / reps);
  return TAPGPU_OK;
}

}  // extern "C"
