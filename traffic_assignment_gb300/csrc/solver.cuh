// solver.cuh - host-side solver context behind the tapgpu_* C ABI.
#pragma once
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdint>
#include <memory>
#include <string>
#include <vector>

#include "fw_kernels.cuh"
#include "hier_kernels.cuh"
#include "tap_gpu.h"

namespace tapgpu {

void set_message(const std::string& m);

// device allocation owned by a context
struct DevMem {
  void* p = nullptr;
  size_t bytes = 0;
};

// default bound of the elimination hierarchy's per-scenario buffers
constexpr size_t kHierBytes = size_t(24) << 30;
// iterations of a scenario after which its spread labels keep it off the hierarchy
constexpr int kSpreadIters = 2;

// predecessor rows of n1 64-bit link indices that the shortest-path API widens at
// once: 64 MiB of them, one at least (n1 up to 2^30 + 1)
inline int64_t rows_at_once(int64_t rows, int n1) {
  return std::max<int64_t>(1, std::min<int64_t>(rows, (int64_t(64) << 20) / (int64_t(8) * n1)));
}

class HierBuilder;

struct Ctx {
  // sizes (internal link order: sorted by (init, term))
  int N = 0, n1 = 0, M = 0, Z = 0, F = 0;
  bool fp64 = true;
  int device = 0, num_sms = 0;
  tapgpu_options opt{};
  std::vector<int64_t> perm;  // internal link k -> caller's link index
  std::vector<int> h_tail, h_head;
  std::vector<double> h_cap, h_fft, h_alpha, h_beta;
  // base capacities on the device for the scenario rows, and the links in
  // order of increasing base capacity (both redone after tapgpu_set_capacity)
  double* base_cap = nullptr;
  std::vector<int> h_cap_order;
  bool base_dirty = true;
  // per-call scenario edits on the device (grown as needed)
  int* ed_ptr = nullptr;
  int* ed_link = nullptr;
  double* ed_val = nullptr;
  double* ed_min = nullptr;
  int64_t ed_scen_cap = 0, ed_cap = 0;

  // device topology and link parameters
  int *row_ptr = nullptr, *head = nullptr, *tail = nullptr, *in_ptr = nullptr, *in_link = nullptr;
  int* in_head = nullptr;  // head node of each reverse-star slot
  int* out_deg = nullptr;  // out-degree of each node
  int* ell_pos = nullptr;  // slot of each link among its tail's first four (-1: beyond)
  unsigned* e4x = nullptr;  // first word of each link's padded record (head | tail degree << 16)
  std::vector<unsigned> h_e4x;
  bool deg16 = false;       // node ids and out-degrees fit 16 bits (16-bit queue ring)
  std::vector<int> h_ell_pos;
  // padded reverse records of the loading kernel's per-node predecessor scan
  // (FP32 paths, nodes and links fitting 16 bits)
  bool rev4 = false;
  int* r4_pos = nullptr;    // slot of each link among its head's first four in-links (-1: beyond)
  unsigned* r4x = nullptr;  // first word of each link's padded reverse record (link << 16 | tail)
  unsigned* r4_more = nullptr;  // bit v: node v has more than four in-links
  double *fft = nullptr, *alpha = nullptr, *beta = nullptr;
  unsigned char* ipow = nullptr;

  // demand
  int *od_ptr = nullptr, *od_dest = nullptr;
  long long* od_q = nullptr;
  double* od_dem = nullptr;
  int* sources = nullptr;
  double inv_scale = 1.0, total_demand = 0.0;
  int scale_bits = 0;
  // demand scenarios (trip modifications): their own OD demand per scenario
  std::vector<double> h_od_dem;  // base demand in device entry order
  long long nnz = 0;
  long long* sc_od_q = nullptr;  // [dem_scen][nnz] fixed point
  double* sc_total = nullptr;    // [dem_scen] demand totals
  int dem_scen = 0;              // scenarios with their own demand (0: none set)
  bool use_dem_scen = false;     // the current batched solve uses them
  // link-record scenarios (ADD / CHANGE records): per-scenario parameter rows
  // [link_scen][M] and a bitmask [link_scen][absent_words] of the links a
  // scenario's network does not have
  double *sc_fft = nullptr, *sc_alpha = nullptr, *sc_beta = nullptr;
  unsigned char* sc_ipow = nullptr;
  unsigned* sc_absent = nullptr;
  std::vector<unsigned> h_absent;
  int absent_words = 0;
  int link_scen = 0;             // scenarios with their own link records (0: none set)
  bool use_link_scen = false;    // the current batched solve uses them

  // per-scenario state (capacity for S_cap scenarios)
  int S_cap = 0;
  double *cap = nullptr, *x = nullptr, *t = nullptr, *d = nullptr, *dtdx = nullptr;
  unsigned long long* yfx = nullptr;
  uint2* e32 = nullptr;  // packed {head, f32 weight} per scenario and link
  uint2* r32 = nullptr;  // packed {tail, f32 weight} per scenario, reverse-star order
  uint2* e4 = nullptr;   // per scenario, the first four records of each node (padded)
  uint2* r4 = nullptr;   // per scenario, the first four in-link records of each node (padded)
  uint4* r4d = nullptr;  // the same for FP64 paths: {link, tail, f64 weight}
  bool aon_c64 = false;  // FP64 loading in the compact layout (predecessor words in the label slot)
  int* rpos = nullptr;   // reverse-star slot of each link
  std::vector<int> h_rpos;
  double* w64 = nullptr;
  bool records_ready = false;  // e32 .. r4 or w64, r4d of S_cap scenarios are there
  ScenState* state = nullptr;
  double* partials = nullptr;
  unsigned* arrive = nullptr;
  double* trace = nullptr;
  int trace_cap = 0;
  int* scen_list = nullptr;
  std::vector<int> h_scen_list;
  double *x_hist = nullptr, *d_hist = nullptr, *lam_hist = nullptr;
  int hist_cap = 0;
  int ckpt_every = 1;
  int ls_mode = kLsReference;
  // adjoint work buffers (allocated on first use)
  double *adj_xbar = nullptr, *adj_cbar = nullptr, *adj_seg = nullptr, *adj_part = nullptr;
  double* adj_scal = nullptr;
  unsigned* adj_arrive = nullptr;

  // scratch
  void* dist = nullptr;
  int64_t dist_tasks = 0;  // tasks the dist buffer holds
  void* path_scratch = nullptr;
  size_t path_scratch_bytes = 0;
  int* counters = nullptr;  // [2]
  int* err = nullptr;       // [1]
  int* err_info = nullptr;  // [2]
  // shortest-path API: sources, predecessors [api_rows][n1] and, api_pred_rows
  // at a time, as the caller's link indices
  int *api_src = nullptr, *pred_buf = nullptr;
  int64_t *api_pred = nullptr, *api_perm = nullptr;
  int64_t api_rows = 0, api_pred_rows = 0;
  unsigned long long* path_stats = nullptr;  // [8] rounds, tasks, expansions, idle polls, batches
  // buffers of the one-shot API (weights in both precisions, loaded volumes)
  uint2* api_e32 = nullptr;
  uint2* api_e4 = nullptr;
  uint2* api_r32 = nullptr;
  double* api_w64 = nullptr;
  unsigned long long* api_yfx = nullptr;

  // elimination hierarchy (hierarchy.h): the solver's shortest paths and
  // loading where the plan suits the network; the label-correction kernels
  // otherwise, and for a scenario whose labels leave the integers' range
  std::shared_ptr<HierBuilder> builder;  // makes the plan, until it is asked for
  bool hier = false;             // the plan is in place
  bool hier_on = false;          // the iterations run on it (choose_paths)
  ScenState* api_state = nullptr;  // of a loading through the API
  int hier_cap = 0;              // scenarios that its buffers were made for
  HierGraph hg{};
  double hier_relaxations = 0;
  std::vector<int> h_tile_ptr;   // first tile of each elimination level
  int u_exp0 = 0;                // exponent of the first labels
  int *h_opos = nullptr, *h_group = nullptr, *h_column = nullptr;  // origins by position
  int *h_chain_ptr = nullptr, *h_chain = nullptr;
  int* h_dest_of = nullptr;      // destination index of each node or -1
  int h_dests = 0, h_width = 0;  // demand by destination: [h_dests][h_width]
  unsigned long long *h_dem = nullptr, *h_sc_dem = nullptr;
  size_t hier_bytes = kHierBytes;  // bound of the buffers below
  int hier_slots = 0;            // scenarios they hold
  unsigned long long *h_w = nullptr, *h_d0 = nullptr, *h_fup = nullptr;
  unsigned long long *h_dlab = nullptr, *h_vol = nullptr;
  unsigned long long *h_mid = nullptr, *h_flow = nullptr;
  unsigned char* h_via = nullptr;
  int *h_from = nullptr, *h_list = nullptr, *h_list_n = nullptr;
  unsigned short* h_arr = nullptr;
  struct HierCourse {
    int iter = -1, pauses = 0;   // the iteration that paused last, and how often
    int spread = 0;              // iterations given to the label-correction kernels for their spread
  };
  std::vector<HierCourse> hier_course;  // by scenario, of the present solve
  // whether scenario s takes its iterations on the hierarchy
  bool on_hierarchy(int s) const {
    return hier_on && (s >= static_cast<int>(hier_course.size()) || hier_course[s].spread < kSpreadIters);
  }

  cudaStream_t stream = nullptr;
  cudaGraphExec_t gexec = nullptr;
  int g_iters = 0, g_nscen = -1;
  bool g_dem = false, g_links = false;
  int solve_max_iters = 0;
  int last_nscen = 1;  // scenarios of the last solve (for run_iterations)

  // kernel timing: event pairs recorded around launches (also inside graphs)
  struct Timed {
    int kind;  // 0 shortest paths, 1 loading, 2 line search, 3 step
    cudaEvent_t a, b;
  };
  bool timing = false;
  std::vector<cudaEvent_t> ev_pool;
  size_t ev_used = 0;
  std::vector<Timed> timed;       // launches of the current graph (or direct enqueue)
  double kt_ms[4] = {0, 0, 0, 0};
  long long kt_n[4] = {0, 0, 0, 0};
  long long launches = 0;         // kernels launched by the solver
  long long g_kernels = 0;        // kernels in the current graph
  long long pending_kernels = 0;  // kernels enqueued directly since the last sync
  bool measuring = false;         // marks enabled for the path kernels of an iteration
  cudaEvent_t next_event();
  int mark(int kind, bool begin);
  int collect_timing();
  void count_launches(long long n);

  // launch shapes
  int sssp_block = 256, aon_block = 512, link_grid = 0;
  // line-search passes and step: block size and blocks per scenario
  int ls_block = 256, ls_link_grid = 0;
  int sssp_variant = kSsspAsync;
  double nf_delta = 1.0;      // near-far threshold step for the solver's costs
  double api_nf_delta = 1.0;  // the same for the weights of the one-shot API
  bool sssp_smem = true, aon_smem = true;
  int sssp_grid = 0, aon_grid = 0;
  // line-search blocks per scenario: about 16 blocks per SM over the whole
  // batch, so that a batch's threads each sum many links and the 16-value
  // block reductions stay a small part of the FP64 work
  int ls_grid(int nscen) const {
    const int want = (16 * num_sms + nscen - 1) / (nscen > 0 ? nscen : 1);
    return want < 1 ? 1 : (want > step_grid(nscen) ? step_grid(nscen) : want);
  }
  // line-search passes over the whole grid; k_ls_rest goes on with what is left
  // (steps below 2^-24, exact roots after six passes).  One pass would save 2 us
  // an iteration of a small network early in a solve, but late most steps are
  // below 2^-12 and the one block takes 20 us longer (416 nodes to relative gap
  // 1e-5, 26,000 iterations: 12,700 -> 17,200 it/s with two).
  int grid_passes() const { return ls_mode == kLsExact ? 6 : 2; }
  // One scenario whose links make up to two blocks per SM: one block per SM, its
  // share longer.  Else some SMs have twice the FP64 work of the others, a step
  // that costs as much at 1.01 as at 1.95 blocks per SM.  Line search of an
  // iteration in FP64 mode, us, by blocks per SM: 1.01 58 -> 44, 1.25 59 -> 45, 1.5
  // 61 -> 47, 1.8 61 -> 49, 1.95 61 -> 51 (FP32 mode 50..53 -> 39..41); at two the
  // grid is full (68 either way).
  int step_grid(int nscen) const {
    return nscen == 1 && ls_link_grid > num_sms && ls_link_grid < 2 * num_sms ? num_sms
                                                                              : ls_link_grid;
  }

  std::vector<DevMem> owned;

  ~Ctx();
  int alloc(void** p, size_t bytes);
  template <class T>
  int alloc_n(T** p, size_t n) {
    return alloc(reinterpret_cast<void**>(p), n * sizeof(T));
  }
  int ensure_scenarios(int S);
  int alloc_scenarios(int S);
  void release_scenarios();
  int plan_launches();

  Graph graph() const;
  LinkParams link_params() const;
  // the parameters of one scenario as a single shared row
  LinkParams link_params_of(int scen) const;
  bool absent_in(int scen, int k) const {
    return use_link_scen && !h_absent.empty() &&
           ((h_absent[static_cast<size_t>(scen) * absent_words + (k >> 5)] >> (k & 31)) & 1u);
  }
  Demand demand() const;
  PathArgs path_args(int nscen_slots) const;
  LinkArgs link_args(int nscen, bool records = false) const;

  // enqueue helpers (stream ordered, capturable)
  int enqueue_paths(int nscen, bool load, const uint2* e32p, const uint2* r32p, const double* w64p,
                    unsigned long long* ydst, bool use_state);
  int enqueue_iteration(int nscen);
  int enqueue_initial(int nscen, bool warm);
  int enqueue_tail(int nscen, bool records = false);
  int run_graph(int iters, int nscen);
  int take_plan();
  int hier_demand(const long long* dev_q, int nscen, unsigned long long** dem);
  void release_hier();
  int ensure_hier(int S);
  int have_hier(int nscen, bool own_demand, bool* there);
  bool hier_pays(int nscen, int levels, double relaxations, int arcs) const;
  bool hier_pays(int nscen) const {
    return hier_pays(nscen, static_cast<int>(h_tile_ptr.size()) - 1, hier_relaxations, hg.arcs);
  }
  int choose_paths(int nscen);
  int ensure_legacy(int S);
  int alloc_records(int S);
  void release_records();
  int ensure_labels();
  // the arrays of the last solve are there
  bool can_iterate() const {
    return S_cap > 0 && (hier_on ? hier_cap > 0 : records_ready);
  }
  int enqueue_hier(int nscen, const double* cost, long long stride, cudaEvent_t between = nullptr);
  HierArgs hier_args(const double* cost, long long stride) const;
  int hier_load_api(bool* loaded);
  int begin_paths(int nscen);
  int set_active(const std::vector<int>& active);
  int resume_paused(int S, std::vector<ScenState>& st);
  int run_corrected(const std::vector<int>& list, int iters);
  int run_active(const std::vector<int>& active, int iters);
  int sync_check();
  int read_states(int S, std::vector<ScenState>& out);
};

}  // namespace tapgpu

// the opaque handle of the C ABI
struct tapgpu_ctx {
  tapgpu::Ctx* c;
};
