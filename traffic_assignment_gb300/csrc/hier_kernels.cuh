// hier_kernels.cuh - arguments and launches of the elimination-hierarchy path
// kernels (hier_kernels.cu; the plan is hierarchy.h's).
#pragma once
#include "fw_kernels.cuh"
#include "hierarchy.h"

namespace tapgpu {

// ScenState::done: labels left the integer range, or used too little of it
// (see hier_kernels.cu); kPausing: left it in the iteration under way, whose
// loading empties the scenario's buffers and then makes it kPaused; kSpread: the
// labels of some pairs have too few bits beside the largest one
constexpr int kPaused = 2, kCoarse = 3, kPausing = 4, kSpread = 5;

// the plan on the device
struct HierGraph {
  int n, arcs, climb;
  const HierChunk* chunks;
  const char* shut;
  const int* idx;
  const unsigned short* idx_climb;  // climb slot of each idx entry
  const unsigned short* arc_climb;  // climb slot of each arc slot's row
  const int *tgt_base, *tgt_rel, *rel;
  const int* arc_link;   // [2 arcs]
  const int *link_arc, *link_next;
  int num_elims, num_marks;
  const HierPlan::Elim* elims;
  const int *elim_pair, *elim_close;
  const HierPlan::Pair* pairs;
  const HierPlan::Item *tiles, *marks;
  int top_rows, top_levels, num_subs;
  const HierPlan::Top* tops;
  const int *top_uidx, *top_dest, *job_ptr, *jobs;
  const HierPlan::Sub* subs;
  const int* sub_ext;
  const HierPlan::SubRow* sub_rows;
  const int* sub_slot;
  const unsigned* sub_ids;
};

struct HierArgs {
  HierGraph h;
  int m, num_sources;
  // scenario slots slot0 .. slot0+nslots-1 of scen_list; the arrays below
  // are indexed by slot - slot0
  const int* scen_list;
  ScenState* state;
  int slot0, nslots;
  const double* cost;           // link costs, row [scenario * cost_stride]
  long long cost_stride;
  const unsigned* absent;       // [S][absent_words] links not in a scenario's network, or null
  int absent_words;
  unsigned long long* w;                      // [slot][3 arcs] integer weights: down, up, closed
  unsigned long long* mid;      // [slot][3 arcs] the two slots a shortcut splits into
  unsigned long long* flow;     // [slot][3 arcs] fixed-point volumes (all zero between loadings,
                                // so scenarios can take turns in a slot)
  unsigned long long* d0;                     // [slot][origin][climb] labels of the climb
  int* from;                    // [slot][origin][climb] the up arc each of them came over
  unsigned char* via;           // [slot][origin][climb] later row of the chunk it came from, or 0xff
  unsigned long long* fup;                    // [slot][origin][climb] volumes that arrive by the climb
  const int* opos;              // [origin] position of its node
  const int *chain_ptr, *chain; // chunks from each origin's to its root's
  const int* group;             // [padded origins] in position order, -1: none
  int groups;
  const unsigned long long* dest_dem;         // [scenario * dest_stride][dest][dest_width] demand by destination,
                                // columns as `group`
  long long dest_stride;
  int dest_width;
  unsigned long long* dlab;                   // [slot][group][top_rows][32] labels
  unsigned long long* vol;                    // [slot][group][top_rows][32] volumes (zero between iterations)
  unsigned short* arr;          // [slot][group][top_rows][32] arrival of each label
  int* list;                    // [slot][2][3 arcs] shortcuts to split
  int* list_n;                  // [slot][4] their counts (zero between iterations)
  unsigned long long* y_fx;     // [S][m]
};

constexpr int kHierWidth = 32;                   // origins per group of the sweep
size_t hier_climb_smem(int climb);               // per warp
constexpr size_t kHierMaxClimb = size_t(96) << 10;  // its bound
// the pairs of `count` nodes of a plan that is otherwise in place (chunk_of: by position)
cudaError_t launch_hier_pairs(const HierGraph& h, const HierPlan::Node* nodes, int count,
                              const int* chunk_of, HierPlan::Pair* pairs, cudaStream_t s);
// tile_ptr: first tile of each elimination level, [num_levels + 1]
cudaError_t launch_hier_eliminate(const HierArgs& a, int num_levels,
                                  const int* tile_ptr, cudaStream_t s);
cudaError_t launch_hier_climb(const HierArgs& a, cudaStream_t s);
cudaError_t launch_hier_sweep(const HierArgs& a, int num_sms, cudaStream_t s);
// demand by destination from the OD entries q [nscen][nnz] of the pairs of two nodes
// with base demand od_dem (dest_of: destination index of a node), `out` zero before
cudaError_t launch_hier_demand(const int* od_ptr, const int* od_dest, const double* od_dem,
                               const int* dest_of, const long long* q, long long nnz, int nscen,
                               int origins, const int* column, unsigned long long* out, int width,
                               long long stride, bool scenarios, cudaStream_t s);
cudaError_t launch_hier_load(const HierArgs& a, int num_sms, cudaStream_t s);
// kernels of one elimination, climb, sweep and loading
int hier_launches(const HierGraph& h, int num_levels);

}  // namespace tapgpu
