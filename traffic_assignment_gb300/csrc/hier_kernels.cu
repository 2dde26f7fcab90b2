// hier_kernels.cu - shortest paths and all-or-nothing loading over the
// elimination hierarchy (hierarchy.h), for FP64 path costs; per scenario and
// iteration
//
//  k_hier_weights    arc weights from the link costs
//  k_hier_bottom     the nodes eliminated from below: w(a, b) = min(w(a, b),
//  k_hier_tiles      w(a, i) + w(i, b)) for every pair of upper neighbours a, b
//                    of i; subtrees, then levels of dense tiles
//  k_hier_mark       at the end, for every arc whose weight comes from such a
//  k_hier_mark_far   pair, the two arcs it splits into
//  k_hier_climb      one warp per origin: labels reached by up arcs alone
//                    (then down within a chunk)
//  k_hier_top        one block per group of 32 origins (lane = origin): labels
//                    of the upper nodes, from the roots down
//  k_hier_subs       one warp per group and subtree below them: labels down,
//                    then the demand carried back up
//  k_hier_volumes    the demand carried up the upper nodes, over the arcs that
//                    gave their labels
//  k_hier_descend    one warp per origin: the volumes that arrive by the climb
//  k_hier_split      shortcut volumes split down to link volumes
//
// Labels are integers (cost x 2^e rounded, 62 bits), so a
// path's label does not depend on how the hierarchy groups its links, equal
// labels are equal exactly, and comparisons against shortcut sums need no
// tolerance.  The exponent of a scenario follows its largest label, which gets
// kBits + 1 bits the next time.  A label that leaves the range pauses the
// scenario (done = kPausing, at the end of the loading kPaused), and so does a
// largest label of less than kMinBits + 1 bits (kCoarse): the host repeats the
// iteration at another exponent.  So a
// link's rounding is at most 2^-54 of the largest label, that of an FP64 sum
// up to 2^-53 of the sum at every link.
//
// One iteration of 10,000 nodes and 1,000 origins (220,000 arcs, 14 million
// relaxations): label correction and tree walks 1.67 ms for one scenario, 21.9
// ms for 16; the hierarchy 1.33 and 5.99 ms.  By kernel, us for 1 and 16
// scenarios: weights 6 / 42, bottom 35 / 82, tiles 38 x 8 / 38 x 16 (from one's end
// to the next one's), mark 46 / 377, mark_far 6 / 35, climb 200 / 1100, top 248 /
// 1520, subs 85 / 1124, volumes 153 / 453, descend 75 / 210, collect 4 / 35,
// passes 12 x 12 / 12 x 32, split 8 / 15, links 5 / 13, exponents 2 / 2.  With one
// scenario every kernel is bound by its chain of dependent steps (levels, chunks
// of an origin's path, rows of a subtree), so they are cut to keep the chain
// short; with many by the 64-bit additions and comparisons of the climb and the
// sweep.
#include "hier_kernels.cuh"

#include <cooperative_groups.h>

#include <algorithm>

namespace tapgpu {

namespace {

namespace cg = cooperative_groups;

constexpr unsigned kFull = 0xffffffffu;
constexpr unsigned long long kNoMid = ~0ull;
constexpr unsigned kNoArc = 0xffffffffu;      // a split into one arc only
// arrivals: the arc's column in its row, or
constexpr int kByClimb = 0xffff;  // label given by the climb
constexpr int kNoLabel = 0xfffe;
constexpr int kMaxExp = 900;

using Int = unsigned long long;  // labels, weights and volumes
constexpr Int kInf = 1ull << 62;
constexpr int kBits = 55;     // the largest label has kBits + 1 bits next time
constexpr int kMinBits = 53;  // with fewer the iteration is repeated
// The smallest label of a pair with demand has at least kLeastBits + 1 bits, so
// a link's rounding is at most 2^-41 of any path's cost; else the label-correction
// kernels take the iteration (kSpread).  City networks, cold and warm, have pairs
// from 1 to 2^7 .. 2^10: their smallest labels keep 46 to 49 bits.
constexpr int kLeastBits = 40;

__device__ __forceinline__ Int addmin(Int a, Int b, Int c) {
  const Int s = a + b;
  return s < c ? s : c;
}

struct alignas(32) Int4 {
  Int v[4];
};

__device__ __forceinline__ Int4 vec_load(const Int* p) { return *reinterpret_cast<const Int4*>(p); }

__device__ __forceinline__ int vload_int(const int* p) {
  return *reinterpret_cast<const volatile int*>(p);
}

__device__ __forceinline__ void weights4(const Int* p, Int (&w)[4]) {
  const ulonglong2 x = __ldg(reinterpret_cast<const ulonglong2*>(p));
  const ulonglong2 y = __ldg(reinterpret_cast<const ulonglong2*>(p) + 1);
  w[0] = x.x;
  w[1] = x.y;
  w[2] = y.x;
  w[3] = y.y;
}

// integer weight of link k of a scenario; kInf when absent or out of range, zero
// for a zero cost only (a label of zero is exact)
__device__ __forceinline__ Int link_weight(const HierArgs& a, int scen, int k, double scale) {
  if (a.absent &&
      ((__ldg(a.absent + static_cast<size_t>(scen) * a.absent_words + (k >> 5)) >> (k & 31)) & 1u))
    return kInf;
  const double c = a.cost[static_cast<size_t>(scen) * static_cast<size_t>(a.cost_stride) + k];
  const double v = __dmul_rn(c, scale);
  if (!(v < static_cast<double>(kInf))) return kInf;
  const Int w = __double2ull_rn(v);
  return w == 0 && c > 0.0 ? Int(1) : w;
}

// the two arc slots (planes included) an arc splits into
__device__ __forceinline__ unsigned long long split_of(int first, unsigned second) {
  return (static_cast<unsigned long long>(first) << 32) | second;
}

// the blocks of a cluster: global writes before are seen after
__device__ __forceinline__ void cluster_barrier(int cluster) {
  if (cluster > 1) {
    __threadfence();
    cg::this_cluster().sync();
  } else {
    __syncthreads();
  }
}

// Programmatic launches: a kernel may start while the one before it in the
// stream still runs, and reads what that one wrote only after the wait (by
// plain or L2 loads; the plan's arrays may be read before).  The next one is let
// in after the wait, so two are under way at most.  For the chains of short
// launches (36 levels of tiles, 12 passes of the splits; 10,000 nodes, one
// scenario: 55 us less of a 1.4 ms iteration).
__device__ __forceinline__ void wait_for_previous() {
  asm volatile("griddepcontrol.wait;" ::: "memory");
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
}

__device__ __forceinline__ void copy16(void* smem, const void* global) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(smem))),
               "l"(global));
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;"); }
template <int N>
__device__ __forceinline__ void copy_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}
__device__ __forceinline__ void copy1(Int* smem, const Int* global) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"(
                   static_cast<unsigned>(__cvta_generic_to_shared(smem))),
               "l"(global), "n"(sizeof(Int)));
}

constexpr int kElimBlock = 256;

// arc weights of the scenarios from their link costs
__global__ void __launch_bounds__(kElimBlock) k_hier_weights(HierArgs a) {
  const HierGraph& h = a.h;
  const int slot = blockIdx.y;
  const int scen = a.scen_list ? a.scen_list[a.slot0 + slot] : 0;
  if (a.state[scen].done) return;
  const double scale = scalbn(1.0, a.state[scen].u_exp);
  Int* w = a.w + static_cast<size_t>(slot) * 3 * h.arcs;
  unsigned long long* mid = a.mid + static_cast<size_t>(slot) * 3 * h.arcs;
  for (int s = blockIdx.x * kElimBlock + threadIdx.x; s < 3 * h.arcs; s += gridDim.x * kElimBlock) {
    Int x = kInf;
    if (s < 2 * h.arcs)
      for (int k = __ldg(h.arc_link + s); k >= 0; k = __ldg(h.link_next + k)) {
        const Int y = link_weight(a, scen, k, scale);
        if (y < x) x = y;
      }
    w[s] = x;
    mid[s] = kNoMid;
  }
}

// One elimination subtree per block, its arcs in shared memory: level by
// level the sums of every pair of a node's upper neighbours, one thread each;
// then the closed plane of its chunks, and the splits of the arcs inside
// (their weights are final here).
__global__ void __launch_bounds__(kElimBlock) k_hier_bottom(HierArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const HierGraph& h = a.h;
  const int slot = blockIdx.y;
  const int scen = a.scen_list ? a.scen_list[a.slot0 + slot] : 0;
  if (a.state[scen].done) return;
  const HierPlan::Elim e = h.elims[blockIdx.x];
  const int arcs = h.arcs;
  Int* w = a.w + static_cast<size_t>(slot) * 3 * arcs;
  unsigned long long* mid = a.mid + static_cast<size_t>(slot) * 3 * arcs;
  Int* dn = reinterpret_cast<Int*>(smem_raw);
  Int* up = dn + e.len;
  for (int i = threadIdx.x; i < e.len; i += kElimBlock) {
    dn[i] = w[e.slot + i];
    up[i] = w[arcs + e.slot + i];
  }
  int p0 = __ldg(h.elim_pair + e.lev);
  for (int l = 0; l < e.num_levels; ++l) {
    const int p1 = __ldg(h.elim_pair + e.lev + l + 1);
    HierPlan::Pair ahead = {};
    if (p0 + static_cast<int>(threadIdx.x) < p1) ahead = h.pairs[p0 + threadIdx.x];
    __syncthreads();
    for (int i = p0 + threadIdx.x; i < p1; i += kElimBlock) {
      const HierPlan::Pair p = ahead;
      if (i + kElimBlock < p1) ahead = h.pairs[i + kElimBlock];
      const Int down = dn[p.b] + up[p.a], upw = dn[p.a] + up[p.b];
      if (p.target >= 0) {
        if (down < dn[p.target]) atomicMin(dn + p.target, down);
        if (upw < up[p.target]) atomicMin(up + p.target, upw);
      } else {
        if (down < kInf) atomicMin(w + ~p.target, down);
        if (upw < kInf) atomicMin(w + arcs + ~p.target, upw);
      }
    }
    p0 = p1;
  }
  __syncthreads();
  for (int i = threadIdx.x; i < e.len; i += kElimBlock) {
    w[e.slot + i] = dn[i];
    w[arcs + e.slot + i] = up[i];
  }
  for (int i = __ldg(h.elim_pair + e.lev) + threadIdx.x; i < p0; i += kElimBlock) {
    const HierPlan::Pair p = h.pairs[i];
    if (p.target < 0) continue;
    const Int down = dn[p.b] + up[p.a], upw = dn[p.a] + up[p.b];
    if (down == dn[p.target] && down < kInf)
      atomicMin(mid + e.slot + p.target, split_of(e.slot + p.b, arcs + e.slot + p.a));
    if (upw == up[p.target] && upw < kInf)
      atomicMin(mid + arcs + e.slot + p.target, split_of(e.slot + p.a, arcs + e.slot + p.b));
  }
  // closed plane: one thread per column, rows from the last
  for (int c = 0; c < e.num_close; ++c) {
    const HierChunk ch = h.chunks[__ldg(h.elim_close + e.close + c)];
    const int at = ch.woff - e.slot;
    for (int col = threadIdx.x; col < ch.r; col += kElimBlock) {
      for (int j = ch.k - 1; j >= 0; --j) {
        const int s = ch.woff + j * ch.ld + col;
        Int x = dn[s - e.slot];
        int via = -1;
        for (int i = j + 1; i < ch.k; ++i) {
          const Int y = w[2 * arcs + ch.woff + i * ch.ld + col] + dn[at + j * ch.ld + ch.r4 + ch.k - 1 - i];
          if (y < x) {
            x = y;
            via = i;
          }
        }
        w[2 * arcs + s] = x;
        if (x < kInf)
          mid[2 * arcs + s] =
              via < 0 ? split_of(s, kNoArc)
                      : split_of(ch.woff + j * ch.ld + ch.r4 + ch.k - 1 - via,
                                 static_cast<unsigned>(2 * arcs + ch.woff + via * ch.ld + col));
      }
    }
    // the down arcs again by upper row, for the climb
    for (int q = threadIdx.x; q < ch.k * ch.k; q += kElimBlock) {
      const int i = q / ch.k, j = q - i * ch.k;
      if (i > j)
        w[2 * arcs + ch.woff + i * ch.ld + ch.r4 + j] = dn[at + j * ch.ld + ch.r4 + ch.k - 1 - i];
    }
  }
}

constexpr int kFarParts = 4;  // blocks per subtree

// splits of the arcs above the subtrees through their nodes: one pair per thread
__global__ void __launch_bounds__(kElimBlock) k_hier_mark_far(HierArgs a) {
  const HierGraph& h = a.h;
  const int slot = blockIdx.y;
  const int scen = a.scen_list ? a.scen_list[a.slot0 + slot] : 0;
  if (a.state[scen].done) return;
  const HierPlan::Elim e = h.elims[blockIdx.x / kFarParts];
  const int arcs = h.arcs;
  const Int* w = a.w + static_cast<size_t>(slot) * 3 * arcs;
  unsigned long long* mid = a.mid + static_cast<size_t>(slot) * 3 * arcs;
  const Int* dn = w + e.slot;
  const Int* up = dn + arcs;
  const int p1 = __ldg(h.elim_pair + e.lev + e.num_levels);
#pragma unroll 2
  for (int i = __ldg(h.elim_pair + e.lev) + (blockIdx.x % kFarParts) * kElimBlock + threadIdx.x;
       i < p1; i += kFarParts * kElimBlock) {
    const HierPlan::Pair p = h.pairs[i];
    if (p.target >= 0) continue;
    const Int down = __ldg(dn + p.b) + __ldg(up + p.a), upw = __ldg(dn + p.a) + __ldg(up + p.b);
    if (down == __ldg(w + ~p.target) && down < kInf)
      atomicMin(mid + ~p.target, split_of(e.slot + p.b, arcs + e.slot + p.a));
    if (upw == __ldg(w + arcs + ~p.target) && upw < kInf)
      atomicMin(mid + arcs + ~p.target, split_of(e.slot + p.a, arcs + e.slot + p.b));
  }
}

// The pairs of the subtrees' nodes (once per plan), one warp per node: its
// upper neighbours in ascending order are its chunk's later nodes, then U.
__global__ void __launch_bounds__(kElimBlock) k_hier_pairs(HierGraph h, const HierPlan::Node* nodes,
                                                           int count, const int* chunk_of,
                                                           HierPlan::Pair* pairs) {
  const int lane = threadIdx.x & 31;
  const int at = blockIdx.x * (kElimBlock / 32) + (threadIdx.x >> 5);
  if (at >= count) return;
  const HierPlan::Node nd = nodes[at];
  const HierChunk ch = h.chunks[chunk_of[nd.pos]];
  const int i = nd.pos - ch.first, row = ch.woff + i * ch.ld;
  const int nl = ch.k - 1 - i, upper = nl + ch.r;
  auto col = [&](int t) { return t < nl ? ch.r4 + nl - 1 - t : t - nl; };
  int out = nd.pair;
  for (int x = 0; x < upper - 1; ++x) {
    const int base = x < nl ? ch.woff + (i + 1 + x) * ch.ld : h.tgt_base[ch.ioff + x - nl];
    const int rel = x < nl ? 0 : h.tgt_rel[ch.ioff + x - nl] - nl;
    for (int y = x + 1 + lane; y < upper; y += 32) {
      const int target = base + (x < nl ? col(y) : h.rel[rel + y]);
      const bool inside = target >= nd.slot && target < nd.slot + nd.len;
      pairs[out + y - x - 1] = {static_cast<unsigned short>(row + col(x) - nd.slot),
                                static_cast<unsigned short>(row + col(y) - nd.slot),
                                inside ? target - nd.slot : ~target};
    }
    out += upper - 1 - x;
  }
}

constexpr int kTileBlock = 4 * kHierTile;

struct TileShared {
  // columns of the tile's two sides: [side][pivot][column]
  alignas(16) Int dn[2][kHierPivots][kHierTile];
  alignas(16) Int up[2][kHierPivots][kHierTile];
  // the pivots' own arcs, i < j: down[i][j] = j -> i and over[i][j] = i -> j
  alignas(16) Int down[kHierPivots][kHierPivots];
  alignas(16) Int over[kHierPivots][kHierPivots];
};

// Up to kHierPivots columns of a chunk and the pairs of the later columns and
// upper neighbours in a kHierTile x kHierTile tile.  Every tile first eliminates
// the pivots' own arcs (one warp, in registers) and its two column blocks
// (one column, side and direction per thread) by itself; writing them back
// is left to the tiles on the diagonal, and a tile that reads values already
// written finds the same minima, so a level is one launch.  Then a min-plus
// product of the panels, 4 x 4 pairs in one direction per thread.  A level is
// bound by the chain of one tile's steps (few tiles, 16 pivots deep): small
// tiles and panels keep the chain short and spread a level over more SMs
// (32 columns and 64 x 64 tiles: 20 us per level).
__global__ void __launch_bounds__(kTileBlock) k_hier_tiles(HierArgs a, int tile0) {
  static_assert(kHierPivots == 16 && kHierTile == 32, "one warp holds 16 x 16 arcs");
  constexpr int P = kHierPivots;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  TileShared& sh = *reinterpret_cast<TileShared*>(smem_raw);
  const HierGraph& h = a.h;
  const HierPlan::Item it = h.tiles[tile0 + blockIdx.x];
  const int slot = blockIdx.y;
  const int scen = a.scen_list ? a.scen_list[a.slot0 + slot] : 0;
  const int arcs = h.arcs;
  Int* w = a.w + static_cast<size_t>(slot) * 3 * arcs;
  Int* wu = w + arcs;
  const HierChunk ch = h.chunks[it.chunk];
  const int k = min(P, ch.k - it.pivot);         // pivots
  const int later = ch.k - it.pivot - k;         // columns after them
  const int n = later + ch.r;
  auto row = [&](int i) { return ch.woff + (it.pivot + i) * ch.ld; };  // (pivot or later column)
  // slot column of the c-th of the later columns and upper neighbours
  auto column = [&](int c) { return c < later ? ch.r4 + later - 1 - c : c - later; };
  auto loc = [&](int i, int j) { return row(i) + ch.r4 + ch.k - 1 - it.pivot - j; };
  const int t = threadIdx.x & (kHierTile - 1);
  const int side = threadIdx.x >> 6;
  const bool upward = (threadIdx.x >> 5) & 1;
  const int c = (side ? it.b : it.a) + t;
  const bool first = it.a == 0 && it.b == 0, diagonal = it.a == it.b;
  // this thread's pairs: 4 x 4, upwards (a -> b) or downwards
  const bool over = threadIdx.x >= kTileBlock / 2;
  const int ty = ((threadIdx.x & 63) >> 3) * 4, tx = (threadIdx.x & 7) * 4;
  const int ca = it.a + ty, cb = it.b + tx;
  int base[4], rel[4];
#pragma unroll
  for (int y = 0; y < 4; ++y) {
    base[y] = -1;
    rel[y] = 0;
    if (ca + y >= later && ca + y < n) {
      base[y] = __ldg(h.tgt_base + ch.ioff + ca + y - later);
      rel[y] = __ldg(h.tgt_rel + ch.ioff + ca + y - later) - later;
    }
  }
  // the pairs' targets
  int target[4][4];
#pragma unroll
  for (int y = 0; y < 4; ++y)
#pragma unroll
    for (int z = 0; z < 4; ++z) {
      target[y][z] = -1;
      if (ca + y < cb + z && cb + z < n)
        target[y][z] = base[y] >= 0 ? base[y] + __ldg(h.rel + rel[y] + cb + z)
                                    : row(k + ca + y) + column(cb + z);
    }
  wait_for_previous();
  if (a.state[scen].done) return;
  Int x[P];
  Int* p = (upward ? wu : w) + row(0) + (c < n ? column(c) : 0);
#pragma unroll
  for (int i = 0; i < P; ++i) x[i] = i < k && c < n ? p[i * ch.ld] : kInf;
  if (threadIdx.x < 32) {
    // lane = (row y, half of the columns): arcs y -> 8 half .. 8 half + 7
    const int y = threadIdx.x & 15, half = threadIdx.x >> 4;
    Int s[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int j = 8 * half + q;
      s[q] = kInf;
      if (y < k && j < k && y != j) s[q] = y < j ? wu[loc(y, j)] : w[loc(j, y)];
    }
    const unsigned open = __ballot_sync(
        kFull, y < k && !__ldg(h.shut + ch.first + it.pivot + (y < k ? y : 0)));
    // (no branches: rows past the last and those not passed through count as
    // out of reach)
#pragma unroll
    for (int i = 0; i < P - 1; ++i) {
      Int to = __shfl_sync(kFull, s[i & 7], y + 16 * (i >> 3));
      to = y > i && ((open >> i) & 1u) ? to : kInf;
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const Int on = __shfl_sync(kFull, s[q], i + 16 * half);
        // (columns up to i are done: their own value changes nothing)
        s[q] = addmin(to, 8 * half + q > i ? on : kInf, s[q]);
      }
    }
#pragma unroll
    for (int q = 0; q < 8; ++q) {
      const int j = 8 * half + q;
      // (what passes through a row that is not passed through does not count)
      if (y < j) sh.over[y][j] = (open >> y) & 1u ? s[q] : kInf;
      if (y > j) sh.down[j][y] = (open >> j) & 1u ? s[q] : kInf;
      if (first && y < k && j < k && y != j && min(y, j) > 0) {
        if (y < j) wu[loc(y, j)] = s[q];
        else w[loc(j, y)] = s[q];
      }
    }
  }
  if (n == 0) return;
  __syncthreads();
  // the column: up: j -> i -> column, down: column -> i -> j
#pragma unroll
  for (int i = 0; i < P - 1; ++i) {
    const Int* s = upward ? sh.down[i] : sh.over[i];
#pragma unroll
    for (int j0 = (i + 1) & ~3; j0 < P; j0 += 4) {
      const Int4 y = vec_load(s + j0);
#pragma unroll
      for (int q = 0; q < 4; ++q)
        if (j0 + q > i) x[j0 + q] = addmin(x[i], y.v[q], x[j0 + q]);
    }
  }
  Int(*panel)[kHierTile] = upward ? sh.up[side] : sh.dn[side];
#pragma unroll
  for (int i = 0; i < P; ++i) {
    if (diagonal && side == 0 && c < n && i > 0 && i < k) p[i * ch.ld] = x[i];
    panel[i][t] = i < k && !__ldg(h.shut + ch.first + it.pivot + i) ? x[i] : kInf;
  }
  __syncthreads();
  if (ca >= n || cb >= n || cb + 3 <= ca) return;
  // downwards: b -> i -> a (the down arc of the lower node a), upwards: a -> i -> b
  Int m[4][4];
#pragma unroll
  for (int y = 0; y < 4; ++y)
#pragma unroll
    for (int z = 0; z < 4; ++z) m[y][z] = kInf;
  const Int(*pa)[kHierTile] = over ? sh.dn[0] : sh.up[0];
  const Int(*pb)[kHierTile] = over ? sh.up[1] : sh.dn[1];
#pragma unroll 4
  for (int i = 0; i < k; ++i) {
    const Int4 va = vec_load(&pa[i][ty]), vb = vec_load(&pb[i][tx]);
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int z = 0; z < 4; ++z) m[y][z] = addmin(va.v[y], vb.v[z], m[y][z]);
  }
  Int* to = over ? wu : w;
#pragma unroll
  for (int y = 0; y < 4; ++y)
#pragma unroll
    for (int z = 0; z < 4; ++z)
      if (target[y][z] >= 0 && m[y][z] < kInf) atomicMin(to + target[y][z], m[y][z]);
}

struct MarkShared {
  alignas(16) Int dn[2][kHierMaxCols][kHierMark];
  alignas(16) Int up[2][kHierMaxCols][kHierMark];
  Int down[kHierMaxCols][kHierMaxCols];
  Int over[kHierMaxCols][kHierMaxCols];
};

// A chunk's kHierMark x kHierMark tile of upper neighbours once all weights
// are final: for every arc whose weight is a sum through this chunk, the split
// through the chunk's first such node (over all chunks the lowest slots are
// kept); and the closed plane of the chunk.
__global__ void __launch_bounds__(kElimBlock) k_hier_mark(HierArgs a) {
  static_assert(kElimBlock == (kHierMark / 4) * (kHierMark / 4) && kElimBlock == 4 * kHierMark,
                "one 4 x 4 block, and one column, side and direction, per thread");
  extern __shared__ __align__(16) unsigned char smem_raw[];
  MarkShared& sh = *reinterpret_cast<MarkShared*>(smem_raw);
  const HierGraph& h = a.h;
  const HierPlan::Item it = h.marks[blockIdx.x];
  const int slot = blockIdx.y;
  const int scen = a.scen_list ? a.scen_list[a.slot0 + slot] : 0;
  if (a.state[scen].done) return;
  const int arcs = h.arcs;
  Int* w = a.w + static_cast<size_t>(slot) * 3 * arcs;
  const Int* wu = w + arcs;
  unsigned long long* mid = a.mid + static_cast<size_t>(slot) * 3 * arcs;
  const HierChunk ch = h.chunks[it.chunk];
  const int k = ch.k, r = ch.r;
  auto row = [&](int i) { return ch.woff + i * ch.ld; };
  auto loc = [&](int i, int j) { return ch.woff + i * ch.ld + ch.r4 + ch.k - 1 - j; };
  const int t = threadIdx.x & (kHierMark - 1);
  const int side = threadIdx.x >> 7;
  const bool upward = (threadIdx.x >> 6) & 1;
  const int col = (side ? it.b : it.a) + t;
  const bool first = it.a == 0 && it.b == 0, diagonal = it.a == it.b;
  {
    const Int* p = w + (upward ? arcs : 0) + ch.woff + col;
    Int(*x)[kHierMark] = upward ? sh.up[side] : sh.dn[side];
    if (col < r) {
#pragma unroll 4
      for (int i = 0; i < k; ++i) copy1(&x[i][t], p + i * ch.ld);
    } else {
#pragma unroll 4
      for (int i = 0; i < k; ++i) x[i][t] = kInf;
    }
    copy_commit();
  }
  const int lane = threadIdx.x & 31;
  const unsigned open =
      __ballot_sync(kFull, lane < k && !__ldg(h.shut + ch.first + (lane < k ? lane : 0)));
  const int ty = (threadIdx.x >> 4) * 4, tx = (threadIdx.x & 15) * 4;
  const int ca = it.a + ty, cb = it.b + tx;
  int target[4][4];
  Int m1[4][4], m2[4][4];
#pragma unroll
  for (int y = 0; y < 4; ++y) {
    int base = 0, rel = 0;
    if (ca + y < r) {
      base = __ldg(h.tgt_base + ch.ioff + ca + y);
      rel = __ldg(h.tgt_rel + ch.ioff + ca + y);
    }
#pragma unroll
    for (int z = 0; z < 4; ++z) {
      target[y][z] = ca + y < cb + z && cb + z < r ? base + __ldg(h.rel + rel + cb + z) : -1;
      m1[y][z] = target[y][z] >= 0 ? w[target[y][z]] : kInf;
      m2[y][z] = target[y][z] >= 0 ? wu[target[y][z]] : kInf;
    }
  }
  if (diagonal)
    for (int e = threadIdx.x; e < kHierMaxCols * kHierMaxCols; e += kElimBlock) {
      const int i = e / kHierMaxCols, j = e % kHierMaxCols;
      if (i < j && j < k) {
        sh.down[i][j] = w[loc(i, j)];
        sh.over[i][j] = wu[loc(i, j)];
      }
    }
  copy_wait<0>();
  __syncthreads();
  if (ca < r && cb < r && cb + 3 > ca) {
    int v1[4][4], v2[4][4];
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int z = 0; z < 4; ++z) v1[y][z] = v2[y][z] = -1;
#pragma unroll 2
    for (int i = k - 1; i >= 0; --i) {
      if (!((open >> i) & 1u)) continue;
      const Int4 da = vec_load(&sh.dn[0][i][ty]), ua = vec_load(&sh.up[0][i][ty]);
      const Int4 db = vec_load(&sh.dn[1][i][tx]), ub = vec_load(&sh.up[1][i][tx]);
#pragma unroll
      for (int y = 0; y < 4; ++y)
#pragma unroll
        for (int z = 0; z < 4; ++z) {
          if (db.v[z] + ua.v[y] == m1[y][z]) v1[y][z] = i;
          if (da.v[y] + ub.v[z] == m2[y][z]) v2[y][z] = i;
        }
    }
#pragma unroll
    for (int y = 0; y < 4; ++y)
#pragma unroll
      for (int z = 0; z < 4; ++z) {
        const int at = target[y][z], u = row(v1[y][z]), v = row(v2[y][z]);
        if (v1[y][z] >= 0 && m1[y][z] < kInf)
          atomicMin(mid + at, split_of(u + cb + z, arcs + u + ca + y));
        if (v2[y][z] >= 0 && m2[y][z] < kInf)
          atomicMin(mid + arcs + at, split_of(v + ca + y, arcs + v + cb + z));
      }
  }
  if (k == 1 || !diagonal) return;
  if (first)
    for (int e = threadIdx.x; e < kHierMaxCols * kHierMaxCols; e += kElimBlock) {
      const int y = e / kHierMaxCols, z = e % kHierMaxCols;
      if (y >= k || z >= k || y == z) continue;
      const Int own = y > z ? sh.down[z][y] : sh.over[y][z];
      // the chunk's own arc y -> z through a row i < y, z
      int via = -1;
#pragma unroll 4
      for (int i = min(y, z) - 1; i >= 0; --i)
        if (sh.down[i][y] + sh.over[i][z] == own && ((open >> i) & 1u)) via = i;
      if (via >= 0 && own < kInf)
        atomicMin(mid + (y > z ? loc(z, y) : arcs + loc(y, z)),
                  split_of(loc(via, y), arcs + loc(via, z)));
      // the down arcs again by upper row, for the climb
      if (y > z) w[2 * arcs + row(y) + ch.r4 + z] = own;
    }
  if (side == 0 && col < r) {
    const Int(*x)[kHierMark] = upward ? sh.up[0] : sh.dn[0];
    const Int(*s)[kHierMaxCols] = upward ? sh.down : sh.over;
    for (int j = k - 1; j >= 1; --j) {
      const Int y = x[j][t];
      int via = -1;
#pragma unroll 4
      for (int i = j - 1; i >= 0; --i)
        if (x[i][t] + s[i][j] == y && ((open >> i) & 1u)) via = i;
      if (via >= 0 && y < kInf)
        atomicMin(mid + (upward ? arcs : 0) + row(j) + col,
                  upward ? split_of(loc(via, j), arcs + row(via) + col)
                         : split_of(row(via) + col, arcs + loc(via, j)));
    }
  }
  // the closed plane of the columns, four rows at a time from the last: the
  // way to row j may pass a later row i, by the chunk's own arc i -> j
  __syncthreads();
  if (side != 1 || upward || col >= r) return;  // (side 1 holds the same columns)
  Int(*x)[kHierMark] = sh.dn[1];
  for (int j0 = (k - 1) & ~3; j0 >= 0; j0 -= 4) {
    Int y[4];
    int via[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      y[q] = j0 + q < k ? x[j0 + q][t] : kInf;
      via[q] = -1;
    }
    auto pass = [&](int q, int i, Int xi) {
      const Int z = xi + sh.down[j0 + q][i];
      if (z < y[q]) {
        y[q] = z;
        via[q] = i;
      }
    };
#pragma unroll 4
    for (int i = j0 + 4; i < k; ++i) {
      const Int xi = x[i][t];
#pragma unroll
      for (int q = 0; q < 4; ++q) pass(q, i, xi);
    }
#pragma unroll
    for (int i = 3; i >= 1; --i)
#pragma unroll
      for (int q = i - 1; q >= 0; --q)
        if (j0 + i < k) pass(q, j0 + i, y[i]);
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      if (j0 + q >= k) continue;
      x[j0 + q][t] = y[q];
      const int at = row(j0 + q) + col;
      w[2 * arcs + at] = y[q];
      if (y[q] < kInf)
        mid[2 * arcs + at] =
            via[q] < 0 ? split_of(at, kNoArc)
                       : split_of(loc(j0 + q, via[q]),
                                  static_cast<unsigned>(2 * arcs + row(via[q]) + col));
    }
  }
}

// ---------------------------------------------------------------------------
// climb
// ---------------------------------------------------------------------------

// The ancestors of an origin are one path of the elimination tree and hold
// the upper neighbours of each of its nodes, so a label is addressed by its
// row's climb slot (rows of all chunks above, then its own).  Chunk by chunk:
// the chunk's own up arcs with lane = row, then lane = upper neighbour, then
// the chunk's own down arcs, which complete the labels the sweep starts from.
__global__ void k_hier_climb(HierArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const HierGraph& h = a.h;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = blockDim.x >> 5;
  const long long task = static_cast<long long>(blockIdx.x) * warps + warp;
  if (task >= static_cast<long long>(a.nslots) * a.num_sources) return;
  const int slot = static_cast<int>(task / a.num_sources);
  // (neighbouring origins together: they climb the same chunks)
  const int o = __ldg(a.group + (task - static_cast<long long>(slot) * a.num_sources));
  const int scen = a.scen_list ? a.scen_list[a.slot0 + slot] : 0;
  if (a.state[scen].done) return;
  const int H = h.climb;
  Int* d = reinterpret_cast<Int*>(smem_raw) + static_cast<size_t>(warp) * H;
  int* from = reinterpret_cast<int*>(reinterpret_cast<Int*>(smem_raw) + static_cast<size_t>(warps) * H) +
              static_cast<size_t>(warp) * H;
  const Int* up = a.w + static_cast<size_t>(slot) * 3 * h.arcs + h.arcs;
  const size_t off = (static_cast<size_t>(slot) * a.num_sources + o) * H;
  Int* dout = a.d0 + off;
  Int* fup = a.fup + off;
  const int src = __ldg(a.opos + o);
  const int p0 = __ldg(a.chain_ptr + o), p1 = __ldg(a.chain_ptr + o + 1);
  HierChunk ch = h.chunks[__ldg(a.chain + p0)];
  int join = src - ch.first;  // the chunk's lowest row on the path
  const int most = ch.coff + ch.k;
  for (int i = lane; i < most; i += 32) {
    d[i] = i == ch.coff + join ? Int(0) : kInf;
    from[i] = -1;
  }
  __syncwarp();
  for (int p = p0; p < p1; ++p) {
    HierChunk next = ch;
    if (p + 1 < p1) next = h.chunks[__ldg(a.chain + p + 1)];  // (in flight during this chunk)
    const int k = ch.k;
    Int x = lane >= join && lane < k ? d[ch.coff + lane] : kInf;
    int fx = -1;
    for (int i0 = 0; i0 < k - 1; i0 += 4) {
      Int w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = i0 + q;
        w[q] = lane > i && lane < k ? __ldg(up + ch.woff + i * ch.ld + ch.r4 + k - 1 - lane) : kInf;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const Int y = __shfl_sync(kFull, x, i0 + q) + w[q];
        if (y < x) {
          x = y;
          fx = ch.woff + (i0 + q) * ch.ld + ch.r4 + k - 1 - lane;
        }
      }
    }
    if (fx >= 0) from[ch.coff + lane] = fx;
    // four columns per lane; the row that gave a label is tracked by fours
    for (int c0 = 0; c0 < ch.r4; c0 += 128) {
      const int col = c0 + 4 * lane;
      Int best[4];
      int blk[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        best[c] = kInf;
        blk[c] = 0;
      }
      const Int* p = up + ch.woff + (col < ch.r4 ? col : 0);
#pragma unroll 2
      for (int i0 = 0; i0 < k; i0 += 4) {
        Int w[4][4];
#pragma unroll
        for (int q = 0; q < 4; ++q)
          weights4(p + (i0 + q < k ? i0 + q : k - 1) * ch.ld, w[q]);  // (past the last: again)
        Int m[4];
#pragma unroll
        for (int c = 0; c < 4; ++c) m[c] = best[c];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const Int xi = __shfl_sync(kFull, x, i0 + q);  // (lanes past the last row: out of reach)
#pragma unroll
          for (int c = 0; c < 4; ++c) m[c] = addmin(xi, w[q][c], m[c]);
        }
#pragma unroll
        for (int c = 0; c < 4; ++c) {
          if (m[c] < best[c]) blk[c] = i0;
          best[c] = m[c];
        }
      }
      int at[4];
      bool better[4];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        at[c] = col + c < ch.r ? __ldg(h.idx_climb + ch.ioff + col + c) : -1;
        better[c] = at[c] >= 0 && best[c] < kInf && best[c] < d[at[c]];
      }
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        if (!__any_sync(kFull, better[c])) continue;
        int row = blk[c];
#pragma unroll
        for (int q = 3; q >= 0; --q) {
          const int i = blk[c] + q;
          const Int xi = __shfl_sync(kFull, x, i & 31);
          if (better[c] && i < k && xi + __ldg(up + ch.woff + i * ch.ld + col + c) == best[c]) row = i;
        }
        if (better[c]) {
          d[at[c]] = best[c];
          from[at[c]] = ch.woff + row * ch.ld + col + c;
        }
      }
    }
    // the same rows reached from a later one
    int via = 0xff;
    for (int i0 = k - 1; i0 >= 1; i0 -= 4) {
      Int w[4];
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int i = i0 - q;
        w[q] = lane < i ? __ldg(up + h.arcs + ch.woff + i * ch.ld + ch.r4 + lane) : kInf;
      }
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        if (i0 - q < 1) break;
        const Int y = __shfl_sync(kFull, x, i0 - q) + w[q];
        if (y < x) {
          x = y;
          via = i0 - q;
        }
      }
    }
    if (lane < k) {
      dout[ch.coff + lane] = x;
      a.via[off + ch.coff + lane] = static_cast<unsigned char>(via);
    }
    __syncwarp();
    if (p + 1 < p1) join = __ldg(h.idx + ch.ioff) - next.first;
    ch = next;
  }
  for (int i = lane; i < most; i += 32) {
    a.from[off + i] = from[i];
    fup[i] = 0;
  }
}

// ---------------------------------------------------------------------------
// sweep
// ---------------------------------------------------------------------------

// Adds val to flow[arc] for every lane of the mask with arc >= 0, lanes of one
// arc summed first (the lanes are neighbouring origins: mostly one or two arcs).
__device__ __forceinline__ void flow_add(unsigned long long* flow, int arc, unsigned long long val,
                                         unsigned mask) {
  const int lane = threadIdx.x & 31;
  unsigned rest = __ballot_sync(mask, arc >= 0) & mask;
  constexpr unsigned kPart = (1u << 27) - 1;  // 32 lanes' parts stay below 2^32
  for (int n = 0; rest && n < 4; ++n) {
    const int lead = __ffs(rest) - 1;
    const int c = __shfl_sync(mask, arc, lead);
    const bool on = arc == c;
    const unsigned same = __ballot_sync(mask, on) & mask;
    const unsigned p0 = __reduce_add_sync(mask, on ? static_cast<unsigned>(val) & kPart : 0u);
    const unsigned p1 =
        __reduce_add_sync(mask, on ? static_cast<unsigned>(val >> 27) & kPart : 0u);
    const unsigned p2 = __reduce_add_sync(mask, on ? static_cast<unsigned>(val >> 54) : 0u);
    if (lane == lead)
      atomicAdd(flow + c, static_cast<unsigned long long>(p0) +
                              (static_cast<unsigned long long>(p1) << 27) +
                              (static_cast<unsigned long long>(p2) << 54));
    rest &= ~same;
  }
  if ((rest >> lane) & 1u) atomicAdd(flow + arc, val);
}

constexpr int kLanes = 32;      // origins per group

// one lane's origin in a group's sweep
struct Lane {
  int op;        // position, -1: none
  size_t chain;  // its climb slots
};

__device__ __forceinline__ Lane lane_of(const HierArgs& a, int slot, int grp) {
  Lane r;
  const int o = __ldg(a.group + grp * kLanes + (threadIdx.x & 31));
  r.op = o >= 0 ? __ldg(a.opos + o) : -1;
  r.chain = (static_cast<size_t>(slot) * a.num_sources + (o >= 0 ? o : 0)) * a.h.climb;
  return r;
}

// a lane's demand at a destination: sums up what it saw of the labels
struct DemandAt {
  Int largest = 0, least = ~Int(0);
  bool out_of_range = false;
  // demand q at label x (all ones: some, below the unit)
  __device__ __forceinline__ Int take(Int q, Int x) {
    if (q == 0) return 0;
    if (x >= kInf) {  // out of the integers' range, or no path: the host finds out
      out_of_range = true;
      return 0;
    }
    if (x > largest) largest = x;
    if (x - 1 < least) least = x - 1;  // (zero wraps round)
    return q == ~Int(0) ? Int(0) : q;
  }
  // by whole warps
  __device__ __forceinline__ void report(ScenState& st) {
    if (out_of_range) st.done = kPausing;
    Int x = largest;
#pragma unroll
    for (int z = 16; z >= 1; z >>= 1) {
      const Int n = __shfl_xor_sync(kFull, x, z);
      if (n > x) x = n;
    }
    if ((threadIdx.x & 31) == 0 && x) atomicMax(&st.maxlab, x);
    x = least;
#pragma unroll
    for (int z = 16; z >= 1; z >>= 1) {
      const Int n = __shfl_xor_sync(kFull, x, z);
      if (n < x) x = n;
    }
    if ((threadIdx.x & 31) == 0 && x != ~Int(0)) atomicMin(&st.minlab, x + 1);
  }
};

// A warp's staging: two tiles of upper neighbours' labels and of the rows'
// weights to them.
template <int T>
struct TopShared {
  Int lab[2][T * kLanes];
  Int w[2][kHierJobRows * T];
};

// Up to RB rows of a top chunk: min over the upper neighbours' labels.  Labels
// and weights are staged a tile ahead (the chain of a level is one job's: with
// the weights read as they are needed, each tile waited twice for the L2); the
// arrival is tracked by blocks of four arcs and resolved once per tile.
template <int RB, int T>
__device__ __forceinline__ void top_rows(const HierArgs& a, const HierPlan::Top& t, int r0, int nr,
                                         const Int* w, const Lane& ln, const Int* d0, Int* Dg,
                                         unsigned short* P, TopShared<T>& sh) {
  constexpr int kIds = (T + 31) / 32;
  constexpr int kPiece = 16 / sizeof(Int), kPieces = kLanes / kPiece, kRows = kLanes / kPieces;
  constexpr int kRowPieces = T / kPiece;  // of a row's weights to a tile
  const HierGraph& h = a.h;
  const int lane = threadIdx.x & 31;
  const int pr = lane / kPieces, pp = (lane % kPieces) * kPiece;
  const bool climbed = ln.op >= t.fd && ln.op <= t.last;
  Int acc[RB];
  int arr[RB];
  const Int* wr = w + t.woff + static_cast<size_t>(r0) * t.ld;
  // the ids of a tile, spread over the lanes
  int ids[kIds];
  auto load_ids = [&](int u0) {
#pragma unroll
    for (int z = 0; z < kIds; ++z) {
      const int u = 32 * z + lane;
      ids[z] = u < T && u0 + u < t.r4 ? __ldg(h.top_uidx + t.uoff + u0 + u) : 0;
    }
  };
  auto stage = [&](int u0, int n) {
    for (int e = lane; e < RB * kRowPieces; e += 32) {
      const int q = e / kRowPieces, c = (e % kRowPieces) * kPiece;
      if (q < nr && u0 + c < t.r4) copy16(&sh.w[n][q * T + c], wr + q * t.ld + u0 + c);
    }
#pragma unroll
    for (int s = 0; s < T; s += kRows) {
      const int u = __shfl_sync(kFull, ids[s / 32], (s + pr) & 31);
      if (u0 + s + pr < t.r4)
        copy16(&sh.lab[n][(s + pr) * kLanes + pp], Dg + static_cast<size_t>(u) * kLanes + pp);
    }
    copy_commit();
  };
  load_ids(0);
  if (t.r4 > 0) stage(0, 0);
  load_ids(T);
#pragma unroll
  for (int q = 0; q < RB; ++q) {
    acc[q] = climbed && q < nr ? __ldg(d0 + ln.chain + t.coff + r0 + q) : kInf;
    arr[q] = acc[q] < kInf ? kByClimb : kNoLabel;
  }
  for (int u0 = 0, n = 0; u0 < t.r4; u0 += T, n ^= 1) {
    if (u0 + T < t.r4) {
      stage(u0 + T, n ^ 1);
      load_ids(u0 + 2 * T);
      copy_wait<1>();
    } else {
      copy_wait<0>();
    }
    __syncwarp();
    const Int* x = sh.lab[n] + lane;
    const Int* y0 = sh.w[n];
    const int nb = min(T, t.r4 - u0) / 4;
    int blk[RB];
#pragma unroll
    for (int q = 0; q < RB; ++q) blk[q] = -1;
#pragma unroll 2
    for (int b = 0; b < nb; ++b) {
      const Int x0 = x[(4 * b) * kLanes], x1 = x[(4 * b + 1) * kLanes],
              x2 = x[(4 * b + 2) * kLanes], x3 = x[(4 * b + 3) * kLanes];
#pragma unroll
      for (int q = 0; q < RB; ++q) {  // (rows past the last: any weights, not stored)
        const Int4 y = vec_load(y0 + q * T + 4 * b);
        const Int m = addmin(
            x3, y.v[3],
            addmin(x2, y.v[2], addmin(x1, y.v[1], addmin(x0, y.v[0], acc[q]))));
        if (m < acc[q]) blk[q] = b;
        acc[q] = m;
      }
    }
#pragma unroll
    for (int q = 0; q < RB; ++q) {
      if (blk[q] < 0) continue;
      const int b = blk[q];
      const Int4 y = vec_load(y0 + q * T + 4 * b);
      const int z = x[(4 * b) * kLanes] + y.v[0] == acc[q]       ? 0
                    : x[(4 * b + 1) * kLanes] + y.v[1] == acc[q] ? 1
                    : x[(4 * b + 2) * kLanes] + y.v[2] == acc[q] ? 2
                                                                 : 3;
      arr[q] = u0 + 4 * b + z;
    }
    __syncwarp();  // (the tile is copied over next)
  }
#pragma unroll
  for (int q = 0; q < RB; ++q)
    if (q < nr) {
      Dg[static_cast<size_t>(t.row + r0 + q) * kLanes + lane] = acc[q];
      P[static_cast<size_t>(t.row + r0 + q) * kLanes + lane] = static_cast<unsigned short>(arr[q]);
    }
}

constexpr int kTopBlock = 256;

// Labels of the top chunks of one scenario and group of origins per cluster,
// level by level from the roots; warps take jobs of a few rows.  One block
// per cluster once the groups fill the chip; four before, with larger tiles
// (a level's time is then one job's).
template <int T>
__global__ void __launch_bounds__(kTopBlock, T * sizeof(Int) > 128 ? 1 : 2)
    k_hier_top(HierArgs a, int cluster) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const HierGraph& h = a.h;
  const int cell = blockIdx.x / cluster;
  const int slot = cell / a.groups, grp = cell - slot * a.groups;
  const int scen = a.scen_list ? a.scen_list[a.slot0 + slot] : 0;
  if (a.state[scen].done) return;  // (the same for the blocks of a cluster)
  const int warp = (blockIdx.x % cluster) * (kTopBlock / 32) + (threadIdx.x >> 5);
  const int warps = cluster * (kTopBlock / 32);
  TopShared<T>& sh = reinterpret_cast<TopShared<T>*>(smem_raw)[threadIdx.x >> 5];
  const size_t at = static_cast<size_t>(cell) * h.top_rows * kLanes;
  Int* Dg = a.dlab + at;
  unsigned short* P = a.arr + at;
  const Int* w = a.w + static_cast<size_t>(slot) * 3 * h.arcs;
  const Int* d0 = a.d0;
  const Lane ln = lane_of(a, slot, grp);
  int i0 = __ldg(h.job_ptr), i1 = __ldg(h.job_ptr + 1);
  int job = i0 + warp < i1 ? __ldg(h.jobs + i0 + warp) : 0;
  HierPlan::Top t = h.tops[job >> 8];
  for (int l = 0; l < h.top_levels; ++l) {
    // (the next level's first job is read before the barrier)
    const int i2 = l + 1 < h.top_levels ? __ldg(h.job_ptr + l + 2) : i1;
    for (int i = i0 + warp; i < i1;) {
      const int r0 = (job >> 3) & 31, nr = (job & 7) + 1;
      i += warps;
      const int next = i < i1 ? i : i1 + warp;
      const int job_next = next < i2 ? __ldg(h.jobs + next) : 0;
      if (nr <= 2)
        top_rows<2, T>(a, t, r0, nr, w, ln, d0, Dg, P, sh);
      else if (nr <= 4)
        top_rows<4, T>(a, t, r0, nr, w, ln, d0, Dg, P, sh);
      else
        top_rows<kHierJobRows, T>(a, t, r0, nr, w, ln, d0, Dg, P, sh);
      job = job_next;
      t = h.tops[job >> 8];
    }
    if (i0 + warp >= i1) {  // (no job in this level)
      job = i1 + warp < i2 ? __ldg(h.jobs + i1 + warp) : 0;
      t = h.tops[job >> 8];
    }
    i0 = i1;
    i1 = i2;
    cluster_barrier(cluster);
  }
}

constexpr int kSubWarps = 4;

// shared memory of one warp's subtree
struct SubShared {
  Int lab[(kHierSubUpper + kHierSubRows) * kLanes];  // outside neighbours, rows; then volumes
  Int w[4 * kHierSubPieces];
  HierPlan::SubRow rows[kHierSubRows];
  int slot[kHierSubPieces];
  unsigned ids[kHierSubPieces];
  unsigned char arr[kHierSubRows * kLanes];
};

// Subtrees below the top chunks, one warp per scenario, group and subtree:
// labels downwards, then the demand of its destinations upwards, all in shared
// memory; what leaves the subtree is added to the top rows' volumes.
__global__ void __launch_bounds__(kSubWarps * 32) k_hier_subs(HierArgs a) {
  constexpr int kPiece = 16 / sizeof(Int), kPieces = kLanes / kPiece, kRows = kLanes / kPieces;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const HierGraph& h = a.h;
  const int lane = threadIdx.x & 31;
  const long long task = static_cast<long long>(blockIdx.x) * kSubWarps + (threadIdx.x >> 5);
  if (task >= static_cast<long long>(a.nslots) * a.groups * h.num_subs) return;
  SubShared& sh = reinterpret_cast<SubShared*>(smem_raw)[threadIdx.x >> 5];
  const int cell = static_cast<int>(task / h.num_subs);  // (slot, group)
  const int slot = cell / a.groups, grp = cell - slot * a.groups;
  const int scen = a.scen_list ? a.scen_list[a.slot0 + slot] : 0;
  if (__shfl_sync(kFull, vload_int(&a.state[scen].done), 0)) return;
  const HierPlan::Sub s = h.subs[task - static_cast<long long>(cell) * h.num_subs];
  const Int* w = a.w + static_cast<size_t>(slot) * 3 * h.arcs;
  unsigned long long* flow = a.flow + static_cast<size_t>(slot) * 3 * h.arcs;
  const size_t at = static_cast<size_t>(cell) * h.top_rows * kLanes;
  const Int* Dg = a.dlab + at;
  Int* F = a.vol + at + lane;
  {
    const int pr = lane / kPieces, pp = (lane % kPieces) * kPiece;
    for (int p = lane; p < 2 * s.num_rows; p += 32)
      copy16(reinterpret_cast<int4*>(sh.rows) + p,
             reinterpret_cast<const int4*>(h.sub_rows + s.row) + p);
    for (int e = pr; e < s.num_ext; e += kRows)
      copy16(sh.lab + e * kLanes + pp,
             Dg + static_cast<size_t>(__ldg(h.sub_ext + s.ext + e)) * kLanes + pp);
    for (int p = lane; p < s.num_pieces; p += 32) {
      const int at_slot = __ldg(h.sub_slot + s.piece + p);
      sh.slot[p] = at_slot;
      sh.ids[p] = __ldg(h.sub_ids + s.piece + p);
#pragma unroll
      for (int z = 0; z < 4; z += kPiece) copy16(sh.w + 4 * p + z, w + at_slot + z);
    }
    copy_commit();
    copy_wait<0>();
    __syncwarp();
  }
  const Lane ln = lane_of(a, slot, grp);
  const Int* d0 = a.d0 + ln.chain;
  Int* fup = a.fup + ln.chain;
  Int* lab = sh.lab + lane;
  for (int i = 0; i < s.num_rows; ++i) {
    const HierPlan::SubRow& r = sh.rows[i];
    Int acc = ln.op >= r.fd && ln.op <= r.last ? __ldg(d0 + r.slot) : kInf;
    int arr = acc < kInf ? 0xff : 0xfe, blk = -1;
    const int np = r.num_pieces, p0 = r.piece;
    for (int p = 0; p < np; ++p) {
      const unsigned ids = sh.ids[p0 + p];
      const Int4 y = vec_load(sh.w + 4 * (p0 + p));
      const Int m = addmin(
          lab[(ids >> 24) * kLanes], y.v[3],
          addmin(lab[((ids >> 16) & 255u) * kLanes], y.v[2],
                        addmin(lab[((ids >> 8) & 255u) * kLanes], y.v[1],
                                      addmin(lab[(ids & 255u) * kLanes], y.v[0], acc))));
      if (m < acc) blk = p;
      acc = m;
    }
    if (blk >= 0) {
      const unsigned ids = sh.ids[p0 + blk];
      const Int4 y = vec_load(sh.w + 4 * (p0 + blk));
      const int z = lab[(ids & 255u) * kLanes] + y.v[0] == acc           ? 0
                    : lab[((ids >> 8) & 255u) * kLanes] + y.v[1] == acc  ? 1
                    : lab[((ids >> 16) & 255u) * kLanes] + y.v[2] == acc ? 2
                                                                         : 3;
      arr = 4 * blk + z;
    }
    lab[(s.num_ext + i) * kLanes] = acc;
    sh.arr[i * kLanes + lane] = static_cast<unsigned char>(arr);
  }
  // volumes in the labels' place: the demand at the rows (four loads in flight)
  DemandAt da;
  Int* vol = reinterpret_cast<Int*>(lab);
  const Int* dem = a.dest_dem +
                 static_cast<size_t>(scen) * static_cast<size_t>(a.dest_stride) + grp * kLanes + lane;
  for (int i0 = 0; i0 < s.num_rows; i0 += 4) {
    Int q[4];
#pragma unroll
    for (int z = 0; z < 4; ++z) {
      const int dest = i0 + z < s.num_rows ? sh.rows[i0 + z].dest : -1;
      q[z] = dest >= 0 ? __ldg(dem + static_cast<size_t>(dest) * a.dest_width) : Int(0);
    }
#pragma unroll
    for (int z = 0; z < 4; ++z)
      if (i0 + z < s.num_rows) {
        const int at_row = (s.num_ext + i0 + z) * kLanes;
        vol[at_row] = da.take(q[z], lab[at_row]);
      }
  }
  for (int e = 0; e < s.num_ext; ++e) vol[e * kLanes] = 0;
  for (int i = s.num_rows - 1; i >= 0; --i) {
    const Int f = vol[(s.num_ext + i) * kLanes];
    if (!__any_sync(kFull, f != 0)) continue;
    const int arr = sh.arr[i * kLanes + lane];
    int arc = -1;
    if (f != 0) {
      if (arr == 0xff) {
        fup[sh.rows[i].slot] = f;
      } else {
        const int p = sh.rows[i].piece + (arr >> 2);
        arc = sh.slot[p] + (arr & 3);
        vol[((sh.ids[p] >> (8 * (arr & 3))) & 255u) * kLanes] += f;
      }
    }
    flow_add(flow, arc, f, kFull);
  }
  for (int e = 0; e < s.num_ext; ++e) {
    const Int f = vol[e * kLanes];
    if (f != 0) atomicAdd(F + static_cast<size_t>(__ldg(h.sub_ext + s.ext + e)) * kLanes, f);
  }
  da.report(a.state[scen]);
}

// Volumes of the top chunks of one scenario and group per cluster, from the
// lowest level; each row's volume goes to the upper neighbour that gave its
// label.  (Runs for a scenario that paused in this iteration too: it leaves
// the volumes zero.  One that paused before has no labels here: the slot may
// hold another scenario's.)
template <int N, bool AHEAD>
__global__ void __launch_bounds__(kTopBlock, AHEAD ? 1 : 4) k_hier_volumes(HierArgs a, int cluster) {
  const HierGraph& h = a.h;
  const int cell = blockIdx.x / cluster;
  const int slot = cell / a.groups, grp = cell - slot * a.groups;
  const int scen = a.scen_list ? a.scen_list[a.slot0 + slot] : 0;
  const int done = a.state[scen].done;
  if (done && done != kPausing) return;
  const int lane = threadIdx.x & 31;
  const int warp = (blockIdx.x % cluster) * (kTopBlock / 32) + (threadIdx.x >> 5);
  const int warps = cluster * (kTopBlock / 32);
  const size_t at = static_cast<size_t>(cell) * h.top_rows * kLanes + lane;
  const Int* D = a.dlab + at;
  Int* F = a.vol + at;
  const unsigned short* P = a.arr + at;
  unsigned long long* flow = a.flow + static_cast<size_t>(slot) * 3 * h.arcs;
  const Lane ln = lane_of(a, slot, grp);
  Int* fup = a.fup + ln.chain;
  const Int* dem = a.dest_dem +
                 static_cast<size_t>(scen) * static_cast<size_t>(a.dest_stride) + grp * kLanes + lane;
  DemandAt da;
  // N rows of a job, their arrivals, targets and demand: none depends on the
  // level above, so with AHEAD the first ones are read before the barrier
  struct Rows {
    int job;
    HierPlan::Top t;
    int p[N], u[N];
    Int q[N];
    Int x[N];
  };
  auto fetch = [&](Rows& r, int z0) {
    const int r0 = ((r.job >> 3) & 31) + z0, nr = (r.job & 7) + 1 - z0;
    int dest[N];
#pragma unroll
    for (int z = 0; z < N; ++z) {
      const size_t row = static_cast<size_t>(r.t.row + r0 + z);
      r.p[z] = z < nr ? P[row * kLanes] : kNoLabel;
      dest[z] = z < nr ? __ldg(h.top_dest + row) : -1;
    }
#pragma unroll
    for (int z = 0; z < N; ++z) {
      const size_t row = static_cast<size_t>(r.t.row + r0 + z);
      r.u[z] = r.p[z] < kNoLabel ? __ldg(h.top_uidx + r.t.uoff + r.p[z]) : 0;
      r.q[z] = 0;
      r.x[z] = 0;
      if (dest[z] >= 0) {
        r.q[z] = __ldg(dem + static_cast<size_t>(dest[z]) * a.dest_width);
        r.x[z] = D[row * kLanes];
      }
    }
  };
  auto open = [&](Rows& r, int i) {
    r.job = __ldg(h.jobs + i);
    r.t = h.tops[r.job >> 8];
    if (AHEAD) fetch(r, 0);
  };
  Rows r;
  int i0 = __ldg(h.job_ptr + h.top_levels - 1), i1 = __ldg(h.job_ptr + h.top_levels);
  if (i0 + warp < i1) open(r, i0 + warp);
  for (int l = h.top_levels - 1; l >= 0; --l) {
    const int im = l > 0 ? __ldg(h.job_ptr + l - 1) : 0;
    for (int i = i0 + warp; i < i1; i += warps) {
      if (i != i0 + warp) open(r, i);
      for (int z0 = 0; z0 <= (r.job & 7); z0 += N) {
        const int r0 = ((r.job >> 3) & 31) + z0, nr = (r.job & 7) + 1 - z0;
        if (!AHEAD || z0 > 0) fetch(r, z0);
        Int f[N];
#pragma unroll
        for (int z = 0; z < N; ++z)
          f[z] = z < nr ? __ldcg(F + static_cast<size_t>(r.t.row + r0 + z) * kLanes) : Int(0);
#pragma unroll
        for (int z = 0; z < N; ++z) {
          if (z >= nr) break;
          if (f[z] != 0) F[static_cast<size_t>(r.t.row + r0 + z) * kLanes] = 0;
          f[z] += da.take(r.q[z], r.x[z]);
          if (!__any_sync(kFull, f[z] != 0)) continue;
          int arc = -1;
          if (f[z] != 0) {
            if (r.p[z] == kByClimb) {
              fup[r.t.coff + r0 + z] = f[z];
            } else {
              arc = r.t.woff + (r0 + z) * r.t.ld + r.p[z];
              atomicAdd(F + static_cast<size_t>(r.u[z]) * kLanes, f[z]);
            }
          }
          flow_add(flow, arc, f[z], kFull);
        }
      }
    }
    i1 = i0;
    i0 = im;
    if (l > 0 && i0 + warp < i1) open(r, i0 + warp);
    cluster_barrier(cluster);
  }
  da.report(a.state[scen]);
}

// ---------------------------------------------------------------------------
// loading: the climb's volumes, then shortcuts split down to links
// ---------------------------------------------------------------------------

// From the root's chunk down the origin's path: within a chunk first the rows
// whose label came from a later row (in row order), then the climb's own
// arrivals from the last row.
__global__ void k_hier_descend(HierArgs a) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  const HierGraph& h = a.h;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int warps = blockDim.x >> 5;
  const long long task = static_cast<long long>(blockIdx.x) * warps + warp;
  if (task >= static_cast<long long>(a.nslots) * a.num_sources) return;
  const int slot = static_cast<int>(task / a.num_sources);
  // (neighbouring origins together: they climb the same chunks)
  const int o = __ldg(a.group + (task - static_cast<long long>(slot) * a.num_sources));
  const int scen = a.scen_list ? a.scen_list[a.slot0 + slot] : 0;
  if (a.state[scen].done) return;
  const int H = h.climb;
  Int* f = reinterpret_cast<Int*>(smem_raw) + static_cast<size_t>(warp) * H;
  const size_t off = (static_cast<size_t>(slot) * a.num_sources + o) * H;
  const Int* fup = a.fup + off;
  unsigned long long* flow = a.flow + static_cast<size_t>(slot) * 3 * h.arcs;
  const int p0 = __ldg(a.chain_ptr + o), p1 = __ldg(a.chain_ptr + o + 1);
  {
    const HierChunk ch = h.chunks[__ldg(a.chain + p0)];
    for (int i = lane; i < ch.coff + ch.k; i += 32) f[i] = fup[i];
  }
  __syncwarp();
  HierChunk next = h.chunks[__ldg(a.chain + p1 - 1)];
  for (int p = p1 - 1; p >= p0; --p) {
    const HierChunk ch = next;
    if (p > p0) next = h.chunks[__ldg(a.chain + p - 1)];
    Int x = lane < ch.k ? f[ch.coff + lane] : Int(0);
    if (!__any_sync(kFull, x != 0)) continue;
    const int via = lane < ch.k ? a.via[off + ch.coff + lane] : 0xff;
    const int arc = lane < ch.k ? a.from[off + ch.coff + lane] : -1;
    const int to = arc >= 0 ? __ldg(h.arc_climb + arc) : -1;
    unsigned rest = __ballot_sync(kFull, via != 0xff);
    while (rest) {
      const int j = __ffs(rest) - 1;
      rest &= rest - 1;
      const Int y = __shfl_sync(kFull, x, j);
      if (y == 0) continue;
      const int i = __shfl_sync(kFull, via, j);
      if (lane == j) {
        x = 0;
        atomicAdd(flow + ch.woff + j * ch.ld + ch.r4 + ch.k - 1 - i, y);
      }
      if (lane == i) x += y;
    }
    rest = __ballot_sync(kFull, arc >= 0);
    while (rest) {
      const int i = 31 - __clz(rest);
      rest &= ~(1u << i);
      const Int y = __shfl_sync(kFull, x, i);
      if (y == 0) continue;
      const int t = __shfl_sync(kFull, to, i);
      if (lane == i) atomicAdd(flow + h.arcs + arc, y);
      if (t >= ch.coff) {
        if (t < ch.coff + ch.k) {
          if (lane == t - ch.coff) x += y;
        } else if (lane == i) {
          f[t] += y;
        }
      }
      __syncwarp();  // (the next row may add to the same slot; shuffles do not order memory)
    }
    __syncwarp();
  }
}

// a shortcut's volume while it is listed (volumes are below 2^61)
constexpr unsigned long long kListed = 1ull << 63;

constexpr int kCollect = 4;  // arcs per thread

// The shortcuts that carry volume, one counter increment per block (one per
// warp serialised on the scenario's counter: 473 us for 64 scenarios of
// 720,000 arcs).
__global__ void __launch_bounds__(kElimBlock) k_hier_collect(HierArgs a) {
  const int slot = blockIdx.y;
  const int scen = a.scen_list ? a.scen_list[a.slot0 + slot] : 0;
  const int done = a.state[scen].done;
  if (done && done != kPausing) return;
  const int arcs3 = 3 * a.h.arcs, lane = threadIdx.x & 31;
  const unsigned long long* mid = a.mid + static_cast<size_t>(slot) * arcs3;
  unsigned long long* flow = a.flow + static_cast<size_t>(slot) * arcs3;
  if (done) {  // paused: what the sweep added is for nobody
    for (int z = 0; z < kCollect; ++z) {
      const int s = blockIdx.x * (kCollect * kElimBlock) + z * kElimBlock + threadIdx.x;
      if (s < arcs3) flow[s] = 0ull;
    }
    return;
  }
  int* list = a.list + static_cast<size_t>(slot) * 2 * arcs3;
  __shared__ int count, base;
  if (threadIdx.x == 0) count = 0;
  const int s0 = blockIdx.x * (kCollect * kElimBlock) + threadIdx.x;
  unsigned long long f[kCollect], md[kCollect];
#pragma unroll
  for (int z = 0; z < kCollect; ++z) {
    const int s = s0 + z * kElimBlock;
    f[z] = s < arcs3 ? flow[s] : 0ull;
    md[z] = s < arcs3 ? mid[s] : kNoMid;
  }
  unsigned m[kCollect];
  int total = 0;
#pragma unroll
  for (int z = 0; z < kCollect; ++z) {
    const bool on = f[z] != 0ull && md[z] != kNoMid;
    if (on) flow[s0 + z * kElimBlock] = f[z] | kListed;
    m[z] = __ballot_sync(kFull, on);
    total += __popc(m[z]);
  }
  __syncthreads();
  int at = 0;
  if (lane == 0 && total) at = atomicAdd(&count, total);
  __syncthreads();
  if (threadIdx.x == 0 && count) base = atomicAdd(a.list_n + slot * 4, count);
  __syncthreads();
  at = __shfl_sync(kFull, at, 0) + base;
#pragma unroll
  for (int z = 0; z < kCollect; ++z) {
    if ((m[z] >> lane) & 1u) list[at + __popc(m[z] & ((1u << lane) - 1u))] = s0 + z * kElimBlock;
    at += __popc(m[z]);
  }
}

constexpr int kSplitBlock = 256;
// Passes launched with the whole grid.  What they leave takes the one block of
// k_hier_split 8 us at 10,000 nodes, 15 at 40,000 and 24 at 100,000, of 1.3, 3.4
// and 7.4 ms an iteration (4 scenarios of 40,000 nodes 15, 2 of 100,000 27).
constexpr int kSplitPasses = 12;

// One pass over a scenario's listed shortcuts: a shortcut's volume passes to
// the two arcs of its split.  The first goes on in the same thread at once,
// with whatever it holds already; the second is listed for the next pass
// unless it is.  (whole warps; tid of nthr threads of the scenario)
__device__ __forceinline__ void split_pass(const HierArgs& a, int slot, int pass, int n, int tid,
                                           int nthr) {
  const int arcs3 = 3 * a.h.arcs;
  const int lane = threadIdx.x & 31;
  int* lists = a.list + static_cast<size_t>(slot) * 2 * arcs3;
  const int* cur = lists + (pass & 1) * arcs3;
  int* nxt = lists + ((pass + 1) & 1) * arcs3;
  int* ncnt = a.list_n + slot * 4 + (pass + 1) % 3;
  const unsigned long long* mid = a.mid + static_cast<size_t>(slot) * arcs3;
  unsigned long long* flow = a.flow + static_cast<size_t>(slot) * arcs3;
  for (int i0 = tid - lane; i0 < n; i0 += nthr) {
    // (from the end: mostly upper arcs first, so that lower ones are met with
    // all they get)
    const int s = i0 + lane < n ? __ldcg(cur + n - 1 - i0 - lane) : -1;
    unsigned long long m = kNoMid, f = 0ull;
    if (s >= 0) {
      m = mid[s];
      f = atomicExch(flow + s, 0ull) & ~kListed;
    }
    bool go = f != 0ull;
    while (__any_sync(kFull, go)) {
      int later = -1;
      if (go) {
        const int c0 = static_cast<int>(m >> 32), c1 = static_cast<int>(m & 0xffffffffu);
        const unsigned long long m0 = mid[c0], m1 = c1 >= 0 ? mid[c1] : kNoMid;
        if (c1 >= 0) {  // (kNoArc: c1 < 0)
          if (m1 == kNoMid) atomicAdd(flow + c1, f);
          else if (!(atomicAdd(flow + c1, f) & kListed) && !(atomicOr(flow + c1, kListed) & kListed))
            later = c1;
        }
        go = m0 != kNoMid;
        if (go) {
          f += atomicAnd(flow + c0, kListed) & ~kListed;  // (it stays listed if it was)
          m = m0;
        } else {
          atomicAdd(flow + c0, f);
        }
      }
      const unsigned on = __ballot_sync(kFull, later >= 0);
      if (on) {
        int at = 0;
        if (lane == __ffs(on) - 1) at = atomicAdd(ncnt, __popc(on));
        at = __shfl_sync(kFull, at, __ffs(on) - 1);
        if (later >= 0) __stcg(nxt + at + __popc(on & ((1u << lane) - 1u)), later);
      }
    }
  }
  if (tid == 0) __stcg(a.list_n + slot * 4 + (pass + 2) % 3, 0);
}

__global__ void __launch_bounds__(kSplitBlock) k_hier_pass(HierArgs a, int pass) {
  const int slot = blockIdx.y;
  wait_for_previous();
  if (a.state[a.scen_list ? a.scen_list[a.slot0 + slot] : 0].done) return;
  const int n = __ldcg(a.list_n + slot * 4 + pass % 3);
  const int tid = blockIdx.x * kSplitBlock + threadIdx.x;
  split_pass(a, slot, pass, n, tid, gridDim.x * kSplitBlock);
}

// What the passes above leave (short chains on a few arcs): until only links
// carry volume, one block per scenario.
__global__ void __launch_bounds__(kSplitBlock) k_hier_split(HierArgs a) {
  const int slot = blockIdx.x;
  if (a.state[a.scen_list ? a.scen_list[a.slot0 + slot] : 0].done) return;
  int* cnt = a.list_n + slot * 4;
  for (int pass = kSplitPasses; pass <= kSplitPasses + a.h.n; ++pass) {
    const int n = __ldcg(cnt + pass % 3);
    if (n == 0) break;
    split_pass(a, slot, pass, n, threadIdx.x, kSplitBlock);
    __threadfence();
    __syncthreads();
  }
  __syncthreads();
  if (threadIdx.x < 3) cnt[threadIdx.x] = 0;
}

// The links' volumes: an arc's goes to the lowest of its parallel links at its
// weight.
__global__ void __launch_bounds__(kElimBlock) k_hier_links(HierArgs a) {
  const HierGraph& h = a.h;
  const int slot = blockIdx.y;
  const int scen = a.scen_list ? a.scen_list[a.slot0 + slot] : 0;
  ScenState& st = a.state[scen];
  if (st.done) return;
  unsigned long long* flow = a.flow + static_cast<size_t>(slot) * 3 * h.arcs;
  const int u_exp = st.u_exp;
  const double scale = scalbn(1.0, u_exp);
  for (int k = blockIdx.x * kElimBlock + threadIdx.x; k < a.m; k += gridDim.x * kElimBlock) {
    const int s = __ldg(h.link_arc + k);
    int best = -1;
    if (s >= 0) {
      best = __ldg(h.arc_link + s);
      if (best != k) continue;  // the first of parallel links writes for all
      Int x = kInf;
      if (__ldg(h.link_next + k) >= 0)
        for (int q = k; q >= 0; q = __ldg(h.link_next + q)) {
          const Int z = link_weight(a, scen, q, scale);
          if (z < x) {
            x = z;
            best = q;
          }
        }
      const unsigned long long y = flow[s];
      for (int q = k; q >= 0; q = __ldg(h.link_next + q))
        a.y_fx[static_cast<size_t>(scen) * a.m + q] = q == best ? y : 0ull;
      flow[s] = 0ull;
    } else {
      a.y_fx[static_cast<size_t>(scen) * a.m + k] = 0ull;
    }
  }
}

// the next iteration's exponents
__global__ void __launch_bounds__(kElimBlock) k_hier_exponents(HierArgs a) {
  const int slot = blockIdx.x * kElimBlock + threadIdx.x;
  if (slot >= a.nslots) return;
  ScenState& st = a.state[a.scen_list ? a.scen_list[a.slot0 + slot] : 0];
  if (st.done == kPausing) st.done = kPaused;
  if (st.done || !st.maxlab) return;
  const int top = 63 - __clzll(static_cast<long long>(st.maxlab));
  const int u_exp = max(-kMaxExp, min(kMaxExp, st.u_exp + kBits - top));
  const bool spread = st.minlab < (Int(1) << kLeastBits);
  if ((top < kMinBits || (spread && top < kBits)) && u_exp != st.u_exp)
    st.done = kCoarse;
  else if (spread)
    st.done = kSpread;
  st.u_exp = u_exp;
  st.maxlab = 0ull;
  st.minlab = ~Int(0);
}

template <typename Fn>
cudaError_t max_smem(Fn fn) {
  return allow_max_smem_of(reinterpret_cast<const void*>(fn));
}

// in clusters (1: none); early: see wait_for_previous
template <typename Fn, typename... Args>
cudaError_t launch_with(Fn fn, dim3 grid, int block, size_t smem, int cluster, bool early,
                        cudaStream_t s, Args... args) {
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = grid;
  cfg.blockDim = dim3(block);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = s;
  cudaLaunchAttribute at[2];
  unsigned n = 0;
  if (cluster > 1) {
    at[n].id = cudaLaunchAttributeClusterDimension;
    at[n].val.clusterDim.x = cluster;
    at[n].val.clusterDim.y = 1;
    at[n++].val.clusterDim.z = 1;
  }
  if (early) {
    at[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[n++].val.programmaticStreamSerializationAllowed = 1;
  }
  cfg.attrs = at;
  cfg.numAttrs = n;
  return cudaLaunchKernelEx(&cfg, fn, args...);
}

}  // namespace

cudaError_t launch_hier_eliminate(const HierArgs& a, int num_levels, const int* tile_ptr, cudaStream_t s) {
  cudaError_t e = max_smem(k_hier_mark);
  if (e != cudaSuccess) return e;
  const int wb = (3 * a.h.arcs + 4 * kElimBlock - 1) / (4 * kElimBlock);
  k_hier_weights<<<dim3(wb, a.nslots), kElimBlock, 0, s>>>(a);
  if (a.h.num_elims > 0)
    k_hier_bottom<<<dim3(a.h.num_elims, a.nslots), kElimBlock, 2 * sizeof(Int) * kHierSubSlots, s>>>(a);
  for (int l = 0; l < num_levels; ++l)
    if ((e = launch_with(k_hier_tiles, dim3(tile_ptr[l + 1] - tile_ptr[l], a.nslots), kTileBlock,
                         sizeof(TileShared), 1, true, s, a, tile_ptr[l])) != cudaSuccess)
      return e;
  if (a.h.num_marks > 0)
    k_hier_mark<<<dim3(a.h.num_marks, a.nslots), kElimBlock, sizeof(MarkShared), s>>>(a);
  if (a.h.num_elims > 0)
    k_hier_mark_far<<<dim3(a.h.num_elims * kFarParts, a.nslots), kElimBlock, 0, s>>>(a);
  return cudaGetLastError();
}

cudaError_t launch_hier_climb(const HierArgs& a, cudaStream_t s) {
  const size_t per = hier_climb_smem(a.h.climb);
  const int warps = static_cast<int>(std::max<size_t>(1, std::min<size_t>(4, kHierMaxClimb / per)));
  cudaError_t e = max_smem(k_hier_climb);
  if (e != cudaSuccess) return e;
  const long long tasks = static_cast<long long>(a.nslots) * a.num_sources;
  k_hier_climb<<<static_cast<unsigned>((tasks + warps - 1) / warps), 32 * warps, per * warps, s>>>(a);
  return cudaGetLastError();
}

static cudaError_t descend_t(const HierArgs& a, cudaStream_t s) {
  const size_t per = sizeof(Int) * static_cast<size_t>(a.h.climb);
  const int warps = static_cast<int>(std::max<size_t>(1, std::min<size_t>(4, kHierMaxClimb / per)));
  cudaError_t e = max_smem(k_hier_descend);
  if (e != cudaSuccess) return e;
  const long long tasks = static_cast<long long>(a.nslots) * a.num_sources;
  k_hier_descend<<<static_cast<unsigned>((tasks + warps - 1) / warps), 32 * warps, per * warps, s>>>(a);
  return cudaGetLastError();
}

template <int T>
static cudaError_t top_t(const HierArgs& a, int cluster, cudaStream_t s) {
  const size_t smem = sizeof(TopShared<T>) * (kTopBlock / 32);
  cudaError_t e = max_smem(k_hier_top<T>);
  if (e != cudaSuccess) return e;
  return launch_with(k_hier_top<T>, dim3(a.nslots * a.groups * cluster), kTopBlock, smem, cluster, false, s, a, cluster);
}

cudaError_t launch_hier_sweep(const HierArgs& a, int num_sms, cudaStream_t s) {
  const int cells = a.nslots * a.groups;
  // A group's blocks in one cluster while there are SMs for all of them (top:
  // a block fills an SM; two waves of clusters of four took 485 us for 64
  // cells, clusters of two 316).  The volumes' blocks share an SM: 64 cells 177
  // us by fours, 212 by twos.
  const int cluster = 4 * cells <= num_sms ? 4 : (2 * cells <= num_sms ? 2 : 1);
  const int vcluster = 2 * cells <= num_sms ? 4 : (cells <= num_sms ? 2 : 1);
  cudaError_t e = cudaSuccess;
  if (a.h.top_levels > 0)
    e = cluster > 1 ? top_t<256 / sizeof(Int)>(a, cluster, s) : top_t<128 / sizeof(Int)>(a, 1, s);
  if (e != cudaSuccess) return e;
  if (a.h.num_subs > 0) {
    const size_t smem = sizeof(SubShared) * kSubWarps;
    if ((e = max_smem(k_hier_subs)) != cudaSuccess) return e;
    const long long tasks = static_cast<long long>(cells) * a.h.num_subs;
    k_hier_subs<<<static_cast<unsigned>((tasks + kSubWarps - 1) / kSubWarps), kSubWarps * 32, smem, s>>>(a);
  }
  if (a.h.top_levels > 0)
    return vcluster > 1 ? launch_with(k_hier_volumes<kHierJobRows, true>, dim3(cells * vcluster), kTopBlock,
                                      0, vcluster, false, s, a, vcluster)
                        : launch_with(k_hier_volumes<4, false>, dim3(cells), kTopBlock, 0, 1, false, s, a, 1);
  return cudaGetLastError();
}

int hier_launches(const HierGraph& h, int num_levels) {
  return 2 + num_levels + 2 * (h.num_elims > 0) + (h.num_marks > 0) + 2 * (h.top_levels > 0) +
         (h.num_subs > 0) + kSplitPasses + 5;
}

size_t hier_climb_smem(int climb) {
  return (sizeof(Int) + sizeof(int)) * static_cast<size_t>(climb);
}

cudaError_t launch_hier_pairs(const HierGraph& h, const HierPlan::Node* nodes, int count,
                              const int* chunk_of, HierPlan::Pair* pairs, cudaStream_t s) {
  if (count > 0)
    k_hier_pairs<<<(count + kElimBlock / 32 - 1) / (kElimBlock / 32), kElimBlock, 0, s>>>(
        h, nodes, count, chunk_of, pairs);
  return cudaGetLastError();
}

// demand by destination: [row][dest][width] (all ones: positive but below the
// fixed point)
__global__ void k_hier_demand(const int* od_ptr, const int* od_dest, const double* od_dem,
                              const int* dest_of, const long long* q, long long nnz, int origins,
                              const int* column, Int* out, int width, long long stride,
                              bool scenarios, bool below) {
  const int s = blockIdx.y;
  for (int o = blockIdx.x; o < origins; o += gridDim.x) {
    for (int j = od_ptr[o] + threadIdx.x; j < od_ptr[o + 1]; j += blockDim.x) {
      if (!(od_dem[j] > 0) || od_dest[j] == o + 1) continue;
      const int dest = dest_of[od_dest[j]];
      const Int x = static_cast<Int>(q[static_cast<size_t>(s) * nnz + j]);
      if (x == 0 && scenarios) continue;  // a demand scenario removed this pair
      Int* p = out + static_cast<size_t>(s) * stride + static_cast<size_t>(dest) * width + column[o];
      // entries of one pair add up; `below`, the second pass: pairs left at zero
      if (x != 0 && !below) atomicAdd(p, x);
      if (x == 0 && below) atomicCAS(p, Int(0), ~Int(0));
    }
  }
}

cudaError_t launch_hier_demand(const int* od_ptr, const int* od_dest, const double* od_dem,
                               const int* dest_of, const long long* q, long long nnz, int nscen,
                               int origins, const int* column, unsigned long long* out, int width,
                               long long stride, bool scenarios, cudaStream_t s) {
  const dim3 grid(std::min(origins, 1024), nscen);
  for (int below = 0; below < 2; ++below)
    k_hier_demand<<<grid, 256, 0, s>>>(od_ptr, od_dest, od_dem, dest_of, q, nnz, origins, column, out,
                                       width, stride, scenarios, below != 0);
  return cudaGetLastError();
}

cudaError_t launch_hier_load(const HierArgs& a, int num_sms, cudaStream_t s) {
  cudaError_t e = descend_t(a, s);
  if (e != cudaSuccess) return e;
  const int cb = (3 * a.h.arcs + kCollect * kElimBlock - 1) / (kCollect * kElimBlock);
  k_hier_collect<<<dim3(cb, a.nslots), kElimBlock, 0, s>>>(a);
  const int pb = std::max(1, (2048 / kSplitBlock) * num_sms / a.nslots);
  for (int p = 0; p < kSplitPasses; ++p)
    if ((e = launch_with(k_hier_pass, dim3(pb, a.nslots), kSplitBlock, 0, 1, true, s, a, p)) != cudaSuccess)
      return e;
  k_hier_split<<<a.nslots, kSplitBlock, 0, s>>>(a);
  k_hier_links<<<dim3((a.m + kElimBlock - 1) / kElimBlock, a.nslots), kElimBlock, 0, s>>>(a);
  k_hier_exponents<<<(a.nslots + kElimBlock - 1) / kElimBlock, kElimBlock, 0, s>>>(a);
  return cudaGetLastError();
}

}  // namespace tapgpu
