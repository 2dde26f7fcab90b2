// hierarchy.h - elimination hierarchy of a network's nodes (host plan).
//
// The nodes are eliminated in a minimum-degree order; eliminating a node
// joins its remaining neighbours by shortcut arcs.  The order depends on the
// topology alone, so it is made once per context; the arcs' weights are made
// anew for every scenario and iteration (hier_kernels.cu).  Every shortest
// path then climbs from its origin to some node and descends from there, so
// one pass over an origin's ancestors and one over all arcs gives its labels
// (customizable contraction hierarchies, Dibbelt, Strasser and Wagner 2016;
// the downward sweep over all nodes is PHAST, Delling et al. 2011).
//
// Nodes are named by their position in the order (0 first eliminated).  The
// upper neighbours of a node are those eliminated after it.  Columns with the
// same upper neighbours are grouped into chunks of at most kHierMaxCols
// consecutive positions, stored as dense panels:
//   idx list of chunk c (ld entries at ioff): its upper neighbours U outside
//     the chunk in ascending order, padded to r4 (a multiple of 4), then the
//     chunk's own positions first+k-1 .. first+1, padded to a multiple of 4
//   row i (node first+i): arcs woff + i*ld + t to idx entry t, t < r for U and
//     r4 <= t < r4 + k-1-i for the chunk's later nodes; the other slots are
//     padding (no link, infinite weight)
// An arc slot has three weights: down (upper node -> row node), up (plane
// arcs..2 arcs) and, in chunks of several columns, closed (2 arcs..3 arcs, U
// only): the way down from an upper neighbour to the row that may pass later
// nodes of the chunk, so that the rows of a chunk need only U's labels.
#pragma once
#include <atomic>
#include <cstdint>
#include <vector>

namespace tapgpu {

constexpr int kHierMaxCols = 32;  // columns of a chunk
constexpr int kHierSubSlots = 1024;  // arc slots of an elimination subtree
constexpr int kHierPivots = 16;   // columns eliminated together
constexpr int kHierTile = 32;     // side of an elimination tile
constexpr int kHierMark = 64;     // side of a tile of the splits
// sweep: rows of a chunk taken together by one group of lanes, and the
// limits of a subtree that one group of lanes handles by itself
constexpr int kHierJobRows = 8;
constexpr int kHierSubRows = 20;    // rows
constexpr int kHierSubUpper = 36;   // upper neighbours outside
constexpr int kHierSubPieces = 80;  // blocks of four arcs

struct alignas(16) HierChunk {
  int first, k, r, r4, ld, ioff, woff;
  int parent;  // chunk of the lowest upper neighbour, -1
  int fd;      // lowest position of its subtree
  int coff;    // rows of all chunks above it: row i has climb slot coff + i
  int pad0, pad1;
};

struct HierPlan {
  int n = 0;                      // nodes (positions)
  int arcs = 0;                   // arc slots
  double relaxations = 0;         // triangle relaxations of one elimination
  int climb = 0;                  // climb slots (largest coff + k)
  std::vector<int> pos, node;     // node -> position and back
  std::vector<HierChunk> chunks;  // ascending positions
  std::vector<int> chunk_of;      // position -> chunk
  std::vector<char> shut;         // position: not passed through
  std::vector<char> active;       // position: a destination in its subtree
  std::vector<int> idx;           // idx lists
  // elimination targets: the arc of upper neighbours a < b of chunk c is
  // tgt_base[ioff+a] + rel[tgt_rel[ioff+a] + b]
  std::vector<int> tgt_base, tgt_rel, rel;
  std::vector<int> arc_link;      // [2*arcs] down then up: lowest link of the slot or -1
  std::vector<int> link_arc;      // link -> slot (up: + arcs), -1 for a self loop
  std::vector<int> link_next;     // next parallel link of the same slot, -1
  // Elimination.  Subtrees of at most kHierSubSlots slots go to one thread
  // block each, node by node: pairs of a node's upper neighbours (levels of
  // independent nodes), the target inside the subtree (slot - first slot) or
  // outside (~slot).  The chunks above go by levels of tiles (a thread
  // block each: first columns a <= b).
  struct Pair {
    unsigned short a, b;  // the node's slots to the lower and the higher neighbour - first slot
    int target;
  };
  // (made on the device from the nodes: a node's pairs in order of the lower
  // neighbour start at `pair`)
  struct alignas(16) Node {
    int pos, pair;
    int slot, len;        // its subtree's slots
  };
  struct alignas(16) Elim {
    int slot, len;        // its slots
    int lev, num_levels;  // pairs of level l: elim_pair[lev + l] .. elim_pair[lev + l + 1]
    int close, num_close; // its chunks of several columns
    int pad0, pad1;
  };
  struct alignas(16) Item {
    int chunk, pivot, a, b;  // first column to eliminate; tile (of later columns, then U)
  };
  std::vector<Elim> elims;
  std::vector<int> elim_pair, elim_close;
  std::vector<Node> nodes;
  int num_pairs = 0;
  int num_levels = 0;
  std::vector<int> tile_ptr;  // [num_levels + 1]
  std::vector<Item> tiles;
  std::vector<Item> marks;    // tiles (of U) of the chunks above the subtrees, for the splits
  // sweep over the active rows: the top chunks level by level from the
  // roots (rows of a chunk are independent of each other: the closed plane),
  // and the subtrees below them
  struct alignas(16) Top {
    int row, k, r, r4;            // first top row
    int uoff, woff, ld, coff;     // upper neighbours' top rows, first slot (plane included)
    int fd, last, pad0, pad1;     // positions of its subtree
  };
  struct alignas(16) Sub {
    int ext, num_ext;             // outside upper neighbours: top rows
    int row, num_rows;            // its rows, upper ones first
    int piece, num_pieces;        // their blocks of four arcs
    int pad0, pad1;
  };
  struct alignas(16) SubRow {
    int piece, num_pieces;        // within the subtree
    int slot;                     // climb slot
    int fd, last;                 // positions of its chunk's subtree
    int dest;                     // destination or -1
    int pad0, pad1;
  };
  int top_rows = 0, top_levels = 0;
  std::vector<Top> tops;
  std::vector<int> top_uidx;      // top rows of the tops' upper neighbours (padded)
  std::vector<int> top_dest;      // [top_rows] destination or -1
  std::vector<int> job_ptr;       // [top_levels + 1]
  std::vector<int> jobs;          // top << 8 | first row << 3 | rows - 1
  std::vector<Sub> subs;
  std::vector<int> sub_ext;
  std::vector<SubRow> sub_rows;
  std::vector<int> sub_slot;      // first slot of each piece (plane included)
  std::vector<unsigned> sub_ids;  // its four local rows: outside neighbours first, then rows
  std::vector<int> dest_node;     // destinations
};

// Build the plan of the graph with n nodes (0..n-1) and m directed links
// tail -> head.  Nodes below first_thru are not passed through; dests marks
// the nodes with demand.  Returns false when the hierarchy does not suit the
// network: links between two nodes that are not passed through, or more arcs
// or elimination work than the limits allow; and soon after *stop is set.
bool hier_build(int n, int m, const int* tail, const int* head, int first_thru,
                const std::vector<char>& dests, double max_arcs, double max_relaxations,
                HierPlan& out, const std::atomic<bool>* stop = nullptr);

}  // namespace tapgpu
