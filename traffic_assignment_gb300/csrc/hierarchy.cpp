// hierarchy.cpp - minimum-degree order and panel layout of the elimination
// hierarchy (see hierarchy.h).
#include "hierarchy.h"

#include <algorithm>
#include <cmath>
#include <numeric>

namespace tapgpu {

namespace {

// Minimum-degree order on the quotient graph with element absorption,
// approximate external degrees and merging of indistinguishable nodes (the
// method of Amestoy, Davis and Duff 1996).  Nodes marked `early` are
// eliminated before all others; hubs, with more than 10 sqrt(n) neighbours, come
// last and are left out of the others' degrees, as that method has it: else every
// leaf of a hub goes through all of them (a star of 50,000 leaves 1.5 s, of
// 100,000 5.6 s; so 21 and 36 ms).  False when the fill exceeds max_arcs.
class MinDegree {
 public:
  MinDegree(int n, const std::vector<int>& ptr, const std::vector<int>& adj,
            const std::vector<char>& early, double max_arcs, const std::atomic<bool>* stop)
      : n_(n), early_(early), max_arcs_(max_arcs), stop_(stop), vars_(n), elems_(n), members_(n), nv_(n, 1),
        deg_(n), state_(n, kVar), mark_(n, 0), w_(n, 0), prev_(n, -1), next_(n, -1),
        head_(2 * static_cast<size_t>(n) + 2, -1), hash_(n, 0), chain_(n, -1) {
    const int most = std::max(16, static_cast<int>(10.0 * std::sqrt(static_cast<double>(n))));
    for (int v = 0; v < n; ++v)
      if (!early[v] && ptr[v + 1] - ptr[v] > most) {
        state_[v] = kDead;
        hubs_.push_back(v);
      }
    std::stable_sort(hubs_.begin(), hubs_.end(),
                     [&](int a, int b) { return ptr[a + 1] - ptr[a] < ptr[b + 1] - ptr[b]; });
    for (int v = 0; v < n; ++v) {
      if (state_[v] != kVar) continue;
      vars_[v].reserve(ptr[v + 1] - ptr[v]);
      for (int i = ptr[v]; i < ptr[v + 1]; ++i)
        if (state_[adj[i]] == kVar) vars_[v].push_back(adj[i]);
      deg_[v] = static_cast<int>(vars_[v].size());
      insert(v);
    }
  }

  bool run(std::vector<int>& order) {
    order.clear();
    order.reserve(n_);
    int stamp = 0, wstamp = 1;
    int lo = 0, left = n_ - static_cast<int>(hubs_.size());
    std::vector<int> lp, dense_hash;
    double fill = 0;
    while (left > 0) {
      while (lo < static_cast<int>(head_.size()) && head_[lo] < 0) ++lo;
      const int p = head_[lo];
      remove(p);
      // the new element: p's live neighbours
      ++stamp;
      mark_[p] = stamp;
      lp.clear();
      int weight = 0;
      auto take = [&](int v) {
        if (state_[v] == kVar && mark_[v] != stamp) {
          mark_[v] = stamp;
          lp.push_back(v);
          weight += nv_[v];
        }
      };
      for (int v : vars_[p]) take(v);
      for (int e : elems_[p]) {
        if (state_[e] != kElem) continue;
        for (int v : vars_[e]) take(v);
        state_[e] = kDead;
        std::vector<int>().swap(vars_[e]);
      }
      std::vector<int>().swap(elems_[p]);
      state_[p] = kElem;
      left -= nv_[p];
      emit(p, order);
      fill += static_cast<double>(nv_[p]) * (weight + 0.5 * (nv_[p] - 1));
      if (fill > max_arcs_ || (stop_ && *stop_)) return false;
      // |L_e \ L_p| of every element next to L_p
      const int base = wstamp;
      for (int v : lp)
        for (int e : elems_[v]) {
          if (state_[e] != kElem) continue;
          if (w_[e] < base) w_[e] = base + deg_[e];
          w_[e] -= nv_[v];
        }
      int max_left = 0;
      size_t live = 0;
      for (int v : lp) {
        remove(v);
        // elements: drop dead and absorbed ones, add p
        size_t ne = 0;
        long long d = 0;
        unsigned h = static_cast<unsigned>(p);
        auto& ev = elems_[v];
        for (int e : ev) {
          if (state_[e] != kElem) continue;
          const int out = w_[e] - base;
          if (out <= 0) {  // every node of e is in L_p: absorbed
            state_[e] = kDead;
            std::vector<int>().swap(vars_[e]);
            continue;
          }
          max_left = std::max(max_left, deg_[e]);
          d += out;
          h += static_cast<unsigned>(e);
          ev[ne++] = e;
        }
        ev.resize(ne);
        size_t na = 0;
        auto& av = vars_[v];
        for (int u : av) {
          if (state_[u] != kVar || mark_[u] == stamp) continue;  // (in L_p: covered by p)
          d += nv_[u];
          h += static_cast<unsigned>(u);
          av[na++] = u;
        }
        av.resize(na);
        if (ne == 0 && na == 0 && early_[v] == early_[p]) {  // p's neighbours only: goes with p
          state_[v] = kDead;
          weight -= nv_[v];
          left -= nv_[v];
          emit(v, order);
          continue;
        }
        ev.push_back(p);
        deg_[v] = static_cast<int>(std::min<long long>(deg_[v], d));
        hash_[v] = h;
        lp[live++] = v;
      }
      lp.resize(live);
      wstamp = base + max_left + n_ + 1;
      if (wstamp > (1 << 30)) {
        std::fill(w_.begin(), w_.end(), 0);
        wstamp = 1;
      }
      // merge indistinguishable nodes of L_p
      const size_t nb = lp.size() * 2 + 1;
      dense_hash.assign(nb, -1);
      for (int v : lp) {
        const size_t b = hash_[v] % nb;
        bool merged = false;
        for (int u = dense_hash[b]; u >= 0 && !merged; u = chain_[u]) {
          if (hash_[u] != hash_[v] || early_[u] != early_[v]) continue;
          if (vars_[u].size() != vars_[v].size() || elems_[u].size() != elems_[v].size()) continue;
          if (!same(u, v, stamp)) continue;
          nv_[u] += nv_[v];
          nv_[v] = 0;
          state_[v] = kDead;
          members_[u].push_back(v);
          std::vector<int>().swap(vars_[v]);
          std::vector<int>().swap(elems_[v]);
          merged = true;
        }
        if (!merged) {
          chain_[v] = dense_hash[b];
          dense_hash[b] = v;
        }
      }
      live = 0;
      for (int v : lp) {
        if (state_[v] != kVar) continue;
        const long long d = static_cast<long long>(deg_[v]) + weight - nv_[v];
        deg_[v] = static_cast<int>(std::max<long long>(0, std::min<long long>(d, left - nv_[v])));
        insert(v);
        lo = std::min(lo, key(v));
        lp[live++] = v;
      }
      lp.resize(live);
      vars_[p] = lp;
      deg_[p] = weight;
      if (lp.empty()) state_[p] = kDead;
    }
    order.insert(order.end(), hubs_.begin(), hubs_.end());
    return true;
  }

 private:
  enum : char { kVar, kElem, kDead };
  int key(int v) const { return early_[v] ? deg_[v] : n_ + deg_[v]; }
  void insert(int v) {
    const int k = key(v);
    next_[v] = head_[k];
    prev_[v] = -1;
    if (head_[k] >= 0) prev_[head_[k]] = v;
    head_[k] = v;
    slot_key(v) = k;
  }
  int& slot_key(int v) { return key_[v]; }
  void remove(int v) {
    const int k = key_[v];
    if (prev_[v] >= 0) next_[prev_[v]] = next_[v];
    else head_[k] = next_[v];
    if (next_[v] >= 0) prev_[next_[v]] = prev_[v];
  }
  void emit(int v, std::vector<int>& order) {
    order.push_back(v);
    for (size_t i = 0; i < members_[v].size(); ++i) emit(members_[v][i], order);
    std::vector<int>().swap(members_[v]);
  }
  bool same(int u, int v, int& stamp) {
    ++stamp;
    for (int x : vars_[u]) mark_[x] = stamp;
    for (int x : elems_[u]) mark_[x] = stamp;
    for (int x : vars_[v])
      if (mark_[x] != stamp) return false;
    for (int x : elems_[v])
      if (mark_[x] != stamp) return false;
    return true;
  }

  int n_;
  const std::vector<char>& early_;
  double max_arcs_;
  const std::atomic<bool>* stop_;
  std::vector<std::vector<int>> vars_, elems_, members_;
  std::vector<int> nv_, deg_, hubs_;
  std::vector<char> state_;
  std::vector<int> mark_, w_, prev_, next_;
  std::vector<int> head_;
  std::vector<unsigned> hash_;
  std::vector<int> chain_;
  std::vector<int> key_ = std::vector<int>(static_cast<size_t>(n_), 0);
};

}  // namespace

bool hier_build(int n, int m, const int* tail, const int* head, int first_thru,
                const std::vector<char>& dests, double max_arcs, double max_relaxations,
                HierPlan& out, const std::atomic<bool>* stop) {
  out = HierPlan();
  out.n = n;
  // undirected neighbours, each once
  std::vector<int> ptr(n + 1, 0), adj;
  {
    std::vector<int> cnt(n + 1, 0);
    for (int k = 0; k < m; ++k) {
      if (tail[k] == head[k]) continue;
      if (tail[k] < first_thru && head[k] < first_thru) return false;
      ++cnt[tail[k]];
      ++cnt[head[k]];
    }
    std::vector<int> start(n + 1, 0);
    for (int v = 0; v < n; ++v) start[v + 1] = start[v] + cnt[v];
    std::vector<int> all(start[n]), fill(start.begin(), start.end() - 1);
    for (int k = 0; k < m; ++k) {
      if (tail[k] == head[k]) continue;
      all[fill[tail[k]]++] = head[k];
      all[fill[head[k]]++] = tail[k];
    }
    adj.reserve(all.size());
    for (int v = 0; v < n; ++v) {
      std::sort(all.begin() + start[v], all.begin() + start[v + 1]);
      for (int i = start[v]; i < start[v + 1]; ++i)
        if (i == start[v] || all[i] != all[i - 1]) adj.push_back(all[i]);
      ptr[v + 1] = static_cast<int>(adj.size());
    }
  }
  std::vector<char> early(n, 0);
  for (int v = 0; v < n && v < first_thru; ++v) early[v] = 1;
  std::vector<int> order;
  if (!MinDegree(n, ptr, adj, early, max_arcs, stop).run(order)) return false;

  // elimination tree of that order, then its postorder
  std::vector<int> rank(n), parent(n, -1);
  for (int i = 0; i < n; ++i) rank[order[i]] = i;
  {
    std::vector<int> top(n, -1);
    for (int i = 0; i < n; ++i)
      for (int e = ptr[order[i]]; e < ptr[order[i] + 1]; ++e) {
        int j = rank[adj[e]];
        if (j >= i) continue;
        while (top[j] >= 0 && top[j] != i) {
          const int t = top[j];
          top[j] = i;
          j = t;
        }
        if (top[j] < 0) {
          top[j] = i;
          parent[j] = i;
        }
      }
  }
  std::vector<int> post(n);  // order index -> position
  {
    std::vector<int> first_child(n, -1), sibling(n, -1), stack;
    for (int i = n - 1; i >= 0; --i)
      if (parent[i] >= 0) {
        sibling[i] = first_child[parent[i]];
        first_child[parent[i]] = i;
      }
    int next = 0;
    for (int root = 0; root < n; ++root) {
      if (parent[root] >= 0) continue;
      stack.push_back(root);
      while (!stack.empty()) {
        const int v = stack.back();
        if (first_child[v] >= 0) {
          stack.push_back(first_child[v]);
          first_child[v] = sibling[first_child[v]];  // (its remaining children)
        } else {
          post[v] = next++;
          stack.pop_back();
        }
      }
    }
  }
  out.pos.resize(n);
  out.node.resize(n);
  for (int i = 0; i < n; ++i) {
    out.node[post[i]] = order[i];
    out.pos[order[i]] = post[i];
  }
  std::vector<int> par(n, -1);
  for (int i = 0; i < n; ++i)
    if (parent[i] >= 0) par[post[i]] = post[parent[i]];

  // upper neighbours of every position: its own links and its children's
  std::vector<int64_t> sptr(n + 1, 0);
  std::vector<int> st;
  st.reserve(static_cast<size_t>(n) * 16);
  {
    std::vector<int> mark(n, -1), last_child(n, -1), older(n, -1);
    for (int j = 0; j < n; ++j) {
      mark[j] = j;
      const int v = out.node[j];
      for (int e = ptr[v]; e < ptr[v + 1]; ++e) {
        const int u = out.pos[adj[e]];
        if (u > j && mark[u] != j) {
          mark[u] = j;
          st.push_back(u);
        }
      }
      for (int c = last_child[j]; c >= 0; c = older[c])
        for (int64_t i = sptr[c]; i < sptr[c + 1]; ++i) {
          const int u = st[static_cast<size_t>(i)];
          if (mark[u] != j) {
            mark[u] = j;
            st.push_back(u);
          }
        }
      sptr[j + 1] = static_cast<int64_t>(st.size());
      if (static_cast<double>(st.size()) > max_arcs || (stop && *stop)) return false;
      if (par[j] >= 0) {
        older[j] = last_child[par[j]];
        last_child[par[j]] = j;
      }
    }
  }

  // chunks
  out.chunk_of.resize(n);
  auto cols = [&](int j) { return static_cast<int>(sptr[j + 1] - sptr[j]); };
  int64_t slots = 0, lists = 0;
  for (int j = 0; j < n;) {
    int e = j + 1;
    while (e < n && e - j < kHierMaxCols && par[e - 1] == e && cols(e) == cols(e - 1) - 1)
      ++e;
    HierChunk c;
    c.first = j;
    c.k = e - j;
    c.r = cols(e - 1);
    c.r4 = (c.r + 3) & ~3;
    c.ld = c.r4 + ((c.k - 1 + 3) & ~3);
    c.ioff = static_cast<int>(lists);
    c.woff = static_cast<int>(slots);
    c.parent = -1;
    lists += c.ld;
    slots += static_cast<int64_t>(c.k) * c.ld;
    if (slots > (int64_t(1) << 28)) return false;
    for (int i = j; i < e; ++i) out.chunk_of[i] = static_cast<int>(out.chunks.size());
    out.chunks.push_back(c);
    out.relaxations += static_cast<double>(c.k) * c.r * c.r;
    j = e;
  }
  if (out.relaxations > max_relaxations) return false;
  out.arcs = static_cast<int>(slots);
  const int nc = static_cast<int>(out.chunks.size());
  out.idx.resize(static_cast<size_t>(lists));
  for (auto& c : out.chunks) {
    int* l = out.idx.data() + c.ioff;
    const int last = c.first + c.k - 1;
    std::copy(st.begin() + sptr[last], st.begin() + sptr[last + 1], l);
    std::sort(l, l + c.r);
    for (int t = c.r; t < c.ld; ++t) l[t] = last;
    for (int j = 1; j < c.k; ++j) l[c.r4 + c.k - 1 - j] = c.first + j;
    if (c.r > 0) c.parent = out.chunk_of[l[0]];
  }
  std::vector<int>().swap(st);

  // subtrees and climb slots
  out.shut.resize(n);
  out.active.resize(n);
  std::vector<int> fd(n);
  for (int j = 0; j < n; ++j) {
    fd[j] = j;
    out.shut[j] = out.node[j] < first_thru;
    out.active[j] = dests[out.node[j]];
  }
  for (int j = 0; j < n; ++j)
    if (par[j] >= 0) {
      fd[par[j]] = std::min(fd[par[j]], fd[j]);
      out.active[par[j]] |= out.active[j];
    }
  for (int c = nc - 1; c >= 0; --c) {
    HierChunk& ch = out.chunks[c];
    ch.fd = fd[ch.first + ch.k - 1];
    ch.coff = ch.parent >= 0 ? out.chunks[ch.parent].coff + out.chunks[ch.parent].k : 0;
    ch.pad0 = ch.pad1 = 0;
    out.climb = std::max(out.climb, ch.coff + ch.k);
  }

  // elimination targets
  out.tgt_base.assign(out.idx.size(), 0);
  out.tgt_rel.assign(out.idx.size(), 0);
  {
    for (const auto& c : out.chunks) {
      const int* u = out.idx.data() + c.ioff;
      for (int t0 = 0; t0 < c.r;) {
        const HierChunk& p = out.chunks[out.chunk_of[u[t0]]];
        int t1 = t0;
        while (t1 < c.r && u[t1] < p.first + p.k) ++t1;
        // columns of u[t0..r) in p's rows: its own nodes, then a merge with its U
        const int off = static_cast<int>(out.rel.size()) - t0;
        const int* pu = out.idx.data() + p.ioff;
        int q = 0;
        for (int t = t0; t < c.r; ++t) {
          if (t < t1) {
            out.rel.push_back(p.r4 + p.k - 1 - (u[t] - p.first));
          } else {
            while (pu[q] != u[t]) ++q;
            out.rel.push_back(q);
          }
        }
        for (int t = t0; t < t1; ++t) {
          out.tgt_base[c.ioff + t] = p.woff + (u[t] - p.first) * p.ld;
          out.tgt_rel[c.ioff + t] = off;
        }
        t0 = t1;
      }
    }
  }

  // links
  out.arc_link.assign(2 * static_cast<size_t>(out.arcs), -1);
  out.link_arc.assign(m, -1);
  out.link_next.assign(m, -1);
  for (int k = m - 1; k >= 0; --k) {
    if (tail[k] == head[k]) continue;
    const int a = out.pos[tail[k]], b = out.pos[head[k]];
    const int lo = std::min(a, b), hi = std::max(a, b);
    const HierChunk& c = out.chunks[out.chunk_of[lo]];
    int t;
    if (hi < c.first + c.k) {
      t = c.r4 + c.k - 1 - (hi - c.first);
    } else {
      const int* u = out.idx.data() + c.ioff;
      t = static_cast<int>(std::lower_bound(u, u + c.r, hi) - u);
    }
    const int slot = c.woff + (lo - c.first) * c.ld + t + (a < b ? out.arcs : 0);
    out.link_arc[k] = slot;
    out.link_next[k] = out.arc_link[slot];
    out.arc_link[slot] = k;
  }

  // elimination: subtrees, then levels of tiles
  {
    std::vector<int> slots_below(nc, 0), height(n, 0), lev(nc, 0);
    for (int c = 0; c < nc; ++c) {
      const HierChunk& ch = out.chunks[c];
      slots_below[c] += ch.k * ch.ld;
      if (ch.parent >= 0)
        slots_below[ch.parent] =
            std::min(slots_below[ch.parent] + slots_below[c], kHierSubSlots + 1);
    }
    for (int j = 0; j < n; ++j)
      if (par[j] >= 0) height[par[j]] = std::max(height[par[j]], height[j] + 1);
    std::vector<char> top(nc, 0);
    std::vector<int> roots;
    for (int c = nc - 1; c >= 0; --c) {
      const int p = out.chunks[c].parent;
      if (p >= 0 && !top[p]) continue;
      if (slots_below[c] > kHierSubSlots) top[c] = 1;
      else roots.push_back(c);
    }
    // the largest subtrees first
    std::stable_sort(roots.begin(), roots.end(),
                     [&](int x, int y) { return slots_below[x] > slots_below[y]; });
    std::vector<std::vector<int>> by_height;
    for (int c : roots) {
      const HierChunk& root = out.chunks[c];
      const int last = root.first + root.k - 1;
      const HierChunk& low = out.chunks[out.chunk_of[root.fd]];
      HierPlan::Elim e = {};
      e.slot = low.woff;
      e.len = root.woff + root.k * root.ld - low.woff;
      if (e.len == 0) continue;
      e.lev = static_cast<int>(out.elim_pair.size());
      e.close = static_cast<int>(out.elim_close.size());
      by_height.assign(height[last] + 1, {});
      for (int j = root.fd; j <= last; ++j)
        if (!out.shut[j]) by_height[height[j]].push_back(j);
      for (int x = out.chunk_of[root.fd]; x <= c; ++x)
        if (out.chunks[x].k > 1) out.elim_close.push_back(x);
      e.num_close = static_cast<int>(out.elim_close.size()) - e.close;
      for (auto& nodes : by_height) {
        out.elim_pair.push_back(out.num_pairs);
        for (int j : nodes) {
          const HierChunk& ch = out.chunks[out.chunk_of[j]];
          const int upper = ch.first + ch.k - 1 - j + ch.r;
          if (upper < 2) continue;
          out.nodes.push_back({j, out.num_pairs, e.slot, e.len});
          out.num_pairs += upper * (upper - 1) / 2;
        }
      }
      out.elim_pair.push_back(out.num_pairs);
      e.num_levels = static_cast<int>(by_height.size());
      out.elims.push_back(e);
    }
    std::vector<std::vector<std::pair<int, int>>> levels;  // (chunk, first pivot)
    for (int c = 0; c < nc; ++c) {
      if (!top[c]) continue;
      const HierChunk& ch = out.chunks[c];
      for (int p = 0; p < ch.k; p += kHierPivots, ++lev[c]) {
        if (lev[c] >= static_cast<int>(levels.size())) levels.resize(lev[c] + 1);
        levels[lev[c]].push_back({c, p});
      }
      if (ch.parent >= 0) lev[ch.parent] = std::max(lev[ch.parent], lev[c]);
      for (int t = 0; t == 0 || t < ch.r; t += kHierMark)
        for (int u = t; u == t || u < ch.r; u += kHierMark) out.marks.push_back({c, 0, t, u});
    }
    out.num_levels = static_cast<int>(levels.size());
    out.tile_ptr.push_back(0);
    for (const auto& l : levels) {
      for (const auto& cp : l) {
        const HierChunk& ch = out.chunks[cp.first];
        const int cols = std::max(0, ch.k - cp.second - kHierPivots) + ch.r;
        for (int t = 0; t == 0 || t < cols; t += kHierTile)
          for (int u = t; u == t || u < cols; u += kHierTile)
            out.tiles.push_back({cp.first, cp.second, t, u});
      }
      out.tile_ptr.push_back(static_cast<int>(out.tiles.size()));
    }
  }

  // sweep
  std::vector<int> dest_of(n, -1);
  for (int v = 0; v < n; ++v)
    if (dests[v]) {
      dest_of[out.pos[v]] = static_cast<int>(out.dest_node.size());
      out.dest_node.push_back(v);
    }
  std::vector<int> rows(nc, 0), pieces(nc, 0);  // active ones of each chunk's subtree
  for (int c = 0; c < nc; ++c) {
    const HierChunk& ch = out.chunks[c];
    for (int i = 0; i < ch.k; ++i)
      if (out.active[ch.first + i]) {
        ++rows[c];
        pieces[c] += ch.r4 / 4;
      }
  }
  for (int c = 0; c < nc; ++c)
    if (out.chunks[c].parent >= 0) {
      rows[out.chunks[c].parent] += rows[c];
      pieces[out.chunks[c].parent] += pieces[c];
    }
  std::vector<int> level(nc, -1), top_of(nc, -1), sub_roots;
  std::vector<std::vector<int>> levels;
  for (int c = nc - 1; c >= 0; --c) {
    const HierChunk& ch = out.chunks[c];
    if ((ch.parent >= 0 && level[ch.parent] < 0) || rows[c] == 0) continue;
    if (rows[c] <= kHierSubRows && ch.r <= kHierSubUpper && pieces[c] <= kHierSubPieces) {
      sub_roots.push_back(c);
      continue;
    }
    level[c] = ch.parent >= 0 ? level[ch.parent] + 1 : 0;
    if (level[c] >= static_cast<int>(levels.size())) levels.resize(level[c] + 1);
    levels[level[c]].push_back(c);
  }
  auto plane = [&](const HierChunk& ch) { return ch.k > 1 ? 2 * out.arcs : 0; };
  std::vector<int> top_row(n, -1);
  out.top_levels = static_cast<int>(levels.size());
  out.job_ptr.push_back(0);
  for (auto& l : levels) {
    // jobs of eight rows where the level has many, else of four; long jobs
    // first, so that the last ones to finish are short
    int level_rows = 0;
    for (int c : l) level_rows += out.chunks[c].k;
    const int rb = level_rows >= 16 * kHierJobRows ? kHierJobRows : 4;
    std::sort(l.begin(), l.end(), [&](int a, int b) {
      const HierChunk &x = out.chunks[a], &y = out.chunks[b];
      return std::make_pair(y.r * std::min(y.k, rb), b) < std::make_pair(x.r * std::min(x.k, rb), a);
    });
    for (int c : l) {
      const HierChunk& ch = out.chunks[c];
      HierPlan::Top t = {};
      t.row = out.top_rows;
      t.k = ch.k;
      t.r = ch.r;
      t.r4 = ch.r4;
      t.uoff = static_cast<int>(out.top_uidx.size());
      t.woff = ch.woff + plane(ch);
      t.ld = ch.ld;
      t.coff = ch.coff;
      t.fd = ch.fd;
      t.last = ch.first + ch.k - 1;
      for (int i = 0; i < ch.r; ++i) out.top_uidx.push_back(top_row[out.idx[ch.ioff + i]]);
      while (out.top_uidx.size() % 4) out.top_uidx.push_back(0);
      for (int i = 0; i < ch.k; ++i) {
        top_row[ch.first + i] = out.top_rows++;
        out.top_dest.push_back(dest_of[ch.first + i]);
      }
      for (int i = 0; i < ch.k; i += rb)
        out.jobs.push_back(static_cast<int>(out.tops.size()) << 8 | i << 3 |
                           (std::min(rb, ch.k - i) - 1));
      out.tops.push_back(t);
    }
    out.job_ptr.push_back(static_cast<int>(out.jobs.size()));
  }
  // the largest subtrees first (they are taken from a counter)
  std::stable_sort(sub_roots.begin(), sub_roots.end(),
                   [&](int a, int b) { return pieces[a] + 4 * rows[a] > pieces[b] + 4 * rows[b]; });
  std::vector<int> local(n, -1);
  for (int c : sub_roots) {
    const HierChunk& root = out.chunks[c];
    HierPlan::Sub s = {};
    s.ext = static_cast<int>(out.sub_ext.size());
    s.num_ext = root.r;
    s.row = static_cast<int>(out.sub_rows.size());
    s.piece = static_cast<int>(out.sub_slot.size());
    for (int i = 0; i < root.r; ++i) {
      local[out.idx[root.ioff + i]] = i;
      out.sub_ext.push_back(top_row[out.idx[root.ioff + i]]);
    }
    for (int j = root.first + root.k - 1; j >= root.fd; --j) {
      if (!out.active[j]) continue;
      const HierChunk& ch = out.chunks[out.chunk_of[j]];
      HierPlan::SubRow r = {};
      r.piece = static_cast<int>(out.sub_slot.size()) - s.piece;
      r.num_pieces = ch.r4 / 4;
      r.slot = ch.coff + (j - ch.first);
      r.fd = ch.fd;
      r.last = ch.first + ch.k - 1;
      r.dest = dest_of[j];
      local[j] = root.r + s.num_rows;
      for (int b = 0; b < ch.r4; b += 4) {
        out.sub_slot.push_back(ch.woff + (j - ch.first) * ch.ld + b + plane(ch));
        unsigned ids = 0;
        for (int q = 0; q < 4; ++q)
          ids |= static_cast<unsigned>(b + q < ch.r ? local[out.idx[ch.ioff + b + q]] : 0) << (8 * q);
        out.sub_ids.push_back(ids);
      }
      out.sub_rows.push_back(r);
      ++s.num_rows;
    }
    s.num_pieces = static_cast<int>(out.sub_slot.size()) - s.piece;
    out.subs.push_back(s);
  }
  return true;
}

}  // namespace tapgpu
