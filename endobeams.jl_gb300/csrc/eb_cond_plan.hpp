// Symbolic part of the preconditioner (host only, no CUDA): which nodes of a
// simulation are eliminated before the inverse or band LU of the others, in which order, and the block
// lists that the numeric kernels and the solves walk.
//
// A beam structure is mostly wire: the interior nodes of a wire segment have
// two neighbours.  Eliminating such a node from the 6x6-block tangent couples
// its two neighbours and nothing else, so whole segments condense onto their
// crossings at next to no fill.  The plan eliminates independent sets (levels)
// of nodes: first all nodes of degree <= 2, level after level (a segment of
// q nodes takes about log2 q levels), then, while it pays, independent sets
// of nodes of degree <= 4 and upwards.  Every level is data-parallel; the
// remaining nodes, a much smaller graph, go to the explicit inverse
// (eb_dense.cuh) or, where they are many, to the band LU in reverse
// Cuthill-McKee order.  A 48-wire stent of 8,664 nodes keeps about 250 nodes,
// and N b² (the band LU's work) falls by two orders of magnitude.
//
// When another level pays (cond_cost, in us of one application): a level costs 5 us, 3 in small systems (about 2.5 in
// each sweep: a barrier of the team and its instructions' latency) and its blocks' bytes (with 2 us
// a 33 x 33 net took 2.10 ms a step, with 5 us 1.94, a 48 x 200 stent 11.4 and 10.8; from 6 us on a
// stent that refactorises twice a step loses 4% to the larger inverse); the explicit inverse reads 4 N² bytes at about 1 TB/s and its 2 N³ operations at 20 TFLOP/s are
// spread over some 30 applications; the band sweeps walk 2 N/32 blocks one after the other on one
// SM, a step taking about 0.9 us + 3.5 ns per DOF of half bandwidth where two blocks fit in shared
// memory, else 6 us + 6 ns (42 x 42 net, b = 593: 3.0 and 10 us); the band LU's N/32 panels, again on
// one SM, take 20 us + 0.3 b + 0.00046 b² each (75 us at b = 125, 337 at 593, 638 at 875), also
// spread over 30 applications.
//
// Towards the inverse the levels are not priced one by one, because only the last one brings it
// within reach.  Where it stays out of reach, a second plan is made for the band alone, every
// level priced, and the cheaper of the two is taken: 50 x 50 net, kept 4,530 at b = 875 by the first
// plan, 49 ms a step; 7,788 at b = 311 by the second, 12.7 (the band of the whole net: 26).
#pragma once
#include <algorithm>
#include <cstdint>
#include <cstdlib>
#include <numeric>
#include <vector>

namespace eb {

// Reverse Cuthill-McKee order of one simulation's node graph (neighbours in
// increasing degree, root a pseudo-peripheral node of each component).
// adj holds local neighbour lists (self excluded).  Returns the half
// bandwidth in nodes of the permuted graph; pos[i] is node i's position.
inline int rcm_order(const std::vector<std::vector<int>>& adj, std::vector<int>& pos) {
  const int n = (int)adj.size();
  std::vector<int> order;
  order.reserve(n);
  std::vector<char> seen(n, 0);
  std::vector<int> level(n, -1), queue;
  auto bfs = [&](int root, std::vector<int>& visited) {
    visited.clear();
    visited.push_back(root);
    level[root] = 0;
    int last = 0;
    for (size_t h = 0; h < visited.size(); ++h) {
      int v = visited[h];
      for (int w : adj[v])
        if (level[w] < 0) {
          level[w] = level[v] + 1;
          last = std::max(last, level[w]);
          visited.push_back(w);
        }
    }
    return last;
  };
  std::vector<int> comp;
  for (int start = 0; start < n; ++start) {
    if (seen[start]) continue;
    int root = start;
    // pseudo-peripheral root (George-Liu iteration)
    // (levels hold the BFS from `root` at the top of every iteration)
    int ecc = bfs(root, comp);
    for (int it = 0; it < 8; ++it) {
      int best = -1;
      for (int v : comp)
        if (level[v] == ecc && (best < 0 || adj[v].size() < adj[best].size())) best = v;
      for (int v : comp) level[v] = -1;
      int e2 = bfs(best, comp);
      if (e2 <= ecc) break;
      ecc = e2;
      root = best;
    }
    for (int v : comp) level[v] = -1;
    // Cuthill-McKee from root
    queue.clear();
    queue.push_back(root);
    seen[root] = 1;
    for (size_t h = 0; h < queue.size(); ++h) {
      int v = queue[h];
      order.push_back(v);
      std::vector<int> nb;
      for (int w : adj[v])
        if (!seen[w]) nb.push_back(w);
      std::sort(nb.begin(), nb.end(), [&](int x, int y) {
        return adj[x].size() != adj[y].size() ? adj[x].size() < adj[y].size() : x < y;
      });
      for (int w : nb) {
        seen[w] = 1;
        queue.push_back(w);
      }
    }
  }
  std::reverse(order.begin(), order.end());
  pos.assign(n, 0);
  for (int k = 0; k < n; ++k) pos[order[k]] = k;
  int bw = 0;
  for (int v = 0; v < n; ++v)
    for (int w : adj[v]) bw = std::max(bw, std::abs(pos[v] - pos[w]));
  return bw;
}

// Plan of one simulation.  Nodes are renumbered by position: eliminated nodes level by
// level, then the kept nodes in band order.  Blocks (6x6) are numbered so that every list a
// solve walks is contiguous: for each eliminated position its diagonal block and its row's
// blocks towards later positions (W), then for each position the blocks of its row towards
// earlier, eliminated positions (L), then the blocks among the kept nodes.
struct CondPlan {
  int n = 0, ne = 0, w = 0;            // nodes, eliminated nodes, half bandwidth (nodes) of the kept graph
  std::vector<int> pos;                // node -> position
  std::vector<int> lev_ptr;            // positions of level l: [lev_ptr[l], lev_ptr[l+1])
  std::vector<int> wptr;               // ne + 1: blocks [wptr[p], wptr[p+1]) = diagonal, W of position p
  std::vector<int> lptr;               // n + 1: L blocks of position p
  std::vector<int> srow, scol;         // per block: positions of its row and column
  int red0 = 0, n_blocks = 0;          // first block among the kept nodes, number of blocks
  // per level: target blocks (increasing), and for each the (L, W) block pairs of the level's nodes
  // whose products are added to it, in elimination order
  std::vector<std::vector<int>> tgt, tptr, cl, cw;

  // block of (row position r, column position c), -1 if outside the pattern
  int find(int r, int c) const {
    int lo, hi;
    if (r < ne && c >= r) { lo = wptr[r]; hi = wptr[r + 1]; }
    else if (c < ne) { lo = lptr[r]; hi = lptr[r + 1]; }
    else { lo = rptr[r - ne]; hi = rptr[r - ne + 1]; }
    auto it = std::lower_bound(scol.begin() + lo, scol.begin() + hi, c);
    return it != scol.begin() + hi && *it == c ? (int)(it - scol.begin()) : -1;
  }
  std::vector<int> rptr;               // kept rows: blocks among the kept nodes
  double cost = 0;                     // us of one application, with its share of the factorisation
};

constexpr int kWholeDofs = 200;  // at most this many DOFs: nothing is eliminated

// us of one application that a level costs.  A small system's team is at most four CTAs, whose barriers
// are cheaper (12 x 12 net, one level instead of none: a step 1.12 -> 1.05 ms, and as 1,024 of them 42.0 -> 36.4; with 3
// us for every size a 33 x 33 net's step 1.84 -> 1.86).
inline double level_cost(int nodes) { return 6 * nodes <= 2048 ? 3.0 : 5.0; }

// The cheaper of the two (past max_dense the explicit inverse is still what the next levels aim
// at); w < 0: the inverse.  stage_b: the widest half bandwidth whose blocks fit in shared memory.
inline double cond_cost(int nodes, int w, int max_dense, int stage_b) {
  const double N = 6.0 * nodes, b = 6.0 * w + 5, step = b <= stage_b ? 0.9 + 0.0035 * b : 6.0 + 0.006 * b;
  const double band = N / 16 * step + N / 960 * (20 + 0.3 * b + 0.00046 * b * b);
  const double dense = 4e-6 * N * N + 2.0 * N * N * N / (20e6 * 30);
  return max_dense <= 0 ? band : w < 0 ? dense : std::min(band, dense);
}

// Symbolic elimination of one simulation's node graph (adj: sorted neighbour lists, self
// excluded).  At least one node is kept.  max_w: the widest band (nodes) the band LU takes;
// max_dense: the most DOFs of an explicit inverse.
inline void cond_plan_for(const std::vector<std::vector<int>>& adj0, int max_w, int max_dense, int stage_b, CondPlan& P) {
  const int n = (int)adj0.size();
  P = CondPlan();
  P.n = n;
  std::vector<std::vector<int>> adj(adj0), nb(n);
  std::vector<int> elim_level(n, -1), order;  // eliminated nodes in order
  std::vector<char> gone(n, 0), blocked(n, 0);
  std::vector<int> left(n);
  std::iota(left.begin(), left.end(), 0);
  P.lev_ptr.assign(1, 0);
  const double level = level_cost(n);

  // One level: a greedy independent set of the nodes of degree <= cap, lowest degree first.
  auto pick = [&](int cap) {
    std::vector<int> cand, set;
    for (int v : left)
      if ((int)adj[v].size() <= cap) cand.push_back(v);
    std::stable_sort(cand.begin(), cand.end(), [&](int a, int b) { return adj[a].size() < adj[b].size(); });
    for (int v : cand) {
      if (blocked[v]) continue;
      if (set.size() + 1 >= left.size()) break;  // one node stays
      set.push_back(v);
      for (int u : adj[v]) blocked[u] = 1;
    }
    for (int v : set)
      for (int u : adj[v]) blocked[u] = 0;
    return set;
  };
  std::vector<int> merged;
  auto eliminate = [&](std::vector<std::vector<int>>& g, int v) {
    const std::vector<int> N = g[v];
    for (int u : N) {
      merged.clear();
      std::set_union(g[u].begin(), g[u].end(), N.begin(), N.end(), std::back_inserter(merged));
      merged.erase(std::remove_if(merged.begin(), merged.end(), [&](int x) { return x == u || x == v; }), merged.end());
      g[u] = merged;
    }
  };
  // band (half bandwidth in nodes, positions) of the graph g over the nodes `ids`
  auto band = [&](const std::vector<std::vector<int>>& g, const std::vector<int>& ids, std::vector<int>& rpos) {
    std::vector<int> loc(n, -1);
    for (size_t k = 0; k < ids.size(); ++k) loc[ids[k]] = (int)k;
    std::vector<std::vector<int>> a(ids.size());
    for (size_t k = 0; k < ids.size(); ++k)
      for (int u : g[ids[k]]) a[k].push_back(loc[u]);
    return rcm_order(a, rpos);
  };
  auto commit = [&](std::vector<int>& set) {
    std::sort(set.begin(), set.end());
    P.cost += level;
    for (int v : set) {
      P.cost += 144e-6 * (1.0 + 2.0 * adj[v].size());
      nb[v] = adj[v];
      eliminate(adj, v);
      adj[v].clear();
      gone[v] = 1;
      order.push_back(v);
    }
    P.lev_ptr.push_back((int)order.size());
    left.erase(std::remove_if(left.begin(), left.end(), [&](int v) { return gone[v] != 0; }), left.end());
  };

  // Very small systems go to the explicit inverse as they are (cantilever of 20 nodes, ten steps: 19.1
  // ms with levels, 17.8 without; 31 nodes 18.2 and 17.1; 45 nodes 18.4 and 18.8; a 64-node ring's
  // step 0.94 and 0.98).
  const bool whole = 6 * n <= kWholeDofs && 6 * n <= max_dense;
  // wire segments: degree <= 2, while a level removes at least 5% of the nodes
  while (left.size() > 1 && !whole) {
    std::vector<int> set = pick(2);
    if (set.empty() || set.size() * 20 < left.size()) break;
    commit(set);
  }
  // half bandwidths only where the explicit inverse does not cost less than the band sweeps of
  // any bandwidth (w < 0: not needed)
  auto needs_band = [&](int nodes) {
    return max_dense <= 0 || cond_cost(nodes, 0, max_dense, stage_b) < cond_cost(nodes, n, max_dense, stage_b);
  };
  std::vector<int> rpos;
  int w = needs_band((int)left.size()) ? band(adj, left, rpos) : -1;
  for (int cap : {4, 8, 12, 16, 24, 32}) {
    while (left.size() > 1 && !whole) {
      std::vector<int> set = pick(cap);
      if (set.empty() || set.size() * 20 < left.size()) break;
      double blocks = 0;
      for (int v : set) blocks += 1.0 + 2.0 * adj[v].size();
      const int m = (int)left.size(), m2 = m - (int)set.size();
      int w2 = -1;
      if (needs_band(m2)) {
        std::vector<std::vector<int>> g(adj);
        std::vector<char> out(n, 0);
        for (int v : set) out[v] = 1;
        std::vector<int> keep, rp;
        for (int v : left)
          if (!out[v]) keep.push_back(v);
        for (int v : set) eliminate(g, v);
        w2 = band(g, keep, rp);
        if (w2 > max_w && w <= max_w && 6 * m2 > max_dense) break;
      }
      // past max_dense there is no inverse yet: go on towards it
      if ((max_dense <= 0 || 6 * m <= max_dense) &&
          cond_cost(m2, w2, max_dense, stage_b) + level + 144e-6 * blocks > cond_cost(m, w, max_dense, stage_b))
        break;
      commit(set);
      w = w2;
    }
  }
  w = band(adj, left, rpos);
  P.w = w;
  P.ne = (int)order.size();
  P.cost += cond_cost((int)left.size(), w, 6 * (int)left.size() <= max_dense ? max_dense : 0, stage_b);

  // ---- positions and block numbers
  const int ne = P.ne;
  P.pos.assign(n, 0);
  for (int k = 0; k < ne; ++k) P.pos[order[k]] = k;
  for (size_t k = 0; k < left.size(); ++k) P.pos[left[k]] = ne + rpos[k];
  std::vector<int> node_at(n);
  for (int v = 0; v < n; ++v) node_at[P.pos[v]] = v;
  std::vector<std::vector<int>> lrow(n);  // per position: earlier eliminated neighbours
  P.wptr.assign(ne + 1, 0);
  auto put = [&](int r, int c) {
    P.srow.push_back(r);
    P.scol.push_back(c);
  };
  std::vector<int> q;
  for (int p = 0; p < ne; ++p) {
    q.clear();
    for (int u : nb[node_at[p]]) q.push_back(P.pos[u]);
    std::sort(q.begin(), q.end());
    put(p, p);
    for (int c : q) {
      put(p, c);
      lrow[c].push_back(p);
    }
    P.wptr[p + 1] = (int)P.scol.size();
  }
  P.lptr.assign(n + 1, 0);
  P.lptr[0] = (int)P.scol.size();
  for (int p = 0; p < n; ++p) {
    for (int c : lrow[p]) put(p, c);
    P.lptr[p + 1] = (int)P.scol.size();
  }
  P.red0 = (int)P.scol.size();
  P.rptr.assign(n - ne + 1, P.red0);
  for (int p = ne; p < n; ++p) {
    q.assign(1, p);
    for (int u : adj[node_at[p]]) q.push_back(P.pos[u]);
    std::sort(q.begin(), q.end());
    for (int c : q) put(p, c);
    P.rptr[p - ne + 1] = (int)P.scol.size();
  }
  P.n_blocks = (int)P.scol.size();

  // ---- update lists
  const int nlev = (int)P.lev_ptr.size() - 1;
  P.tgt.resize(nlev);
  P.tptr.resize(nlev);
  P.cl.resize(nlev);
  P.cw.resize(nlev);
  std::vector<int> ut, cnt(P.n_blocks + 1, 0), touched;
  for (int l = 0; l < nlev; ++l) {
    ut.clear();
    touched.clear();
    for (int p = P.lev_ptr[l]; p < P.lev_ptr[l + 1]; ++p)
      for (int a = P.wptr[p] + 1; a < P.wptr[p + 1]; ++a)
        for (int b = P.wptr[p] + 1; b < P.wptr[p + 1]; ++b) {
          const int t = P.find(P.scol[a], P.scol[b]);
          if (cnt[t]++ == 0) touched.push_back(t);
          ut.push_back(t);
        }
    std::sort(touched.begin(), touched.end());
    P.tgt[l] = touched;
    P.tptr[l].assign(1, 0);
    for (int t : touched) {
      P.tptr[l].push_back(P.tptr[l].back() + cnt[t]);
      cnt[t] = P.tptr[l][P.tptr[l].size() - 2];  // next free entry of the target
    }
    P.cl[l].resize(ut.size());
    P.cw[l].resize(ut.size());
    size_t u = 0;
    for (int p = P.lev_ptr[l]; p < P.lev_ptr[l + 1]; ++p)
      for (int a = P.wptr[p] + 1; a < P.wptr[p + 1]; ++a) {
        const int left_block = P.find(P.scol[a], p);
        for (int b = P.wptr[p] + 1; b < P.wptr[p + 1]; ++b) {
          const int k = cnt[ut[u++]]++;
          P.cl[l][k] = left_block;
          P.cw[l][k] = b;
        }
      }
    for (int t : touched) cnt[t] = 0;
  }
}

// The plan of one simulation (arguments as above).
inline void cond_plan(const std::vector<std::vector<int>>& adj, int max_w, int max_dense, CondPlan& P, int stage_b = 1 << 30) {
  cond_plan_for(adj, max_w, max_dense, stage_b, P);
  if (max_dense <= 0 || 6 * (P.n - P.ne) <= max_dense) return;
  CondPlan B;
  cond_plan_for(adj, max_w, 0, stage_b, B);
  if (B.w <= max_w && (P.w > max_w || B.cost < P.cost)) P = std::move(B);
}

}  // namespace eb
