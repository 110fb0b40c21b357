// Tiled pipeline schedule of a sparse triangular sweep: chains, tiles, steps,
// shared-memory ring codes and cross-tile waits (see fc_schedule.hpp).
#include "fc_schedule.hpp"

#include <algorithm>
#include <atomic>
#include <cmath>
#include <deque>
#include <limits>
#include <mutex>
#include <numeric>
#include <set>
#include <system_error>
#include <thread>
#include <utility>

namespace {

struct Deps {
  const int *ia, *ja, *dg;
  bool fwd;
  int begin(int i) const { return fwd ? ia[i] : dg[i] + 1; }
  int end(int i) const { return fwd ? dg[i] : ia[i + 1]; }
};

}  // namespace

// Rows from which the choice of the tiles uses threads: one takes 30 us to
// start, as long as a trial on 3,000 rows (1,386 rows on 16 Arm cores: 0.6 ms
// more with threads).
#define FC_THREADS_ROWS 8192

// body(i) for i in [0, count) on up to `most` and hardware_concurrency threads,
// this one among them; on fewer where no more can be started
template <class F>
static void parallel_items(int count, int most, F body) {
  std::atomic<int> next{0};
  auto work = [&]() {
    for (int i = next++; i < count; i = next++) body(i);
  };
  std::vector<std::thread> th;
  const int nt = std::min(std::min(count, most), (int)std::thread::hardware_concurrency());
  try {
    for (int k = 1; k < nt; ++k) th.emplace_back(work);
  } catch (const std::system_error&) {
  }
  work();
  for (std::thread& t : th) t.join();
}

// Slabs along the axes for T nearly cubic cells.  ext: extents of the chain
// centroids; an axis along which they hardly spread (the direction of the grid
// lines) and axis nocut (>= 0) are not cut.  Returns the axes that are.
static int cut_counts(int T, const double (&ext)[3], int nocut, int (&slabs)[3]) {
  const double emax = std::max(ext[0], std::max(ext[1], ext[2]));
  int axes[3], dims = 0;
  double vol = 1.0;
  for (int a = 0; a < 3; ++a) {
    slabs[a] = 1;
    if (a == nocut || !(ext[a] > 0.05 * emax)) continue;
    vol *= ext[a];
    axes[dims++] = a;
  }
  // the longest axes first; the last one takes what is left of T
  std::stable_sort(axes, axes + dims, [&](int p, int q) { return ext[p] > ext[q]; });
  int left = T, used = 0;
  for (int l = 0; l < dims; ++l) {
    const double side = std::pow(vol / left, 1.0 / (dims - l));  // of a cubic cell of what is left
    const int want = l + 1 == dims ? left : (int)std::lround(ext[axes[l]] / side);
    slabs[axes[l]] = std::max(1, std::min(left, want));
    left = (left + slabs[axes[l]] - 1) / slabs[axes[l]];
    vol /= ext[axes[l]];
    used += slabs[axes[l]] > 1;
  }
  return used;
}

// Cuts items (chains) weighted by rows into T parts: slabs along axis ax[0],
// each of them along ax[1], each of those along ax[2].  The parts are shared
// out evenly over the slabs, whose weights follow.  A cut goes to the
// position nearest to the balanced one, within half a slab, where the gap in
// the coordinate is at least half the widest gap there, so that grid lines
// sharing a coordinate stay on one side.  Slabs of a structured mesh with as
// many parts are then cut at the same places: a dependency passes through as
// few tiles one after the other as the counts allow, and the tiles have the
// same number of lines to within one in each direction (bisecting the chains
// over and over left tiles of 6,400 to 25,088 rows at 128^3, 37 of them one
// after the other, where this leaves 12,288 to 14,976 rows and 23 tiles).
// With `threads` the slabs of the first axis are cut concurrently (they write
// disjoint entries of part_of).
static void axis_cuts(std::vector<int>& items, const std::vector<double>* const (&c)[3], const std::vector<int>& w,
                      const int (&ax)[3], const int (&slabs)[3], int level, int T, int first_part,
                      std::vector<int>& part_of, bool threads) {
  while (level < 3 && slabs[ax[level]] == 1) ++level;
  if (level == 3 || T == 1) {
    for (int i : items) part_of[i] = first_part;
    return;
  }
  bool last = true;
  for (int l = level + 1; l < 3; ++l) last = last && slabs[ax[l]] == 1;
  const int np = last ? T : std::min(T, slabs[ax[level]]);
  const std::vector<double>& key = *c[ax[level]];
  std::vector<std::pair<double, int>> kv(items.size());
  for (size_t q = 0; q < items.size(); ++q) kv[q] = {key[items[q]], items[q]};
  std::stable_sort(kv.begin(), kv.end(),
                   [](const std::pair<double, int>& a, const std::pair<double, int>& b) { return a.first < b.first; });
  std::vector<long long> before(kv.size() + 1, 0);  // weight of the first q items
  for (size_t q = 0; q < kv.size(); ++q) before[q + 1] = before[q] + w[kv[q].second];
  const long long tot = before.back();
  auto parts_before = [&](int s) { return (int)((long long)T * s / np); };  // parts of the first s slabs
  std::vector<size_t> cut(np + 1, 0);
  cut[np] = kv.size();
  for (int s = 1; s < np; ++s) {
    const long long want = tot * parts_before(s) / T, tol = std::max<long long>(1, tot / np / 2);
    auto at = [&](long long x) { return (size_t)(std::lower_bound(before.begin(), before.end(), x) - before.begin()); };
    const size_t lo = std::max(at(want - tol), cut[s - 1]), hi = std::min(at(want + tol), kv.size());
    double widest = 0.0;
    for (size_t q = std::max<size_t>(1, lo); q < hi; ++q) widest = std::max(widest, kv[q].first - kv[q - 1].first);
    size_t best = std::max(at(want), cut[s - 1]);
    long long best_dist = -1;
    for (size_t q = std::max<size_t>(1, lo); q < hi; ++q) {
      if (kv[q].first - kv[q - 1].first < 0.5 * widest) continue;
      const long long dist = before[q] > want ? before[q] - want : want - before[q];
      if (best_dist < 0 || dist < best_dist) { best_dist = dist; best = q; }
    }
    cut[s] = best;
  }
  std::vector<std::vector<int>> slab(np);
  for (int s = 0; s < np; ++s)
    for (size_t q = cut[s]; q < cut[s + 1]; ++q) slab[s].push_back(kv[q].second);
  kv.clear();
  kv.shrink_to_fit();
  auto run = [&](int s) {
    const int p0 = parts_before(s);
    axis_cuts(slab[s], c, w, ax, slabs, level + 1, parts_before(s + 1) - p0, first_part + p0, part_of, false);
  };
  if (threads && !last && items.size() > 4096) {
    parallel_items(np, np, run);
  } else {
    for (int s = 0; s < np; ++s) run(s);
  }
}

// runs body(lo, hi) over [0, n) in contiguous chunks on up to
// hardware_concurrency threads
template <class F>
static void parallel_chunks(int n, F body) {
  const int nt = std::max(1, std::min<int>((int)std::thread::hardware_concurrency(), std::max(1, n / 4)));
  if (nt <= 1) {
    body(0, n);
    return;
  }
  std::vector<std::thread> th;
  for (int k = 0; k < nt; ++k) {
    const int lo = (int)((long long)n * k / nt), hi = (int)((long long)n * (k + 1) / nt);
    th.emplace_back([&body, lo, hi]() { body(lo, hi); });
  }
  for (std::thread& t : th) t.join();
}

namespace {

// The dependency chains of a system, what its tiles are made of; the same for
// every tile count.
struct Chains {
  int n, count = 0;
  Deps D;
  std::vector<int> of;       // chain of each row
  std::vector<int> rows;     // rows per chain
  std::vector<double> cen[3];  // centroids and their extents (with coordinates)
  double ext[3] = {0.0, 0.0, 0.0};
  // undirected adjacency of the chains through dependencies, built only where
  // tiles are grown or merged over it: cuts along the axes give at most the
  // target count by themselves
  std::once_flag graph_once;
  std::vector<int> adj_ptr, adj;

  // a row continues the chain of its latest dependency
  Chains(int n_, const Deps& D_, const std::vector<int>& lev, const double* xyz) : n(n_), D(D_), of(n_, -1) {
    std::vector<char> has_succ(n, 0);
    for (int t = 0; t < n; ++t) {
      const int i = D.fwd ? t : n - 1 - t;
      int best = -1;
      for (int k = D.begin(i); k < D.end(i); ++k) {
        const int j = D.ja[k];
        if (has_succ[j]) continue;
        if (best < 0 || lev[j] > lev[best] || (lev[j] == lev[best] && (D.fwd ? j > best : j < best))) best = j;
      }
      if (best >= 0) {
        has_succ[best] = 1;
        of[i] = of[best];
        rows[of[i]]++;
      } else {
        of[i] = count++;
        rows.push_back(1);
      }
    }
    if (!xyz) return;
    for (int a = 0; a < 3; ++a) {
      cen[a].assign(count, 0.0);
      for (int i = 0; i < n; ++i) cen[a][of[i]] += xyz[(size_t)a * n + i];
      for (int c = 0; c < count; ++c) cen[a][c] /= rows[c];
      const auto mm = std::minmax_element(cen[a].begin(), cen[a].end());
      ext[a] = *mm.second - *mm.first;
    }
  }

  void graph() {
    std::call_once(graph_once, [&]() {
      std::vector<std::pair<int, int>> edges;
      edges.reserve((size_t)n * 2);
      for (int i = 0; i < n; ++i)
        for (int k = D.begin(i); k < D.end(i); ++k) {
          const int a = of[i], b = of[D.ja[k]];
          if (a != b) { edges.push_back({a, b}); edges.push_back({b, a}); }
        }
      std::sort(edges.begin(), edges.end());
      edges.erase(std::unique(edges.begin(), edges.end()), edges.end());
      adj_ptr.assign(count + 1, 0);
      for (auto& e : edges) adj_ptr[e.first + 1]++;
      for (int c = 0; c < count; ++c) adj_ptr[c + 1] += adj_ptr[c];
      adj.resize(edges.size());
      for (size_t q = 0; q < edges.size(); ++q) adj[q] = edges[q].second;  // sorted by (first, second)
    });
  }
};

// Tiles of the chains: cuts along the axes, or regions grown over the chain
// graph in breadth-first order.  Returns their count (0: stopped, see
// FC_CUT_UNLESS_3) and the axes that were cut.
int tiles_of_chains(Chains& G, int ntiles_target, int nocut, bool threads, std::vector<int>& tile_of_chain,
                    int& cut_axes) {
  cut_axes = 0;
  const int n = G.n, nch = G.count, T = std::max(1, std::min(ntiles_target, nch));
  const long long target = (n + T - 1) / T;
  tile_of_chain.assign(nch, -1);
  std::vector<long long> tile_rows;
  // chains that lie in one point (or nowhere) cannot be told apart by
  // coordinates: their tiles are grown as well
  bool cut = false;
  if (!G.cen[0].empty()) {
    int slabs[3];
    cut_axes = cut_counts(T, G.ext, nocut, slabs);
    if (nocut == FC_CUT_UNLESS_3 && cut_axes == 3) return 0;
    cut = cut_axes > 0 || T == 1;
    if (cut) {
      int ax[3] = {0, 1, 2};  // the longest axes first
      std::stable_sort(ax, ax + 3, [&](int p, int q) { return G.ext[p] > G.ext[q]; });
      std::vector<int> items(nch);
      std::iota(items.begin(), items.end(), 0);
      const std::vector<double>* const cen[3] = {&G.cen[0], &G.cen[1], &G.cen[2]};
      axis_cuts(items, cen, G.rows, ax, slabs, 0, T, 0, tile_of_chain, threads);
      // drop empty parts
      std::vector<int> used(T, 0);
      for (int c = 0; c < nch; ++c) used[tile_of_chain[c]] = 1;
      std::vector<int> nid(T, -1);
      int m = 0;
      for (int t = 0; t < T; ++t)
        if (used[t]) nid[t] = m++;
      for (int c = 0; c < nch; ++c) tile_of_chain[c] = nid[tile_of_chain[c]];
      tile_rows.assign(m, 0);
      for (int c = 0; c < nch; ++c) tile_rows[tile_of_chain[c]] += G.rows[c];
    }
  }
  if (!cut) {
    G.graph();
    std::deque<int> q;
    int next_seed = 0;
    while (true) {
      while (next_seed < nch && tile_of_chain[next_seed] >= 0) ++next_seed;
      if (next_seed >= nch) break;
      const int t = (int)tile_rows.size();
      tile_rows.push_back(0);
      q.clear();
      q.push_back(next_seed);
      tile_of_chain[next_seed] = t;
      while (!q.empty() && tile_rows[t] < target) {
        const int c = q.front();
        q.pop_front();
        if (tile_of_chain[c] != t) continue;
        tile_rows[t] += G.rows[c];
        for (int e = G.adj_ptr[c]; e < G.adj_ptr[c + 1] && tile_rows[t] < target; ++e) {
          const int d = G.adj[e];
          if (tile_of_chain[d] < 0) { tile_of_chain[d] = t; q.push_back(d); }
        }
      }
      // chains queued but not consumed go back to the pool
      for (int c : q)
        if (tile_of_chain[c] == t) tile_of_chain[c] = -1;
    }
  }
  // every chain now has a tile; merge the smallest tiles until at most T remain
  int ntiles = (int)tile_rows.size();
  if (ntiles > T) {
    G.graph();
    std::vector<int> remap(ntiles);
    std::iota(remap.begin(), remap.end(), 0);
    auto find = [&](int x) { while (remap[x] != x) x = remap[x] = remap[remap[x]]; return x; };
    // tile adjacency through chain edges
    std::vector<std::pair<int, int>> tedges;
    for (int c = 0; c < nch; ++c)
      for (int e = G.adj_ptr[c]; e < G.adj_ptr[c + 1]; ++e) {
        int a = tile_of_chain[c], b = tile_of_chain[G.adj[e]];
        if (a != b) tedges.push_back({a, b});
      }
    std::sort(tedges.begin(), tedges.end());
    tedges.erase(std::unique(tedges.begin(), tedges.end()), tedges.end());
    int alive = ntiles;
    while (alive > T) {
      int small = -1;
      for (int t = 0; t < ntiles; ++t)
        if (find(t) == t && (small < 0 || tile_rows[t] < tile_rows[small])) small = t;
      int best = -1;
      for (auto& e : tedges) {
        if (find(e.first) != small) continue;
        int o = find(e.second);
        if (o != small && (best < 0 || tile_rows[o] < tile_rows[best])) best = o;
      }
      if (best < 0)  // isolated: merge into the smallest other tile
        for (int t = 0; t < ntiles; ++t)
          if (find(t) == t && t != small && (best < 0 || tile_rows[t] < tile_rows[best])) best = t;
      remap[small] = best;
      tile_rows[best] += tile_rows[small];
      --alive;
    }
    std::vector<int> newid(ntiles, -1);
    int m = 0;
    for (int t = 0; t < ntiles; ++t)
      if (find(t) == t) newid[t] = m++;
    for (int c = 0; c < nch; ++c) tile_of_chain[c] = newid[find(tile_of_chain[c])];
    ntiles = m;
  }
  return ntiles;
}

}  // namespace

void build_sweep_schedule(int n, const int* ia, const int* ja, const int* dg, const std::vector<int>& lev, int nlev,
                          bool forward, int ntiles_target, const double* xyz, SweepSchedule& S,
                          std::vector<int>& code, bool with_waits, int nocut) {
  S = SweepSchedule();
  S.n = n;
  S.nlev = nlev;
  const Deps D{ia, ja, dg, forward};
  // ---- chains, tiles
  Chains G(n, D, lev, xyz);
  std::vector<int> tile_of_chain;
  const int ntiles = tiles_of_chains(G, ntiles_target, nocut, true, tile_of_chain, S.cut_axes);
  if (ntiles == 0 && n > 0) return;
  const int nch = G.count;
  const std::vector<int>& chain_of = G.of;
  S.ntiles = ntiles;
  // ---- per tile: steps (distinct levels) and slots (chains sharing a slot
  //         when their level ranges do not overlap)
  std::vector<int> chain_lo(nch, 1 << 30), chain_hi(nch, -1);
  for (int i = 0; i < n; ++i) {
    const int c = chain_of[i];
    chain_lo[c] = std::min(chain_lo[c], lev[i]);
    chain_hi[c] = std::max(chain_hi[c], lev[i]);
  }
  std::vector<std::vector<int>> tile_chains(ntiles);
  for (int c = 0; c < nch; ++c) tile_chains[tile_of_chain[c]].push_back(c);
  std::vector<int> slot_of_chain(nch, 0);
  std::vector<int> row_tile(n), row_step(n), row_slot(n);
  // slots, tile by tile (concurrently): the chains in order of their first
  // level each take the free slot (its last chain ended before that level)
  // that was freed last, the lowest such slot on ties, else a new slot; the
  // free slots are kept ordered by (level after which free, -slot)
  S.tile_slots.assign(ntiles, 1);
  parallel_chunks(ntiles, [&](int t0, int t1) {
    for (int t = t0; t < t1; ++t) {
      auto& ch = tile_chains[t];
      std::sort(ch.begin(), ch.end(), [&](int a, int b) {
        return chain_lo[a] != chain_lo[b] ? chain_lo[a] < chain_lo[b] : a < b;
      });
      std::set<std::pair<int, int>> slot_free;
      int nslots = 0;
      for (int c : ch) {
        auto it = slot_free.lower_bound({chain_lo[c], std::numeric_limits<int>::min()});
        int sl;
        if (it != slot_free.begin()) {
          --it;
          sl = -it->second;
          slot_free.erase(it);
        } else {
          sl = nslots++;
        }
        slot_free.insert({chain_hi[c], -sl});
        slot_of_chain[c] = sl;
      }
      S.tile_slots[t] = std::max(1, nslots);
    }
  });
  for (int t = 0; t < ntiles; ++t) S.max_slots = std::max(S.max_slots, S.tile_slots[t]);
  // the distinct levels of every tile, ascending: marked in a (tile, level)
  // table that then maps a row's level to its step, or sorted per tile when
  // that table would be large
  std::vector<std::vector<int>> tile_levels(ntiles);
  const size_t tab_cells = (size_t)ntiles * (size_t)std::max(1, nlev);
  std::vector<int> step_tab;
  if (tab_cells <= ((size_t)1 << 24)) {
    step_tab.assign(tab_cells, -1);
    for (int i = 0; i < n; ++i) step_tab[(size_t)tile_of_chain[chain_of[i]] * nlev + lev[i]] = -2;
    for (int t = 0; t < ntiles; ++t) {
      int* tab = step_tab.data() + (size_t)t * nlev;
      for (int l = 0; l < nlev; ++l)
        if (tab[l] == -2) {
          tab[l] = (int)tile_levels[t].size();
          tile_levels[t].push_back(l);
        }
    }
  } else {
    for (int i = 0; i < n; ++i) tile_levels[tile_of_chain[chain_of[i]]].push_back(lev[i]);
    for (int t = 0; t < ntiles; ++t) {
      auto& L = tile_levels[t];
      std::sort(L.begin(), L.end());
      L.erase(std::unique(L.begin(), L.end()), L.end());
    }
  }
  S.R = std::max(1, std::min(4, (int)((160 * 1024) / (8LL * std::max(1, S.max_slots)))));
  S.tile_step_ptr.assign(ntiles + 1, 0);
  for (int t = 0; t < ntiles; ++t) S.tile_step_ptr[t + 1] = S.tile_step_ptr[t] + (int)tile_levels[t].size();
  const int nsteps = S.tile_step_ptr[ntiles];
  S.step_level.resize(nsteps);
  S.step_row_ptr.assign(nsteps + 1, 0);
  for (int t = 0; t < ntiles; ++t)
    for (size_t s = 0; s < tile_levels[t].size(); ++s) {
      const int gs = S.tile_step_ptr[t] + (int)s;
      S.step_level[gs] = tile_levels[t][s];
      S.step_row_ptr[gs + 1] = S.step_row_ptr[gs] + S.tile_slots[t];
    }
  S.rows.assign(S.step_row_ptr[nsteps], -1);
  // place every row (its tile's level -> step from the table, else by binary search)
  for (int i = 0; i < n; ++i) {
    const int t = tile_of_chain[chain_of[i]];
    int s;
    if (!step_tab.empty()) {
      s = step_tab[(size_t)t * nlev + lev[i]];
    } else {
      const auto& L = tile_levels[t];
      s = (int)(std::lower_bound(L.begin(), L.end(), lev[i]) - L.begin());
    }
    const int slot = slot_of_chain[chain_of[i]];
    row_tile[i] = t;
    row_step[i] = s;
    row_slot[i] = slot;
    S.rows[S.step_row_ptr[S.tile_step_ptr[t] + s] + slot] = i;
  }
  if (!with_waits) return;
  // ---- entry codes and waits
  std::vector<std::vector<std::pair<int, int>>> waits(nsteps);
  for (int i = 0; i < n; ++i) {
    const int t = row_tile[i], s = row_step[i];
    const int gs = S.tile_step_ptr[t] + s;
    for (int k = D.begin(i); k < D.end(i); ++k) {
      const int j = ja[k];
      if (row_tile[j] == t && s - row_step[j] < S.R) {
        code[k] = (row_step[j] % S.R) * S.tile_slots[t] + row_slot[j];
        S.ring_entries++;
      } else {
        code[k] = -j - 2;
        if (row_tile[j] != t) {
          waits[gs].push_back({row_tile[j], lev[j] + 1});
          S.cross_tile_entries++;
        } else {
          S.global_same_tile_entries++;
        }
      }
    }
  }
  S.wait_ptr.assign(nsteps + 1, 0);
  for (int gs = 0; gs < nsteps; ++gs) {
    auto& w = waits[gs];
    std::sort(w.begin(), w.end());
    // keep the largest requirement per producer tile
    std::vector<std::pair<int, int>> m;
    for (auto& p : w) {
      if (!m.empty() && m.back().first == p.first) m.back().second = std::max(m.back().second, p.second);
      else m.push_back(p);
    }
    for (auto& p : m) { S.wait_tile.push_back(p.first); S.wait_level.push_back(p.second); }
    S.wait_ptr[gs + 1] = (int)S.wait_tile.size();
  }
}

// Critical-path estimate of a sweep: every level of a tile costs tau0 per
// FC_STEP_ROWS rows begun and per_row * rows; it starts when the tile's
// previous level is done and, for each producer it waits on, hop microseconds
// after the producer published the needed progress.  Returns microseconds.
double estimate_sweep_us(const SweepSchedule& S, double tau0, double per_row, double hop) {
  std::vector<std::vector<double>> pub(S.ntiles);
  std::vector<int> cur(S.ntiles, 0);
  // steps of all tiles in level order (a valid processing order)
  std::vector<std::pair<int, int>> order;  // (level, global step)
  for (int t = 0; t < S.ntiles; ++t)
    for (int gs = S.tile_step_ptr[t]; gs < S.tile_step_ptr[t + 1]; ++gs) order.push_back({S.step_level[gs], gs});
  std::sort(order.begin(), order.end());
  std::vector<int> tile_of_step(S.step_level.size());
  for (int t = 0; t < S.ntiles; ++t)
    for (int gs = S.tile_step_ptr[t]; gs < S.tile_step_ptr[t + 1]; ++gs) tile_of_step[gs] = t;
  double tmax = 0.0;
  for (auto& o : order) {
    const int gs = o.second, t = tile_of_step[gs];
    double st = pub[t].empty() ? 0.0 : pub[t].back();
    for (int w = S.wait_ptr[gs]; w < S.wait_ptr[gs + 1]; ++w) {
      const int q = S.wait_tile[w], need = S.wait_level[w];
      const int q0 = S.tile_step_ptr[q];
      // first published step of q whose next level reaches need
      int lo = 0, hi = (int)pub[q].size() - 1, found = -1;
      while (lo <= hi) {
        const int mid = (lo + hi) / 2;
        const int nxt = (q0 + mid + 1 < S.tile_step_ptr[q + 1]) ? S.step_level[q0 + mid + 1] : S.nlev;
        if (nxt >= need) { found = mid; hi = mid - 1; } else lo = mid + 1;
      }
      if (found >= 0) st = std::max(st, pub[q][found] + hop);
    }
    int rowsn = 0;
    for (int sl = 0; sl < S.tile_slots[t]; ++sl) rowsn += S.rows[S.step_row_ptr[gs] + sl] >= 0;
    const double end = st + tau0 * ((rowsn + FC_STEP_ROWS - 1) / FC_STEP_ROWS) + per_row * rowsn;
    pub[t].push_back(end);
    tmax = std::max(tmax, end);
  }
  return tmax;
}

namespace {

// Rows renumbered by level, with their chains and dependencies: what an
// estimate reads then lies in a row, or in the levels just before.
struct LevelOrder {
  std::vector<int> level_ptr, chain, dep_ptr, dep;

  LevelOrder(const Chains& G, const std::vector<int>& lev, int nlev)
      : level_ptr(nlev + 1, 0), chain(G.n), dep_ptr(G.n + 1, 0) {
    const int n = G.n;
    for (int i = 0; i < n; ++i) level_ptr[lev[i] + 1]++;
    for (int l = 0; l < nlev; ++l) level_ptr[l + 1] += level_ptr[l];
    std::vector<int> row(n), pos(n), at(level_ptr.begin(), level_ptr.end() - 1);
    for (int i = 0; i < n; ++i) row[pos[i] = at[lev[i]]++] = i;
    for (int q = 0; q < n; ++q) dep_ptr[q + 1] = dep_ptr[q] + G.D.end(row[q]) - G.D.begin(row[q]);
    dep.resize(dep_ptr[n]);
    auto fill = [&](int lo, int hi) {
      for (int q = lo; q < hi; ++q) {
        const int i = row[q], k0 = G.D.begin(i);
        chain[q] = G.of[i];
        for (int e = dep_ptr[q]; e < dep_ptr[q + 1]; ++e) dep[e] = pos[G.D.ja[k0 + e - dep_ptr[q]]];
      }
    };
    if (n > FC_THREADS_ROWS) parallel_chunks(n, fill);
    else fill(0, n);
  }
};

// The same estimate (to the last bit) from the tiles alone, without a schedule:
// the rows of a level in a tile are one step of it, which waits for the steps
// of the rows that its own depend on.
double estimate_tiles_us(const LevelOrder& L, const std::vector<int>& tile_of_chain, int ntiles, double tau0,
                         double per_row, double hop) {
  const int n = (int)L.chain.size();
  std::vector<double> end(ntiles, 0.0), start(ntiles, 0.0), row_end(n, 0.0);
  std::vector<int> rows(ntiles, 0), active, tile(n);
  for (int q = 0; q < n; ++q) tile[q] = tile_of_chain[L.chain[q]];
  double tmax = 0.0;
  for (size_t l = 0; l + 1 < L.level_ptr.size(); ++l) {
    const int q0 = L.level_ptr[l], q1 = L.level_ptr[l + 1];
    for (int q = q0; q < q1; ++q) {
      const int t = tile[q];
      if (rows[t]++ == 0) { active.push_back(t); start[t] = end[t]; }
      for (int e = L.dep_ptr[q]; e < L.dep_ptr[q + 1]; ++e)
        if (tile[L.dep[e]] != t) start[t] = std::max(start[t], row_end[L.dep[e]] + hop);
    }
    for (int t : active) {
      end[t] = start[t] + tau0 * ((rows[t] + FC_STEP_ROWS - 1) / FC_STEP_ROWS) + per_row * rows[t];
      tmax = std::max(tmax, end[t]);
      rows[t] = 0;
    }
    active.clear();
    for (int q = q0; q < q1; ++q) row_end[q] = end[tile[q]];
  }
  return tmax;
}

}  // namespace

// ---------------------------------------------------------------------------
int pick_sweep_tiles(int n, const int* ia, const int* ja, const int* dg, const double* xyz, const std::vector<int>& cand,
                     double tau0, double per_row, double hop, double* best_est, int* nocut) {
  std::vector<int> lev;
  const int nls = symmetric_levels(n, ia, ja, dg, lev);
  const int nc = (int)cand.size();
  // what all trials share: the chains and the rows by level.  A trial is then
  // the cuts and one pass over the entries.  A whole schedule for each, on a
  // thread of its own, took 79 ms for 58,212 tetrahedra on 8 cores (20 trials of
  // 9 counts; the four counts tried before them 17), now 15; 750,000: 303 and 99.
  Chains G(n, Deps{ia, ja, dg, true}, lev, xyz);
  const LevelOrder L(G, lev, nls);
  struct Trial { int c, out; double est; bool cut3; };
  auto run = [&](std::vector<Trial>& tr) {
    parallel_items((int)tr.size(), n > FC_THREADS_ROWS ? (int)tr.size() : 1, [&](int k) {
      Trial& t = tr[k];
      std::vector<int> tile_of_chain;
      int cut_axes = 0;
      const int ntiles = tiles_of_chains(G, cand[t.c], t.out, false, tile_of_chain, cut_axes);
      t.cut3 = cut_axes == 3;
      if (ntiles > 0) t.est = estimate_tiles_us(L, tile_of_chain, ntiles, tau0, per_row, hop);
    });
  };
  std::vector<int> counts;  // candidates to try, without duplicates
  for (int c = 0; c < nc; ++c)
    if (cand[c] >= 1 && std::find(cand.begin(), cand.begin() + c, cand[c]) == cand.begin() + c) counts.push_back(c);
  std::vector<Trial> tr;
  for (int c : counts) tr.push_back({c, nocut ? FC_CUT_UNLESS_3 : -1, 1e300, false});
  run(tr);
  if (nocut && std::any_of(tr.begin(), tr.end(), [](const Trial& t) { return t.cut3; })) {
    // the trials that would have cut all three axes stopped there
    std::vector<Trial> more;
    for (size_t k = 0; k < counts.size(); k += 2)
      for (int out = 0; out < 3; ++out) more.push_back({counts[k], out, 1e300, false});
    for (size_t k = 0; k < counts.size() && k < 2; ++k) more.push_back({counts[k], -1, 1e300, false});
    run(more);
    tr.insert(tr.end(), more.begin(), more.end());
  }
  const Trial* best = nullptr;
  for (const Trial& t : tr)
    if (!best || t.est < best->est) best = &t;
  if (nocut) *nocut = best && best->out >= 0 ? best->out : -1;
  if (best_est) *best_est = best ? best->est : 0.0;
  return best && best->est < 1e300 ? cand[best->c] : (nc ? std::max(1, cand[0]) : 1);
}

int symmetric_levels(int n, const int* ia, const int* ja, const int* dg, std::vector<int>& lev) {
  lev.assign(n, 0);
  for (int i = 0; i < n; ++i) {
    int l = lev[i];
    for (int k = ia[i]; k < dg[i]; ++k) l = std::max(l, lev[ja[k]] + 1);
    lev[i] = l;
    for (int k = dg[i] + 1; k < ia[i + 1]; ++k) lev[ja[k]] = std::max(lev[ja[k]], l + 1);
  }
  int nlev = 0;
  for (int i = 0; i < n; ++i) nlev = std::max(nlev, lev[i] + 1);
  return nlev;
}

// Splits the rows of every (tile, level) step wider than wmax into sub-levels:
// lev(i) becomes lev(i) * M + chunk(i), chunk = rank of the row in its step /
// wmax, then the levels are renumbered densely.  Rows of one level do not
// depend on each other, so every dependency still points to a lower level.
// The tiling is recomputed from the new levels (it may move rows between
// tiles), so the split is repeated until no step is wider than wmax (a few
// passes).  Returns the number of levels.
static int split_wide_levels(int n, const int* ia, const int* ja, const int* dg, int ntiles, const double* xyz,
                             int wmax, std::vector<int>& lev, int nlev, int nocut) {
  std::vector<int> code_tmp;  // not written by a layout-only build
  for (int pass = 0; pass < 8; ++pass) {
    SweepSchedule T;
    build_sweep_schedule(n, ia, ja, dg, lev, nlev, true, ntiles, xyz, T, code_tmp, false, nocut);
    std::vector<int> chunk(n, 0);
    int maxc = 0;
    const int nsteps = T.tile_step_ptr[T.ntiles];
    for (int gs = 0; gs < nsteps; ++gs) {
      int cnt = 0;
      for (int q = T.step_row_ptr[gs]; q < T.step_row_ptr[gs + 1]; ++q) {
        const int i = T.rows[q];
        if (i < 0) continue;
        chunk[i] = cnt / wmax;
        ++cnt;
      }
      maxc = std::max(maxc, (cnt - 1) / wmax);
    }
    if (maxc == 0) break;
    const long long M = maxc + 1;
    if ((long long)nlev * M <= (1LL << 26)) {
      // dense ranks of the keys lev * M + chunk through a table of all keys
      std::vector<int> rank((size_t)nlev * M, 0);
      for (int i = 0; i < n; ++i) rank[(size_t)lev[i] * M + chunk[i]] = 1;
      int r = 0;
      for (int& v : rank) v = v ? r++ : -1;
      for (int i = 0; i < n; ++i) lev[i] = rank[(size_t)lev[i] * M + chunk[i]];
      nlev = r;
    } else {
      std::vector<long long> key(n);
      for (int i = 0; i < n; ++i) key[i] = (long long)lev[i] * M + chunk[i];
      std::vector<long long> uk(key);
      std::sort(uk.begin(), uk.end());
      uk.erase(std::unique(uk.begin(), uk.end()), uk.end());
      for (int i = 0; i < n; ++i) lev[i] = (int)(std::lower_bound(uk.begin(), uk.end(), key[i]) - uk.begin());
      nlev = (int)uk.size();
    }
  }
  return nlev;
}

bool build_ordered_sweep(int n, const int* ia, const int* ja, const int* dg, const int* ts, int ntiles,
                         const double* xyz, int R, OrderedSweep& O, SweepSchedule& S, std::string& err, int wmax,
                         int chunk, int nocut, bool checks) {
  O = OrderedSweep();
  O.n = n;
  O.R = std::max(2, R);
  std::vector<int> lev;
  int nlev = symmetric_levels(n, ia, ja, dg, lev);
  if (wmax > 0) nlev = split_wide_levels(n, ia, ja, dg, ntiles, xyz, wmax, lev, nlev, nocut);
  O.nlev = nlev;
  std::vector<int> code_tmp((size_t)ia[n], 0);
  build_sweep_schedule(n, ia, ja, dg, lev, nlev, true, ntiles, xyz, S, code_tmp, true, nocut);
  // ---- new numbering: tile, step, slot order, empty slots dropped; a level
  // wider than chunk rows takes several steps
  const int T = S.ntiles;
  O.ntiles = T;
  O.tile_step_ptr.assign(T + 1, 0);
  O.step_ptr.reserve(S.tile_step_ptr[T] + 1);
  O.tile_W.assign(T, 1);
  O.perm.reserve(n);
  O.iperm.assign(n, -1);
  // per old row: new index, tile, step within the tile, position in the
  // step, kept together so that a dependency costs one cache line
  struct RowInfo { int q, tile, ls, pos; };
  std::vector<RowInfo> rinfo(n);
  std::vector<int> row_tile(n), row_ls(n);
  for (int t = 0; t < T; ++t) {
    const int first = (int)O.step_ptr.size();
    for (int gs = S.tile_step_ptr[t]; gs < S.tile_step_ptr[t + 1]; ++gs) {
      O.step_ptr.push_back((int)O.perm.size());
      int pos = 0, rows = 0;
      for (int q = S.step_row_ptr[gs]; q < S.step_row_ptr[gs + 1]; ++q) {
        const int i = S.rows[q];
        if (i < 0) continue;
        if (chunk > 0 && pos == chunk) {
          O.step_ptr.push_back((int)O.perm.size());
          pos = 0;
        }
        O.iperm[i] = (int)O.perm.size();
        O.perm.push_back(i);
        row_tile[i] = t;
        row_ls[i] = (int)O.step_ptr.size() - 1 - first;
        rinfo[i] = {O.iperm[i], t, row_ls[i], pos++};
        ++rows;
        O.tile_W[t] = std::max(O.tile_W[t], pos);
      }
      O.max_level_rows = std::max(O.max_level_rows, rows);
    }
    O.tile_step_ptr[t + 1] = (int)O.step_ptr.size();
    O.max_tile_steps = std::max(O.max_tile_steps, O.tile_step_ptr[t + 1] - O.tile_step_ptr[t]);
  }
  O.nsteps = (int)O.step_ptr.size();
  O.step_ptr.push_back((int)O.perm.size());
  O.rp_ptr.assign(O.nsteps + 1, 0);
  for (int gs = 0; gs < O.nsteps; ++gs)
    O.rp_ptr[gs + 1] = O.rp_ptr[gs] + ((O.step_ptr[gs + 1] - O.step_ptr[gs] + 3) & ~3);
  if ((int)O.perm.size() != n) { err = "ordered sweep: schedule does not cover every row once"; return false; }
  for (int t = 0; t < T; ++t) O.maxW = std::max(O.maxW, O.tile_W[t]);
  if (chunk > 0) {
    int per_level = 1;  // steps of the widest level, rounded up to a power of two
    while (per_level * chunk < O.max_level_rows) per_level *= 2;
    while (per_level > 1 && (long long)O.R * per_level * O.maxW * 8 > FC_RING_BYTES) per_level /= 2;
    O.R *= per_level;
  }
  const int nE = (n + 3) & ~3;
  O.nE = nE;
  const size_t E = (size_t)FC_ELL * nE;
  // ---- per triangle: entries, codes, exchange and push blocks
  std::vector<int> row_step(n);  // global step of every new row
  for (int gs = 0; gs < O.nsteps; ++gs)
    for (int q = O.step_ptr[gs]; q < O.step_ptr[gs + 1]; ++q) row_step[q] = gs;
  // the two triangles are independent: built concurrently
  auto build_dir = [&](int dirn, std::string& derr) -> bool {
    OrderedDir& D = O.dir[dirn];
    D.ne.assign(nE, 0);
    if (checks) {
      D.slot.assign(E, -1);
      D.col.assign(E, 0);
      D.srec.assign((size_t)4 * nE, 0);
    }
    D.rec.assign((size_t)4 * nE, 0);
    D.ovf_ptr.assign(n + 1, 0);
    for (int q = 0; q < n; ++q) {
      const int i = O.perm[q];
      const int k0 = dirn == 0 ? ia[i] : dg[i] + 1, k1 = dirn == 0 ? dg[i] : ia[i + 1];
      D.ne[q] = k1 - k0;
      D.ovf_ptr[q + 1] = D.ovf_ptr[q] + std::max(0, k1 - k0 - FC_ELL);
    }
    const int novf = D.ovf_ptr[n];
    D.ovf_slot.assign(novf, -1);
    D.ovf_code.assign(novf, 0);
    D.ovf_col.assign(novf, 0);
    std::vector<int> nx(n, 0);  // exchange slots of each consumer row
    // pushes in the order they arise (consumer row ascending, entries in CSR
    // order): producer row, consumer row, the consumer's slot number; grouped
    // by producer below (a counting sort keeps that order within a producer)
    std::vector<int> push_src, push_dst, push_m;
    for (int q = 0; q < n; ++q) {
      const int i = O.perm[q], t = row_tile[i];
      const int nst = O.tile_step_ptr[t + 1] - O.tile_step_ptr[t];
      const int W = O.tile_W[t];
      const int my = dirn == 0 ? row_ls[i] : nst - 1 - row_ls[i];
      const int k0 = dirn == 0 ? ia[i] : dg[i] + 1;
      int codes[FC_ELL] = {0, 0, 0, 0};
      for (int e = 0; e < D.ne[q]; ++e) {
        const int k = k0 + e, j = ja[k];
        const RowInfo rj = rinfo[j];
        const int qj = rj.q;
        int c;
        if (rj.tile == t) {
          const int pj = dirn == 0 ? rj.ls : nst - 1 - rj.ls;
          if (pj >= my) { derr = "ordered sweep: dependency not before its consumer in the tile"; return false; }
          if (my - pj <= O.R - 1) c = (pj % O.R) * W + rj.pos;
          else c = -1;
        } else {
          c = -1;
          D.cross_tile_entries++;
        }
        if (c > 65534) { derr = "ordered sweep: ring index does not fit 16 bits"; return false; }
        if (c < 0) {
          push_src.push_back(qj);
          push_dst.push_back(q);
          push_m.push_back(nx[q]++);
          D.pushed_entries++;
        } else {
          D.ring_entries++;
        }
        if (e < FC_ELL) {
          codes[e] = c + 1;
          if (checks) {
            D.slot[(size_t)e * nE + q] = k;
            D.col[(size_t)e * nE + q] = qj;
          }
        } else {
          const int o = D.ovf_ptr[q] + e - FC_ELL;
          D.ovf_slot[o] = k;
          D.ovf_code[o] = c;
          D.ovf_col[o] = qj;
        }
      }
      // the codes wait where the places will be
      D.rec[4 * (size_t)q + 1] = codes[0] | (codes[1] << 16);
      D.rec[4 * (size_t)q + 2] = codes[2] | (codes[3] << 16);
    }
    std::vector<int> cons_ptr(n + 1, 0), cons_q(push_src.size()), cons_m(push_src.size());
    for (int qj : push_src) cons_ptr[qj + 1]++;
    for (int q = 0; q < n; ++q) cons_ptr[q + 1] += cons_ptr[q];
    {
      std::vector<int> fill(cons_ptr.begin(), cons_ptr.end() - 1);
      for (size_t u = 0; u < push_src.size(); ++u) {
        const int o = fill[push_src[u]]++;
        cons_q[o] = push_dst[u];
        cons_m[o] = push_m[u];
      }
    }
    std::vector<int>().swap(push_src);
    std::vector<int>().swap(push_dst);
    std::vector<int>().swap(push_m);
    // exchange blocks (consumer side) and push blocks (producer side, copied
    // in bulk: each starts on a multiple of 4 elements), one per step
    D.xv_ptr.assign(O.nsteps + 1, 0);
    D.push_ptr.assign(O.nsteps + 1, 0);
    std::vector<int> xoff(n, 0), poff(n, 0);
    for (int gs = 0; gs < O.nsteps; ++gs) {
      int xs = 0, ps = 0;
      for (int q = O.step_ptr[gs]; q < O.step_ptr[gs + 1]; ++q) {
        xoff[q] = xs;
        poff[q] = ps;
        xs += nx[q];
        ps += cons_ptr[q + 1] - cons_ptr[q];
      }
      if (xs > 65534 - O.R * O.maxW || ps > 65535) { derr = "ordered sweep: exchange block of a step too large"; return false; }
      D.xv_ptr[gs + 1] = D.xv_ptr[gs] + xs;
      D.push_ptr[gs + 1] = D.push_ptr[gs] + ((ps + 3) & ~3);
    }
    D.push.assign(D.push_ptr[O.nsteps], 0);
    for (int q = 0; q < n; ++q) {
      const int np = cons_ptr[q + 1] - cons_ptr[q];
      if (nx[q] > 255 || np > 255) { derr = "ordered sweep: more than 255 exchanged entries in a row"; return false; }
      if (D.ne[q] > FC_REC_MAX_ENTRIES) { derr = "ordered sweep: more than 8191 entries in a row"; return false; }
      int* r = D.rec.data() + 4 * (size_t)q;
      if (checks) {
        int* const s = D.srec.data() + 4 * (size_t)q;
        s[0] = D.ne[q] | (np << 8) | (xoff[q] << 16);
        s[1] = poff[q];
        s[2] = r[1];
        s[3] = r[2];
      }
      {
        const int rw = O.R * O.tile_W[row_tile[O.perm[q]]];
        unsigned place[FC_ELL];
        int mx = 0;
        for (int e = 0; e < FC_ELL; ++e) {
          const unsigned c1 = ((unsigned)r[1 + e / 2] >> (16 * (e & 1))) & 0xFFFFu;
          if (c1 > 0) place[e] = c1 - 1;
          else if (e < D.ne[q]) place[e] = rw + 1 + xoff[q] + mx++;
          else place[e] = rw;
        }
        r[0] = np | (poff[q] << 8);
        r[1] = (int)(place[0] | (place[1] << 16));
        r[2] = (int)(place[2] | (place[3] << 16));
        r[3] = FC_REC_PACK(D.ne[q], mx, xoff[q]);
      }
      for (int m = 0; m < np; ++m) {
        const int qc = cons_q[cons_ptr[q] + m], mc = cons_m[cons_ptr[q] + m];
        D.push[D.push_ptr[row_step[q]] + poff[q] + m] = D.xv_ptr[row_step[qc]] + xoff[qc] + mc;
      }
    }
    return true;
  };
  std::string err1;
  bool ok1 = true;
  std::thread th1([&]() { ok1 = build_dir(1, err1); });
  const bool ok0 = build_dir(0, err);
  th1.join();
  if (!ok0) return false;
  if (!ok1) { err = err1; return false; }
  for (int d = 0; d < 2; ++d)
    for (int q = 0; q < n; ++q) O.max_entries = std::max(O.max_entries, O.dir[d].ne[q]);
  // ---- DILU transpose slots of the lower entries, diagonal slots, matrix
  O.lo_tslot.assign(E, 0);
  O.lo_ovf_tslot.assign(O.dir[0].ovf_ptr[n], 0);
  if (checks) O.dslot.assign(nE, 0);
  O.p_ptr.assign(n + 1, 0);
  for (int q = 0; q < n; ++q) {
    const int i = O.perm[q];
    if (checks) O.dslot[q] = dg[i];
    O.p_ptr[q + 1] = O.p_ptr[q] + (ia[i + 1] - ia[i]);
    for (int e = 0; e < O.dir[0].ne[q]; ++e) {
      const int k = ia[i] + e;
      const int tsk = ts ? ts[k] : k;
      if (e < FC_ELL) O.lo_tslot[(size_t)e * nE + q] = tsk;
      else O.lo_ovf_tslot[O.dir[0].ovf_ptr[q] + e - FC_ELL] = tsk;
    }
  }
  O.p_col.resize(ia[n]);
  O.p_slot.resize(ia[n]);
  for (int q = 0; q < n; ++q) {
    const int i = O.perm[q];
    int o = O.p_ptr[q];
    for (int k = ia[i]; k < ia[i + 1]; ++k, ++o) {
      O.p_col[o] = O.iperm[ja[k]];
      O.p_slot[o] = k;
    }
  }
  return true;
}
