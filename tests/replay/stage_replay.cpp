// Staging of the schedule-ordered sweeps without a GPU.
//
//   stage_replay model K G rule
// plays the hand-over of K stage buffers of G steps between the stager, the
// importers and the sets of compute warps (csrc/fc_sweep.cuh) in many random
// orders, one actor or another held up for a while: barriers that are waited
// for by parity, named barriers of the steps, copies that land late; then sweeps
// of other modes (other K) on the same barriers and words.  rule
// "code": the importers wait as fc_stage.hpp has it; "parity": always by the
// parity of `empty`.  Reports buffers written before they were read, read
// before they were written, named barriers arrived at twice and dead ends.
//
//   stage_replay fits file tiles
// the widest steps that get their buffers, as the pattern analysis looks for
// them.
//
//   stage_replay groups file tiles chunk
// reads a pattern (n, nnz, ia, ja, diagonal places; 0-based) and prints the
// groups and buffers of its sweeps; checks the steps' descriptors for G = 1, 2
// and 4 against the schedule.
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <string>
#include <vector>

#include "fc_stage.hpp"

using namespace fcdev;

namespace {

struct MBar {  // an mbarrier: completed phases, arrivals still missing
  int done = 0, need = 0, left = 0;
  void init(int n) { need = left = n; }
  void arrive(int n = 1) {
    left -= n;
    if (left == 0) { ++done; left = need; }
  }
  bool passes(int parity) const { return (done & 1) != parity; }  // of the phase with this parity, or of the one before
};

struct Shared {  // what the sweeps of a kernel hand on
  MBar empty[FC_MAX_STAGES], full[FC_MAX_STAGES];
  unsigned parity = 0;  // bit b: of the next use of buffer b; bit 31: of the next sweep
  int word[2] = {0, 0};
  explicit Shared(int G) {
    for (MBar& b : empty) b.init(G);
    for (MBar& b : full) b.init(1);
  }
};

struct Model {
  Shared& sh;
  int K, G, ns, ng, ahead;
  bool parity_rule;
  std::mt19937& rng;
  MBar *empty, *full;
  std::vector<int> land;                  // buffers whose copy is under way: its group, else -1
  std::vector<int> copied, imported;      // group whose records / exchanged values a buffer holds
  std::vector<int> read, back;            // per group: steps that have read their values, given their buffer back
  std::vector<char> set_rel, imp_rel, passed;  // named barrier of step k
  bool cleared = false;
  int set_k[FC_SETS], set_at[FC_SETS], imp_g[FC_IMP_WARPS], imp_rel_k[FC_IMP_WARPS], stag_g = 0;
  bool imp_in[FC_IMP_WARPS];
  std::string bad;

  Model(Shared& s, int K_, int G_, int ns_, bool parity_rule_, std::mt19937& r)
      : sh(s), K(K_), G(G_), ns(ns_), ng((ns_ + G_ - 1) / G_), ahead(import_ahead(K_, G_)), parity_rule(parity_rule_), rng(r),
        empty(s.empty), full(s.full), land(K_, -1), copied(K_, -1), imported(K_, -1), read(ng, 0), back(ng, 0),
        set_rel(ns_ + 1, 0), imp_rel(ns_, 0), passed(ns_, 0) {
    for (int s = 0; s < FC_SETS; ++s) { set_k[s] = s; set_at[s] = 0; }
    for (int w = 0; w < FC_IMP_WARPS; ++w) { imp_g[w] = w; imp_in[w] = false; imp_rel_k[w] = 0; }
    set_rel[0] = 1;
  }
  int steps(int g) const { return std::min(G, ns - g * G); }
  int par(int g) const { return (int)(((sh.parity >> (g % K)) ^ (unsigned)(g / K)) & 1u); }
  int& word() { return sh.word[sh.parity >> 31]; }
  void fail(const char* what, int g) {
    if (bad.empty()) bad = std::string(what) + " (group " + std::to_string(g) + ")";
  }
  // one move of an actor; false if it has to wait or is done
  bool set(int s) {
    const int k = set_k[s];
    if (k >= ns) return false;
    const int g = k / G, b = g % K;
    switch (set_at[s]) {
      case 0:
        if (!full[b].passes(par(g))) return false;
        if (copied[b] != g) fail("records not landed", g);
        break;
      case 1:
        if (!set_rel[k] || !imp_rel[k]) return false;
        passed[k] = 1;
        break;
      case 2:
        if (imported[b] != g) fail("wrong exchanged values", g);
        ++read[g];
        break;
      case 3:
        set_rel[k + 1] = 1;
        break;
      default:
        if (copied[b] != g) fail("push targets overwritten", g);
        ++back[g];
        empty[b].arrive();
        set_k[s] += FC_SETS;
        set_at[s] = -1;
    }
    ++set_at[s];
    return true;
  }
  bool importer(int w) {
    const int g = imp_g[w];
    if (g >= ng) return false;
    const int b = g % K;
    if (!imp_in[w]) {
      if (g >= ahead) {
        if (parity_rule || import_by_parity(K, G)) {
          if (!empty[(g - ahead) % K].passes(par(g - ahead))) return false;
        } else if (word() < g + 1) {
          return false;
        }
      }
      if (g >= K && read[g - K] != steps(g - K)) fail("exchanged values written over unread ones", g);
      imported[b] = g;
      imp_in[w] = true;
      imp_rel_k[w] = g * G;
      return true;
    }
    const int k = imp_rel_k[w]++;
    if (k >= FC_STEP_BARS && !passed[k - FC_STEP_BARS]) fail("named barrier arrived at twice", g);
    imp_rel[k] = 1;
    if (imp_rel_k[w] == g * G + steps(g)) { imp_in[w] = false; imp_g[w] += FC_IMP_WARPS; }
    return true;
  }
  bool stager() {
    const int g = stag_g;
    if (g >= ng) return false;
    if (!cleared) {
      sh.word[(sh.parity >> 31) ^ 1u] = 0;
      return cleared = true;
    }
    const int b = g % K;
    if (g >= K && !empty[b].passes(par(g) ^ 1)) return false;
    if (g >= K && back[g - K] != steps(g - K)) fail("records copied over ones in use", g);
    if (!import_by_parity(K, G)) word() = g + 1;
    copied[b] = -1;
    land[b] = g;
    if (steps(g) < G) empty[b].arrive(G - steps(g));
    ++stag_g;
    return true;
  }
  bool copy(int b) {
    if (land[b] < 0) return false;
    copied[b] = land[b];
    land[b] = -1;
    full[b].arrive();
    return true;
  }
  bool run() {
    const int actors = FC_SETS + FC_IMP_WARPS + 1 + K;
    int held = -1, left = 0, idle = 0;
    while (bad.empty()) {
      if (left == 0) { held = (int)(rng() % actors); left = 1 + (int)(rng() % 200); }
      --left;
      const int a = (int)(rng() % actors);
      bool moved = false;
      if (a != held || idle > 40 * actors) {
        if (a < FC_SETS) moved = set(a);
        else if (a < FC_SETS + FC_IMP_WARPS) moved = importer(a - FC_SETS);
        else if (a == FC_SETS + FC_IMP_WARPS) moved = stager();
        else moved = copy(a - FC_SETS - FC_IMP_WARPS - 1);
      }
      idle = moved ? 0 : idle + 1;
      bool over = stag_g >= ng;
      for (int s = 0; s < FC_SETS; ++s) over = over && set_k[s] >= ns;
      if (over) {
        const unsigned first = (1u << (ng % K)) - 1u, all = (1u << K) - 1u;
        sh.parity ^= first ^ ((ng / K) & 1 ? all : 0u) ^ 0x80000000u;
        return true;
      }
      if (idle > 400 * actors) fail("nobody can move", stag_g);
    }
    return false;
  }
};

int model(int K, int G, const std::string& rule) {
  std::mt19937 rng(1234);
  for (int t = 0; t < 2000; ++t) {
    Shared sh(G);
    const int sweeps = 1 + (int)(rng() % 4);
    for (int s = 0; s < sweeps; ++s) {
      const int Ks = s == 0 ? K : 4 << (rng() % 3);  // another mode
      Model m(sh, Ks, G, 1 + (int)(rng() % 90), rule == "parity", rng);
      if (!m.run()) {
        std::printf("K %d G %d run %d sweep %d: %s\n", Ks, G, t, s, m.bad.c_str());
        return 1;
      }
    }
  }
  std::printf("OK\n");
  return 0;
}

int build(const char* file, int tiles, int chunk, OrderedSweep& O) {
  FILE* f = std::fopen(file, "rb");
  if (!f) return 2;
  int head[2];
  std::vector<int> ia, ja, dg;
  auto get = [&](std::vector<int>& v, size_t m) {
    v.resize(m);
    return std::fread(v.data(), sizeof(int), m, f) == m;
  };
  const bool ok = std::fread(head, sizeof(int), 2, f) == 2 && get(ia, head[0] + 1) && get(ja, head[1]) && get(dg, head[0]);
  std::fclose(f);
  if (!ok) return 2;
  SweepSchedule S;
  std::string err;
  if (!build_ordered_sweep(head[0], ia.data(), ja.data(), dg.data(), nullptr, tiles, nullptr, 4, O, S, err, 0, chunk)) {
    std::printf("%s\n", err.c_str());
    return 1;
  }
  return 0;
}

int fits(const char* file, int tiles) {
  for (int chunk = FC_SET_ROWS; chunk > 0; chunk = narrower_steps(chunk)) {
    OrderedSweep O;
    const int st = build(file, tiles, chunk, O);
    if (st) return st;
    const int G = steps_per_buffer(O, false), G_gs = steps_per_buffer(O, true);
    if (!G || !G_gs) continue;
    std::printf("rows %d G %d %d\n", chunk, G, G_gs);
    return 0;
  }
  std::printf("no buffers\n");
  return 1;
}

int groups(const char* file, int tiles, int chunk) {
  OrderedSweep O;
  const int st = build(file, tiles, chunk, O);
  if (st) return st;
  int bad = 0, most = 0;
  for (int d = 0; d < 2; ++d)
    for (int q = 0; q < O.n; ++q) most = std::max(most, O.dir[d].rec[4 * (size_t)q] & 255);
  for (int G = 1; G <= FC_SETS; G *= 2) {
    StepGroups V;
    std::vector<int> desc[2];
    if (!group_steps(O, G, V, desc)) continue;
    for (int d = 0; d < 2; ++d)
      for (int t = 0; t < O.ntiles; ++t) {
        const OrderedDir& H = O.dir[d];
        const int s0 = O.tile_step_ptr[t], ns = O.tile_step_ptr[t + 1] - s0;
        int rows = 0, pushes = 0, xs = 0;
        for (int k = 0; k < ns; ++k) {  // in the order of the sweep
          const int s = s0 + (d ? ns - 1 - k : k), k0 = k / G * G, k1 = std::min(k0 + G, ns);
          const int lo = s0 + (d ? ns - k1 : k0);
          if (k == k0) rows = pushes = xs = 0;
          const int* q = desc[d].data() + 4 * (size_t)s;
          const int cnt = q[1] & 0xFFFF, np = (int)((unsigned)q[1] >> 16);
          bad += q[0] != O.step_ptr[s] || cnt != O.step_ptr[s + 1] - O.step_ptr[s] || np != H.push_ptr[s + 1] - H.push_ptr[s];
          bad += (q[2] & 0xFFFF) != O.rp_ptr[s] - O.rp_ptr[lo] || (int)((unsigned)q[2] >> 16) != H.push_ptr[s] - H.push_ptr[lo];
          bad += (q[3] & 0xFFFF) != O.step_ptr[s] - (O.step_ptr[lo] & ~3) || (int)((unsigned)q[3] >> 16) != H.xv_ptr[s] - H.xv_ptr[lo];
          rows += (cnt + 3) & ~3;
          pushes += np;
          xs += H.xv_ptr[s + 1] - H.xv_ptr[s];
          bad += (q[3] & 0xFFFF) + cnt > V.g_rows + 8 || rows > V.g_padded || pushes > V.g_push || xs > V.g_x;
        }
      }
  }
  const size_t area = ordered_stage_area(O.R, O.maxW);
  std::printf("tiles %d steps %d width %d pushes %d bad %d\n", O.ntiles, O.max_tile_steps, O.max_level_rows, most, bad);
  for (int gs = 0; gs < 2; ++gs) {
    const int G = steps_per_buffer(O, gs != 0);
    std::printf("gs %d G %d", gs, G);
    StepGroups V;
    if (G && group_steps(O, G, V, nullptr))
      for (int m = gs ? OS_GS : OS_SETUP_DIC; m <= (gs ? OS_GS : OS_BWD_DOT); ++m)
        std::printf(" K%d %d %d", m, stages_in(area, StageLayout::of<double>(V, m).bytes),
                    stages_in(area, StageLayout::of<float>(V, m).bytes));
    std::printf("\n");
  }
  return bad != 0;
}

}  // namespace

int main(int argc, char** argv) {
  if (argc > 4 && !std::strcmp(argv[1], "model")) return model(std::atoi(argv[2]), std::atoi(argv[3]), argv[4]);
  if (argc > 3 && !std::strcmp(argv[1], "fits")) return fits(argv[2], std::atoi(argv[3]));
  if (argc > 4 && !std::strcmp(argv[1], "groups")) return groups(argv[2], std::atoi(argv[3]), std::atoi(argv[4]));
  return 2;
}
