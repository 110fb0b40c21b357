// CPU replay of the schedule-ordered sweeps from the row records as the kernels
// read them (OrderedDir::rec, csrc/fc_sweep.cuh): a row's entry count, the place
// of each of its first FC_ELL values (ring, the zero past it, exchange block),
// the exchanged values of its further entries, its pushes.  Forward and backward
// substitution, bit for bit against the plain ones in the original numbering.
//
//   record_replay file tiles chunk [coords]    (pattern: n, nnz, ia, ja, diagonal places; 0-based)
//
// coords: none; or "same", "nan", "inf": rows that all lie in one point, or nowhere.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <limits>
#include <random>
#include <string>
#include <vector>

#include "fc_schedule.hpp"

int main(int argc, char** argv) {
  if (argc < 4) return 2;
  std::FILE* f = std::fopen(argv[1], "rb");
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
  const int n = head[0];
  OrderedSweep O;
  SweepSchedule S;
  std::string err;
  const std::string where = argc > 4 ? argv[4] : "";
  const double at = where == "nan" ? std::nan("") : where == "inf" ? std::numeric_limits<double>::infinity() : 1.5;
  const std::vector<double> xyz(where.empty() ? 0 : 3 * (size_t)n, at);
  if (!build_ordered_sweep(n, ia.data(), ja.data(), dg.data(), nullptr, std::atoi(argv[2]),
                           where.empty() ? nullptr : xyz.data(), 4, O, S, err, 0, std::atoi(argv[3]))) {
    std::printf("refused: %s\n", err.c_str());
    return 0;
  }
  std::mt19937 rng(11);
  std::uniform_real_distribution<double> U(-1.0, 1.0);
  std::vector<double> a(ja.size()), rhs(n);
  for (double& v : a) v = 0.1 * U(rng);
  for (double& v : rhs) v = U(rng);
  long long bad = 0, most = 0, ring_served = 0;
  for (int dirn = 0; dirn < 2; ++dirn) {
    std::vector<double> ref(n), out(n, NAN), xv(O.dir[dirn].xv_ptr[O.nsteps], NAN);
    for (int s = 0; s < n; ++s) {
      const int i = dirn ? n - 1 - s : s;
      double v = rhs[i];
      for (int k = dirn ? dg[i] + 1 : ia[i]; k < (dirn ? ia[i + 1] : dg[i]); ++k) v = std::fma(-a[k], ref[ja[k]], v);
      ref[i] = v;
    }
    const OrderedDir& D = O.dir[dirn];
    std::vector<std::vector<double>> ring(O.ntiles);
    std::vector<int> next(O.ntiles, 0);
    for (int t = 0; t < O.ntiles; ++t) ring[t].assign((size_t)O.R * O.tile_W[t] + 1, NAN);
    for (int t = 0; t < O.ntiles; ++t) ring[t].back() = 0.0;
    for (int left = O.nsteps; left > 0;) {
      const int before = left;
      for (int t = 0; t < O.ntiles; ++t)
        for (;;) {  // as many steps of the tile as can run
          const int s0 = O.tile_step_ptr[t], ns = O.tile_step_ptr[t + 1] - s0, k = next[t], W = O.tile_W[t];
          if (k >= ns) break;
          const int s = s0 + (dirn ? ns - 1 - k : k), base = O.step_ptr[s], cnt = O.step_ptr[s + 1] - base;
          double* const x = xv.data() + D.xv_ptr[s];
          bool ready = true;
          for (int j = 0; j < D.xv_ptr[s + 1] - D.xv_ptr[s]; ++j) ready = ready && !std::isnan(x[j]);
          if (!ready) break;
          std::vector<double> val(cnt);
          for (int sl = 0; sl < cnt; ++sl) {
            const int q = base + sl, i = O.perm[q], k0 = dirn ? dg[i] + 1 : ia[i];
            const int* r = D.rec.data() + 4 * (size_t)q;
            const int ne = FC_REC_ENTRIES(r[3]);
            int m = FC_REC_EXCHANGED(r[3]);
            const unsigned place[FC_ELL] = {(unsigned)r[1] & 0xFFFFu, (unsigned)r[1] >> 16, (unsigned)r[2] & 0xFFFFu,
                                            (unsigned)r[2] >> 16};
            const unsigned rw = (unsigned)(O.R * W);
            bad += ne != (dirn ? ia[i + 1] - dg[i] - 1 : dg[i] - ia[i]);
            most = std::max<long long>(most, ne);
            double v = rhs[i];
            for (int e = 0; e < FC_ELL; ++e) {
              const double y = place[e] <= rw ? ring[t][place[e]] : x[place[e] - rw - 1];
              v = std::fma(e < ne ? -a[k0 + e] : 0.0, y, v);
              ring_served += e < ne && place[e] < rw;
            }
            for (int e = FC_ELL; e < ne; ++e) {
              const int o = D.ovf_ptr[q] + e - FC_ELL, c = D.ovf_code[o];
              bad += D.ovf_slot[o] != k0 + e;
              v = std::fma(-a[k0 + e], c >= 0 ? ring[t][c] : x[FC_REC_OFFSET(r[3]) + m++], v);
              ring_served += c >= 0;
            }
            val[sl] = v;
          }
          for (int j = 0; j < D.xv_ptr[s + 1] - D.xv_ptr[s]; ++j) x[j] = NAN;
          for (int sl = 0; sl < cnt; ++sl) {
            const int* r = D.rec.data() + 4 * (size_t)(base + sl);
            ring[t][(size_t)(k % O.R) * W + sl] = out[base + sl] = val[sl];
            for (int m = 0; m < (r[0] & 255); ++m) xv[D.push[D.push_ptr[s] + ((unsigned)r[0] >> 8) + m]] = val[sl];
          }
          ++next[t];
          --left;
        }
      if (left == before) { std::printf("dead end in direction %d\n", dirn); return 1; }
    }
    for (int q = 0; q < n; ++q) bad += out[q] != ref[O.perm[q]];
  }
  std::printf("tiles %d most %lld ring %lld bad %lld\n", O.ntiles, most, ring_served, bad);
  return bad != 0;
}
