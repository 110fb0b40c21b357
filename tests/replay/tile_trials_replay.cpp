// Choice of the sweeps' tiles on meshes whose chains spread along all three axes:
// pick_sweep_tiles, which estimates its trials from the tiles alone, against a
// whole schedule built for every trial, and the threads that it runs at most.
// argv: nx ny nz seed sms; rows on a jittered nx x ny x nz lattice, coupled to
// the six neighbours and some of the diagonal ones, numbered along a random
// axis order.  Prints "tiles nocut est" of both, then threads and cores.
#include <dirent.h>

#include <algorithm>
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <random>
#include <thread>
#include <vector>

#include "fc_schedule.hpp"

static int tasks() {
  int n = 0;
  if (DIR* d = opendir("/proc/self/task")) {
    while (dirent* e = readdir(d)) n += e->d_name[0] != '.';
    closedir(d);
  }
  return n;
}

int main(int argc, char** argv) {
  if (argc < 6) return 2;
  const int nx = std::atoi(argv[1]), ny = std::atoi(argv[2]), nz = std::atoi(argv[3]), sms = std::atoi(argv[5]);
  std::mt19937 rng(std::atoi(argv[4]));
  std::uniform_real_distribution<double> U(-0.3, 0.3);
  const int n = nx * ny * nz;
  std::vector<double> xyz(3 * (size_t)n);
  std::vector<std::vector<int>> cols(n);
  auto id = [&](int i, int j, int k) { return (i * ny + j) * nz + k; };
  for (int i = 0; i < nx; ++i)
    for (int j = 0; j < ny; ++j)
      for (int k = 0; k < nz; ++k) {
        const int r = id(i, j, k);
        xyz[r] = i + U(rng); xyz[n + r] = j + U(rng); xyz[2 * (size_t)n + r] = k + U(rng);
        cols[r].push_back(r);
        const int nb[7][3] = {{1, 0, 0}, {0, 1, 0}, {0, 0, 1}, {1, 1, 0}, {0, 1, 1}, {1, 0, 1}, {1, 1, 1}};
        for (int e = 0; e < 7; ++e) {
          if (e > 2 && rng() % 2) continue;
          const int a = i + nb[e][0], b = j + nb[e][1], c = k + nb[e][2];
          if (a >= nx || b >= ny || c >= nz) continue;
          cols[r].push_back(id(a, b, c));
          cols[id(a, b, c)].push_back(r);
        }
      }
  std::vector<int> ia(n + 1, 0), ja, dg(n);
  for (int r = 0; r < n; ++r) {
    std::sort(cols[r].begin(), cols[r].end());
    for (int c : cols[r]) {
      if (c == r) dg[r] = (int)ja.size();
      ja.push_back(c);
    }
    ia[r + 1] = (int)ja.size();
  }
  const std::vector<int> cand = {sms, (3 * sms) / 4, sms / 2, sms / 2, sms / 4, sms / 8};
  std::vector<int> lev, scratch(ia[n], 0);
  const int nls = symmetric_levels(n, ia.data(), ja.data(), dg.data(), lev);
  double best = 1e300;
  int tiles = 0, out = -1;
  auto trial = [&](int count, int nocut) {
    SweepSchedule S;
    build_sweep_schedule(n, ia.data(), ja.data(), dg.data(), lev, nls, true, count, xyz.data(), S, scratch, true, nocut);
    const double e = S.ntiles > 0 ? estimate_sweep_us(S, 0.15, 0.0006, 1.2) : 1e300;
    if (e < best) { best = e; tiles = count; out = nocut; }
    return S.cut_axes == 3;
  };
  const int counts[5] = {cand[0], cand[1], cand[2], cand[4], cand[5]};
  bool three = false;
  for (int c : counts) three = trial(c, FC_CUT_UNLESS_3) || three;
  if (three) {
    for (int c = 0; c < 5; c += 2)
      for (int a = 0; a < 3; ++a) trial(counts[c], a);
    for (int c = 0; c < 2; ++c) trial(counts[c], -1);
  }
  std::atomic<int> most{0}, stop{0};
  std::thread watch([&]() {
    while (!stop) most = std::max(most.load(), tasks());
  });
  double est = 0;
  int nocut = -1;
  const int t2 = pick_sweep_tiles(n, ia.data(), ja.data(), dg.data(), xyz.data(), cand, 0.15, 0.0006, 1.2, &est, &nocut);
  stop = 1;
  watch.join();
  std::printf("%d %d %.17g\n%d %d %.17g\n%d %u\n", tiles, out < 0 ? -1 : out, best, t2, nocut, est, most.load(),
              std::thread::hardware_concurrency());
  return 0;
}
