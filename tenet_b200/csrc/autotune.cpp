// Tile-shape autotuner state and per-job shape choice (see autotune.hpp).
#include "autotune.hpp"

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <queue>

namespace tnt {

namespace {

constexpr int64_t kF64Bk = 16;

int64_t ceil_div(int64_t a, int64_t b) { return (a + b - 1) / b; }

int64_t ksteps(const GemmJob& j) { return ceil_div(j.k, kF64Bk) + 1; }

}  // namespace

std::mutex& tuning_mutex() {
  static std::mutex m;
  return m;
}

DeviceTuning& device_tuning(int device) {
  static std::map<int, DeviceTuning> table;
  return table[device];
}

bool autotune_enabled() {
  const char* e = getenv("TNT_AUTOTUNE");
  return !(e && std::strcmp(e, "0") == 0);
}

std::vector<int32_t> choose_f64_shapes(const std::vector<GemmJob>& jobs, const double cost[4]) {
  std::vector<int32_t> shapes(jobs.size(), kShape64x64);
  for (size_t j = 0; j < jobs.size(); ++j) {
    const GemmJob& J = jobs[j];
    double best = 0.0;
    for (int s = 0; s < 4; ++s) {
      const double t = (double)(ceil_div(std::max<int64_t>(J.m, 1), kShapeM[s]) *
                                ceil_div(std::max<int64_t>(J.n, 1), kShapeN[s])) *
                       (double)ksteps(J) * cost[s];
      if (s == 0 || t < best) {
        best = t;
        shapes[j] = s;
      }
    }
  }
  return shapes;
}

namespace {

int blocks16(int64_t n) { return (int)ceil_div(n, 16); }

// First block and size of piece i of n blocks cut into equal pieces of at most cap.
void piece(int n, int cap, int i, int& first, int& size) {
  const int t = (n + cap - 1) / cap, base = n / t, rem = n % t;
  first = i * base + (i < rem ? i : rem);
  size = base + (i < rem ? 1 : 0);
}

int tile_blocks(const GemmTile& t) { return ((t.shape >> 3) + 1) * ((t.shape & 7) + 1); }

}  // namespace

std::vector<GemmTile> build_f64_tiles(const std::vector<GemmJob>& jobs, int64_t nbatch, int cap, double g, double b) {
  std::vector<std::pair<double, GemmTile>> v;
  for (int64_t q = 0; q < nbatch; ++q)
    for (size_t j = 0; j < jobs.size(); ++j) {
      const GemmJob& J = jobs[j];
      const int mb = blocks16(J.m), nb = blocks16(J.n);
      const int mt = (mb + cap - 1) / cap, nt = (nb + cap - 1) / cap;
      if (mt == 0 || nt == 0) continue;
      // one cost per job (its largest tile's), so a job's tiles stay adjacent
      const double c = (double)ksteps(J) * (g + b * ceil_div(mb, mt) * ceil_div(nb, nt));
      for (int x = 0; x < mt; ++x)
        for (int y = 0; y < nt; ++y) {
          int m0, h, n0, w;
          piece(mb, cap, x, m0, h);
          piece(nb, cap, y, n0, w);
          v.push_back({c, GemmTile{(int32_t)j, (int32_t)q, m0, n0, f64_tile_code(16 * h, 16 * w), 0}});
        }
    }
  std::stable_sort(v.begin(), v.end(), [](const auto& x, const auto& y) { return x.first > y.first; });
  std::vector<GemmTile> out;
  out.reserve(v.size());
  for (auto& x : v) out.push_back(x.second);
  return out;
}

void f64_tile_units(const std::vector<GemmJob>& jobs, const std::vector<GemmTile>& tiles, double& ktiles,
                    double& block_ktiles) {
  ktiles = block_ktiles = 0.0;
  for (const GemmTile& t : tiles) {
    ktiles += (double)ksteps(jobs[t.job]);
    block_ktiles += (double)ksteps(jobs[t.job]) * tile_blocks(t);
  }
}

int choose_f64_cap(const std::vector<GemmJob>& jobs, int64_t nbatch, double g, double b, int sms) {
  // More tiles than this keep every SM busy at any cap: the sums decide.
  constexpr size_t kDeal = 20000;
  int best = kF64MaxBlocks;
  double best_t = 0.0;
  for (int cap = kF64MaxBlocks; cap >= 2; --cap) {
    const std::vector<GemmTile> tiles = build_f64_tiles(jobs, nbatch, cap, g, b);
    double kt, bkt;
    f64_tile_units(jobs, tiles, kt, bkt);
    double t = (g * kt + b * bkt) / sms;
    if (tiles.size() <= kDeal) {
      // Longest-first deal to the SMs, and the longest chain: alone on its SM a tile
      // still takes its latency (about six block times) per k-tile.
      std::priority_queue<double, std::vector<double>, std::greater<double>> load;
      for (int i = 0; i < sms; ++i) load.push(0.0);
      double top = 0.0;
      for (const GemmTile& x : tiles) {
        const double ks = (double)ksteps(jobs[x.job]), c = ks * (g + b * tile_blocks(x));
        const double l = load.top() + c;
        load.pop();
        load.push(l);
        top = std::max({top, l, ks * b * (6.0 + tile_blocks(x))});
      }
      t = top;
    }
    if (cap == kF64MaxBlocks || t < best_t) {
      best = cap;
      best_t = t;
    }
  }
  return best;
}

}  // namespace tnt
