// Tile-shape autotuner state and per-job shape choice (see autotune.hpp).
#include "autotune.hpp"

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <functional>
#include <map>
#include <tuple>

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
  // Jobs by falling cost (a job's largest tile's), so that only they are sorted and
  // the tiles are written in place; a job's tiles stay adjacent, and of jobs of one
  // cost each batch entry's come together.
  struct Cut {
    double cost;
    int32_t job;
    int mb, nb, mt, nt;
  };
  std::vector<Cut> cuts;
  cuts.reserve(jobs.size());
  size_t total = 0;
  for (size_t j = 0; j < jobs.size(); ++j) {
    const GemmJob& J = jobs[j];
    Cut c{0.0, (int32_t)j, blocks16(J.m), blocks16(J.n), 0, 0};
    c.mt = (c.mb + cap - 1) / cap;
    c.nt = (c.nb + cap - 1) / cap;
    if (c.mt == 0 || c.nt == 0) continue;
    c.cost = (double)ksteps(J) * (g + b * ceil_div(c.mb, c.mt) * ceil_div(c.nb, c.nt));
    total += (size_t)c.mt * c.nt;
    cuts.push_back(c);
  }
  std::stable_sort(cuts.begin(), cuts.end(), [](const Cut& x, const Cut& y) { return x.cost > y.cost; });
  std::vector<GemmTile> out;
  out.reserve(total * (size_t)nbatch);
  for (size_t i = 0, e; i < cuts.size(); i = e) {
    for (e = i + 1; e < cuts.size() && cuts[e].cost == cuts[i].cost;) ++e;
    for (int64_t q = 0; q < nbatch; ++q)
      for (size_t c = i; c < e; ++c)
        for (int x = 0; x < cuts[c].mt; ++x)
          for (int y = 0; y < cuts[c].nt; ++y) {
            int m0, h, n0, w;
            piece(cuts[c].mb, cap, x, m0, h);
            piece(cuts[c].nb, cap, y, n0, w);
            out.push_back(GemmTile{cuts[c].job, (int32_t)q, m0, n0, f64_tile_code(16 * h, 16 * w), 0});
          }
  }
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
  constexpr double kDeal = 20000;
  // Jobs of one size count as one: this runs on the first compose of every plan.
  struct Size {
    int64_t ks, count;
    int mb, nb;
  };
  std::vector<Size> sizes;
  sizes.reserve(jobs.size());
  for (const GemmJob& J : jobs)
    if (J.m > 0 && J.n > 0) sizes.push_back({ksteps(J), nbatch, blocks16(J.m), blocks16(J.n)});
  auto key = [](const Size& x) { return std::make_tuple(x.ks, x.mb, x.nb); };
  std::sort(sizes.begin(), sizes.end(), [&](const Size& x, const Size& y) { return key(x) > key(y); });
  size_t kinds = 0;
  for (size_t i = 0; i < sizes.size(); ++i)
    if (kinds > 0 && key(sizes[kinds - 1]) == key(sizes[i]))
      sizes[kinds - 1].count += nbatch;
    else
      sizes[kinds++] = sizes[i];
  sizes.resize(kinds);

  // Per cap: bounds on the time of a longest-first deal of its tiles to the SMs: at least
  // the SMs' mean load and the longest tile's chain (alone on its SM a tile still takes
  // its latency, about six block times, per k-tile), at most the mean and one tile more.
  struct Option {
    double tiles = 0.0, mean = 0.0, chain = 0.0, least = 0.0, most = 0.0;
  };
  Option opt[kF64MaxBlocks + 1];
  double bound = 0.0;
  for (int cap = kF64MaxBlocks; cap >= 2; --cap) {
    Option& o = opt[cap];
    double top = 0.0;
    for (const Size& z : sizes) {
      const int mt = (z.mb + cap - 1) / cap, nt = (z.nb + cap - 1) / cap;
      for (int h = 1; h >= 0; --h)      // pieces one block taller than the others, then these
        for (int w = 1; w >= 0; --w) {  // and wider
          const int64_t n = z.count * (h ? z.mb % mt : mt - z.mb % mt) * (w ? z.nb % nt : nt - z.nb % nt);
          if (n == 0) continue;
          const double blocks = (double)(z.mb / mt + h) * (z.nb / nt + w), c = (double)z.ks * (g + b * blocks);
          o.tiles += (double)n;
          o.mean += c * (double)n / sms;
          top = std::max(top, c);
          o.chain = std::max(o.chain, (double)z.ks * b * (6.0 + blocks));
        }
    }
    const bool deal = o.tiles <= kDeal;
    o.least = deal ? std::max({o.mean, o.chain, top}) : o.mean;
    o.most = deal ? std::max(o.mean + top, o.chain) : o.mean;
    bound = cap == kF64MaxBlocks ? o.most : std::min(bound, o.most);
  }
  // Only caps that can still be the best, with other tiles than the next larger one, are dealt
  // out, in the order of their lists (a deal by classes of equal tiles took another cap for an
  // SU(2) map with sectors of 768 and 1024: 214 us, this one's 195).
  std::vector<int> open;
  for (int cap = kF64MaxBlocks; cap >= 2; --cap)
    if (opt[cap].least <= bound && (cap == kF64MaxBlocks || opt[cap].tiles != opt[cap + 1].tiles)) open.push_back(cap);
  int best = open.empty() ? kF64MaxBlocks : open[0];
  if (open.size() < 2) return best;
  double best_t = 0.0;
  for (const int cap : open) {
    const Option& o = opt[cap];
    double t = o.mean;
    if (o.tiles <= kDeal) {
      std::vector<double> load(sms, 0.0);  // a heap, least loaded SM first
      double top = 0.0;
      for (const GemmTile& x : build_f64_tiles(jobs, nbatch, cap, g, b)) {
        std::pop_heap(load.begin(), load.end(), std::greater<double>());
        top = std::max(top, load.back() += (double)ksteps(jobs[x.job]) * (g + b * tile_blocks(x)));
        std::push_heap(load.begin(), load.end(), std::greater<double>());
      }
      t = std::max(top, o.chain);
    }
    if (cap == open[0] || t < best_t) {
      best = cap;
      best_t = t;
    }
  }
  return best;
}

}  // namespace tnt
