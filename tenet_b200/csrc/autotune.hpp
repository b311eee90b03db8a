// Tile-shape autotuner for the grouped GEMMs, keyed on the block-size
// histogram of a compose plan.
//
// FP64 path: a job's rows and columns are cut into equal tiles of at most `cap`
// 16 x 16 blocks a side (cap 2 .. 5), one cap per plan and batch count.  A tile
// costs g + b * blocks per k-tile (its SM's time); the cap is the one whose tile
// list, dealt longest first to the SMs, is estimated to end first.  g and b are
// measured once per device by timing the first sufficiently large compose with
// caps 4 and 2; before that they take model defaults (g / b = 3.2, as measured
// on a B200).  Large batches take the largest tiles, a single small compose the
// smallest: there the longest tile's chain of k-tiles is the whole time.
//
// The four uniform shapes (64x64, 64x32, 32x64, 32x32) and choose_f64_shapes are
// what tnt_tuning_info and tnt_cplan_tile_shapes report.
//
// Split path: the output tile width (64 or 128 columns) is picked by the
// measured time per padded multiply-accumulate of each width.
#pragma once

#include <cstdint>
#include <mutex>
#include <vector>

#include "kernels.cuh"

namespace tnt {

struct DeviceTuning {
  bool f64_calibrated = false;
  double f64_g = 0.67, f64_b = 0.212;  // per tile k-tile and per block k-tile (relative until calibrated)
  double f64_cost[4] = {1.0, 0.6, 0.6, 0.4};  // g + b * blocks of the uniform shapes, kShape* order
  bool split_calibrated = false;
  double split_eff64 = 0.8;  // per-MAC throughput of 64-wide tiles relative to 128-wide
};

// Per-device tuning state (process-wide); lock tuning_mutex() around access.
DeviceTuning& device_tuning(int device);
std::mutex& tuning_mutex();

// Autotuning is on unless TNT_AUTOTUNE=0.
bool autotune_enabled();

// Per-job FP64 tile shapes for the given per-shape costs.
std::vector<int32_t> choose_f64_shapes(const std::vector<GemmJob>& jobs, const double cost[4]);

// The FP64 tile list of `nbatch` batch entries at a cap, longest first by the
// model's cost; a job's tiles of one cost stay adjacent, so its operands are
// read from HBM once.
std::vector<GemmTile> build_f64_tiles(const std::vector<GemmJob>& jobs, int64_t nbatch, int cap, double g, double b);

// Sums over the list of k-tiles (+ 1 for the start and end of a tile) and of
// k-tiles times blocks: the units g and b are quoted in.
void f64_tile_units(const std::vector<GemmJob>& jobs, const std::vector<GemmTile>& tiles, double& ktiles,
                    double& block_ktiles);

// The cap with the smallest estimated time on `sms` SMs.
int choose_f64_cap(const std::vector<GemmJob>& jobs, int64_t nbatch, double g, double b, int sms);

}  // namespace tnt
