// FP64 grouped GEMM for products whose K is a few: C = alpha A B + beta C with
// K <= kThinMaxK in every job (an MPO or gate contraction over physical legs).
//
// Bound by HBM: each output costs K <= 8 FMAs against its own 8-byte store, so
// the work is one streaming pass that reads A (or B) once and writes C once.
// The tensor-core tiles of gemm_f64.cu pad K and the short side of such a
// product to 16 and give every 64 rows a CTA of its own: the MPO step of the
// full-size SU(2) effective Hamiltonian (K and N of 1 and 3, 271 MB in and 271
// MB out per product) took 1610 us there, 4% of the measured copy rate.
//
// Three mappings, chosen per job when the tile list is built:
//  * tall (m >= kThinTall): a tile is 512 rows (2048 for up to 8 columns, where 512 move
//    too few bytes to cover a tile's start: 150 against 90.5 us above) by up to 32
//    columns; a thread keeps 2 to 8 rows of A in registers, all loads in flight before
//    the first store, B's columns sit in shared memory, and each warp writes 256
//    contiguous bytes per column.
//  * middle (kThinWide <= m < kThinTall): a tile is `lanes` rows, a divisor of m rounded up
//    that leaves few of the 256 threads idle, by a range of columns dealt to the 256 / lanes
//    groups of threads; a thread keeps its row of A.  As tall tiles such rows left
//    most threads idle (40 x 50000 x 8: 60 us, 10 as tensor-core tiles, now 7).
//  * wide (m < kThinWide, a gate's 1 x 1 sectors against a long row): a tile is a
//    range of columns, walked flat over (row, column) so that short columns
//    still give contiguous stores; A sits in shared memory.
// A thread walks its columns one after the other, so a plan of few tiles is as long as
// one of them: columns per thread are halved, from 32 to 4, until there is a tile for
// nearly every SM (600 x 512 x 8: 16.5 us at 32, 3.6 as tensor-core tiles, now 3.8).
#include <algorithm>

#include "kernels.cuh"

namespace tnt {

namespace {

template <bool BETA>
__device__ __forceinline__ void thin_store(double* p, double acc, double alpha, double beta) {
  const double v = alpha * acc;
  *p = BETA ? fma(beta, *p, v) : v;
}

// Rows [row, rend) of a tall tile, RPT of them per thread at a time: all of a
// group's loads of A are in flight before its first store.  K is exact (K = 0: A is
// not read), so that no test stands between the loads of B and the products.
template <int K, int RPT, bool BETA>
__device__ __forceinline__ void tall_rows(const double* __restrict__ a, int64_t lda, double* __restrict__ c, int64_t ldc,
                                          int64_t row, int64_t rend, int ncol, const double* sm, double alpha,
                                          double beta) {
  for (int64_t r0 = row + threadIdx.x; r0 < rend; r0 += RPT * kThinThreads) {
    double x[RPT][K + 1];
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
      for (int l = 0; l < K; ++l)
        x[r][l] = r0 + r * kThinThreads < rend ? __ldg(a + r0 + r * kThinThreads + l * lda) : 0.0;
#pragma unroll 2
    for (int j = 0; j < ncol; ++j) {
      double s[RPT];
#pragma unroll
      for (int r = 0; r < RPT; ++r) s[r] = 0.0;
#pragma unroll
      for (int l = 0; l < K; ++l) {
        const double y = sm[j * kThinPitch + l];
#pragma unroll
        for (int r = 0; r < RPT; ++r) s[r] = fma(x[r][l], y, s[r]);
      }
#pragma unroll
      for (int r = 0; r < RPT; ++r)
        if (r0 + r * kThinThreads < rend) thin_store<BETA>(c + r0 + r * kThinThreads + j * ldc, s[r], alpha, beta);
    }
  }
}

// One row of a middle tile per thread, columns first, first + step, ..
template <int K, bool BETA>
__device__ __forceinline__ void row_columns(const double* __restrict__ a, int64_t lda, double* __restrict__ c,
                                            int64_t ldc, int first, int step, int ncol, const double* sm, double alpha,
                                            double beta) {
  double x[K + 1];
#pragma unroll
  for (int l = 0; l < K; ++l) x[l] = __ldg(a + l * lda);
#pragma unroll 4
  for (int j = first; j < ncol; j += step) {
    double s = 0.0;
#pragma unroll
    for (int l = 0; l < K; ++l) s = fma(x[l], sm[j * kThinPitch + l], s);
    thin_store<BETA>(c + j * ldc, s, alpha, beta);
  }
}

template <bool BETA>
__global__ void __launch_bounds__(kThinThreads) gemm_thin_kernel(const GemmJob* __restrict__ jobs,
                                                                 const ThinTile* __restrict__ tiles, int32_t ntiles,
                                                                 double* __restrict__ C, int64_t sc,
                                                                 const double* __restrict__ A, int64_t sa,
                                                                 const double* __restrict__ B, int64_t sb, double alpha,
                                                                 double beta) {
  __shared__ double sm[kThinCols * kThinPitch];  // B's columns, or A (wide: fewer than kThinWide rows)
  static_assert(kThinWide * kThinMaxK <= kThinCols * kThinPitch, "A of a wide job fits the staging");
  const int tid = threadIdx.x;
  for (int32_t it = blockIdx.x; it < ntiles; it += gridDim.x) {
    const ThinTile tile = tiles[it];
    const GemmJob J = jobs[tile.job];
    const int k = (int)J.k;  // 0 .. kThinMaxK
    static_assert(kThinMaxK == 8, "the cases below");
    const double* a = A + tile.batch * sa + J.a_off;
    const double* b = B + tile.batch * sb + J.b_off + tile.col * J.ldb;
    double* c = C + tile.batch * sc + J.c_off + tile.col * J.ldc;
    __syncthreads();  // the previous tile's readers of sm are done
    if (J.m >= kThinWide) {
      const int ncol = tile.ncol;
      for (int e = tid; e < ncol * k; e += kThinThreads) {
        const int j = e / k, l = e - j * k;
        sm[j * kThinPitch + l] = b[l + j * J.ldb];
      }
      __syncthreads();
      const int64_t rend = tile.row + tile.nrow < J.m ? tile.row + tile.nrow : J.m;
      if (tile.lanes < kThinThreads) {
        const int group = tid / tile.lanes, groups = kThinThreads / tile.lanes;
        const int64_t row = tile.row + (tid - group * tile.lanes);
        if (group < groups && row < rend) {
          const double* ar = a + row;
          double* cr = c + row;
#define TNT_THIN_K(n) \
  case n: row_columns<n, BETA>(ar, J.lda, cr, J.ldc, group, groups, ncol, sm, alpha, beta); break;
          switch (k) {
            TNT_THIN_K(0) TNT_THIN_K(1) TNT_THIN_K(2) TNT_THIN_K(3) TNT_THIN_K(4)
            TNT_THIN_K(5) TNT_THIN_K(6) TNT_THIN_K(7) TNT_THIN_K(8)
          }
#undef TNT_THIN_K
        }
        continue;
      }
#define TNT_THIN_K(n, rows) \
  case n: tall_rows<n, rows, BETA>(a, J.lda, c, J.ldc, tile.row, rend, ncol, sm, alpha, beta); break;
      switch (k) {
        TNT_THIN_K(0, 8) TNT_THIN_K(1, 8) TNT_THIN_K(2, 4) TNT_THIN_K(3, 4) TNT_THIN_K(4, 4)
        TNT_THIN_K(5, 2) TNT_THIN_K(6, 2) TNT_THIN_K(7, 2) TNT_THIN_K(8, 2)
      }
#undef TNT_THIN_K
    } else {
      const int m = (int)J.m;
      for (int e = tid; e < m * k; e += kThinThreads) sm[e] = a[e % m + (int64_t)(e / m) * J.lda];
      __syncthreads();
      const int total = m * tile.ncol;  // at most kThinWideElems
#pragma unroll 4
      for (int e = tid; e < total; e += kThinThreads) {
        const int j = e / m, i = e - j * m;
        double s = 0.0;
        for (int l = 0; l < k; ++l) s = fma(sm[l * m + i], __ldg(b + l + j * J.ldb), s);
        thin_store<BETA>(c + i + j * J.ldc, s, alpha, beta);
      }
    }
  }
}

// Rows of a middle tile: m in equal parts of at least 64 rows (one part below 128) that
// leave the fewest threads without a row.
int thin_lanes(int64_t m) {
  int best = (int)std::min<int64_t>(m, kThinThreads - 1);
  double most = 0.0;
  for (int64_t parts = 1; parts == 1 || (m + parts - 1) / parts >= 64; ++parts) {
    const int64_t rows = (m + parts - 1) / parts;
    if (rows >= kThinThreads) continue;
    const double busy = (double)(kThinThreads / rows) * (double)m / (double)parts;
    if (busy > 1.05 * most) {
      most = busy;
      best = (int)rows;
    }
  }
  return best;
}

}  // namespace

// The thin path takes a plan only as a whole: a plan that mixes thin and thick products
// keeps the one launch of gemm_f64.cu.  Beside thick sectors a second launch costs more
// than a few thin ones; one thick sector beside large thin ones loses the stream, which
// takes no plan that it cannot finish.
bool thin_plan(const std::vector<GemmJob>& jobs) {
  for (const GemmJob& j : jobs)
    if (j.k > kThinMaxK) return false;
  return !jobs.empty();
}

std::vector<ThinTile> build_thin_tiles(const std::vector<GemmJob>& jobs, int64_t nbatch) {
  constexpr size_t kFill = 128;  // more, smaller tiles lose to their start (280: 300000 x 1 x 1 from 3.0 to 4.1 us)
  std::vector<ThinTile> out;
  for (int per = 32;; per /= 2) {  // columns per thread
    out.clear();
    for (int64_t b = 0; b < nbatch; ++b)
      for (size_t j = 0; j < jobs.size(); ++j) {
        const GemmJob& J = jobs[j];
        if (J.m <= 0 || J.n <= 0) continue;
        const bool wide = J.m < kThinWide, tall = J.m >= kThinTall;
        const int lanes = wide || tall ? kThinThreads : thin_lanes(J.m);
        const int64_t nr = wide ? J.m : !tall ? lanes : J.n <= 8 && per == 32 ? 4 * kThinRows : kThinRows;
        const int64_t nc = wide ? kThinWideElems * per / 32 / J.m
                                : std::min<int64_t>(kThinCols, (int64_t)per * (kThinThreads / lanes));
        for (int64_t col = 0; col < J.n; col += nc)
          for (int64_t row = 0; row < J.m; row += nr)
            out.push_back(ThinTile{(int32_t)j, (int32_t)b, row, col, (int32_t)nr,
                                   (int32_t)std::min<int64_t>(nc, J.n - col), lanes});
      }
    if (per == 4 || out.size() >= kFill) return out;
  }
}

cudaError_t launch_gemm_thin(const GemmJob* jobs, const ThinTile* tiles, int32_t ntiles, double* c, int64_t sc,
                             const double* a, int64_t sa, const double* b, int64_t sb, double alpha, double beta,
                             cudaStream_t stream) {
  if (ntiles == 0) return cudaSuccess;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int grid = ntiles < sms * 8 ? ntiles : sms * 8;  // eight resident CTAs per SM
  if (beta == 0.0)
    gemm_thin_kernel<false><<<grid, kThinThreads, 0, stream>>>(jobs, tiles, ntiles, c, sc, a, sa, b, sb, alpha, beta);
  else
    gemm_thin_kernel<true><<<grid, kThinThreads, 0, stream>>>(jobs, tiles, ntiles, c, sc, a, sa, b, sb, alpha, beta);
  return cudaGetLastError();
}

}  // namespace tnt
