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
// Two mappings, chosen per job when the tile list is built:
//  * tall (m >= kThinWide): a tile is kThinRows rows (four times that for up to
//    8 columns, where a tile of 512 rows moves too few bytes to cover its
//    start: 150 against 90.5 us above) by up to kThinCols columns; a thread keeps
//    2 to 8 rows of A in registers, all loads in flight before the first
//    store, B's columns sit in shared memory, and each warp writes 256
//    contiguous bytes per column.
//  * wide (m < kThinWide, a gate's 1 x 1 sectors against a long row): a tile is a
//    range of columns, walked flat over (row, column) so that short columns
//    still give contiguous stores; A sits in shared memory.
#include <algorithm>

#include "kernels.cuh"

namespace tnt {

namespace {

constexpr int kThinThreads = 256;

template <bool BETA>
__device__ __forceinline__ void thin_store(double* p, double acc, double alpha, double beta) {
  const double v = alpha * acc;
  *p = BETA ? fma(beta, *p, v) : v;
}

// Rows [row, rend) of a tall tile, RPT of them per thread at a time: all of a
// group's loads of A (K <= KM columns) are in flight before its first store.
template <int KM, int RPT, bool BETA>
__device__ __forceinline__ void tall_rows(const double* __restrict__ a, int64_t lda, double* __restrict__ c, int64_t ldc,
                                          int64_t row, int64_t rend, int k, int ncol, const double* sm, double alpha,
                                          double beta) {
  for (int64_t r0 = row + threadIdx.x; r0 < rend; r0 += RPT * kThinThreads) {
    double x[RPT][KM];
#pragma unroll
    for (int r = 0; r < RPT; ++r)
#pragma unroll
      for (int l = 0; l < KM; ++l)
        x[r][l] = (l < k && r0 + r * kThinThreads < rend) ? __ldg(a + r0 + r * kThinThreads + l * lda) : 0.0;
    for (int j = 0; j < ncol; ++j) {
      double s[RPT];
#pragma unroll
      for (int r = 0; r < RPT; ++r) s[r] = 0.0;
#pragma unroll
      for (int l = 0; l < KM; ++l)
        if (l < k) {
          const double y = sm[j * kThinMaxK + l];
#pragma unroll
          for (int r = 0; r < RPT; ++r) s[r] = fma(x[r][l], y, s[r]);
        }
#pragma unroll
      for (int r = 0; r < RPT; ++r)
        if (r0 + r * kThinThreads < rend) thin_store<BETA>(c + r0 + r * kThinThreads + j * ldc, s[r], alpha, beta);
    }
  }
}

template <bool BETA>
__global__ void __launch_bounds__(kThinThreads) gemm_thin_kernel(const GemmJob* __restrict__ jobs,
                                                                 const ThinTile* __restrict__ tiles, int32_t ntiles,
                                                                 double* __restrict__ C, int64_t sc,
                                                                 const double* __restrict__ A, int64_t sa,
                                                                 const double* __restrict__ B, int64_t sb, double alpha,
                                                                 double beta) {
  __shared__ double sm[kThinCols * kThinMaxK];  // B's columns (tall) or A (wide: fewer than kThinWide rows)
  static_assert(kThinWide * kThinMaxK <= kThinCols * kThinMaxK, "A of a wide job fits the staging");
  const int tid = threadIdx.x;
  for (int32_t it = blockIdx.x; it < ntiles; it += gridDim.x) {
    const ThinTile tile = tiles[it];
    const GemmJob J = jobs[tile.job];
    const int k = (int)J.k;
    const double* a = A + tile.batch * sa + J.a_off;
    const double* b = B + tile.batch * sb + J.b_off + tile.col * J.ldb;
    double* c = C + tile.batch * sc + J.c_off + tile.col * J.ldc;
    __syncthreads();  // the previous tile's readers of sm are done
    if (J.m >= kThinWide) {
      const int ncol = tile.ncol;
      for (int e = tid; e < ncol * k; e += kThinThreads) {
        const int j = e / k, l = e - j * k;
        sm[j * kThinMaxK + l] = b[l + j * J.ldb];
      }
      __syncthreads();
      const int64_t rend = tile.row + tile.nrow < J.m ? tile.row + tile.nrow : J.m;
      switch (k) {
        case 0: case 1: tall_rows<1, 8, BETA>(a, J.lda, c, J.ldc, tile.row, rend, k, ncol, sm, alpha, beta); break;
        case 2: tall_rows<2, 4, BETA>(a, J.lda, c, J.ldc, tile.row, rend, k, ncol, sm, alpha, beta); break;
        case 3: tall_rows<3, 4, BETA>(a, J.lda, c, J.ldc, tile.row, rend, k, ncol, sm, alpha, beta); break;
        case 4: tall_rows<4, 4, BETA>(a, J.lda, c, J.ldc, tile.row, rend, k, ncol, sm, alpha, beta); break;
        default: tall_rows<kThinMaxK, 2, BETA>(a, J.lda, c, J.ldc, tile.row, rend, k, ncol, sm, alpha, beta); break;
      }
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

}  // namespace

// The thin path takes a plan only as a whole: a plan that mixes thin and thick
// products keeps the one launch of gemm_f64.cu (a second launch costs more
// than its few thin sectors).
bool thin_plan(const std::vector<GemmJob>& jobs) {
  for (const GemmJob& j : jobs)
    if (j.k > kThinMaxK) return false;
  return !jobs.empty();
}

std::vector<ThinTile> build_thin_tiles(const std::vector<GemmJob>& jobs, int64_t nbatch) {
  std::vector<ThinTile> out;
  for (int64_t b = 0; b < nbatch; ++b)
    for (size_t j = 0; j < jobs.size(); ++j) {
      const GemmJob& J = jobs[j];
      if (J.m <= 0 || J.n <= 0) continue;
      const bool wide = J.m < kThinWide;
      const int64_t nr = wide ? J.m : J.n <= 8 ? 4 * kThinRows : kThinRows;
      const int64_t nc = wide ? std::max<int64_t>(1, kThinWideElems / J.m) : kThinCols;
      for (int64_t col = 0; col < J.n; col += nc)
        for (int64_t row = 0; row < J.m; row += nr)
          out.push_back(ThinTile{(int32_t)j, (int32_t)b, row, col, (int32_t)nr, (int32_t)std::min<int64_t>(nc, J.n - col)});
    }
  return out;
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
