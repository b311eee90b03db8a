// FP64 Krylov building blocks on the device: weighted inner products against
// many vectors, many-vector axpy, scaling and a small symmetric eigensolver.
//
// The reference's Krylov crate offers CG over the KrylovVector /
// LinearOperator traits (tenet-krylov/src/{cg,vector,operator}.rs); the
// inner product of block-sparse tensors is the quantum-dimension-weighted
// sum <x, y> = sum_c d_c tr(x_c^T y_c) (TensorKit semantics, as pinned by
// tenet/tests/semantic_suite.rs).  These kernels keep a Lanczos iteration
// resident on the GPU in FP64: orthogonalisation (weighted dots + axpy) and
// the tridiagonal eigenproblem (cyclic Jacobi by one warp).
#include <cfloat>

#include "kernels.cuh"

namespace tnt {

namespace {

constexpr int kDotThreads = 256;
constexpr int kDotMaxVecs = 64;
// Elements per CTA of a weighted dot: eight per thread, so a 0.5 M element vector
// (3.7 MB) makes 230 CTAs; at 8192 it made 58, which left most SMs idle (66 us per
// dot against 15 vectors, 0.8 TB/s; now 8.6 us).
constexpr int kChunk = 2048;
constexpr int kPer = kChunk / kDotThreads;
constexpr int kVecs = 4;  // vectors per pass: 32 loads in flight per thread

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Partial weighted dots of chunk `blockIdx.x`: part[blockIdx.x * k + j] =
// sum_{e in chunk} w(e) V_j[e] y[e], with w constant per coupled sector.
__global__ void __launch_bounds__(kDotThreads) wdot_kernel(const SvdJob* __restrict__ sectors, int32_t nsectors,
                                                           const int64_t* __restrict__ chunk_sector,
                                                           const int64_t* __restrict__ chunk_start, int32_t k,
                                                           const double* __restrict__ V, int64_t ldv,
                                                           const double* __restrict__ y, double* __restrict__ part) {
  __shared__ double red[kDotMaxVecs][kDotThreads / 32];
  const int64_t c = blockIdx.x;
  const SvdJob S = sectors[chunk_sector[c]];
  const int64_t begin = chunk_start[c];
  const int64_t size = S.m * S.n;
  const int64_t end = begin + kChunk < size ? begin + kChunk : size;
  const double w = S.weight;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t at = S.a_off + begin + threadIdx.x;
  const int left = (int)(end - begin) - (int)threadIdx.x;  // elements from this thread's first on
  double ye[kPer];
#pragma unroll
  for (int i = 0; i < kPer; ++i) ye[i] = i * kDotThreads < left ? y[at + i * kDotThreads] : 0.0;
  for (int j0 = 0; j0 < k; j0 += kVecs) {
    double v[kVecs][kPer];
#pragma unroll
    for (int j = 0; j < kVecs; ++j)
#pragma unroll
      for (int i = 0; i < kPer; ++i)
        v[j][i] = (j0 + j < k && i * kDotThreads < left) ? V[(int64_t)(j0 + j) * ldv + at + i * kDotThreads] : 0.0;
#pragma unroll
    for (int j = 0; j < kVecs; ++j) {
      double acc = 0.0;
#pragma unroll
      for (int i = 0; i < kPer; ++i) acc = fma(v[j][i], ye[i], acc);
      acc = warp_sum(acc);
      if (lane == 0 && j0 + j < k) red[j0 + j][warp] = acc;
    }
  }
  __syncthreads();
  for (int j = threadIdx.x; j < k; j += blockDim.x) {
    double s = 0.0;
    for (int q = 0; q < kDotThreads / 32; ++q) s += red[j][q];
    part[c * k + j] = w * s;
  }
}

// out[j] = sum over chunks of part[c * k + j] (fixed order: deterministic).
__global__ void wdot_reduce_kernel(const double* __restrict__ part, int64_t nchunks, int32_t k,
                                   double* __restrict__ out) {
  const int j = blockIdx.x;
  double s = 0.0;
  for (int64_t c = threadIdx.x; c < nchunks; c += blockDim.x) s += part[c * k + j];
  __shared__ double red[32];
  s = warp_sum(s);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = s;
  __syncthreads();
  if (threadIdx.x < 32) {
    double t = threadIdx.x < (blockDim.x >> 5) ? red[threadIdx.x] : 0.0;
    t = warp_sum(t);
    if (threadIdx.x == 0) out[j] = t;
  }
}

// y = a * y + sum_j coef[j] V_j   (a = 1: Gram-Schmidt update with coef = -h).
__global__ void axpy_many_kernel(int64_t n, int32_t k, const double* __restrict__ V, int64_t ldv,
                                 const double* __restrict__ coef, double a, const double* __restrict__ a_dev,
                                 double* __restrict__ y) {
  const double aa = a_dev ? *a_dev : a;
  for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    double v = aa * y[e];
    for (int j = 0; j < k; ++j) v = fma(coef[j], V[(int64_t)j * ldv + e], v);
    y[e] = v;
  }
}

// Cyclic Jacobi eigen-decomposition of a symmetric m x m matrix (m <= 48) by one
// warp, two rows per lane; eigenvalues ascending, eigenvectors as columns
// (column-major).  A chain of m (m - 1) / 2 rotations per sweep: with 256 threads a
// rotation cost four CTA barriers and 1400 cycles, 1.87 ms at m = 30; now 1.38 ms.
__global__ void __launch_bounds__(32) symeig_kernel(int32_t m, const double* __restrict__ Ain,
                                                    double* __restrict__ evals, double* __restrict__ evecs,
                                                    int32_t* __restrict__ status) {
  __shared__ double A[48][49];
  __shared__ double Q[48][49];
  __shared__ double ev[48];
  const int lane = threadIdx.x;
  for (int i = lane; i < m * m; i += 32) {
    const int r = i % m, c = i / m;
    A[r][c] = Ain[i];
    Q[r][c] = r == c ? 1.0 : 0.0;
  }
  __syncwarp();
  const double tol = 4.0 * sqrt((double)m) * DBL_EPSILON;
  const int i0 = lane, i1 = lane + 32;
  const bool on0 = i0 < m, on1 = i1 < m;
  const int r0 = on0 ? i0 : 0, r1 = on1 ? i1 : 0;  // rows beyond m read a valid one and write nothing
  int sweep = 0;
  for (; sweep < 60; ++sweep) {
    bool rot = false;
    for (int p = 0; p < m - 1; ++p) {
      for (int q = p + 1; q < m; ++q) {
        const double apq = A[p][q], app = A[p][p], aqq = A[q][q];
        if (!(fabs(apq) > 1e-300 && fabs(apq) > tol * sqrt(fabs(app * aqq)) + 1e-300)) continue;
        rot = true;
        const double theta = (aqq - app) / (2.0 * apq);
        const double t = (theta >= 0 ? 1.0 : -1.0) / (fabs(theta) + sqrt(theta * theta + 1.0));
        const double c = rsqrt(t * t + 1.0), s = t * c;
        // Q <- Q J; A <- A J on columns p, q, then A <- J^T A on rows p, q
        const double u0 = A[r0][p], v0 = A[r0][q], u1 = A[r1][p], v1 = A[r1][q];
        const double g0 = Q[r0][p], h0 = Q[r0][q], g1 = Q[r1][p], h1 = Q[r1][q];
        __syncwarp();
        if (on0) {
          A[i0][p] = c * u0 - s * v0;
          A[i0][q] = s * u0 + c * v0;
          Q[i0][p] = c * g0 - s * h0;
          Q[i0][q] = s * g0 + c * h0;
        }
        if (on1) {
          A[i1][p] = c * u1 - s * v1;
          A[i1][q] = s * u1 + c * v1;
          Q[i1][p] = c * g1 - s * h1;
          Q[i1][q] = s * g1 + c * h1;
        }
        __syncwarp();
        const double x0 = A[p][r0], y0 = A[q][r0], x1 = A[p][r1], y1 = A[q][r1];
        __syncwarp();
        if (on0) {
          A[p][i0] = c * x0 - s * y0;
          A[q][i0] = s * x0 + c * y0;
        }
        if (on1) {
          A[p][i1] = c * x1 - s * y1;
          A[q][i1] = s * x1 + c * y1;
        }
        __syncwarp();
      }
    }
    if (!rot) break;
  }
  if (lane == 0 && sweep == 60) *status = 1;
  for (int i = lane; i < m; i += 32) ev[i] = A[i][i];
  __syncwarp();
  for (int i = lane; i < m; i += 32) {
    int pos = 0;
    for (int j = 0; j < m; ++j) pos += (ev[j] < ev[i] || (ev[j] == ev[i] && j < i)) ? 1 : 0;
    evals[pos] = ev[i];
    for (int r = 0; r < m; ++r) evecs[r + (int64_t)pos * m] = Q[r][i];
  }
}

}  // namespace

int64_t wdot_chunks(const SvdJob* host_sectors, int32_t nsectors, std::vector<int64_t>& sector_of_chunk,
                    std::vector<int64_t>& start_of_chunk) {
  sector_of_chunk.clear();
  start_of_chunk.clear();
  for (int32_t s = 0; s < nsectors; ++s) {
    const int64_t size = host_sectors[s].m * host_sectors[s].n;
    for (int64_t b = 0; b < size; b += kChunk) {
      sector_of_chunk.push_back(s);
      start_of_chunk.push_back(b);
    }
  }
  return (int64_t)sector_of_chunk.size();
}

cudaError_t launch_wdot(const SvdJob* sectors, int32_t nsectors, const int64_t* chunk_sector,
                        const int64_t* chunk_start, int64_t nchunks, int32_t k, const double* V, int64_t ldv,
                        const double* y, double* part, double* out, cudaStream_t stream) {
  if (k <= 0) return cudaSuccess;
  if (k > kDotMaxVecs) return cudaErrorInvalidValue;
  if (nchunks > 0)
    wdot_kernel<<<(unsigned)nchunks, kDotThreads, 0, stream>>>(sectors, nsectors, chunk_sector, chunk_start, k, V,
                                                              ldv, y, part);
  wdot_reduce_kernel<<<k, 256, 0, stream>>>(part, nchunks, k, out);
  return cudaGetLastError();
}

cudaError_t launch_axpy_many(int64_t n, int32_t k, const double* V, int64_t ldv, const double* coef, double a,
                             const double* a_dev, double* y, cudaStream_t stream) {
  if (n == 0) return cudaSuccess;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int64_t blocks = (n + 255) / 256;
  const unsigned grid = (unsigned)(blocks < (int64_t)sms * 16 ? blocks : (int64_t)sms * 16);
  axpy_many_kernel<<<grid, 256, 0, stream>>>(n, k, V, ldv, coef, a, a_dev, y);
  return cudaGetLastError();
}

cudaError_t launch_symeig(int32_t m, const double* A, double* evals, double* evecs, int32_t* status,
                          cudaStream_t stream) {
  if (m <= 0) return cudaSuccess;
  if (m > 48) return cudaErrorInvalidValue;
  symeig_kernel<<<1, 32, 0, stream>>>(m, A, evals, evecs, status);
  return cudaGetLastError();
}

}  // namespace tnt
