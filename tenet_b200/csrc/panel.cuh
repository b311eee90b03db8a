// Shared by the cluster Householder QR (qr.cu) and the one-sided Jacobi engine
// (jacobi.cu): per-sector scratch layout, cluster barrier, FP64 MMA, pairing.
#pragma once

#include <cfloat>

#include "kernels.cuh"

namespace tnt {

// Per-sector scratch of the factorisations, in doubles from work_off:
//   W (rows x k, leading dimension rows = max(m, n)), J (k x k), column norms (k),
//   ranks (k), T of the two QR passes (kFacT(k) each), meta (kFacMeta).
// meta: [0] the power of two the sector was scaled by, [1] and [2] eigh's norms
// ([2] also the cluster's maximum in the QR), from [4] on: 32-bit words of the
// sweeps' reductions.
constexpr int kPanel = 32;  // widest reflector panel
constexpr int kFacMeta = 16;
__host__ __device__ inline int64_t fac_t_elems(int64_t k) { return (k + kPanel) * kPanel; }
__host__ __device__ inline int64_t fac_work_elems(int64_t rows, int64_t k) {
  return rows * k + k * k + 2 * k + 2 * fac_t_elems(k) + kFacMeta;
}
struct FacWork {
  double *W, *J, *sv, *rk, *T[2], *meta;
};
__host__ __device__ inline FacWork fac_work(double* base, int64_t rows, int64_t k) {
  FacWork f;
  f.W = base;
  f.J = f.W + rows * k;
  f.sv = f.J + k * k;
  f.rk = f.sv + k;
  f.T[0] = f.rk + k;
  f.T[1] = f.T[0] + fac_t_elems(k);
  f.meta = f.T[1] + fac_t_elems(k);
  return f;
}

#ifdef __CUDACC__
namespace panel {

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// All threads of the cluster (of the CTA when it is alone); writes before it
// are visible to L2 reads (ld.global.cg) after it.
__device__ __forceinline__ void cluster_barrier(int cl) {
  if (cl == 1) {
    __syncthreads();
    return;
  }
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;\n" ::: "memory");
}

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};\n"
               : "+d"(d0), "+d"(d1)
               : "d"(a), "d"(b));
}

// Whether a sector of this call was refused (status, bit 1; bad, of the general eigh
// kernels, may be null) or has not converged (status, bit 0).
__device__ __forceinline__ bool factor_failed(const int32_t* status, const int32_t* bad) {
  return *status != 0 || (bad != nullptr && *bad != 0);
}

// Round-robin pairing of k2 (even) players: round r, pair i.
__device__ __forceinline__ void tournament_pair(int r, int i, int k2, int& p, int& q) {
  int a, b;
  if (i == 0) {
    a = k2 - 1;
    b = r;
  } else {
    a = r + i;
    if (a >= k2 - 1) a -= k2 - 1;
    b = r - i;
    if (b < 0) b += k2 - 1;
  }
  p = a < b ? a : b;
  q = a < b ? b : a;
}

}  // namespace panel
#endif

}  // namespace tnt
