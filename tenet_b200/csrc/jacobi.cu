// One-sided Jacobi on a thread-block cluster per sector: the engine of the
// batched SVD and of the symmetric eigendecomposition.
//
// In: W (k x k, leading dimension ldw) in the sector's scratch, for the SVD the
// transposed R factor of the sector (qr.cu), for eigh the shifted matrix.  Out:
// W J = columns orthogonal to 4 sqrt(k) eps, J (SVD only) in the scratch, column
// norms in sv.
//
// The rounding of some 10 k rotations moves the length of J's columns by a random walk
// and a small bias, and W J's with them (k = 300: -13 eps on average, -34 eps at most; a
// value's error 25 eps of the largest).  So at the end both are divided by the length
// of J's column, which leaves the values 4 eps and the product of the factors 23
// (38 before, 24 by the general kernels).
//
// Columns are split into nb blocks (nb even, w columns each); a sweep is a
// round-robin tournament of the blocks, one pair per CTA and round, with the
// pairs inside each block rotated in the first round.  What bounds a round is
// the latency of the rotation chain (dot product, reduction, angle, update) and,
// for the largest sectors, the FP64 units, so:
//  * the w columns of one block stay in registers (G lanes per column) while the
//    other block's columns pass by in shared memory: per rotation one column is
//    read and written there instead of two read twice and written once;
//  * short columns take few lanes each (G = 8 up to k = 64, 16 up to 128), so the
//    reduction and the angle are shared by several pairs of a warp;
//  * columns carry a scale (fast rotations: p - a q and q + b p, two FMAs per
//    element instead of two products and two FMAs), taken out once per block pair;
//  * squared norms are formed once and updated per rotation, so a pair needs one
//    dot product;
//  * tests and the tangent run in single precision (its error only leaves 1e-6 of
//    the pair's cosine behind); the scale factor (1 + t^2)^{-1/2} comes from one
//    third-order step in FP64, so a rotation is orthogonal to FP64 rounding;
//  * the sweep that only confirms convergence is left out when the sweep
//    before it cannot have left a cosine above the tolerance (below).
//
// Two kernels.  While all columns, with J's rows stacked below W's, fit the
// cluster's shared memory twice (k <= 320, or 448 without J), they never leave it:
// blocks move to the CTA of their next pair through distributed shared memory.
// Beyond, blocks are staged through L2, the rotations of a block pair accumulate
// in a 2w x 2w matrix below the staged columns, and J's columns are multiplied by
// it on the FP64 tensor cores.  (Handing columns from warp to warp on a count of
// their rounds instead of a CTA-wide barrier measured the same there.)
// Measured on a B200 against the general kernels of svd.cu and a two-sided
// Jacobi in shared memory: truncated SVD of the D = 2048 chain (six sectors of
// 586, two of 293) 94.9 -> 22.6 ms, a whole two-site update at D = 224 (104 x 104)
// 5.2 -> 1.13 ms, eigh at D = 224 6.4 -> 0.89 ms with eigenvalues to 4e-16 (1.4e-14).
#include <algorithm>

#include "panel.cuh"

namespace tnt {

namespace {

using namespace panel;

constexpr int kMaxSweeps = 40;
constexpr size_t kJacobiSmem = 216 * 1024;

// Stride of a staged column: its rows, the zr rows of its accumulator, and a pad
// that keeps the MMA fragments of the accumulator conflict-free (4 mod 16).
__host__ __device__ constexpr int col_stride(int rows, int zr) { return rows + zr + 4; }

// Block width and (even) block count for k columns of `rows` rows on cl CTAs of
// `owners` column owners each.
__host__ __device__ __forceinline__ void block_split(int k, int rows, int cl, int owners, int zr, int& w, int& nb) {
  int cap = (int)(kJacobiSmem / 8 / (2 * col_stride(rows, zr)));
  if (cap > owners) cap = owners;
  if (cap > zr / 2) cap = zr / 2;
  int per = 1;  // block pairs per CTA and round
  while ((k + 2 * cl * per - 1) / (2 * cl * per) > cap) ++per;
  w = (k + 2 * cl * per - 1) / (2 * cl * per);
  nb = (k + w - 1) / w;
  nb = nb < 2 ? 2 : (nb + 1) & ~1;
}

struct Thresholds {
  float tol, noise2, floor;
};

// Tangent t, (1 + t^2)^{-1/2} and its inverse, t * gamma (the norms' change).
struct Rotation {
  double t, c, ic, tg;
};

__device__ __forceinline__ float rcp_approx(float x) {
  float y;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float rsqrt_approx(float x) {
  float y;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}
__device__ __forceinline__ float sqrt_approx(float x) {
  float y;
  asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
  return y;
}

// The rotation that makes the pair orthogonal (squared norms al, be, dot ga);
// false when the pair counts as orthogonal already.  The sector is scaled to a
// largest entry below 1, so every float here is in range: squared norms lie
// between noise2 (about 1e-30) and k^2, |ga| above floor (about 1e-33).
__device__ __forceinline__ bool rotation(double al, double be, double ga, const Thresholds& th, Rotation& R,
                                         float& cosmax, float& fillmax) {
  const float gf = (float)ga, af = (float)al, bf = (float)be;
  const float rr = rsqrt_approx(af) * rsqrt_approx(bf), cosine = fabsf(gf) * rr;
  if (!(cosine > th.tol && fminf(af, bf) > th.noise2 && fabsf(gf) > th.floor)) return false;
  const float z = 0.5f * (float)(be - al) * rcp_approx(gf), az = fabsf(z);
  float t = rcp_approx(az < 1e4f ? az + sqrt_approx(fmaf(z, z, 1.0f)) : az + az);
  t = z < 0.0f ? -t : t;
  const double td = (double)t, y = (double)rsqrt_approx(fmaf(t, t, 1.0f)), x = fma(td, td, 1.0);
  const double e = fma(-x * y, y, 1.0);  // y (1 + e/2 + 3 e^2 / 8) = x^{-1/2} up to e^3
  R.t = td;
  R.c = fma(y * e, fma(0.375, e, 0.5), y);
  R.ic = x * R.c;
  R.tg = td * ga;
  // Cosine of the pair, and the most this rotation can put back between one of
  // its columns and a third per unit of the other's cosine with it.
  cosmax = fmaxf(cosmax, cosine);
  fillmax = fmaxf(fillmax, fabsf(t) * rr * fmaxf(af, bf));
  return true;
}

// 1 / d from an estimate good to a few roundings: the product of the rotations' inverse
// factors walks away from the inverse of the product, and a rotation whose two
// coefficients disagree is not orthogonal.
__device__ __forceinline__ double reciprocal_step(double d, double id) { return fma(id, fma(-d, id, 1.0), id); }

// Sum over the G lanes of a column.
template <int G>
__device__ __forceinline__ double group_sum(double v) {
#pragma unroll
  for (int o = G / 2; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// Squared norm, scale and inverse scale of the columns of a block pair (block bi's
// at 0 .. w - 1, block bj's from w on): true column = scale * stored column.
struct Columns {
  double *nrm, *d, *id;
};

// Both columns in shared memory (pairs inside a block); every lane of the warp
// calls it.  PW elements per lane enter the dot product, NZ further ones (G apart
// from row G PW on) only rotate, when acc.  KEEP: all of them are loaded before
// the first store (the compiler cannot move a load over one).
template <int G, int PW, int NZ, bool KEEP>
__device__ __forceinline__ void rotate_smem(bool live, double* base, int ls, int ip, int iq, const Columns& col, bool acc,
                                            const Thresholds& th, float& cosmax, float& fillmax) {
  const int gl = threadIdx.x % G;
  double ga = 0.0, gb = 0.0, al = 0.0, be = 0.0, dp = 1.0, dq = 1.0;
  double u[KEEP ? PW : 1], v[KEEP ? PW : 1], uz[NZ], vz[NZ];
  double* p = base + (live ? ip : 0) * ls + gl;
  double* q = base + (live ? iq : 0) * ls + gl;
#pragma unroll
  for (int j = 0; j < PW; ++j) {
    const double x = p[G * j], y = q[G * j];
    if constexpr (KEEP) {
      u[j] = x;
      v[j] = y;
    }
    if (j & 1) gb = fma(x, y, gb);
    else ga = fma(x, y, ga);
  }
  if (live) {
    al = col.nrm[ip];
    be = col.nrm[iq];
    dp = col.d[ip];
    dq = col.d[iq];
  }
  ga = group_sum<G>(ga + gb) * (dp * dq);
  Rotation R;
  if (live && rotation(al, be, ga, th, R, cosmax, fillmax)) {
    const double ip_ = col.id[ip], iq_ = col.id[iq];
    const double a = -R.t * (dq * ip_), b = R.t * (dp * iq_);
    if constexpr (!KEEP) asm volatile("" ::: "memory");
    if (acc) {
#pragma unroll
      for (int j = 0; j < NZ; ++j) {
        uz[j] = p[G * (PW + j)];
        vz[j] = q[G * (PW + j)];
      }
    }
#pragma unroll
    for (int j = 0; j < PW; ++j) {
      const double x = KEEP ? u[KEEP ? j : 0] : p[G * j], y = KEEP ? v[KEEP ? j : 0] : q[G * j];
      p[G * j] = fma(a, y, x);
      q[G * j] = fma(b, x, y);
    }
    if (acc) {
#pragma unroll
      for (int j = 0; j < NZ; ++j) {
        p[G * (PW + j)] = fma(a, vz[j], uz[j]);
        q[G * (PW + j)] = fma(b, uz[j], vz[j]);
      }
    }
    if (gl == 0) {
      col.nrm[ip] = al - R.tg;
      col.nrm[iq] = be + R.tg;
      const double d0 = dp * R.c, d1 = dq * R.c;
      col.d[ip] = d0;
      col.d[iq] = d1;
      col.id[ip] = reciprocal_step(d0, ip_ * R.ic);
      col.id[iq] = reciprocal_step(d1, iq_ * R.ic);
    }
  }
  __syncwarp();
}

// The pairs inside the two blocks: a round robin in each, all warps.
template <int G, int PW, int NZ, int NW, bool KEEP>
__device__ __forceinline__ void rotate_within(double* base, int ls, int w, int np, int nq, const Columns& col, bool acc,
                                              const Thresholds& th, float& cosmax, float& fillmax) {
  constexpr int PP = 32 / G;
  const int warp = threadIdx.x >> 5, sub = (threadIdx.x & 31) / G;
  const int n2 = (w + 1) & ~1, half = n2 / 2;
  for (int r = 0; r < n2 - 1; ++r) {
    for (int e0 = warp * PP; e0 < n2; e0 += NW * PP) {
      const int e = e0 + sub, b = e >= half;
      int p = 0, q = 0;
      bool live = e < n2;
      if (live) {
        tournament_pair(r, b ? e - half : e, n2, p, q);
        live = q < (b ? nq : np);
        p += b ? w : 0;
        q += b ? w : 0;
      }
      rotate_smem<G, PW, NZ, KEEP>(live, base, ls, p, q, col, acc, th, cosmax, fillmax);
    }
    __syncthreads();
  }
}

// Thresholds from ||W||_F^2 (the same sum in the same order in every CTA): a pair
// is rotated only while its cosine exceeds the rounding level of a length-k dot
// product and both columns stand above the rounding noise k eps ||A||_F (columns of
// the null space shrink to that level, and every rotation refills them with
// noise whose cosine is O(1)).  Every warp leaves its columns' squared norms in
// sv first.
__device__ __forceinline__ double make_thresholds(const FacWork& f, int64_t ldw, int k, int rank, int cl,
                                                  Thresholds& th) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (int c = rank * nwarps + warp; c < k; c += cl * nwarps) {
    double s = 0.0;
    for (int x = lane; x < k; x += 32) {
      const double v = __ldcg(f.W + (int64_t)c * ldw + x);
      s = fma(v, v, s);
    }
    s = warp_sum(s);
    if (lane == 0) f.sv[c] = s;
  }
  cluster_barrier(cl);
  double frob2 = 0.0;  // every warp the same sum in the same order, whatever the CTA's size
  for (int c = lane; c < k; c += 32) frob2 += __ldcg(f.sv + c);
  frob2 = warp_sum(frob2);
  const double tol = 4.0 * sqrt((double)k) * DBL_EPSILON;
  th.tol = (float)tol;
  th.noise2 = (float)(((double)k * DBL_EPSILON) * ((double)k * DBL_EPSILON) * frob2);
  th.floor = (float)(1e-33 * frob2);  // below every gamma above the tolerance of two columns above the noise
  return tol;
}

// After a sweep with these largest values: no pair above the tolerance means
// done.  Otherwise, a cosine zeroed in the sweep can only come back through later
// rotations of its two columns (at most 2 k of them), each adding at most
// fill * cosine, and the single-precision tangent leaves at most 2e-6 of a cosine
// behind: when both stay below the tolerance, a further sweep would rotate nothing.
__device__ __forceinline__ bool converged(int k, double tol, float cosmax, float fillmax) {
  return cosmax == 0.0f || (2.0 * k * (double)fillmax * (double)cosmax <= tol && 2e-6 * (double)cosmax <= tol);
}

// ---------------------------------------------------------------------------
// Columns resident in the cluster's shared memory
// ---------------------------------------------------------------------------

// CTA and slot half (0: block bi's, 1: block bj's) of block x in round r.
__device__ __forceinline__ void block_place(int x, int r, int nb, int& cta, int& side) {
  const int m = nb - 1;
  int other;
  if (x == m) {
    cta = 0;
    other = r;
  } else {
    int d = x - r;
    if (d < 0) d += m;
    cta = d <= m / 2 ? d : m - d;  // nb even: m / 2 = nb / 2 - 1 pairs beside the fixed player's
    if (d == 0) {
      other = m;
    } else {
      other = 2 * r - x;
      if (other < 0) other += m;
      if (other >= m) other -= m;
    }
  }
  side = x < other ? 0 : 1;
}

__device__ __forceinline__ uint32_t remote_smem(const void* p, int rank) {
  uint32_t a = (uint32_t)__cvta_generic_to_shared(p), o;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(o) : "r"(a), "r"(rank));
  return o;
}
__device__ __forceinline__ void st_remote(uint32_t a, double v) {
  asm volatile("st.shared::cluster.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory");
}
__device__ __forceinline__ void st_remote(uint32_t a, int v) {
  asm volatile("st.shared::cluster.s32 [%0], %1;" ::"r"(a), "r"(v) : "memory");
}

// Columns per block and stride of a stored column.
__host__ __device__ __forceinline__ int ring_width(int k, int cl) { return (k + 2 * cl - 1) / (2 * cl); }
__host__ __device__ constexpr int ring_stride(int rows, bool acc, int g) {
  return rows * (acc ? 2 : 1) + (g == 8 ? 8 : 4);
}

// G lanes per column, PW elements of W (and of J, ACC) each (columns padded with
// zeros to G PW rows, so that every loop has a constant length); NW warps own
// 32 / G columns each.
template <int G, int PW, int NW, bool ACC>
__global__ void __launch_bounds__(NW * 32, 1)
    jacobi_ring_kernel(const SvdJob* __restrict__ jobs, double* __restrict__ work, const int64_t* __restrict__ work_off,
                       int32_t* __restrict__ status, int cl) {
  constexpr int PP = 32 / G, PJ = ACC ? PW : 1, kSlots = 2 * NW * PP, kp = G * PW, ls = ring_stride(kp, ACC, G);
  constexpr int kCopy = ((ACC ? 2 : 1) * kp + 31) / 32;  // elements of a whole column per lane
  const int rank = (int)(blockIdx.x % cl);
  const SvdJob S = jobs[blockIdx.x / cl];
  const int k = (int)S.k;
  const int64_t ldw = S.m > S.n ? S.m : S.n;
  if (k == 0) return;
  const FacWork f = fac_work(work + work_off[blockIdx.x / cl], ldw, k);
  extern __shared__ __align__(16) double sm[];
  __shared__ double s_nrm[2][kSlots], s_d[kSlots], s_id[kSlots];
  __shared__ int s_max[2][16][2], s_cos, s_fill;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int gl = lane % G, owner = warp * PP + lane / G;
  const int w = ring_width(k, cl), set_len = 2 * w * ls;
  int nb = (k + w - 1) / w;
  nb = nb < 2 ? 2 : (nb + 1) & ~1;
  const bool active = rank < nb / 2;
  auto bsize = [&](int b) {
    const int n = k - b * w;
    return n < 0 ? 0 : n < w ? n : w;
  };
  Thresholds th;
  const double tol = make_thresholds(f, ldw, k, rank, cl, th);

  // The first round's pair of blocks from the scratch, J = I.
  int bi = 0, bj = 0;
  if (active) {
    tournament_pair(0, rank, nb, bi, bj);
    for (int c = warp; c < 2 * w; c += NW) {
      const int g = c < w ? bi * w + c : bj * w + c - w;
      if (c < w ? c >= bsize(bi) : c - w >= bsize(bj)) continue;
      double* d = sm + (int64_t)c * ls;
      for (int x = lane; x < kp; x += 32) {
        d[x] = x < k ? __ldcg(f.W + (int64_t)g * ldw + x) : 0.0;
        if (ACC) d[kp + x] = x == g ? 1.0 : 0.0;
      }
    }
  }
  if (cl > 1) cluster_barrier(cl);  // every CTA has started (its shared memory can be written) before the first exchange
  __syncthreads();

  int set = 0, sweep = 0;
  for (; sweep < kMaxSweeps && k > 1; ++sweep) {
    float cosmax = 0.0f, fillmax = 0.0f;
    if (tid == 0) {
      s_cos = 0;
      s_fill = 0;
    }
    for (int t = 0; t < nb - 1; ++t) {
      if (active) {
        tournament_pair(t, rank, nb, bi, bj);
        const int np = bsize(bi), nq = bsize(bj);
        double* C = sm + set * set_len;
        double* Q = C + w * ls;
        const Columns col{s_nrm[set], s_d, s_id};
        if (t == 0)
          for (int c = warp; c < 2 * w; c += NW) {
            if (c < w ? c >= np : c - w >= nq) continue;
            double s = 0.0;
            for (int x = lane; x < kp; x += 32) s = fma(C[c * ls + x], C[c * ls + x], s);
            s = warp_sum(s);
            if (lane == 0) col.nrm[c] = s;
          }
        for (int c = tid; c < 2 * w; c += NW * 32) s_d[c] = s_id[c] = 1.0;
        __syncthreads();
        if (t == 0) rotate_within<G, PW, PJ, NW, true>(C, ls, w, np, nq, col, ACC, th, cosmax, fillmax);
        // Cross pairs: G lanes keep column `owner` of block bi in registers.
        double p[PW], pj[PJ];
        const bool own = owner < np;
        const double* po = C + (own ? owner : 0) * ls + gl;  // others load a column they never use
#pragma unroll
        for (int j = 0; j < PW; ++j) {
          p[j] = po[G * j];
          if constexpr (ACC) pj[j] = po[kp + G * j];
        }
        double al = own ? col.nrm[owner] : 0.0, dp = own ? s_d[owner] : 1.0, idp = own ? s_id[owner] : 1.0;
        __syncthreads();
        for (int r = 0; r < w; ++r) {
          int jq = owner + r;
          if (jq >= w) jq -= w;
          const bool live = own && jq < nq;
          double* q = Q + (live ? jq : 0) * ls + gl;
          double ga = 0.0, gb = 0.0, qv[PW], qj[PJ];
#pragma unroll
          for (int j = 0; j < PW; ++j) {
            qv[j] = q[G * j];
            if (j & 1) gb = fma(p[j], qv[j], gb);
            else ga = fma(p[j], qv[j], ga);
          }
          const double be = live ? col.nrm[w + jq] : 0.0, dq = live ? s_d[w + jq] : 1.0, idq = live ? s_id[w + jq] : 1.0;
          if constexpr (ACC)
#pragma unroll
            for (int j = 0; j < PW; ++j) qj[j] = q[kp + G * j];
          const double dd = dp * dq;
          ga = group_sum<G>(ga + gb) * dd;
          Rotation R;
          if (live && rotation(al, be, ga, th, R, cosmax, fillmax)) {
            const double a = -R.t * (dq * idp), b = R.t * (dp * idq);
#pragma unroll
            for (int j = 0; j < PW; ++j) {
              const double u = p[j];
              p[j] = fma(a, qv[j], u);
              q[G * j] = fma(b, u, qv[j]);
            }
            if constexpr (ACC)
#pragma unroll
              for (int j = 0; j < PW; ++j) {
                const double u = pj[j];
                pj[j] = fma(a, qj[j], u);
                q[kp + G * j] = fma(b, u, qj[j]);
              }
            al -= R.tg;
            dp *= R.c;
            idp = reciprocal_step(dp, idp * R.ic);
            if (gl == 0) {
              col.nrm[w + jq] = be + R.tg;
              const double d = dq * R.c;
              s_d[w + jq] = d;
              s_id[w + jq] = reciprocal_step(d, idq * R.ic);
            }
          }
          __syncthreads();
        }
        // On to the next round's places, scales taken out.
        int ci = 0, si = 0, cj = 0, sj = 1;
        if (cl > 1) {
          const int tn = t + 1 < nb - 1 ? t + 1 : 0;
          block_place(bi, tn, nb, ci, si);
          block_place(bj, tn, nb, cj, sj);
        }
        double* N = sm + (cl > 1 ? (set ^ 1) * set_len : 0);
        double* nn = s_nrm[cl > 1 ? set ^ 1 : 0];
        if (own) {
          const int slot = si * w + owner;
          const uint32_t a = remote_smem(N + slot * ls + gl, ci);
#pragma unroll
          for (int j = 0; j < PW; ++j) {
            st_remote(a + 8 * G * j, dp * p[j]);
            if constexpr (ACC) st_remote(a + 8 * (kp + G * j), dp * pj[j]);
          }
          if (gl == 0) st_remote(remote_smem(nn + slot, ci), al);
        }
        for (int c = warp; c < nq; c += NW) {
          const double d = s_d[w + c];
          const int slot = sj * w + c;
          const uint32_t a = remote_smem(N + slot * ls, cj);
          double v[kCopy];
#pragma unroll
          for (int i = 0; i < kCopy; ++i)
            if (lane + 32 * i < (ACC ? 2 : 1) * kp) v[i] = d * Q[c * ls + lane + 32 * i];
#pragma unroll
          for (int i = 0; i < kCopy; ++i)
            if (lane + 32 * i < (ACC ? 2 : 1) * kp) st_remote(a + 8 * (lane + 32 * i), v[i]);
          if (lane == 0 && cl > 1) st_remote(remote_smem(nn + slot, cj), col.nrm[w + c]);
        }
      }
      if (t == nb - 2) {  // the sweep's largest values, to every CTA
        const int wc = __reduce_max_sync(0xffffffffu, __float_as_int(cosmax));  // non-negative: ordered like their bits
        const int wf = __reduce_max_sync(0xffffffffu, __float_as_int(fillmax));
        if (lane == 0) {
          atomicMax(&s_cos, wc);
          atomicMax(&s_fill, wf);
        }
        __syncthreads();
        if (tid < cl) {
          st_remote(remote_smem(&s_max[sweep & 1][rank][0], tid), s_cos);
          st_remote(remote_smem(&s_max[sweep & 1][rank][1], tid), s_fill);
        }
      }
      cluster_barrier(cl);
      if (cl > 1) set ^= 1;
    }
    int mc = 0, mf = 0;
    for (int i = 0; i < cl; ++i) {
      mc = max(mc, s_max[sweep & 1][i][0]);
      mf = max(mf, s_max[sweep & 1][i][1]);
    }
    __syncthreads();  // s_cos and s_fill are cleared next
    if (converged(k, tol, __int_as_float(mc), __int_as_float(mf))) {
      ++sweep;
      break;
    }
  }
  if (rank == 0 && tid == 0) {
    if (sweep == kMaxSweeps) atomicOr(status, 1);
    atomicMax(status + 1, sweep);
  }
  // Columns, norms and J (eigh: the normalised columns) back to the scratch.
  if (active) {
    tournament_pair(0, rank, nb, bi, bj);
    for (int c = warp; c < 2 * w; c += NW) {
      const int g = c < w ? bi * w + c : bj * w + c - w;
      if (c < w ? c >= bsize(bi) : c - w >= bsize(bj)) continue;
      const double* d = sm + set * set_len + (int64_t)c * ls;
      double s = 0.0, jj = 0.0;
      for (int x = lane; x < k; x += 32) {
        s = fma(d[x], d[x], s);
        if (ACC) jj = fma(d[kp + x], d[kp + x], jj);
      }
      s = sqrt(warp_sum(s));
      const double in = ACC ? 1.0 / sqrt(warp_sum(jj)) : 0.0;
      if (lane == 0) f.sv[g] = ACC ? s * in : s;
      for (int x = lane; x < k; x += 32) {
        if (ACC) f.W[(int64_t)g * ldw + x] = d[x] * in;
        f.J[(int64_t)g * k + x] = ACC ? d[kp + x] * in : d[x] / s;
      }
    }
  }
}

// ---------------------------------------------------------------------------
// Columns staged through L2
// ---------------------------------------------------------------------------

// Columns of blocks bi and bj of J times the accumulated rotations: J[:, cols] <-
// J[:, cols] Z, rows split over the warps in strips of 8 (a strip is read whole
// before it is written).  Z's column c starts at zs + c * ls, c < w for block bi's
// columns and w + (index) for block bj's.
template <int ZR>
__device__ __forceinline__ void apply_z(double* J, int k, int w, int p0, int np, int q0, int nq, const double* zs,
                                        int ls) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int kt = (2 * w + 3) / 4, nt = (2 * w + 7) / 8;
  for (int x0 = warp * 8; x0 < k; x0 += nwarps * 8) {
    const bool row = x0 + g < k;
    double a[ZR / 4];
#pragma unroll
    for (int i = 0; i < ZR / 4; ++i) {
      const int z = 4 * i + t4;
      const bool in = z < w ? z < np : z - w < nq;
      a[i] = (i < kt && row && in) ? __ldcg(J + (int64_t)(z < w ? p0 + z : q0 + z - w) * k + x0 + g) : 0.0;
    }
    for (int n = 0; n < nt; ++n) {
      double d0 = 0.0, d1 = 0.0;
      const double* zc = zs + (int64_t)(8 * n + g) * ls;
      const bool col = 8 * n + g < 2 * w;
#pragma unroll
      for (int i = 0; i < ZR / 4; ++i)
        if (i < kt) dmma(d0, d1, a[i], col ? zc[4 * i + t4] : 0.0);
      const int c = 8 * n + 2 * t4;  // output columns c, c + 1 of row g
      if (row) {
        if (c < w ? c < np : c - w < nq) J[(int64_t)(c < w ? p0 + c : q0 + c - w) * k + x0 + g] = d0;
        const int c1 = c + 1;
        if (c1 < w ? c1 < np : c1 - w < nq) J[(int64_t)(c1 < w ? p0 + c1 : q0 + c1 - w) * k + x0 + g] = d1;
      }
    }
  }
}

// One warp per column, at most PW elements of W (pw of them used) and ZR / 32 of the
// accumulator per lane; HOLD: the passing column stays in registers between its
// dot product and its update.  (Two columns of block bi per warp, which reads and
// writes a passing column once for two rotations, measured slower: 2570 cycles a
// round at k = 400 against 2 x 1190, and it spills from k = 576 on.)
template <int PW, int ZR, int NW, bool HOLD>
__global__ void __launch_bounds__(NW * 32, 1)
    jacobi_kernel(const SvdJob* __restrict__ jobs, double* __restrict__ work, const int64_t* __restrict__ work_off,
                  int32_t* __restrict__ status, int cl, int acc) {
  constexpr int PZ = ZR / 32, kp = 32 * PW, ls = col_stride(kp, ZR);
  const int rank = (int)(blockIdx.x % cl);
  const SvdJob S = jobs[blockIdx.x / cl];
  const int k = (int)S.k;
  const int64_t ldw = S.m > S.n ? S.m : S.n;
  if (k == 0) return;
  const bool acc_j = acc != 0;
  const FacWork f = fac_work(work + work_off[blockIdx.x / cl], ldw, k);
  double* W = f.W;
  double* J = f.J;
  int* words = reinterpret_cast<int*>(f.meta + 4);  // per sweep parity: cosine, fill (float bits)
  extern __shared__ __align__(16) double sm[];
  __shared__ double nrm[ZR], s_d[ZR], s_id[ZR];
  __shared__ int s_cos, s_fill;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  int w, nb;
  block_split(k, kp, cl, NW, ZR, w, nb);
  const int pw = (k + 31) / 32;
  const Columns col{nrm, s_d, s_id};
  auto bsize = [&](int b) {
    const int n = k - b * w;
    return n < 0 ? 0 : n < w ? n : w;
  };
  if (acc_j)
    for (int c = rank * NW + warp; c < k; c += cl * NW)
      for (int x = lane; x < k; x += 32) J[(int64_t)c * k + x] = x == c ? 1.0 : 0.0;
  if (rank == 0 && tid < 4) words[tid] = 0;
  Thresholds th;
  const double tol = make_thresholds(f, ldw, k, rank, cl, th);

  int sweep = 0;
  for (; sweep < kMaxSweeps && k > 1; ++sweep) {
    float cosmax = 0.0f, fillmax = 0.0f;
    if (tid == 0) {
      s_cos = 0;
      s_fill = 0;
    }
    for (int t = 0; t < nb - 1; ++t) {
      for (int i = rank; i < nb / 2; i += cl) {
        int bi, bj;
        tournament_pair(t, i, nb, bi, bj);
        const int np = bsize(bi), nq = bsize(bj), p0 = bi * w, q0 = bj * w;
        const bool within = t == 0;
        double* Q = sm + w * ls;  // block bj's columns; block bi's at sm while within its own pairs
        // Stage: block bj (and bi in the first round) in shared memory, one warp per
        // column; norms on the way.
        for (int c = within ? warp : w + warp; c < 2 * w; c += NW) {
          if (lane == 0) s_d[c] = s_id[c] = 1.0;
          if (c < w ? c >= np : c - w >= nq) continue;
          const double* src = W + (int64_t)(c < w ? p0 + c : q0 + c - w) * ldw;
          double* d = sm + c * ls;
          double s = 0.0;
          for (int x = lane; x < kp; x += 32) {
            const double v = x < k ? __ldcg(src + x) : 0.0;
            d[x] = v;
            s = fma(v, v, s);
          }
          if (acc_j)
            for (int z = lane; z < ZR; z += 32) d[kp + z] = z == c ? 1.0 : 0.0;
          s = warp_sum(s);
          if (lane == 0) nrm[c] = s;
        }
        if (within) {
          __syncthreads();
          rotate_within<32, PW, PZ, NW, false>(sm, ls, w, np, nq, col, acc_j, th, cosmax, fillmax);
        }
        // Cross pairs: warp i keeps column i of block bi in registers.
        double p[PW], pz[PZ];
        double al = 0.0, dp = 1.0, idp = 1.0;
        const bool own = warp < np;
        if (within) {
          const double* d = sm + (own ? warp : 0) * ls + lane;
#pragma unroll
          for (int j = 0; j < PW; ++j) p[j] = (own && j < pw) ? d[32 * j] : 0.0;
#pragma unroll
          for (int h = 0; h < PZ; ++h) pz[h] = (own && acc_j) ? d[kp + 32 * h] : 0.0;
          if (own) {
            al = nrm[warp];
            dp = s_d[warp];
            idp = s_id[warp];
          }
        } else {
          const double* d = W + (int64_t)(p0 + (own ? warp : 0)) * ldw;
#pragma unroll
          for (int j = 0; j < PW; ++j) {
            p[j] = (own && lane + 32 * j < k) ? __ldcg(d + lane + 32 * j) : 0.0;
            al = fma(p[j], p[j], al);
          }
          al = warp_sum(al);
#pragma unroll
          for (int h = 0; h < PZ; ++h) pz[h] = lane + 32 * h == warp ? 1.0 : 0.0;  // accumulator row of a block-bi column
        }
        __syncthreads();
        for (int r = 0; r < w; ++r) {
          int jq = warp + r;
          if (jq >= w) jq -= w;
          if (own && jq < nq) {
            double* q = Q + jq * ls + lane;
            double ga = 0.0, gb = 0.0;
            double qv[HOLD ? PW : 1];
#pragma unroll
            for (int j = 0; j < PW; ++j) {
              const double v = j < pw ? q[32 * j] : 0.0;
              if constexpr (HOLD) qv[j] = v;
              if (j & 1) gb = fma(p[j], v, gb);
              else ga = fma(p[j], v, ga);
            }
            const double be = nrm[w + jq], dq = s_d[w + jq], idq = s_id[w + jq];
            ga = warp_sum(ga + gb) * (dp * dq);
            Rotation R;
            if (rotation(al, be, ga, th, R, cosmax, fillmax)) {
              const double a = -R.t * (dq * idp), b = R.t * (dp * idq);
              if constexpr (!HOLD) asm volatile("" ::: "memory");  // read q again: holding it would spill
#pragma unroll
              for (int j = 0; j < PW; ++j)
                if (j < pw) {
                  const double u = p[j], v = HOLD ? qv[HOLD ? j : 0] : q[32 * j];
                  p[j] = fma(a, v, u);
                  q[32 * j] = fma(b, u, v);
                }
              if (acc_j) {
#pragma unroll
                for (int h = 0; h < PZ; ++h) {
                  const double u = pz[h], v = q[kp + 32 * h];
                  pz[h] = fma(a, v, u);
                  q[kp + 32 * h] = fma(b, u, v);
                }
              }
              al -= R.tg;
              dp *= R.c;
              idp = reciprocal_step(dp, idp * R.ic);
              if (lane == 0) {
                nrm[w + jq] = be + R.tg;
                const double d = dq * R.c;
                s_d[w + jq] = d;
                s_id[w + jq] = reciprocal_step(d, idq * R.ic);
              }
            }
          }
          __syncthreads();
        }
        // Back, scales taken out: block bi from registers, block bj from shared memory.
        if (own) {
          double* d = W + (int64_t)(p0 + warp) * ldw;
#pragma unroll
          for (int j = 0; j < PW; ++j)
            if (lane + 32 * j < k) d[lane + 32 * j] = dp * p[j];
          if (acc_j)
#pragma unroll
            for (int h = 0; h < PZ; ++h) sm[warp * ls + kp + 32 * h + lane] = dp * pz[h];
        }
        for (int c = warp; c < nq; c += NW) {
          double* d = Q + c * ls;
          const double dq = s_d[w + c];
          for (int x = lane; x < k; x += 32) W[(int64_t)(q0 + c) * ldw + x] = dq * d[x];
          if (acc_j)
            for (int z = lane; z < ZR; z += 32) d[kp + z] *= dq;
        }
        if (acc_j) {
          __syncthreads();
          apply_z<ZR>(J, k, w, p0, np, q0, nq, sm + kp, ls);
        }
        __syncthreads();  // the staging area is reused by the next pair
      }
      cluster_barrier(cl);
    }
    // The sweep's largest cosine before rotation and largest fill factor, over the cluster.
    const int wc = __reduce_max_sync(0xffffffffu, __float_as_int(cosmax));  // non-negative: ordered like their bits
    const int wf = __reduce_max_sync(0xffffffffu, __float_as_int(fillmax));
    if (lane == 0) {
      atomicMax(&s_cos, wc);
      atomicMax(&s_fill, wf);
    }
    __syncthreads();
    int* wd = words + 2 * (sweep & 1);
    if (tid == 0) {
      atomicMax(wd, s_cos);
      atomicMax(wd + 1, s_fill);
      if (rank == 0) {  // the other parity's words: last read before the previous barrier
        words[2 * ((sweep & 1) ^ 1)] = 0;
        words[2 * ((sweep & 1) ^ 1) + 1] = 0;
      }
    }
    cluster_barrier(cl);
    cosmax = __int_as_float(__ldcg(wd));
    fillmax = __int_as_float(__ldcg(wd + 1));
    cluster_barrier(cl);  // read by all before the next sweep clears or adds
    if (converged(k, tol, cosmax, fillmax)) {
      ++sweep;
      break;
    }
  }
  if (rank == 0 && tid == 0) {
    if (sweep == kMaxSweeps) atomicOr(status, 1);
    atomicMax(status + 1, sweep);
  }
  for (int c = rank * NW + warp; c < k; c += cl * NW) {
    double* wc = W + (int64_t)c * ldw;
    double* jc = J + (int64_t)c * k;
    double s = 0.0, jj = 0.0;
    for (int x = lane; x < k; x += 32) {
      const double v = __ldcg(wc + x), j = acc_j ? __ldcg(jc + x) : 0.0;
      s = fma(v, v, s);
      jj = fma(j, j, jj);
    }
    s = sqrt(warp_sum(s));
    const double in = acc_j ? 1.0 / sqrt(warp_sum(jj)) : 0.0;
    if (lane == 0) f.sv[c] = acc_j ? s * in : s;
    for (int x = lane; x < k; x += 32) {
      if (acc_j) {
        wc[x] = __ldcg(wc + x) * in;
        jc[x] = __ldcg(jc + x) * in;
      } else {
        jc[x] = __ldcg(wc + x) / s;  // eigh: the normalised columns
      }
    }
  }
}

// The kernel's limit on dynamic shared memory belongs to the device, not to the call:
// always the engine's bound, never this launch's own need, which another thread's
// larger launch would find between its own set and its launch.
template <class F, class... A>
cudaError_t launch_cluster(F fn, int njobs, int cl, int threads, size_t smem, cudaStream_t st, A... args) {
  if (smem > kJacobiSmem) return cudaErrorInvalidValue;
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kJacobiSmem);
  if (e != cudaSuccess) return e;
  if (cl > 8) {
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(njobs * cl));
  cfg.blockDim = dim3((unsigned)threads);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fn, args...);
}

// ---------------------------------------------------------------------------
// Outputs
// ---------------------------------------------------------------------------

template <class X>
__device__ __forceinline__ int64_t warp_argmax_abs(int64_t len, X&& x) {
  const int lane = threadIdx.x & 31;
  double best = -1.0;
  int64_t at = 0;
  for (int64_t i = lane; i < len; i += 32) {
    const double v = fabs(x(i));
    if (v > best) {
      best = v;
      at = i;
    }
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const double ob = __shfl_xor_sync(0xffffffffu, best, o);
    const int64_t oi = __shfl_xor_sync(0xffffffffu, at, o);
    if (ob > best || (ob == best && oi < at)) {
      best = ob;
      at = oi;
    }
  }
  return at;
}

constexpr int kFinishWarps = 8;

// Singular triplets in descending order, one warp per column: W's column over its
// norm and J's column (rows back from the places of the QR pass), the left vector's largest-|.| entry positive
// (factorize.rs:3836-3852, 3945-3962; the first maximum wins).
__global__ void __launch_bounds__(kFinishWarps * 32)
    svd_finish_kernel(const SvdJob* __restrict__ jobs, double* __restrict__ U, double* __restrict__ SV,
                      double* __restrict__ VH, double* __restrict__ work, const int64_t* __restrict__ work_off) {
  const SvdJob S = jobs[blockIdx.x];
  const int64_t m = S.m, n = S.n, k = S.k;
  const int lane = threadIdx.x & 31;
  const int64_t c = (int64_t)blockIdx.y * kFinishWarps + (threadIdx.x >> 5);
  if (c >= k) return;
  const bool wide = m < n;
  const int64_t ldw = wide ? n : m;
  const FacWork f = fac_work(work + work_off[blockIdx.x], ldw, k);
  // A sector with an entry that is not finite has values that are not: they come first,
  // so that every place is written.
  auto value = [&](int64_t x) { return isnan(f.sv[x]) ? DBL_MAX * 2.0 : f.sv[x]; };
  const double sc = f.sv[c], top = value(c);
  int64_t pos = 0;
  for (int64_t o = lane; o < k; o += 32) {
    const double so = value(o);
    pos += (so > top || (so == top && o < c)) ? 1 : 0;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) pos += __shfl_xor_sync(0xffffffffu, pos, o);
  const double inv = sc > 0.0 ? 1.0 / sc : 0.0;
  const double* wc = f.W + c * ldw;
  const double* jc = f.J + c * k;
  double* u = U + S.u_off + pos * m;
  double* vh = VH + S.v_off + pos;
  auto j = [&](int64_t x) { return jc[(int)f.rk[x]]; };
  auto left = [&](int64_t x) { return wide ? j(x) : wc[x]; };
  const double sign = left(warp_argmax_abs(m, left)) < 0.0 ? -1.0 : 1.0;
  for (int64_t x = lane; x < m; x += 32) u[x] = wide ? sign * j(x) : sign * wc[x] * inv;
  for (int64_t x = lane; x < n; x += 32) vh[x * k] = wide ? sign * wc[x] * inv : sign * j(x);
  if (lane == 0) SV[S.s_off + pos] = sc / f.meta[0];
}

// eigh runs on B = A + c I with c above the spectral radius rho: B is positive
// definite, its columns after the sweeps, divided by their norms lambda + c, are A's
// eigenvectors, and no rotations need accumulating.  Every error scales with
// c, so c is min(9/8 ||A||_F, 17/16 ||A^2||_inf^{1/2}): within a small factor of
// rho, where ||A||_F alone can be sqrt(n) times it.  Condition number of B: at
// most 33.
//
// Scan: scale (a power of two, largest entry below 1) and ||A||_F to meta[0],
// meta[1].  Sectors that fail the reference's Hermiticity check
// (normwise_hermitian, factorize.rs:5999-6021: ||A - A^T||_F <= 2 * 64 eps ||A||_F,
// every entry finite) set bit 1 of *status.
__device__ void eigh_scan(const double* a, int64_t n, const FacWork& f, int32_t* status) {
  __shared__ double red[2][32];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  double mx = 0.0;
  int finite = 1;
  for (int64_t i = tid; i < n * n; i += blockDim.x) {
    mx = fmax(mx, fabs(a[i]));
    finite &= isfinite(a[i]) ? 1 : 0;
  }
  finite = __syncthreads_and(finite);
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
  if (lane == 0) red[0][warp] = mx;
  __syncthreads();
  for (int i = 0; i < nwarps; ++i) mx = fmax(mx, red[0][i]);
  __syncthreads();
  double scale = 1.0;
  if (finite && mx > 0.0) {
    int e;
    frexp(mx, &e);
    scale = ldexp(1.0, e < -1022 ? 1022 : -e);
  }
  double f2 = 0.0, d2 = 0.0;
  for (int64_t i = tid; i < n * n; i += blockDim.x) {
    const int64_t c = i / n, r = i - c * n;
    const double v = a[i] * scale, d = v - a[c + r * n] * scale;
    f2 = fma(v, v, f2);
    d2 = fma(d, d, d2);
  }
  f2 = warp_sum(f2);
  d2 = warp_sum(d2);
  if (lane == 0) {
    red[0][warp] = f2;
    red[1][warp] = d2;
  }
  __syncthreads();
  if (tid == 0) {
    f2 = d2 = 0.0;
    for (int i = 0; i < nwarps; ++i) {
      f2 += red[0][i];
      d2 += red[1][i];
    }
    const double frob = sqrt(f2);
    if (!finite || sqrt(d2) > 128.0 * DBL_EPSILON * frob) atomicOr(status, 2);
    f.meta[0] = scale;
    f.meta[1] = frob;
    reinterpret_cast<unsigned long long*>(f.meta)[2] = 0ull;  // ||A^2||_inf, by bits
  }
}

__global__ void __launch_bounds__(1024) eigh_scan_kernel(const SvdJob* __restrict__ jobs, const double* __restrict__ A,
                                                         double* __restrict__ work,
                                                         const int64_t* __restrict__ work_off,
                                                         int32_t* __restrict__ status) {
  const SvdJob S = jobs[blockIdx.x];
  if (S.m == 0) return;
  eigh_scan(A + S.a_off, S.m, fac_work(work + work_off[blockIdx.x], S.m, S.m), status);
}

constexpr int kBoundWarps = 8;

// Row sums of |A^2| for the 16 rows from r0 on, by kBoundWarps warps (8 x 8 tiles on the
// FP64 tensor cores, A's symmetry giving rows as columns); their maximum to meta[2].
// Every thread of the CTA calls it (rows beyond n: no work).
__device__ void eigh_bound(const double* a, int n, const FacWork& f, int r0, int warp, double (*rows)[16]) {
  const double scale = f.meta[0];
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  double sum[2] = {0.0, 0.0};
  for (int c0 = 16 * warp; c0 < n && r0 < n; c0 += 16 * kBoundWarps) {
    double d[2][2][2] = {};
#pragma unroll 2
    for (int x0 = 0; x0 < n; x0 += 4) {
      const int x = x0 + t4;
      double u[2], v[2];
#pragma unroll
      for (int h = 0; h < 2; ++h) {
        const int r = r0 + 8 * h + g, c = c0 + 8 * h + g;
        u[h] = (x < n && r < n) ? __ldg(a + x + (int64_t)r * n) * scale : 0.0;
        v[h] = (x < n && c < n) ? __ldg(a + x + (int64_t)c * n) * scale : 0.0;
      }
#pragma unroll
      for (int h = 0; h < 2; ++h)
#pragma unroll
        for (int i = 0; i < 2; ++i) dmma(d[h][i][0], d[h][i][1], u[h], v[i]);
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 2; ++i) sum[h] += fabs(d[h][i][0]) + fabs(d[h][i][1]);
  }
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 1);
    sum[h] += __shfl_xor_sync(0xffffffffu, sum[h], 2);
    if (t4 == 0) rows[warp][8 * h + g] = sum[h];
  }
  __syncthreads();
  if (warp == 0 && lane < 16 && r0 < n) {
    double t = 0.0;
    for (int i = 0; i < kBoundWarps; ++i) t += rows[i][lane];
    atomicMax(reinterpret_cast<unsigned long long*>(f.meta) + 2, (unsigned long long)__double_as_longlong(t));
  }
}

__global__ void __launch_bounds__(kBoundWarps * 32)
    eigh_bound_kernel(const SvdJob* __restrict__ jobs, const double* __restrict__ A, double* __restrict__ work,
                      const int64_t* __restrict__ work_off) {
  const SvdJob S = jobs[blockIdx.x];
  if (16 * (int64_t)blockIdx.y >= S.m) return;
  __shared__ double rows[kBoundWarps][16];
  eigh_bound(A + S.a_off, (int)S.m, fac_work(work + work_off[blockIdx.x], S.m, S.m), 16 * (int)blockIdx.y,
             threadIdx.x >> 5, rows);
}

__device__ __forceinline__ double eigh_shift(const double* meta) {  // meta[2] comes from atomics
  const double c = fmin(1.125 * meta[1], 1.0625 * sqrt(__ldcg(meta + 2)));
  return c > 0.0 ? c : 1.0;  // a zero sector (or one that failed the scan)
}

__global__ void __launch_bounds__(256) eigh_form_kernel(const SvdJob* __restrict__ jobs, const double* __restrict__ A,
                                                        double* __restrict__ work,
                                                        const int64_t* __restrict__ work_off) {
  const SvdJob S = jobs[blockIdx.x];
  const int64_t n = S.m;
  if (n == 0) return;
  const FacWork f = fac_work(work + work_off[blockIdx.x], n, n);
  const double scale = f.meta[0], c = eigh_shift(f.meta);
  const double* a = A + S.a_off;
  for (int64_t i = (int64_t)blockIdx.y * 256 + threadIdx.x; i < n * n; i += (int64_t)gridDim.y * 256)
    f.W[i] = fma(a[i], scale, (i % n) == (i / n) ? c : 0.0);
}

// Sectors up to kEighSmall: scan, bound and shifted matrix in one launch, and all of the
// output stage in another, a CTA per sector.  In launches of their own the seven steps
// were most of the time (n = 4: 70 us, 45 so).
constexpr int64_t kEighSmall = 64;
constexpr int kSmallThreads = 512;

__global__ void __launch_bounds__(kSmallThreads) eigh_prepare_small_kernel(const SvdJob* __restrict__ jobs,
                                                                           const double* __restrict__ A,
                                                                           double* __restrict__ work,
                                                                           const int64_t* __restrict__ work_off,
                                                                           int32_t* __restrict__ status) {
  const SvdJob S = jobs[blockIdx.x];
  const int n = (int)S.m;
  if (n == 0) return;
  const FacWork f = fac_work(work + work_off[blockIdx.x], n, n);
  const double* a = A + S.a_off;
  __shared__ double rows[kSmallThreads / 32][16];
  eigh_scan(a, n, f, status);
  __syncthreads();  // meta
  const int warp = threadIdx.x >> 5, part = warp / kBoundWarps;
  for (int r0 = 0; r0 < n; r0 += 16 * (kSmallThreads / 32 / kBoundWarps)) {
    eigh_bound(a, n, f, r0 + 16 * part, warp % kBoundWarps, rows + part * kBoundWarps);
    __syncthreads();  // rows are used again, and the maxima are in place
  }
  const double scale = f.meta[0], c = eigh_shift(f.meta);
  for (int i = threadIdx.x; i < n * n; i += kSmallThreads) f.W[i] = fma(a[i], scale, (i % n) == (i / n) ? c : 0.0);
}

// One refinement step of the eigenvectors V (Ogita and Aishima, "Iterative
// refinement for symmetric eigenvalue decomposition", 2018): the sweeps' rounding
// errors, a random walk of about 12 n rotations at the scale of c, are replaced by
// those of three products.  With S = V^T A V and R = I - V^T V,
// lambda_i = S_ii / (V^T V)_ii and V <- V + V X,
// X_ij = (S_ij + lambda_j R_ij) / (lambda_j - lambda_i), written as R_ij / 2 plus an
// antisymmetric part (S symmetrised, so that its rounding cannot cost
// orthogonality over a small gap).  Where that part exceeds 1e-8 (a cluster within
// the errors) it is left out.

// Fragments of an m x 4 slice: rows g of a matrix walked down its columns (TR) or
// across them.  OWN: the matrix was written by this launch.
template <bool OWN>
__device__ __forceinline__ double frag(const double* a, int64_t ld, int r, int x, int n, bool tr) {
  if (r >= n || x >= n) return 0.0;
  const double* p = tr ? a + x + (int64_t)r * ld : a + r + (int64_t)x * ld;
  return OWN ? *p : __ldg(p);
}

constexpr int kRefineWarps = 4;  // a CTA takes a 32 x 32 tile, a warp 16 x 16 of it

// The 16 x 16 tile at r0, c0, by one warp.  step 0: W = scale A V.  step 1: X (into vec).
// step 2: W[:, rank] = V + V X.
template <bool OWN>
__device__ __forceinline__ void eigh_refine(const double* a, double* vec, const FacWork& f, int n, int r0, int c0,
                                            int step) {
  const int lane = threadIdx.x & 31, g = lane >> 2, t4 = lane & 3;
  if (r0 >= n || c0 >= n) return;
  const double* V = f.J;
  const double* lhs = step == 0 ? a : V;
  const double* rhs = step == 0 ? V : step == 1 ? f.W : vec;
  double d[2][2][2] = {}, e[2][2][2] = {}, t[2][2][2] = {};
#pragma unroll 2
  for (int x0 = 0; x0 < n; x0 += 4) {
    const int x = x0 + t4;
    double u[2], v[2], w[2], z[2];
#pragma unroll
    for (int h = 0; h < 2; ++h) {
      u[h] = frag<OWN>(lhs, n, r0 + 8 * h + g, x, n, step == 1);
      v[h] = frag<OWN>(rhs, n, c0 + 8 * h + g, x, n, true);
      w[h] = step == 1 ? frag<OWN>(V, n, c0 + 8 * h + g, x, n, true) : 0.0;
      z[h] = step == 1 ? frag<OWN>(f.W, n, r0 + 8 * h + g, x, n, true) : 0.0;
    }
#pragma unroll
    for (int h = 0; h < 2; ++h)
#pragma unroll
      for (int i = 0; i < 2; ++i) {
        dmma(d[h][i][0], d[h][i][1], u[h], v[i]);
        if (step == 1) {
          dmma(e[h][i][0], e[h][i][1], u[h], w[i]);
          dmma(t[h][i][0], t[h][i][1], z[h], w[i]);
        }
      }
  }
  const double scale = f.meta[0];
#pragma unroll
  for (int h = 0; h < 2; ++h)
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int r = r0 + 8 * h + g, c = c0 + 8 * i + 2 * t4 + q;
        if (r >= n || c >= n) continue;
        if (step == 0) {
          f.W[r + (int64_t)c * n] = scale * d[h][i][q];
        } else if (step == 1) {
          const double lr = f.sv[r], lc = f.sv[c], res = (r == c ? 1.0 : 0.0) - e[h][i][q];
          const double mid = 0.5 * (d[h][i][q] + t[h][i][q] + (lr + lc) * res), gap = lc - lr;
          double x = 0.5 * res;
          if (r != c && fabs(mid) < 1e-8 * fabs(gap)) x += mid / gap;
          vec[r + (int64_t)c * n] = x;
        } else {
          f.W[r + (int64_t)f.rk[c] * n] = V[r + (int64_t)c * n] + d[h][i][q];
        }
      }
}

// From step 1 on the outputs are written, so every kernel leaves a call that has
// failed alone (a sector that is not Hermitian, or sweeps that did not converge).
__global__ void __launch_bounds__(kRefineWarps * 32)
    eigh_refine_kernel(const SvdJob* __restrict__ jobs, const double* __restrict__ A, double* __restrict__ VEC,
                       double* __restrict__ work, const int64_t* __restrict__ work_off,
                       const int32_t* __restrict__ status, const int32_t* __restrict__ bad, int step) {
  if (factor_failed(status, bad)) return;
  const SvdJob S = jobs[blockIdx.x];
  const int n = (int)S.m, warp = threadIdx.x >> 5;
  if (n == 0) return;
  eigh_refine<false>(A + S.a_off, VEC + S.u_off, fac_work(work + work_off[blockIdx.x], n, n), n,
                     32 * (int)blockIdx.y + 16 * (warp & 1), 32 * (int)blockIdx.z + 16 * (warp >> 1), step);
}

// lambda_c = (v_c, A v_c) / (v_c, v_c) into sv; ranks by descending |lambda| (ties:
// ascending value, then index) into rk; the sorted values out.
__device__ void eigh_values(const FacWork& f, int n, double* val, double* mag) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  for (int c = warp; c < n; c += nwarps) {
    const double *v = f.J + (int64_t)c * n, *w = f.W + (int64_t)c * n;
    double s = 0.0, q = 0.0;
    for (int x = lane; x < n; x += 32) {
      s = fma(v[x], w[x], s);
      q = fma(v[x], v[x], q);
    }
    s = warp_sum(s);
    q = warp_sum(q);
    if (lane == 0) f.sv[c] = s / q;
  }
  __syncthreads();
  for (int c = warp; c < n; c += nwarps) {
    const double lc = f.sv[c], ac = fabs(lc);
    int pos = 0;
    for (int o = lane; o < n; o += 32) {
      const double lo = f.sv[o], ao = fabs(lo);
      pos += (ao > ac || (ao == ac && (lo < lc || (lo == lc && o < c)))) ? 1 : 0;
    }
    pos = __reduce_add_sync(0xffffffffu, pos);
    if (lane == 0) {
      f.rk[c] = (double)pos;
      val[pos] = lc / f.meta[0];
      if (mag) mag[pos] = ac / f.meta[0];
    }
  }
}

__global__ void __launch_bounds__(1024) eigh_values_kernel(const SvdJob* __restrict__ jobs, double* __restrict__ VAL,
                                                           double* __restrict__ MAG, double* __restrict__ work,
                                                           const int64_t* __restrict__ work_off,
                                                           const int32_t* __restrict__ status,
                                                           const int32_t* __restrict__ bad) {
  const SvdJob S = jobs[blockIdx.x];
  if (S.m == 0 || factor_failed(status, bad)) return;
  eigh_values(fac_work(work + work_off[blockIdx.x], S.m, S.m), (int)S.m, VAL + S.s_off, MAG ? MAG + S.s_off : nullptr);
}

// Column c of a sector, its largest-|.| entry positive (factorize.rs:3902-3913), by one warp.
__device__ __forceinline__ void eigh_column(const FacWork& f, int64_t n, int64_t c, double* vec) {
  const double* wc = f.W + c * n;
  const double sign = wc[warp_argmax_abs(n, [&](int64_t x) { return wc[x]; })] < 0.0 ? -1.0 : 1.0;
  for (int64_t x = threadIdx.x & 31; x < n; x += 32) vec[c * n + x] = sign * wc[x];
}

__global__ void __launch_bounds__(kFinishWarps * 32)
    eigh_finish_kernel(const SvdJob* __restrict__ jobs, double* __restrict__ VEC, double* __restrict__ work,
                       const int64_t* __restrict__ work_off, const int32_t* __restrict__ status,
                       const int32_t* __restrict__ bad) {
  if (factor_failed(status, bad)) return;
  const SvdJob S = jobs[blockIdx.x];
  const int64_t c = (int64_t)blockIdx.y * kFinishWarps + (threadIdx.x >> 5);
  if (c >= S.m) return;
  eigh_column(fac_work(work + work_off[blockIdx.x], S.m, S.m), S.m, c, VEC + S.u_off);
}

__global__ void __launch_bounds__(kSmallThreads)
    eigh_finish_small_kernel(const SvdJob* __restrict__ jobs, const double* __restrict__ A, double* __restrict__ VEC,
                             double* __restrict__ VAL, double* __restrict__ MAG, double* __restrict__ work,
                             const int64_t* __restrict__ work_off, const int32_t* __restrict__ status,
                             const int32_t* __restrict__ bad) {
  const SvdJob S = jobs[blockIdx.x];
  const int n = (int)S.m;
  if (n == 0 || factor_failed(status, bad)) return;
  const FacWork f = fac_work(work + work_off[blockIdx.x], n, n);
  const int warp = threadIdx.x >> 5, nwarps = kSmallThreads / 32, nt = (n + 15) / 16;
  double* vec = VEC + S.u_off;
  for (int step = 0; step < 3; ++step) {
    for (int t = warp; t < nt * nt; t += nwarps)
      eigh_refine<true>(A + S.a_off, vec, f, n, 16 * (t % nt), 16 * (t / nt), step);
    __syncthreads();
    if (step == 0) {
      eigh_values(f, n, VAL + S.s_off, MAG ? MAG + S.s_off : nullptr);
      __syncthreads();
    }
  }
  for (int c = warp; c < n; c += nwarps) eigh_column(f, n, c, vec);
}

}  // namespace

// CTAs per sector for a largest k of the launch: one while a round is a single
// wave of rotations on one SM (k <= 64), four while it is a few, then as many as
// the device can co-schedule.  A round costs its latency whatever the width, and
// a sweep takes k rounds plus an exchange per block pair, so wider clusters
// add exchanges where they no longer shorten the rounds.
int jacobi_cluster(int64_t k, int wide) { return k <= 64 ? 1 : k <= 128 ? 4 : wide > 0 ? 16 : 8; }

int64_t jacobi_class(int64_t k, int wide, bool acc_j) {
  if (k <= 64) return 64;    // 8 lanes a column
  if (k <= 128) return 128;  // 16 lanes
  if (wide > 0 && k <= (acc_j ? 320 : 448)) return acc_j ? 320 : 448;  // 32 lanes, columns resident
  for (int64_t c : {384, 448, 512, 608, 768, 1024})
    if (k <= c) return c;
  return kJacobiMaxK;
}

cudaError_t launch_jacobi(const SvdJob* jobs, int32_t njobs, int64_t max_k, double* work, const int64_t* work_off,
                          int32_t* status, bool acc_j, cudaStream_t st) {
  if (njobs == 0) return cudaSuccess;
  const int cl = jacobi_cluster(max_k, svd_wide_cluster_size());
  const int k = (int)max_k;
#define TNT_RING(g, pw, nw)                                                                                          \
  if (k <= g * pw) {                                                                                                 \
    const size_t smem = (size_t)(cl > 1 ? 4 : 2) * ring_width(k, cl) * ring_stride(g * pw, acc_j, g) * sizeof(double); \
    return acc_j ? launch_cluster(jacobi_ring_kernel<g, pw, nw, true>, njobs, cl, nw * 32, smem, st, jobs, work,      \
                                  work_off, status, cl)                                                              \
                 : launch_cluster(jacobi_ring_kernel<g, pw, nw, false>, njobs, cl, nw * 32, smem, st, jobs, work,     \
                                  work_off, status, cl);                                                             \
  }
#define TNT_RING_EIGH(g, pw, nw)                                                                                     \
  if (k <= g * pw && !acc_j)                                                                                         \
    return launch_cluster(jacobi_ring_kernel<g, pw, nw, false>, njobs, cl, nw * 32,                                  \
                          (size_t)4 * ring_width(k, cl) * ring_stride(g * pw, false, g) * sizeof(double), st, jobs,  \
                          work, work_off, status, cl);
#define TNT_STAGED(pw, zr, nw, hold)                                                                                  \
  if (k <= 32 * pw)                                                                                                  \
    return launch_cluster(jacobi_kernel<pw, zr, nw, hold>, njobs, cl, nw * 32, kJacobiSmem, st, jobs, work, work_off,  \
                          status, cl, acc_j ? 1 : 0);
  // Ring widths grow with k, so the largest sector's need covers the launch.
  TNT_RING(8, 2, 2) TNT_RING(8, 4, 4) TNT_RING(8, 6, 6) TNT_RING(8, 8, 8)
  TNT_RING(16, 6, 6) TNT_RING(16, 7, 7) TNT_RING(16, 8, 8)
  if (cl == 16) {
    TNT_RING(32, 5, 5) TNT_RING(32, 6, 6) TNT_RING(32, 7, 7) TNT_RING(32, 8, 8) TNT_RING(32, 9, 9) TNT_RING(32, 10, 10)
    TNT_RING_EIGH(32, 12, 12) TNT_RING_EIGH(32, 14, 14)
  }
  // Staged classes, on 16 CTAs: elements of a column per lane, accumulator rows, warps
  // (columns of one block), passing column held.  To 608 columns a round is one block pair
  // per CTA (block_split: 2 x 19 columns of 608 + 64 + 4 elements, 25688 of the 27648 doubles that
  // fit; 2 x 20 of 640 do not), so a warp for each of ceil(k / 32) columns and the accumulator's 2 w
  // rows rounded up to 32: 64 from 17 columns on.  Beyond, a CTA takes two pairs of 10 to 12
  // columns a round up to 768, three of 9 to 11 up to 1024, then five or six of 7 or 8 (on 8
  // CTAs 13 to 15, 10 to 12, 8): 15, 12 and 8 warps, within what shared memory (17, 13, 8) and the
  // registers of a lane's part of a column (48, 64, 96 of 136, 170, 255) allow.
  // From 17 elements a lane on a held column spills, so it is read again for its update.
  TNT_STAGED(12, 32, 16, true) TNT_STAGED(14, 32, 16, true) TNT_STAGED(16, 32, 16, true)
  TNT_STAGED(19, 64, 19, false) TNT_STAGED(24, 32, 15, false) TNT_STAGED(32, 32, 12, false) TNT_STAGED(48, 32, 8, false)
  return cudaErrorInvalidValue;
#undef TNT_RING
#undef TNT_RING_EIGH
#undef TNT_STAGED
}

cudaError_t launch_svd_finish(const SvdJob* jobs, int32_t njobs, int64_t max_k, double* u, double* s, double* vh,
                              double* work, const int64_t* work_off, cudaStream_t st) {
  if (njobs == 0 || max_k == 0) return cudaSuccess;
  const dim3 grid((unsigned)njobs, (unsigned)((max_k + kFinishWarps - 1) / kFinishWarps));
  svd_finish_kernel<<<grid, kFinishWarps * 32, 0, st>>>(jobs, u, s, vh, work, work_off);
  return cudaGetLastError();
}

cudaError_t launch_eigh_prepare(const SvdJob* jobs, int32_t njobs, int64_t max_n, const double* a, double* work,
                                const int64_t* work_off, int32_t* status, cudaStream_t st) {
  if (njobs == 0 || max_n == 0) return cudaSuccess;
  if (max_n <= kEighSmall) {
    eigh_prepare_small_kernel<<<njobs, kSmallThreads, 0, st>>>(jobs, a, work, work_off, status);
    return cudaGetLastError();
  }
  eigh_scan_kernel<<<njobs, 1024, 0, st>>>(jobs, a, work, work_off, status);
  eigh_bound_kernel<<<dim3((unsigned)njobs, (unsigned)((max_n + 15) / 16)), kBoundWarps * 32, 0, st>>>(jobs, a, work,
                                                                                                     work_off);
  const unsigned gy = (unsigned)std::min<int64_t>(64, (max_n * max_n + 1023) / 1024);
  eigh_form_kernel<<<dim3((unsigned)njobs, gy), 256, 0, st>>>(jobs, a, work, work_off);
  return cudaGetLastError();
}

cudaError_t launch_eigh_finish(const SvdJob* jobs, int32_t njobs, int64_t max_n, const double* a, double* vecs,
                               double* vals, double* mags, double* work, const int64_t* work_off,
                               const int32_t* status, const int32_t* bad, cudaStream_t st) {
  if (njobs == 0 || max_n == 0) return cudaSuccess;
  if (max_n <= kEighSmall) {
    eigh_finish_small_kernel<<<njobs, kSmallThreads, 0, st>>>(jobs, a, vecs, vals, mags, work, work_off, status, bad);
    return cudaGetLastError();
  }
  const unsigned nt = (unsigned)((max_n + 31) / 32);
  const dim3 tiles((unsigned)njobs, nt, nt);
  eigh_refine_kernel<<<tiles, kRefineWarps * 32, 0, st>>>(jobs, a, vecs, work, work_off, status, bad, 0);
  eigh_values_kernel<<<njobs, 1024, 0, st>>>(jobs, vals, mags, work, work_off, status, bad);
  eigh_refine_kernel<<<tiles, kRefineWarps * 32, 0, st>>>(jobs, a, vecs, work, work_off, status, bad, 1);
  eigh_refine_kernel<<<tiles, kRefineWarps * 32, 0, st>>>(jobs, a, vecs, work, work_off, status, bad, 2);
  const dim3 grid((unsigned)njobs, (unsigned)((max_n + kFinishWarps - 1) / kFinishWarps));
  eigh_finish_kernel<<<grid, kFinishWarps * 32, 0, st>>>(jobs, vecs, work, work_off, status, bad);
  return cudaGetLastError();
}

}  // namespace tnt
