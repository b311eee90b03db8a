// Householder QR of every sector on a thread-block cluster, and the products
// with its Q: tnt_qr, and the SVD's reduction to a triangular factor.
//
// X (rows x ncols) is reduced in panels of PWD reflectors (compact WY form,
// H_p ... H_{p + PWD - 1} = I - V T V^T).  The chain of reflectors is what
// bounds it: one CTA of the cluster factors a panel with one warp per column,
// the column in registers, so a reflector costs one barrier (the next column's
// warp updates, takes its norm and publishes the next reflector); then every CTA
// of the cluster updates its share of the trailing columns on the FP64 tensor
// cores (m8n8k4), V in its shared memory.  A cluster barrier stands between the
// two.  Products with Q need no exchange: each CTA carries its own columns
// through all panels.
//
// Measured: QR of the D = 1024 chain's bond matrix (six sectors of 293) 3.56 -> 0.79 ms
// of kernels against one CTA per sector.
//
// The SVD factors X^T = Q R once (twice for a rectangular sector, whose first pass
// makes it square; in the last pass the rows of X^T in falling order) and gives R^T to the
// Jacobi engine: its columns are graded and nearly orthogonal, which takes 9 to 10 sweeps
// where the sector's own columns take 11 (N(0, 1)) to 18 (a spectrum over three decades)
// at 104 x 104.
#include <algorithm>
#include <functional>

#include "panel.cuh"

namespace tnt {

namespace {

using namespace panel;

constexpr int kSlots = 16;   // partial products of the split first multiply
constexpr int kGroups = 4;   // 8-column groups updated at once by a CTA
constexpr int kSplits = kSlots / kGroups;  // of the rows, in every product: the order of its sum is the sector's own
constexpr int kW2Stride = 12;

// What a launch factors and where its reflectors, T and outputs live.
struct QrView {
  double* Y;    // reflectors below the diagonal, R on and above it
  double* T;    // one PWD x PWD block per panel, column-major
  int64_t ldy;
  int rows, ncols, nref;
};

__device__ __forceinline__ QrView qr_view(int mode, const SvdJob& S, const FacWork& f, double* U, double* VH) {
  QrView v;
  const bool wide = S.m < S.n;
  const int rows = (int)(wide ? S.n : S.m), k = (int)S.k;
  if (mode == kQrFactor) {
    v.Y = f.W;
    v.T = f.T[0];
    v.ldy = S.m;
    v.rows = (int)S.m;
    v.ncols = (int)S.n;
  } else if (mode == kQrSvdFirst) {  // the long side's output region holds rows x k
    v.Y = wide ? VH + S.v_off : U + S.u_off;
    v.T = f.T[0];
    v.ldy = rows;
    v.rows = rows;
    v.ncols = k;
  } else {  // the short side's output region holds k x k
    v.Y = wide ? U + S.u_off : VH + S.v_off;
    v.T = f.T[1];
    v.ldy = k;
    v.rows = k;
    v.ncols = k;
  }
  v.nref = k;
  return v;
}

template <int PWD, int PLR>
struct QrSmem {
  static constexpr int ldv = 32 * PLR + 4;  // = 4 mod 16: conflict-free MMA fragments
  static constexpr int slot = PWD * 8;
  double *V, *T, *W2, *part;
  __device__ explicit QrSmem(double* s) {
    V = s;
    T = V + PWD * ldv;
    W2 = T + PWD * PWD;
    part = W2 + kGroups * PWD * kW2Stride;
  }
  static constexpr size_t bytes() {
    return (size_t)(PWD * ldv + PWD * PWD + kGroups * PWD * kW2Stride + kSlots * slot) * sizeof(double);
  }
};

// Panel p0's V (unit diagonal, zeros above) and T into shared memory.
template <int PWD, int PLR>
__device__ void load_panel(const QrView& v, int p0, const QrSmem<PWD, PLR>& s) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
  const int pw = v.nref - p0 < PWD ? v.nref - p0 : PWD, nrows = v.rows - p0;
  const int xend = (nrows + 31) / 32 * 32;
  for (int j = warp; j < PWD; j += nwarps)
#pragma unroll 4
    for (int x = lane; x < xend; x += 32)
      s.V[j * s.ldv + x] = (j < pw && x > j && x < nrows) ? __ldcg(v.Y + p0 + x + (int64_t)(p0 + j) * v.ldy)
                           : (j < pw && x == j)           ? 1.0
                                                          : 0.0;
  for (int i = threadIdx.x; i < PWD * PWD; i += blockDim.x) s.T[i] = __ldcg(v.T + (int64_t)p0 * PWD + i);
  __syncthreads();
}

// X[p0.., group columns] <- (I - V M V^T) X for the CTA's column groups
// first, first + step, ... (8 columns each, below ncols); M = T^T or T.
template <int PWD, int PLR, bool TRANS>
__device__ void apply_block(double* X, int64_t ldx, int c0, int ncols, int p0, int nrows, int first, int step,
                            const QrSmem<PWD, PLR>& s) {
  constexpr int MT = PWD / 8;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  const int ngroups = (ncols - c0 + 7) / 8;
  for (int base = first; base < ngroups; base += kGroups * step) {
    int gb = (ngroups - base + step - 1) / step;
    if (gb > kGroups) gb = kGroups;
    auto group_col = [&](int q) { return c0 + 8 * (base + q * step); };
    // Warps left over by fewer groups take fewer of the reflectors each.
    const int parts = gb * kSplits * 4 <= nwarps && MT == 4 ? 4 : gb * kSplits * 2 <= nwarps ? 2 : 1;
    if (warp < gb * kSplits * parts) {  // W1 = V^T X, the rows split over kSplits warps per group
      const int q = warp % gb, sp = warp / gb % kSplits, part = warp / (gb * kSplits);
      const int col = group_col(q) + g;
      const double* x0 = X + p0 + (int64_t)col * ldx;
      const int kst = (nrows + 3) / 4, per = (kst + kSplits - 1) / kSplits;
      const int k0 = sp * per, k1 = k0 + per < kst ? k0 + per : kst;
      const int m0 = part * (MT / parts), m1 = m0 + MT / parts;
      double acc[MT][2];
#pragma unroll
      for (int m = 0; m < MT; ++m) acc[m][0] = acc[m][1] = 0.0;
      const bool live = col < ncols;
      for (int st = k0; st < k1; st += 4) {
        double b[4];
#pragma unroll
        for (int u = 0; u < 4; ++u) {
          const int x = 4 * (st + u) + t4;
          b[u] = (live && st + u < k1 && x < nrows) ? __ldcg(x0 + x) : 0.0;
        }
#pragma unroll
        for (int u = 0; u < 4; ++u)
          if (st + u < k1)
#pragma unroll
            for (int m = 0; m < MT; ++m)
              if (m >= m0 && m < m1) dmma(acc[m][0], acc[m][1], s.V[(8 * m + g) * s.ldv + 4 * (st + u) + t4], b[u]);
      }
      double* o = s.part + (sp * gb + q) * s.slot;
#pragma unroll
      for (int m = 0; m < MT; ++m)
        if (m >= m0 && m < m1) {
          o[(8 * m + g) * 8 + 2 * t4] = acc[m][0];
          o[(8 * m + g) * 8 + 2 * t4 + 1] = acc[m][1];
        }
    }
    __syncthreads();
    for (int e = tid; e < gb * s.slot; e += blockDim.x) {
      double w = s.part[e];
      for (int sp = 1; sp < kSplits; ++sp) w += s.part[sp * gb * s.slot + e];
      s.part[e] = w;
    }
    __syncthreads();
    for (int e = tid; e < gb * s.slot; e += blockDim.x) {  // W2 = -M W1
      const int q = e / s.slot, r = (e % s.slot) >> 3, c = e & 7;
      const double* w1 = s.part + q * s.slot + c;
      double a0 = 0.0, a1 = 0.0;
#pragma unroll
      for (int l = 0; l < PWD; l += 2) {
        a0 = fma(TRANS ? s.T[l + r * PWD] : s.T[r + l * PWD], w1[8 * l], a0);
        a1 = fma(TRANS ? s.T[l + 1 + r * PWD] : s.T[r + (l + 1) * PWD], w1[8 * l + 8], a1);
      }
      s.W2[(q * PWD + r) * kW2Stride + c] = -(a0 + a1);
    }
    __syncthreads();
    const int rt = (nrows + 7) / 8;
    for (int it = warp; it < gb * rt; it += nwarps) {  // X += V W2
      const int q = it / rt, x0 = 8 * (it - q * rt);
      const int col = group_col(q) + 2 * t4, x = x0 + g;
      double* xp = X + p0 + x + (int64_t)col * ldx;
      const bool in0 = x < nrows && col < ncols, in1 = x < nrows && col + 1 < ncols;
      double d0 = in0 ? __ldcg(xp) : 0.0, d1 = in1 ? __ldcg(xp + ldx) : 0.0;
#pragma unroll
      for (int i = 0; i < PWD / 4; ++i)
        dmma(d0, d1, s.V[(4 * i + t4) * s.ldv + x0 + g], s.W2[(q * PWD + 4 * i + t4) * kW2Stride + g]);
      if (in0) *xp = d0;
      if (in1) xp[ldx] = d1;
    }
    __syncthreads();
  }
}

// T of the panel in s.V from the Gram matrix V^T V: 8 x 8 diagonal blocks
// column by column, then T = [T1, -T1 G12 T2; 0, T2] twice (once for PWD = 16).
template <int PWD, int PLR>
__device__ void panel_t(const QrSmem<PWD, PLR>& s, const double* taus, int nrows) {
  constexpr int NT = PWD / 8, NTILES = NT * (NT + 1) / 2;
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nwarps = blockDim.x >> 5;
  const int g = lane >> 2, t4 = lane & 3;
  double* G = s.W2;  // PWD x PWD, column-major
  static_assert(kGroups * PWD * kW2Stride >= PWD * PWD + PWD * PWD / 2, "Gram matrix and the combine buffer fit");
  const int avail = nwarps < kSlots * PWD / 8 ? nwarps : kSlots * PWD / 8, splits = avail / NTILES;
  if (warp < splits * NTILES) {
    const int tile = warp % NTILES, sp = warp / NTILES;
    int tj = 0, at = tile;
    while (at > tj) at -= ++tj;
    const int ti = at;
    const int kst = (nrows + 3) / 4, per = (kst + splits - 1) / splits;
    const int k1 = (sp + 1) * per < kst ? (sp + 1) * per : kst;
    double d0 = 0.0, d1 = 0.0;
#pragma unroll 4
    for (int st = sp * per; st < k1; ++st)
      dmma(d0, d1, s.V[(8 * ti + g) * s.ldv + 4 * st + t4], s.V[(8 * tj + g) * s.ldv + 4 * st + t4]);
    double* o = s.part + (sp * NTILES + tile) * 64;
    o[g * 8 + 2 * t4] = d0;
    o[g * 8 + 2 * t4 + 1] = d1;
  }
  for (int i = tid; i < PWD * PWD; i += blockDim.x) s.T[i] = 0.0;
  __syncthreads();
  for (int e = tid; e < NTILES * 64; e += blockDim.x) {
    const int tile = e >> 6, r = (e >> 3) & 7, c = e & 7;
    int tj = 0, at = tile;
    while (at > tj) at -= ++tj;
    double v = 0.0;
    for (int sp = 0; sp < splits; ++sp) v += s.part[(sp * NTILES + tile) * 64 + (e & 63)];
    G[8 * at + r + (8 * tj + c) * PWD] = v;
  }
  __syncthreads();
  if (warp < NT && lane < 8) {
    const int b = 8 * warp;
    double row[8];  // row b + lane of the block
#pragma unroll
    for (int c = 0; c < 8; ++c) {
      double acc = 0.0;
#pragma unroll
      for (int l = 0; l < c; ++l)
        if (l >= lane) acc = fma(row[l], G[b + l + (b + c) * PWD], acc);
      row[c] = c < lane ? 0.0 : c == lane ? taus[b + c] : -taus[b + c] * acc;
      s.T[b + lane + (b + c) * PWD] = row[c];
    }
  }
  __syncthreads();
  double* M = G + PWD * PWD;
  for (int sz = 8; sz < PWD; sz *= 2) {
    const int total = sz * PWD / 2;  // (PWD / 2 sz) blocks of sz x sz
    for (int e = tid; e < total; e += blockDim.x) {
      const int blk = e / (sz * sz), r = e % sz, c = (e / sz) % sz, a = blk * 2 * sz, b = a + sz;
      double v = 0.0;
      for (int l = 0; l <= c; ++l) v = fma(G[a + r + (b + l) * PWD], s.T[b + l + (b + c) * PWD], v);
      M[e] = v;
    }
    __syncthreads();
    for (int e = tid; e < total; e += blockDim.x) {
      const int blk = e / (sz * sz), r = e % sz, c = (e / sz) % sz, a = blk * 2 * sz, b = a + sz;
      double v = 0.0;
      for (int l = r; l < sz; ++l) v = fma(s.T[a + r + (a + l) * PWD], M[blk * sz * sz + l + c * sz], v);
      s.T[a + r + (b + c) * PWD] = -v;
    }
    __syncthreads();
  }
}

template <int PWD, int PLR>
__global__ void __launch_bounds__(PWD * 32, 1)
    qr_factor_kernel(const SvdJob* __restrict__ jobs, const double* __restrict__ A, double* __restrict__ U,
                     double* __restrict__ VH, double* __restrict__ work, const int64_t* __restrict__ work_off, int cl,
                     int mode) {
  const int rank = (int)(blockIdx.x % cl);
  const SvdJob S = jobs[blockIdx.x / cl];
  if (S.k == 0 || (mode == kQrSvdFirst && S.m == S.n)) return;
  const bool wide = S.m < S.n, square = S.m == S.n;
  const int64_t ldw = wide ? S.n : S.m;
  const FacWork f = fac_work(work + work_off[blockIdx.x / cl], ldw, S.k);
  const QrView v = qr_view(mode, S, f, U, VH);
  extern __shared__ __align__(16) double sm[];
  const QrSmem<PWD, PLR> s(sm);
  __shared__ double taus[PWD];
  __shared__ double red[PWD];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const double* a = A + S.a_off;
  const int64_t gt = (int64_t)rank * blockDim.x + tid, gn = (int64_t)cl * blockDim.x;

  // The SVD's last pass takes the rows of X by falling largest entry: Householder QR
  // is accurate row by row only in that order, and X's rows (a sector's columns, which
  // can stand decades apart) carry the relative accuracy of the small singular values.
  // Without it ten decades in random order left 1e-8 of a value, with it 1e-14.
  // Largest entries to sv, and every CTA counts every row's place (k^2 comparisons in
  // shared memory); places to rk, for svd_finish_kernel.
  double mx = 0.0;
  const int* place = reinterpret_cast<const int*>(s.V + v.nref);
  if (mode == kQrSvdSecond) {
    const QrView f1 = qr_view(kQrSvdFirst, S, f, U, VH);
    const double* rows = square ? a : f1.Y;  // row x of X: contiguous from x * ld
    const int64_t ld = square ? S.m : f1.ldy;
    for (int x = rank * PWD + warp; x < v.rows; x += cl * PWD) {
      double top = 0.0;
      for (int c = lane; c < (square ? v.ncols : x + 1); c += 32) top = fmax(top, fabs(__ldcg(rows + c + x * ld)));
#pragma unroll
      for (int o = 16; o > 0; o >>= 1) top = fmax(top, __shfl_xor_sync(0xffffffffu, top, o));
      if (lane == 0) f.sv[x] = top;
    }
    cluster_barrier(cl);
    static_assert(PWD * QrSmem<PWD, PLR>::ldv >= 2 * 32 * PLR, "keys and places fit V");
    for (int x = tid; x < v.rows; x += PWD * 32) s.V[x] = __ldcg(f.sv + x);
    __syncthreads();
    for (int x = tid; x < v.rows; x += PWD * 32) {
      const double top = s.V[x];
      int at = 0;
      for (int o = 0; o < v.rows; ++o) at += (s.V[o] > top || (s.V[o] == top && o < x)) ? 1 : 0;
      reinterpret_cast<int*>(s.V + v.nref)[x] = at;
      if (rank == 0) f.rk[x] = (double)at;
      if (at == 0) red[0] = top;
    }
    __syncthreads();
    mx = red[0];
  } else if (mode == kQrSvdFirst) {
    for (int64_t i = gt; i < S.m * S.n; i += gn) mx = fmax(mx, fabs(a[i]));
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) mx = fmax(mx, __shfl_xor_sync(0xffffffffu, mx, o));
    if (lane == 0) red[warp] = mx;
    unsigned long long* slot = reinterpret_cast<unsigned long long*>(f.meta + 2);
    if (rank == 0 && tid == 0) *slot = 0ull;
    cluster_barrier(cl);
    if (tid == 0) {
      for (int i = 1; i < PWD; ++i) mx = fmax(mx, red[i]);
      atomicMax(slot, (unsigned long long)__double_as_longlong(mx));  // non-negative doubles order like their bits
    }
    cluster_barrier(cl);
    mx = __longlong_as_double((long long)__ldcg(slot));
  }
  // The SVD scales the sector by a power of two to a largest magnitude in
  // [1/2, 1), so no product of its Jacobi sweeps leaves the range of a float.
  double scale = 1.0;
  if (mode == kQrSvdFirst || (mode == kQrSvdSecond && square)) {
    if (mx > 0.0 && mx <= DBL_MAX) {
      int e;
      frexp(mx, &e);
      // 2^-e can overflow for a subnormal maximum: stop at the largest power of two.
      scale = ldexp(1.0, e < -1022 ? 1022 : -e);
    }
    if (rank == 0 && tid == 0) f.meta[0] = scale;
  }

  // X into Y, walked so that reads are contiguous.
  const int64_t total = (int64_t)v.rows * v.ncols;
  if (mode == kQrFactor || (mode == kQrSvdFirst && !wide)) {
    for (int64_t i = gt; i < total; i += gn) v.Y[i] = a[i] * scale;  // ldy = rows
  } else if (mode == kQrSvdFirst || square) {  // A^T: X(x, c) = A[c + x ncols]
    for (int64_t i = gt; i < total; i += gn) {
      const int64_t x = i / v.ncols, c = i - x * v.ncols;
      v.Y[(mode == kQrSvdSecond ? place[x] : x) + c * v.ldy] = a[i] * scale;
    }
  } else {  // R1^T of the first pass, lower triangular
    const QrView f1 = qr_view(kQrSvdFirst, S, f, U, VH);
    for (int64_t i = gt; i < total; i += gn) {
      const int64_t x = i / v.ncols, c = i - x * v.ncols;
      v.Y[place[x] + c * v.ldy] = c <= x ? __ldcg(f1.Y + c + x * f1.ldy) : 0.0;
    }
  }
  cluster_barrier(cl);

  for (int p0 = 0, pi = 0; p0 < v.nref; p0 += PWD, ++pi) {
    const int pw = v.nref - p0 < PWD ? v.nref - p0 : PWD, nrows = v.rows - p0;
    const bool last = p0 + pw >= v.ncols;  // nothing trails
    const bool owner = pi % cl == rank;
    if (owner) {
      const int nq = (nrows + 31) / 32;  // registers in use: rows fall by PWD per panel
      double y[PLR];
      double* yc = v.Y + p0 + (int64_t)(p0 + warp) * v.ldy;
      const bool own = warp < pw;
#pragma unroll
      for (int q = 0; q < PLR; ++q) {
        const int x = lane + 32 * q;
        y[q] = (own && x < nrows) ? __ldcg(yc + x) : 0.0;
      }
      if (!own) {
        if (warp < PWD) taus[warp] = 0.0;
#pragma unroll
        for (int q = 0; q < PLR; ++q)
          if (q < nq) s.V[warp * s.ldv + lane + 32 * q] = 0.0;
      }
      for (int j = 0; j < pw; ++j) {
        double* vj = s.V + j * s.ldv + lane;
        if (warp == j) {
          double ss = lane > j ? y[0] * y[0] : 0.0, s2 = 0.0;
#pragma unroll
          for (int q = 1; q < PLR; ++q)
            if (q < nq) {
              if (q & 1) s2 = fma(y[q], y[q], s2);
              else ss = fma(y[q], y[q], ss);
            }
          const double sigma = warp_sum(ss + s2);
          const double alpha = __shfl_sync(0xffffffffu, y[0], j);
          double t = 0.0, beta = alpha, inv = 0.0;
          if (sigma > 0.0) {
            const double nrm = sqrt(fma(alpha, alpha, sigma));
            beta = alpha >= 0.0 ? -nrm : nrm;
            t = (beta - alpha) / beta;
            inv = 1.0 / (alpha - beta);
          }
          y[0] = lane > j ? y[0] * inv : y[0];
          vj[0] = lane > j ? y[0] : lane == j ? 1.0 : 0.0;
          if (lane == j) y[0] = beta;
#pragma unroll
          for (int q = 1; q < PLR; ++q)
            if (q < nq) {
              y[q] *= inv;
              vj[32 * q] = y[q];
            }
          if (lane == 0) taus[j] = t;
        }
        __syncthreads();
        const double t = taus[j];
        if (warp > j && own && t != 0.0) {
          // v is read again for the update where holding it would spill
          constexpr bool kHold = PLR <= 8;
          double d = 0.0, d2 = 0.0;
          double vv[kHold ? PLR : 1];
#pragma unroll
          for (int q = 0; q < PLR; ++q)
            if (q < nq) {
              const double x = vj[32 * q];
              if constexpr (kHold) vv[q] = x;
              if (q & 1) d2 = fma(x, y[q], d2);
              else d = fma(x, y[q], d);
            }
          d = warp_sum(d + d2) * t;
          if constexpr (!kHold) asm volatile("" ::: "memory");
#pragma unroll
          for (int q = 0; q < PLR; ++q)
            if (q < nq) y[q] = fma(-d, kHold ? vv[kHold ? q : 0] : vj[32 * q], y[q]);
        }
      }
      if (own) {
#pragma unroll
        for (int q = 0; q < PLR; ++q) {
          const int x = lane + 32 * q;
          if (x < nrows) yc[x] = y[q];
        }
      }
      panel_t(s, taus, nrows);
      for (int i = tid; i < PWD * PWD; i += blockDim.x) v.T[(int64_t)p0 * PWD + i] = s.T[i];
    }
    cluster_barrier(cl);
    if (last) continue;
    if (!owner) load_panel(v, p0, s);
    apply_block<PWD, PLR, true>(v.Y, v.ldy, p0 + pw, v.ncols, p0, nrows, rank, cl, s);
    cluster_barrier(cl);
  }

  if (mode == kQrFactor) {  // R (k x n) with a non-negative diagonal
    double* r = VH + S.v_off;
    for (int64_t i = gt; i < (int64_t)v.nref * v.ncols; i += gn) {
      const int64_t c = i / v.nref, row = i - c * v.nref;
      const double sgn = __ldcg(v.Y + row + row * v.ldy) < 0.0 ? -1.0 : 1.0;
      r[i] = row <= c ? sgn * __ldcg(v.Y + row + c * v.ldy) : 0.0;
    }
  } else if (mode == kQrSvdSecond) {  // W = R^T over zeros
    for (int64_t i = gt; i < ldw * v.nref; i += gn) {
      const int64_t c = i / ldw, x = i - c * ldw;
      f.W[i] = (x >= c && x < v.nref) ? __ldcg(v.Y + c + x * v.ldy) : 0.0;
    }
  }
}

// X <- Q X on the CTA's columns (8-column groups cta, cta + ncta, ...):
// kQrFactor forms Q itself (X = the columns of I with R's diagonal signs),
// kQrSvdFirst takes W to the sector's long side, kQrSvdSecond takes J.
template <int PWD, int PLR>
__global__ void __launch_bounds__(PWD * 32, 1)
    qr_apply_kernel(const SvdJob* __restrict__ jobs, double* __restrict__ U, double* __restrict__ VH,
                    double* __restrict__ work, const int64_t* __restrict__ work_off, int ncta, int mode) {
  const SvdJob S = jobs[blockIdx.x / ncta];
  const int cta = (int)(blockIdx.x % ncta);
  if (S.k == 0 || (mode == kQrSvdFirst && S.m == S.n)) return;
  const int64_t ldw = S.m > S.n ? S.m : S.n;
  const FacWork f = fac_work(work + work_off[blockIdx.x / ncta], ldw, S.k);
  const QrView v = qr_view(mode, S, f, U, VH);
  extern __shared__ __align__(16) double sm[];
  const QrSmem<PWD, PLR> s(sm);
  const int k = v.nref;
  if (8 * cta >= k) return;
  double* X = mode == kQrFactor ? U + S.u_off : mode == kQrSvdFirst ? f.W : f.J;
  const int64_t ldx = v.rows;
  if (mode == kQrFactor) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5, nwarps = blockDim.x >> 5;
    for (int c = warp; c < k; c += nwarps) {
      if ((c >> 3) % ncta != cta) continue;
      const double d = v.Y[c + c * v.ldy] < 0.0 ? -1.0 : 1.0;
      for (int x = lane; x < v.rows; x += 32) X[x + (int64_t)c * ldx] = x == c ? d : 0.0;
    }
    __syncthreads();
  }
  for (int p0 = (k - 1) / PWD * PWD; p0 >= 0; p0 -= PWD) {
    int first = cta;
    if (mode == kQrFactor)
      while (8 * first + 7 < p0) first += ncta;  // columns left of the panel are still those of I
    if (8 * first >= k) continue;
    load_panel(v, p0, s);
    apply_block<PWD, PLR, false>(X, ldx, 0, k, p0, v.rows - p0, first, ncta, s);
  }
}

template <int PWD, int PLR>
cudaError_t factor_class(const SvdJob* jobs, int32_t njobs, const double* a, double* u, double* vh, double* work,
                         const int64_t* work_off, int cl, int mode, cudaStream_t st) {
  auto fn = qr_factor_kernel<PWD, PLR>;
  constexpr size_t smem = QrSmem<PWD, PLR>::bytes();
  static_assert(smem <= 226 * 1024, "panel fits shared memory");
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  if (cl > 8) {
    e = cudaFuncSetAttribute(fn, cudaFuncAttributeNonPortableClusterSizeAllowed, 1);
    if (e != cudaSuccess) return e;
  }
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(njobs * cl));
  cfg.blockDim = dim3(PWD * 32);
  cfg.dynamicSmemBytes = smem;
  cfg.stream = st;
  cudaLaunchAttribute attr[1];
  attr[0].id = cudaLaunchAttributeClusterDimension;
  attr[0].val.clusterDim.x = (unsigned)cl;
  attr[0].val.clusterDim.y = 1;
  attr[0].val.clusterDim.z = 1;
  cfg.attrs = attr;
  cfg.numAttrs = 1;
  return cudaLaunchKernelEx(&cfg, fn, jobs, a, u, vh, work, work_off, cl, mode);
}

template <int PWD, int PLR>
cudaError_t apply_class(const SvdJob* jobs, int32_t njobs, int64_t max_k, double* u, double* vh, double* work,
                        const int64_t* work_off, int mode, cudaStream_t st) {
  auto fn = qr_apply_kernel<PWD, PLR>;
  constexpr size_t smem = QrSmem<PWD, PLR>::bytes();
  cudaError_t e = cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) return e;
  const int ncta = (int)((max_k + 8 * kGroups - 1) / (8 * kGroups));  // up to four column groups each
  fn<<<(unsigned)(njobs * ncta), PWD * 32, smem, st>>>(jobs, u, vh, work, work_off, ncta, mode);
  return cudaGetLastError();
}

}  // namespace

// A launch's cluster width, by a longest-first deal of its sectors.  A CTA fills its SM;
// eight clusters of 16, 16 of 8, 36 of 4 or 74 of 2 fit 148 SMs in their GPCs.  A sector is a
// chain of reflectors of about 2 us each, which no width shortens, and trailing updates,
// which the width divides.  300 x 300 sectors, 1 / 10 / 37 / 80 of them, in ms: 16 CTAs
// 0.79 / 1.48 / 4.40 / 8.80, 8 0.82 / 0.82 / 2.42 / 4.83, 4 0.88 / 0.89 / 1.83 / 2.86,
// 2 1.01 / 1.02 / 1.18 / 2.34, 1 1.27 / 1.27 / 1.44 / 1.75.
int qr_cluster(const std::vector<QrSize>& sizes, int wide) {
  struct Width {
    int cl, fits;
  };
  int best = 1;
  double best_t = 0.0;
  std::vector<double> load;
  for (const Width& w : {Width{1, 148}, Width{2, 74}, Width{4, 36}, Width{8, 16}, Width{16, 8}}) {
    if (w.cl > 8 && wide <= 0) break;
    load.assign(w.fits, 0.0);  // a heap, the first cluster to be free in front
    double top = 0.0;
    for (const QrSize& z : sizes) {
      const double r = (double)z.rows, n = (double)std::min(z.rows, z.cols);
      const double t = 2.0 * n * (1.0 + r / 1500.0) + 1.9e-5 * r * (double)z.cols * n / w.cl;
      std::pop_heap(load.begin(), load.end(), std::greater<double>());
      top = std::max(top, load.back() += t);
      std::push_heap(load.begin(), load.end(), std::greater<double>());
    }
    if (w.cl == 1 || top < 0.98 * best_t) {  // a wider cluster also pays for its barriers
      best = w.cl;
      best_t = top;
    }
  }
  return best;
}

cudaError_t launch_qr_factor(const SvdJob* jobs, int32_t njobs, int64_t max_rows, int cl, int mode, const double* a,
                             double* u, double* vh, double* work, const int64_t* work_off, cudaStream_t st) {
  if (njobs == 0) return cudaSuccess;
  if (max_rows <= 64) return factor_class<32, 2>(jobs, njobs, a, u, vh, work, work_off, cl, mode, st);
  if (max_rows <= 256) return factor_class<32, 8>(jobs, njobs, a, u, vh, work, work_off, cl, mode, st);
  if (max_rows <= 640) return factor_class<32, 20>(jobs, njobs, a, u, vh, work, work_off, cl, mode, st);
  if (max_rows <= kQrMaxRows) return factor_class<16, 44>(jobs, njobs, a, u, vh, work, work_off, cl, mode, st);
  return cudaErrorInvalidValue;
}

cudaError_t launch_qr_apply(const SvdJob* jobs, int32_t njobs, int64_t max_rows, int64_t max_k, int mode, double* u,
                            double* vh, double* work, const int64_t* work_off, cudaStream_t st) {
  if (njobs == 0) return cudaSuccess;
  if (max_rows <= 64) return apply_class<32, 2>(jobs, njobs, max_k, u, vh, work, work_off, mode, st);
  if (max_rows <= 256) return apply_class<32, 8>(jobs, njobs, max_k, u, vh, work, work_off, mode, st);
  if (max_rows <= 640) return apply_class<32, 20>(jobs, njobs, max_k, u, vh, work, work_off, mode, st);
  if (max_rows <= kQrMaxRows) return apply_class<16, 44>(jobs, njobs, max_k, u, vh, work, work_off, mode, st);
  return cudaErrorInvalidValue;
}

}  // namespace tnt
