// Recoupling transform kernel: dst = alpha * U . P(src) + beta * dst per group.
//
// Replaces the Host replay of tenet-operations/src/transform_replay.rs:
// Single blocks (4428-4517, a permuted strided copy times one coefficient) and
// Multi groups (4519-4800: pack every source block of a group into a column,
// one GEMM with U^T, scatter back).  Both compute, for every element position
// of the group's common block shape, dst_d = alpha * sum_s U[d, s] src_s (+ beta
// dst_d); here that sum is formed in registers, so each source element is read
// once and each destination element written once.
//
// A group's blocks are viewed as d0 x C matrices: d0 = the extent of
// destination axis 0 (stride 1 in every destination block, contiguous runs of
// the codomain), C = the product of the other extents ("columns").  A CTA
// takes a tile of columns; it stages the group's coefficients, the block
// offsets/strides and the multi-index of each of its columns in shared
// memory, then maps threads as (W lanes along axis 0) x (256/W columns), with
// W the power of two covering min(d0, 32).  Address arithmetic per element is
// a few multiply-adds from shared memory; no division in the element loop.
//
// Tiles come sorted by kernel path (xform_kind); one launch deals its CTAs to the
// paths, and each path has its own loop over its tiles: abelian copies
// with short rows unroll across columns; abelian copies with long rows and
// groups up to 4 x 4 (the SU(2) case) walk each column down axis 0 with
// paired 16-byte accesses where aligned; transposing abelian copies (source
// strided along axis 0, contiguous along another axis) stage planes through
// shared memory in a kernel of their own; everything else takes the general loop.
#include "kernels.cuh"

namespace tnt {

namespace {

constexpr int kXThreads = 256;
constexpr int kRegSrc = 8;        // source values cached in registers per element
constexpr int kSmemCoef = 1024;   // coefficients staged in shared memory
constexpr int kSmemEntries = 48;  // source + destination entries staged in shared memory
constexpr int kMaxTileCols = 256; // columns per tile (multi-indices staged in shared memory)
constexpr int kSmallGroup = 4;    // groups up to 4 x 4 take the register path

struct SmemEntry {
  int64_t offset;
  int64_t strides[kMaxRank];
};

struct XShared {
  XGroup g;
  XTile tile;
  double U[kSmemCoef];
  SmemEntry ent[kSmemEntries];
  uint16_t cidx[kMaxTileCols][kMaxRank - 1];
  int64_t cbase[kMaxTileCols][2];  // abelian groups: per-column source / destination base offsets
};

// Tiles first, first + step, .. of one kernel path.
template <int KIND>
__device__ __forceinline__ void xform_tiles(XShared& sh, const XTile* __restrict__ tiles, int32_t ntiles, int32_t first,
                                            int32_t step, const XGroup* __restrict__ groups,
                                            const XEntry* __restrict__ src_e, const XEntry* __restrict__ dst_e,
                                            const double* __restrict__ coef, const double* __restrict__ src,
                                            double* __restrict__ dst, double alpha, double beta) {
  XGroup& g = sh.g;
  XTile& tile = sh.tile;
  auto& U = sh.U;
  auto& ent = sh.ent;
  auto& cidx = sh.cidx;
  auto& cbase = sh.cbase;
  const int tid = threadIdx.x;
  for (int32_t t = first; t < ntiles; t += step) {
    __syncthreads();
    if (tid == 0) {
      tile = tiles[t];
      g = groups[tile.group];
    }
    __syncthreads();
    const int nsrc = g.nsrc, ndst = g.ndst, rank = g.rank;
    const int ncoef = nsrc * ndst;
    const bool coef_smem = ncoef <= kSmemCoef;
    const bool ent_smem = nsrc + ndst <= kSmemEntries;
    const int d0 = rank > 0 ? g.dims[0] : 1;
    const int ncols = (int)tile.count;
    if (coef_smem)
      for (int i = tid; i < ncoef; i += kXThreads) U[i] = coef[g.coef_off + i];
    if (ent_smem) {
      for (int i = tid; i < nsrc + ndst; i += kXThreads) {
        const XEntry& e = i < nsrc ? src_e[g.src_first + i] : dst_e[g.dst_first + (i - nsrc)];
        ent[i].offset = e.offset;
#pragma unroll
        for (int k = 0; k < kMaxRank; ++k) ent[i].strides[k] = k < rank ? e.strides[k] : 0;
      }
    }
    const bool abelian = KIND == 0 || KIND == 3;
    for (int c = tid; c < ncols; c += kXThreads) {
      int64_t col = tile.start + c;
      int64_t sb = 0, db = 0;
      const XEntry* es = abelian ? &src_e[g.src_first] : nullptr;
      const XEntry* ed = abelian ? &dst_e[g.dst_first] : nullptr;
#pragma unroll
      for (int k = 1; k < kMaxRank; ++k) {
        uint16_t v = 0;
        if (k < rank) {
          const int32_t dk = g.dims[k];
          const int64_t q = col / dk;
          v = (uint16_t)(col - q * dk);
          col = q;
          if (abelian) {
            sb += (int64_t)v * es->strides[k];
            db += (int64_t)v * ed->strides[k];
          }
        }
        cidx[c][k - 1] = v;
      }
      if (abelian) {
        cbase[c][0] = es->offset + sb;
        cbase[c][1] = ed->offset + db;
      }
    }
    __syncthreads();

    const double* Ug = coef_smem ? U : coef + g.coef_off;
    int W = 1;
    while (W < d0 && W < 32) W <<= 1;
    const int H = kXThreads / W;
    const int tx = tid % W, ty = tid / W;

    if constexpr (KIND == 0) {
      // Abelian groups: a scaled permuted copy.  Each thread issues kUnroll
      // independent loads before its stores so enough bytes are in flight to
      // cover HBM latency; column bases come precomputed from shared memory.
      constexpr int kUnroll = 8;
      const double scale = alpha * Ug[0];
      const int64_t s0 = src_e[g.src_first].strides[0];
      for (int i0 = tx; i0 < d0; i0 += W) {
        const int64_t si = (int64_t)i0 * s0;
        for (int cl0 = ty; cl0 < ncols; cl0 += H * kUnroll) {
          double v[kUnroll];
          int64_t od[kUnroll];
#pragma unroll
          for (int u = 0; u < kUnroll; ++u) {
            const int cl = cl0 + u * H;
            od[u] = -1;
            if (cl < ncols) {
              v[u] = __ldg(src + cbase[cl][0] + si);
              od[u] = cbase[cl][1] + i0;
            }
          }
          if (beta != 0.0) {  // added in place before the first is written
#pragma unroll
            for (int u = 0; u < kUnroll; ++u)
              if (od[u] >= 0) v[u] = fma(beta, dst[od[u]], scale * v[u]);
          } else {
#pragma unroll
            for (int u = 0; u < kUnroll; ++u) v[u] *= scale;
          }
#pragma unroll
          for (int u = 0; u < kUnroll; ++u)
            if (od[u] >= 0) dst[od[u]] = v[u];
        }
      }
      continue;
    }

    if constexpr (KIND == 3) {
      // Abelian groups with long rows: a scaled copy of each column down
      // destination axis 0 (column bases precomputed in shared memory).  Each
      // thread issues four loads before its stores, 16-byte pairs when the
      // source runs along that axis and both bases are 16-byte aligned.
      const double u = alpha * Ug[0];
      const int64_t s0 = src_e[g.src_first].strides[0];
      for (int cl = ty; cl < ncols; cl += H) {
        const int64_t sbase = cbase[cl][0], dbase = cbase[cl][1];
        const bool vec = s0 == 1 && (d0 & 1) == 0 &&
                         ((reinterpret_cast<uintptr_t>(src + sbase) | reinterpret_cast<uintptr_t>(dst + dbase)) & 15) == 0;
        if (vec) {
          const int np = d0 >> 1;
          const double2* sp = reinterpret_cast<const double2*>(src + sbase);
          double2* op = reinterpret_cast<double2*>(dst + dbase);
          for (int p0 = tx; p0 < np; p0 += 4 * W) {
            double2 v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (p0 + q * W < np) v[q] = __ldg(sp + p0 + q * W);
            if (beta != 0.0) {  // added in place before the first is written
#pragma unroll
              for (int q = 0; q < 4; ++q)
                if (p0 + q * W < np) {
                  const double2 b = op[p0 + q * W];
                  v[q] = make_double2(fma(beta, b.x, u * v[q].x), fma(beta, b.y, u * v[q].y));
                }
            } else {
#pragma unroll
              for (int q = 0; q < 4; ++q) v[q] = make_double2(u * v[q].x, u * v[q].y);
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (p0 + q * W < np) op[p0 + q * W] = v[q];
          }
        } else {
          for (int i0 = tx; i0 < d0; i0 += 4 * W) {
            double v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (i0 + q * W < d0) v[q] = __ldg(src + sbase + (int64_t)(i0 + q * W) * s0);
            double* op = dst + dbase + i0;
            if (beta != 0.0) {
#pragma unroll
              for (int q = 0; q < 4; ++q)
                if (i0 + q * W < d0) v[q] = fma(beta, op[q * W], u * v[q]);
            } else {
#pragma unroll
              for (int q = 0; q < 4; ++q) v[q] *= u;
            }
#pragma unroll
            for (int q = 0; q < 4; ++q)
              if (i0 + q * W < d0) op[q * W] = v[q];
          }
        }
      }
      continue;
    }

    if constexpr (KIND == 1) {
      // Small recoupling groups (the SU(2) case, and abelian groups with long
      // rows): per column, the block base offsets are formed once and the loop
      // runs down destination axis 0 (stride 1 in every destination block).
      // When every source is contiguous along that axis and every base is
      // 16-byte aligned, elements move in pairs (16-byte loads and stores).
      for (int cl = ty; cl < ncols; cl += H) {
        int64_t sb[kSmallGroup], db[kSmallGroup];
        bool vec = (d0 & 1) == 0;
#pragma unroll
        for (int e = 0; e < kSmallGroup; ++e) {
          sb[e] = 0;
          db[e] = 0;
          if (e < nsrc) {
            const SmemEntry& en = ent[e];
            int64_t o = en.offset;
#pragma unroll
            for (int k = 1; k < kMaxRank; ++k) o += (int64_t)cidx[cl][k - 1] * en.strides[k];
            sb[e] = o;
            vec = vec && en.strides[0] == 1 && ((reinterpret_cast<uintptr_t>(src + o) & 15) == 0);
          }
          if (e < ndst) {
            const SmemEntry& en = ent[nsrc + e];
            int64_t o = en.offset;
#pragma unroll
            for (int k = 1; k < kMaxRank; ++k) o += (int64_t)cidx[cl][k - 1] * en.strides[k];
            db[e] = o;
            vec = vec && ((reinterpret_cast<uintptr_t>(dst + o) & 15) == 0);
          }
        }
        if (vec) {
          const int np = d0 >> 1;
          for (int p0 = tx; p0 < np; p0 += 2 * W) {
            const int p1 = p0 + W;
            const bool two = p1 < np;
            double2 v0[kSmallGroup], v1[kSmallGroup];
#pragma unroll
            for (int e = 0; e < kSmallGroup; ++e) {
              v0[e] = make_double2(0.0, 0.0);
              v1[e] = make_double2(0.0, 0.0);
              if (e < nsrc) {
                const double2* sp = reinterpret_cast<const double2*>(src + sb[e]);
                v0[e] = __ldg(sp + p0);
                if (two) v1[e] = __ldg(sp + p1);
              }
            }
#pragma unroll
            for (int d = 0; d < kSmallGroup; ++d) {
              if (d < ndst) {
                double2 a0 = make_double2(0.0, 0.0), a1 = make_double2(0.0, 0.0);
#pragma unroll
                for (int e = 0; e < kSmallGroup; ++e)
                  if (e < nsrc) {
                    const double u = alpha * Ug[d * nsrc + e];
                    a0.x = fma(u, v0[e].x, a0.x);
                    a0.y = fma(u, v0[e].y, a0.y);
                    a1.x = fma(u, v1[e].x, a1.x);
                    a1.y = fma(u, v1[e].y, a1.y);
                  }
                double2* o = reinterpret_cast<double2*>(dst + db[d]);
                if (beta == 0.0) {
                  o[p0] = a0;
                  if (two) o[p1] = a1;
                } else {
                  double2 b0 = o[p0];
                  o[p0] = make_double2(fma(beta, b0.x, a0.x), fma(beta, b0.y, a0.y));
                  if (two) {
                    double2 b1 = o[p1];
                    o[p1] = make_double2(fma(beta, b1.x, a1.x), fma(beta, b1.y, a1.y));
                  }
                }
              }
            }
          }
          continue;
        }
        for (int i0 = tx; i0 < d0; i0 += 2 * W) {
          const int i1 = i0 + W;
          const bool two = i1 < d0;
          double v0[kSmallGroup], v1[kSmallGroup];
#pragma unroll
          for (int e = 0; e < kSmallGroup; ++e) {
            v0[e] = 0.0;
            v1[e] = 0.0;
            if (e < nsrc) {
              const int64_t s0 = ent[e].strides[0];
              v0[e] = __ldg(src + sb[e] + (int64_t)i0 * s0);
              if (two) v1[e] = __ldg(src + sb[e] + (int64_t)i1 * s0);
            }
          }
#pragma unroll
          for (int d = 0; d < kSmallGroup; ++d) {
            if (d < ndst) {
              double a0 = 0.0, a1 = 0.0;
#pragma unroll
              for (int e = 0; e < kSmallGroup; ++e)
                if (e < nsrc) {
                  const double u = Ug[d * nsrc + e];
                  a0 = fma(u, v0[e], a0);
                  a1 = fma(u, v1[e], a1);
                }
              double* o = dst + db[d] + i0;
              if (beta == 0.0) {
                o[0] = alpha * a0;
                if (two) o[W] = alpha * a1;
              } else {
                o[0] = fma(beta, o[0], alpha * a0);
                if (two) o[W] = fma(beta, o[W], alpha * a1);
              }
            }
          }
        }
      }
      continue;
    }

    if constexpr (KIND == 2) {
    for (int cl = ty; cl < ncols; cl += H) {
      int32_t ci[kMaxRank - 1];
#pragma unroll
      for (int k = 0; k < kMaxRank - 1; ++k) ci[k] = cidx[cl][k];
      for (int i0 = tx; i0 < d0; i0 += W) {
        auto place = [&](int e, bool is_src) -> int64_t {
          if (ent_smem) {
            const SmemEntry& en = ent[is_src ? e : nsrc + e];
            int64_t off = en.offset + (int64_t)i0 * en.strides[0];
#pragma unroll
            for (int k = 1; k < kMaxRank; ++k) off += (int64_t)ci[k - 1] * en.strides[k];
            return off;
          }
          const XEntry& en = is_src ? src_e[g.src_first + e] : dst_e[g.dst_first + e];
          int64_t off = en.offset + (int64_t)i0 * en.strides[0];
          for (int k = 1; k < rank; ++k) off += (int64_t)ci[k - 1] * en.strides[k];
          return off;
        };
        if (nsrc == 1 && ndst == 1) {  // abelian groups: one scaled permuted copy
          const double v = alpha * Ug[0] * __ldg(src + place(0, true));
          const int64_t o = place(0, false);
          dst[o] = beta == 0.0 ? v : fma(beta, dst[o], v);
        } else if (nsrc == 0) {
          for (int d = 0; d < ndst; ++d) {
            const int64_t o = place(d, false);
            dst[o] = beta == 0.0 ? 0.0 : beta * dst[o];
          }
        } else if (nsrc <= kRegSrc) {
          double v[kRegSrc];
#pragma unroll
          for (int s = 0; s < kRegSrc; ++s)
            if (s < nsrc) v[s] = __ldg(src + place(s, true));
          for (int d = 0; d < ndst; ++d) {
            double acc = 0.0;
#pragma unroll
            for (int s = 0; s < kRegSrc; ++s)
              if (s < nsrc) acc = fma(Ug[d * nsrc + s], v[s], acc);
            const int64_t o = place(d, false);
            dst[o] = beta == 0.0 ? alpha * acc : fma(beta, dst[o], alpha * acc);
          }
        } else {
          for (int d = 0; d < ndst; ++d) {
            double acc = 0.0;
            for (int s = 0; s < nsrc; ++s) acc = fma(Ug[d * nsrc + s], __ldg(src + place(s, true)), acc);
            const int64_t o = place(d, false);
            dst[o] = beta == 0.0 ? alpha * acc : fma(beta, dst[o], alpha * acc);
          }
        }
      }
    }
    }
  }
}

// Where each path's tiles and CTAs begin.
struct XParts {
  int32_t tile[kXKinds + 1], cta[kXKinds + 1];
};

// All tiles but the transposing ones, in one launch whose CTAs are dealt to the
// paths in turn.  With a launch per path a permute of small tensors paid three of
// them and three tails: 17 us in a Lanczos step on 34 MB intermediates, now 11; the largest permute of the full-size network 101 -> 94.
__global__ void __launch_bounds__(kXThreads, 3) xform_kernel(const XTile* __restrict__ tiles, XParts parts,
                                                          const XGroup* __restrict__ groups,
                                                          const XEntry* __restrict__ src_e,
                                                          const XEntry* __restrict__ dst_e,
                                                          const double* __restrict__ coef,
                                                          const double* __restrict__ src, double* __restrict__ dst,
                                                          double alpha, double beta) {
  __shared__ XShared sh;
  const int32_t b = (int32_t)blockIdx.x;
#define TNT_XFORM_PATH(k)                                                                                       \
  if (b < parts.cta[k + 1]) {                                                                                   \
    xform_tiles<k>(sh, tiles + parts.tile[k], parts.tile[k + 1] - parts.tile[k], b - parts.cta[k],              \
                   parts.cta[k + 1] - parts.cta[k], groups, src_e, dst_e, coef, src, dst, alpha, beta);         \
    return;                                                                                                     \
  }
  TNT_XFORM_PATH(0) TNT_XFORM_PATH(1) TNT_XFORM_PATH(2) TNT_XFORM_PATH(3)
#undef TNT_XFORM_PATH
}

__device__ __forceinline__ void cp_async8(double* smem, const double* gmem) {
  asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem)
               : "memory");
}

// Transposing copies (one source and one destination block, source stride 1 along
// a destination axis k* > 0, not along axis 0).  A tile's planes of r rows (axis 0)
// x jn columns (axis k*) are loaded along k* and written along axis 0, both
// contiguous, through shared memory with rows of odd length.
//
// Bound by memory: what it takes is enough bytes in flight and few instructions
// per element.  Loads are cp.async into the second of two buffers while the first
// is written, positions step by additions (two divisions per tile and thread, not
// two per element), and folded axes make the planes large.  0.6 GB U(1) tensor,
// (a, b | c, d) -> (c, d | a, b): 186 -> 129 us, of 93 at the copy rate.
template <bool kAdd>
__global__ void __launch_bounds__(kXThreads, 3) xform_transpose_kernel(
    const XTrTile* __restrict__ tiles, int32_t ntiles, const XGroup* __restrict__ groups,
    const XEntry* __restrict__ src_e, const XEntry* __restrict__ dst_e, const double* __restrict__ coef,
    const double* __restrict__ src, double* __restrict__ dst, double alpha, double beta, int cap) {
  extern __shared__ double tbuf[];              // [2][cap]
  __shared__ int64_t pbase[3][kTrPlanes][2];    // first element of each plane, source and destination
  const int tid = threadIdx.x;

  auto place = [&](const XTrTile& T, int slot) {
    if (tid >= T.np) return;
    int64_t sb = T.src, db = T.dst;
    if (T.np > 1) {
      const XGroup& g = groups[T.group];
      const XEntry &es = src_e[g.src_first], &ed = dst_e[g.dst_first];
      int64_t rem = T.first + tid;
      for (int k = 1; k < g.rank; ++k) {
        if (k == T.ks) continue;
        const int32_t dk = g.dims[k];
        const int64_t q = rem / dk, v = rem - q * dk;
        rem = q;
        sb += v * es.strides[k];
        db += v * ed.strides[k];
      }
    }
    pbase[slot][tid][0] = sb;
    pbase[slot][tid][1] = db;
  };
  // Visits the elements e = tid, tid + 256, .. of np planes of b x a, position x
  // along a (fastest), y along b, plane p.  np * a * b <= 4096, so the quotients by
  // float reciprocal are exact: the error is below 2^-11, under half of 1 / a.
  auto walk = [&](int a, int b, int np, auto&& f) {
    const int n = np * a * b;
    const float inv_a = 1.0f / (float)a, inv_b = 1.0f / (float)b;
    int y = __float2int_rz(((float)tid + 0.5f) * inv_a), x = tid - y * a;
    const int dy = __float2int_rz(((float)kXThreads + 0.5f) * inv_a), dx = kXThreads - dy * a;
    if (np == 1) {
#pragma unroll 4
      for (int e = tid; e < n; e += kXThreads) {
        f(x, y, 0);
        x += dx;
        y += dy;
        if (x >= a) {
          x -= a;
          ++y;
        }
      }
      return;
    }
    int p = __float2int_rz(((float)y + 0.5f) * inv_b);
    y -= p * b;
    const int dp = __float2int_rz(((float)dy + 0.5f) * inv_b), dyb = dy - dp * b;
#pragma unroll 4
    for (int e = tid; e < n; e += kXThreads) {
      f(x, y, p);
      x += dx;
      y += dyb;
      p += dp;
      if (x >= a) {
        x -= a;
        ++y;
      }
      if (y >= b) {
        y -= b;
        ++p;
      }
    }
  };
  auto load = [&](const XTrTile& T, double* buf, int slot) {
    const int jp = T.jn | 1, ps = T.r * jp;
    if (T.np == 1) {
      const double* q = src + T.src;
      walk(T.jn, T.r, 1, [&](int j, int i, int) { cp_async8(buf + i * jp + j, q + i * T.s0 + j); });
    } else {
      walk(T.jn, T.r, T.np, [&](int j, int i, int p) {
        cp_async8(buf + p * ps + i * jp + j, src + pbase[slot][p][0] + i * T.s0 + j);
      });
    }
  };
  auto store = [&](const XTrTile& T, const double* buf, int slot) {
    const int jp = T.jn | 1, ps = T.r * jp;
    const double u = alpha * coef[T.coef];
    auto visit = [&](auto&& put) {
      if (T.np == 1) {
        double* q = dst + T.dst;
        walk(T.r, T.jn, 1, [&](int i, int j, int) { put(q + j * T.dks + i, u * buf[i * jp + j]); });
      } else {
        walk(T.r, T.jn, T.np, [&](int i, int j, int p) {
          put(dst + pbase[slot][p][1] + j * T.dks + i, u * buf[p * ps + i * jp + j]);
        });
      }
    };
    if constexpr (!kAdd) {
      visit([](double* at, double x) { *at = x; });
    } else {
      // Four elements are read before they are written: otherwise every load waits for
      // the store before it (24 MB of ragged U(1) blocks 20 us, now 14).
      double* at[4];
      double v[4];
      int have = 0;
      auto flush = [&] {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (q < have) v[q] = fma(beta, *at[q], v[q]);
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (q < have) *at[q] = v[q];
        have = 0;
      };
      visit([&](double* o, double x) {
#pragma unroll
        for (int q = 0; q < 4; ++q)
          if (q == have) {
            at[q] = o;
            v[q] = x;
          }
        if (++have == 4) flush();
      });
      flush();
    }
  };

  int32_t t = blockIdx.x;
  if (t >= ntiles) return;
  XTrTile cur = tiles[t], nxt = cur;
  if (t + (int32_t)gridDim.x < ntiles) nxt = tiles[t + gridDim.x];
  place(cur, 0);
  __syncthreads();
  load(cur, tbuf, 0);
  asm volatile("cp.async.commit_group;\n" ::: "memory");
  for (int it = 0;; ++it) {
    const bool more = t + (int32_t)gridDim.x < ntiles;
    // Three sets of plane positions: a thread that is ahead writes the next one
    // while another still stores with this one's.
    if (more) place(nxt, (it + 1) % 3);
    __syncthreads();  // positions are in place, and the other buffer has been written out
    if (more) load(nxt, tbuf + ((it + 1) & 1) * cap, (it + 1) % 3);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 1;\n" ::: "memory");
    __syncthreads();  // every thread's part of this tile has arrived
    const XTrTile done = cur;
    cur = nxt;
    t += gridDim.x;
    if (t + (int32_t)gridDim.x < ntiles) nxt = tiles[t + gridDim.x];
    store(done, tbuf + (it & 1) * cap, it % 3);
    if (!more) break;
  }
}

}  // namespace

cudaError_t launch_xform(const DevXform& x, double* dst, const double* src, double alpha, double beta,
                         cudaStream_t stream) {
  if (x.ntiles == 0 && x.ntr == 0) return cudaSuccess;
  int dev = 0, sms = 148;
  cudaGetDevice(&dev);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (x.ntiles > 0) {
    XParts parts{};
    for (int k = 0; k < kXKinds; ++k) {
      const int32_t n = x.kind_count[k];
      parts.tile[k + 1] = parts.tile[k] + n;
      parts.cta[k + 1] = parts.cta[k] + (n < sms * 8 ? n : sms * 8);
    }
    xform_kernel<<<parts.cta[kXKinds], kXThreads, 0, stream>>>(x.tiles, parts, x.groups, x.src, x.dst, x.coef, src, dst,
                                                              alpha, beta);
  }
  if (x.ntr > 0) {
    const int smem = 2 * x.tr_cap * (int)sizeof(double);
    const auto kernel = beta != 0.0 ? xform_transpose_kernel<true> : xform_transpose_kernel<false>;
    if (smem > 40 * 1024) {  // beyond what a launch may ask for without it, next to the plane positions
      // Always the largest tile's need: the limit is the device's, and another thread's plan
      // may be launched between this call and the launch.
      const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 2 * kTrCap * (int)sizeof(double));
      if (e != cudaSuccess) return e;
    }
    const int grid = x.ntr < sms * 3 ? x.ntr : sms * 3;
    kernel<<<grid, kXThreads, smem, stream>>>(x.tr_tiles, x.ntr, x.groups, x.src, x.dst, x.coef, src, dst, alpha, beta,
                                              x.tr_cap);
  }
  return cudaGetLastError();
}

}  // namespace tnt
