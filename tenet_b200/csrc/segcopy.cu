// Strided block copies with optional row scaling, many blocks per launch.
//
// Used to publish truncated factorisation outputs in place: every segment
// copies a rows x cols column-major block (source leading dimension src_ld)
// into a destination block (leading dimension dst_ld), optionally scaling row
// i by scales[scale_off + i] (the S Vh product of a truncated SVD).
#include "kernels.cuh"

namespace tnt {

namespace {

// Bound by HBM for large blocks, by the launch for small ones.  kSplit CTAs share
// a segment (one CTA of 256 threads took 0.2 ms over a 586 x 293 block), lanes run
// down the rows, and short columns share a warp.  Columns too few for the warps of
// kSplit CTAs are cut into pieces of at least 128 rows (100000 x 1: 521 us with a warp
// a column, 113 with one CTA, now 9).
constexpr int kSplit = 16;

__global__ void __launch_bounds__(256) segcopy_kernel(const SegCopy* __restrict__ segs, const double* __restrict__ src,
                                                      double* __restrict__ dst, const double* __restrict__ scales) {
  const SegCopy S = segs[blockIdx.x];
  int w = 1;  // lanes per column
  while (w < 32 && w < S.rows) w <<= 1;
  const int per = 256 / w, i0 = threadIdx.x % w;
  const double* s = src + S.src_off;
  double* d = dst + S.dst_off;
  auto copy = [&](int64_t j, int64_t first, int64_t end) {
#pragma unroll 4
    for (int64_t i = first; i < end; i += w) {
      double v = s[i + j * S.src_ld];
      if (S.scale_off >= 0) v *= scales[S.scale_off + i];
      d[i + j * S.dst_ld] = v;
    }
  };
  const int64_t from = (int64_t)blockIdx.y * per + threadIdx.x / w, step = (int64_t)kSplit * per;
  if (S.cols > 0 && S.cols * 2 <= step && S.rows >= 256) {  // then w = 32
    const int64_t fill = step / S.cols, most = S.rows / 128, pieces = fill < most ? fill : most;
    const int64_t len = ((S.rows + pieces - 1) / pieces + 31) & ~31LL;
    for (int64_t q = from; q < S.cols * pieces; q += step) {
      const int64_t j = q / pieces, first = (q - j * pieces) * len, end = first + len;
      copy(j, first + i0, end < S.rows ? end : S.rows);
    }
  } else {
    for (int64_t j = from; j < S.cols; j += step) copy(j, i0, S.rows);
  }
}

}  // namespace

cudaError_t launch_segcopy(const SegCopy* segs, int64_t nseg, const double* src, double* dst, const double* scales,
                           cudaStream_t stream) {
  if (nseg == 0) return cudaSuccess;
  if (nseg > 0x7fffffff) return cudaErrorInvalidValue;
  segcopy_kernel<<<dim3((unsigned)nseg, kSplit), 256, 0, stream>>>(segs, src, dst, scales);
  return cudaGetLastError();
}

}  // namespace tnt
