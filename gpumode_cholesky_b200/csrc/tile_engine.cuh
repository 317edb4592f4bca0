// The warp factorization of the n <= 32 kernel: one warp factors a 32x32 block
// held one row per lane in registers (right-looking, column by column).  The
// pivot column crosses lanes through a double-buffered 32-float shared array,
// so one __syncwarp per pivot orders it.
//
// The algorithm is the textbook right-looking Cholesky that LAPACK's potrf
// (called by the reference's ref_kernel, reference/reference.py:129-130, and
// its cuSOLVER routes, submission.py:4268) computes; pivots use a refined
// reciprocal square root instead of a divide.
#pragma once

#include "common.cuh"

namespace b2p {

// Factor the 32x32 block x[] (row `lane`), columns >= w / rows >= w are
// identity padding.  On return x holds L (lower part valid, upper part is
// don't-care).  Returns the first local pivot index that was not positive, or
// -1.  All 32 lanes must call.
//
// Step k takes the pivot d = x[k] of lane k and, in the same round of
// shuffles, lane k+1's unscaled column-k value e; every lane then forms
// L[k+1][k] = e / sqrt(d) itself and updates its column k+1 at once, so the
// next pivot depends only on shuffles and registers.  The rest of the rank-1
// update (columns k+2..31) goes through a double-buffered shared-memory copy
// of column k and is deferred by one step: step k+1 applies it, two columns an
// instruction, right after shuffling out its own pivot, in the shadow of that
// pivot's reciprocal square root.  The arithmetic is the same as the textbook
// right-looking update, value for value and in the same order.
//
// One form for all pivots: the rsqrt that takes normal ones only saves 23 cycles
// in each step, but a warp whose matrix has another pivot starts again, and the
// two forms' code together cost more than that (us in a graph, two forms / this
// one / before the packed pairs: 20000x32 48.8 / 46.0 / 48.3, 20000x1 21.2 / 18.7
// / 20.0, 4096x32 12.2 / 12.1 / 12.5, 20000x24 53.4 / 54.3 / 58.7; every matrix
// failing, 20000x32 83.7 / 46.0 / 48.3).
__device__ __forceinline__ int warp_factor32(float (&x)[32], int lane, int w, float* colbuf) {
  int bad = -1;
  float nlprev = 0.0f;  // minus this lane's L[lane][k-1]
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    if (k < w) {  // warp-uniform
      const float d = __shfl_sync(kFullMask, x[k], k);
      const float e = (k + 1 < 32) ? __shfl_sync(kFullMask, x[k], k + 1) : 0.0f;
      // Column k-1's update of columns k+1.. (column k had it by look-ahead).
      if (k >= 1 && k + 1 < 32) {
        const float* cb = colbuf + ((k - 1) & 1) * 32;
#pragma unroll
        for (int j4 = (k + 1) / 4; j4 < 8; ++j4) {
          const float4 c = reinterpret_cast<const float4*>(cb)[j4];
          const float cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
          for (int q = 0; q < 4; q += 2) {
            const int j = 4 * j4 + q;
            if (j > k)
              fma2(x[j], x[j + 1], nlprev, cv[q], cv[q + 1]);
            else if (j + 1 > k)
              x[j + 1] = fmaf(nlprev, cv[q + 1], x[j + 1]);
          }
        }
      }
      if (bad < 0 && pivot_bad(d)) bad = k;
      const float y = rsqrt_refined(d);
      x[k] = (lane == k) ? d * y : x[k] * y;
      nlprev = -x[k];
      if (k + 1 < 32) x[k + 1] = fmaf(nlprev, e * y, x[k + 1]);
      if (k + 2 < 32) {
        colbuf[(k & 1) * 32 + lane] = x[k];
        __syncwarp();
      }
    }
  }
  return bad;
}

}  // namespace b2p
