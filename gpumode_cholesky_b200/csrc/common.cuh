// Shared helpers for the B200 potrf kernels (sm_100a only).
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "../../include/b200_potrf.h"

#if defined(__CUDA_ARCH__) && (__CUDA_ARCH__ < 1000)
#error "this library targets sm_100a (B200) only"
#endif

namespace b2p {

constexpr unsigned kFullMask = 0xffffffffu;

// Records a detail message for b2p_last_error() and returns `status`.
int set_error(int status, const char* fmt, ...);

// Returns B2P_ERR_CUDA with a message if the last launch failed.
int check_launch(const char* what);

// Reciprocal square root refined by one Newton-Raphson step
// y <- y * (1.5 - 0.5 * d * y * y), starting from the hardware estimate.
// One step brings the MUFU estimate to about one ulp.  A non-positive or NaN
// pivot yields NaN/Inf, which the factorization propagates.
// NORMAL: the caller checks that d is a normal number (pivot_normal), for
// which the flush-to-zero estimate gives rsqrtf's bits without its scaling of
// subnormal ones (17 against 40 cycles of latency on B200, once per pivot).
template <bool NORMAL = false>
__device__ __forceinline__ float rsqrt_refined(float d) {
  float y;
  if (NORMAL)
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(d));
  else
    y = rsqrtf(d);
  float h = 0.5f * d;
  float t = fmaf(-h * y, y, 0.5f);  // 0.5 - 0.5*d*y^2
  return fmaf(y, t, y);             // y + y*(0.5 - 0.5*d*y^2)
}
__device__ __forceinline__ bool pivot_normal(float d) { return d >= 1.17549435e-38f; }

__device__ __forceinline__ bool pivot_bad(float d) { return !(d > 0.0f); }

// x0 += a b0, x1 += a b1, each one fused multiply-add as fmaf rounds it, in one
// two-lane instruction.  On B200 a 64x64x64 product in shared memory, three
// CTAs of 128 threads per SM, takes 1540 cycles this way and 2890 with fmaf
// (twice the multiply-adds per issue slot), provided that (b0, b1) come out of
// one vector load: packing them from separate registers costs more than it
// gains (3160 to 3590 cycles).
__device__ __forceinline__ void fma2(float& x0, float& x1, float a, float b0, float b1) {
  asm("{\n\t.reg .b64 ra, rb, rx;\n\t"
      "mov.b64 ra, {%2, %2};\n\t"
      "mov.b64 rb, {%3, %4};\n\t"
      "mov.b64 rx, {%0, %1};\n\t"
      "fma.rn.f32x2 rx, ra, rb, rx;\n\t"
      "mov.b64 {%0, %1}, rx;\n\t}"
      : "+f"(x0), "+f"(x1)
      : "f"(a), "f"(b0), "f"(b1));
}

// 64-bit element offset of matrix `b` in a contiguous batch of n x n matrices.
__device__ __forceinline__ int64_t mat_offset(int64_t b, int n) { return b * (int64_t)n * n; }

}  // namespace b2p
