// Whole-matrix kernels for small orders.
//
//   potrf_warp32_kernel  n <= 32: one warp per matrix, one row per lane in
//                        registers.  HBM-bound: A's lower triangle is read
//                        once with coalesced 128-bit loads through a padded
//                        shared staging tile, L (zeros above the diagonal) is
//                        written once with 128-bit streaming stores.
//   potrf_cta128_kernel  32 < n <= 128: one CTA per matrix, the matrix
//                        resident in shared memory, on the 64x64 diagonal
//                        engine (128 threads up to 64, else 256).
//
// These replace the reference's exact-shape kernels chol32_register_rank2
// (submission.py:100-171), cholesky64_rank2 (submission.py:204-290) and
// cholesky128_block16 (submission.py:316-411,555-608) for every order <= 128.
#include <algorithm>

#include "diag64.cuh"
#include "launch.h"
#include "matrix_list.cuh"

namespace b2p {

constexpr int kWarp32Warps = 4;
constexpr int kStageLd = 36;  // staging row stride: 16-byte rows, conflict-free float4

__device__ __forceinline__ float4 ld_stream(const float4* p) {
  float4 v;
  asm volatile("ld.global.nc.L1::no_allocate.v4.f32 {%0,%1,%2,%3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "l"(p));
  return v;
}

__device__ __forceinline__ void st_stream(float4* p, float4 v) {
  asm volatile("st.global.cs.v4.f32 [%0], {%1,%2,%3,%4};" ::"l"(p), "f"(v.x), "f"(v.y), "f"(v.z),
               "f"(v.w)
               : "memory");
}

__global__ void __launch_bounds__(kWarp32Warps * 32, 7)
    potrf_warp32_kernel(const float* __restrict__ a, float* __restrict__ l, MatrixList ml,
                        int32_t* __restrict__ info) {
  __shared__ __align__(16) float stage[kWarp32Warps][32 * kStageLd];
  __shared__ __align__(16) float colbuf[kWarp32Warps][64];
  const int lane = threadIdx.x & 31;
  const int warp = threadIdx.x >> 5;
  float* t = stage[warp];
  for (int64_t item = (int64_t)blockIdx.x * kWarp32Warps + warp; item < ml.count;
       item += (int64_t)gridDim.x * kWarp32Warps) {
    int64_t mat, off;
    int n;
    ml.get(item, mat, off, n);
    const float* src = a + off;
    float* dst = l + off;
    if (n == 32) {
      const float4* s4 = reinterpret_cast<const float4*>(src);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int idx = q * 32 + lane;  // float4 index: row idx>>3, cols 4*(idx&7)..
        const int r = idx >> 3, c = (idx & 7) * 4;
        if (c <= r) *reinterpret_cast<float4*>(t + r * kStageLd + c) = ld_stream(s4 + idx);
      }
    } else {
      for (int r = 0; r < n; ++r)
        if (lane <= r) t[r * kStageLd + lane] = src[(size_t)r * n + lane];
    }
    __syncwarp();
    float x[32];
#pragma unroll
    for (int c4 = 0; c4 < 8; ++c4) {
      const float4 v = *reinterpret_cast<const float4*>(t + lane * kStageLd + 4 * c4);
      x[4 * c4 + 0] = v.x;
      x[4 * c4 + 1] = v.y;
      x[4 * c4 + 2] = v.z;
      x[4 * c4 + 3] = v.w;
    }
    if (n < 32) {
#pragma unroll
      for (int j = 0; j < 32; ++j)
        if (lane >= n || j >= n) x[j] = (lane == j) ? 1.0f : 0.0f;
    }
    const int bad = warp_factor32(x, lane, n, colbuf[warp]);
    __syncwarp();
#pragma unroll
    for (int c4 = 0; c4 < 8; ++c4) {
      float4 v;
      v.x = (4 * c4 + 0 <= lane) ? x[4 * c4 + 0] : 0.0f;
      v.y = (4 * c4 + 1 <= lane) ? x[4 * c4 + 1] : 0.0f;
      v.z = (4 * c4 + 2 <= lane) ? x[4 * c4 + 2] : 0.0f;
      v.w = (4 * c4 + 3 <= lane) ? x[4 * c4 + 3] : 0.0f;
      *reinterpret_cast<float4*>(t + lane * kStageLd + 4 * c4) = v;
    }
    __syncwarp();
    if (n == 32) {
      float4* d4 = reinterpret_cast<float4*>(dst);
#pragma unroll
      for (int q = 0; q < 8; ++q) {
        const int idx = q * 32 + lane;
        const int r = idx >> 3, c = (idx & 7) * 4;
        st_stream(d4 + idx, *reinterpret_cast<const float4*>(t + r * kStageLd + c));
      }
    } else {
      for (int r = 0; r < n; ++r)
        if (lane < n) dst[(size_t)r * n + lane] = t[r * kStageLd + lane];
    }
    if (info != nullptr && lane == 0) info[mat] = bad < 0 ? 0 : bad + 1;
    __syncwarp();
  }
}

// ---- 32 < n <= 128 ------------------------------------------------------------
// The matrix as 64-wide block columns in shared memory, factored by the
// diagonal engine (diag64.cuh): the first with the rows below it along (warps
// 4..7), then A22 -= L21 L21^T on all threads, then the second.  Orders up to
// 64 need the first block alone, on four warps.  Latency bounds it: one chain
// of n pivots.  Measured on B200, us per call in a graph, against warp
// factorizations of 32-wide blocks with a row solve and a 4x4-tile update
// between them: 16x64 14.7 -> 6.9, 16x100 31.4 -> 15.5, 256x128 39.7 -> 23.6,
// 2000x64 99.5 -> 35.0, 8000x48 392 -> 102, 3000x100 382 -> 215.
template <bool BIG>
constexpr int kCtaThreads = BIG ? 256 : kD64Threads;
template <bool BIG>
constexpr int kCtaRows = BIG ? 128 : 64;  // rows of the first block column
template <bool BIG>
constexpr size_t kCtaSmem = sizeof(float) * (size_t)((kCtaRows<BIG> + 64 + (BIG ? 64 : 0)) * kD64Ld + 64 + 8);

__device__ __forceinline__ void cp_async(float* dst, const float* src, int bytes) {
  const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
  if (bytes == 16)
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(d), "l"(src) : "memory");
  else
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(d), "l"(src) : "memory");
}

// S2[i][j] -= sum_m L21[i][m] L21[j][m] for j <= i < 64, m < 64; thread (ti, tj)
// has rows ti + 16 r and columns tj + 16 c (neighbouring threads, neighbouring
// rows: no bank conflicts), of which only r >= c matter.  A panel's products in
// sums as in the block's own updates (Sums).
__device__ __forceinline__ void lower_update64(float* S2, const float* L21) {
  const int ti = threadIdx.x >> 4, tj = threadIdx.x & 15;
  float x[4][4], acc[4][4];
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c <= r; ++c) {
      x[r][c] = S2[(ti + 16 * r) * kD64Ld + tj + 16 * c];
      acc[r][c] = 0.0f;
    }
  auto subtract = [&] {
#pragma unroll
    for (int r = 0; r < 4; ++r)
#pragma unroll
      for (int c = 0; c <= r; ++c) {
        x[r][c] -= acc[r][c];
        acc[r][c] = 0.0f;
      }
  };
  // Columns m .. m + 3; `ends` as kFirstSumEnds, for these four.
  auto products = [&](int m, uint32_t ends) {
    float a[4][4], b[4][4];
#pragma unroll
    for (int r = 0; r < 4; ++r) {
      const float4 v = *reinterpret_cast<const float4*>(L21 + (ti + 16 * r) * kD64Ld + m);
      a[r][0] = v.x, a[r][1] = v.y, a[r][2] = v.z, a[r][3] = v.w;
      const float4 u = *reinterpret_cast<const float4*>(L21 + (tj + 16 * r) * kD64Ld + m);
      b[r][0] = u.x, b[r][1] = u.y, b[r][2] = u.z, b[r][3] = u.w;
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
#pragma unroll
      for (int r = 0; r < 4; ++r)
#pragma unroll
        for (int c = 0; c <= r; ++c) acc[r][c] = fmaf(a[r][p], b[c][p], acc[r][c]);
      if ((ends >> p & 1u) != 0) subtract();
    }
  };
#pragma unroll
  for (int m = 0; m < 16; m += 4) products(m, kFirstSumEnds >> m & 15u);
#pragma unroll 1
  for (int g = 16; g < 64; g += 16) {
#pragma unroll 2
    for (int m = 0; m < 16; m += 4) products(g + m, 0u);
    subtract();
  }
#pragma unroll
  for (int r = 0; r < 4; ++r)
#pragma unroll
    for (int c = 0; c <= r; ++c) S2[(ti + 16 * r) * kD64Ld + tj + 16 * c] = x[r][c];
}

template <bool BIG>
__global__ void __launch_bounds__(kCtaThreads<BIG>, BIG ? 2 : 4)
    potrf_cta128_kernel(const float* __restrict__ a, float* __restrict__ l, MatrixList ml,
                        int32_t* __restrict__ info) {
  extern __shared__ __align__(16) float smem[];
  constexpr int NT = kCtaThreads<BIG>, ROWS = kCtaRows<BIG>;
  float* S1 = smem;                     // columns 0..63
  float* Lt = S1 + ROWS * kD64Ld;       // L^T view of the block being factored
  float* S2 = Lt + 64 * kD64Ld;         // BIG: rows and columns 64..127
  float* invd = S2 + (BIG ? 64 * kD64Ld : 0);
  int* bad = reinterpret_cast<int*>(invd + 64);
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int64_t item = blockIdx.x; item < ml.count; item += gridDim.x) {
    int64_t mat, off;
    int n;
    ml.get(item, mat, off, n);
    const float* src = a + off;
    float* dst = l + off;
    const bool vec = (n & 3) == 0;
    auto at = [&](int r, int c) -> float* {
      return BIG && c >= 64 ? S2 + (r - 64) * kD64Ld + c - 64 : S1 + r * kD64Ld + c;
    };
    // The lower triangle (to the next multiple of four), every copy in flight.
    if (vec) {
      const int c = 4 * lane;
#pragma unroll 4
      for (int r = warp; r < n; r += NT / 32)
        if (c <= r) cp_async(at(r, c), src + (size_t)r * n + c, 16);
    } else {
      for (int r = warp; r < n; r += NT / 32)
#pragma unroll 4
        for (int c = lane; c <= r; c += 32) cp_async(at(r, c), src + (size_t)r * n + c, 4);
    }
    // Identity beyond n (zero below the first block).
    const int pad = n <= 64 ? 64 : 128;
    for (int e = tid; e < (ROWS - n) * 64; e += NT) {
      const int r = n + (e >> 6), c = e & 63;
      S1[r * kD64Ld + c] = r == c ? 1.0f : 0.0f;
      if (BIG && n > 64) S2[(r - 64) * kD64Ld + c] = r - 64 == c ? 1.0f : 0.0f;
    }
    asm volatile("cp.async.wait_all;" ::: "memory");
    __syncthreads();
    diag64_panels<false, BIG, true>(S1, Lt, nullptr, invd, bad, pad == 64 ? (n + 15) / 16 : 4, CtaBarrier(), true);
    if (BIG && n > 64) {
      lower_update64(S2, S1 + 64 * kD64Ld);
      __syncthreads();
      diag64_panels<false, false, true>(S2, Lt, nullptr, invd, bad + 4, (n - 64 + 15) / 16, CtaBarrier());
    }
    if (vec) {
      const int c = 4 * lane;
#pragma unroll 4
      for (int r = warp; r < n; r += NT / 32) {
        if (c >= n) continue;
        float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
        if (c <= r) {
          v = *reinterpret_cast<const float4*>(at(r, c));
          if (c + 1 > r) v.y = 0.f;
          if (c + 2 > r) v.z = 0.f;
          if (c + 3 > r) v.w = 0.f;
        }
        *reinterpret_cast<float4*>(dst + (size_t)r * n + c) = v;
      }
    } else {
      for (int r = warp; r < n; r += NT / 32)
#pragma unroll 4
        for (int c = lane; c < n; c += 32) dst[(size_t)r * n + c] = c <= r ? *at(r, c) : 0.0f;
    }
    if (info != nullptr && tid == 0) {
      int first = 0;
      for (int p = 0; p < (BIG && n > 64 ? 8 : 4) && first == 0; ++p)
        if (bad[p] >= 0) first = 16 * p + bad[p] + 1;
      info[mat] = first <= n ? first : 0;  // beyond: padding behind a pivot that is infinite
    }
    __syncthreads();
  }
}

int launch_warp32(const float* a, float* l, const MatrixList& ml, int32_t* info, cudaStream_t s) {
  if (ml.count == 0) return B2P_OK;
  const int64_t ctas = (ml.count + kWarp32Warps - 1) / kWarp32Warps;
  const int grid = (int)std::min<int64_t>(ctas, (int64_t)device_sms() * 8 * 16);
  {
    TraceScope ts(kKWarp32, s, ml.ns ? 0.0 : 8.0 * (double)ml.count * ml.n * ml.n);
    potrf_warp32_kernel<<<grid, kWarp32Warps * 32, 0, s>>>(a, l, ml, info);
  }
  return check_launch("potrf_warp32_kernel");
}

int launch_cta128(const float* a, float* l, const MatrixList& ml, int32_t* info, cudaStream_t s) {
  if (ml.count == 0) return B2P_OK;
  // A list's orders are not known here: it takes the form that covers them all.
  const bool big = ml.ns != nullptr || ml.n > 64;
  const void* k = big ? (const void*)potrf_cta128_kernel<true> : (const void*)potrf_cta128_kernel<false>;
  const size_t smem = big ? kCtaSmem<true> : kCtaSmem<false>;
  if (int st = ensure_smem_attr(k, smem, big ? kSlotCta128 : kSlotCta64)) return st;
  const int grid = (int)std::min<int64_t>(ml.count, (int64_t)device_sms() * (big ? 2 : 4) * 64);
  {
    TraceScope ts(kKCta128, s, ml.ns ? 0.0 : (double)ml.count * ml.n * ml.n * ml.n / 3.0);
    if (big)
      potrf_cta128_kernel<true><<<grid, kCtaThreads<true>, smem, s>>>(a, l, ml, info);
    else
      potrf_cta128_kernel<false><<<grid, kCtaThreads<false>, smem, s>>>(a, l, ml, info);
  }
  return check_launch("potrf_cta128_kernel");
}

}  // namespace b2p
