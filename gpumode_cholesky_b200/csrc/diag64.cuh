// Factor (and invert) one 64x64 diagonal block with four warps.
//
// Right-looking over four panels of 16 columns.  The rows of a panel are dealt
// to warps 16 at a time: lanes 16..31 of panel warp w hold one row each of the
// w-th 16-row block below the diagonal block, and lanes 0..15 of every panel
// warp hold the diagonal block's own rows.  So each warp factors the 16x16
// diagonal block itself (redundantly) and solves its rows in the same
// instructions, and no value crosses warps inside a panel.  Four pivots at a
// time, the 4x4 diagonal piece is shuffled to every lane and every lane runs
// its little factorization, so that the chain from one pivot to the next is a
// reciprocal square root, a multiply and a fused multiply-add; solved columns
// reach the rest of the panel by shuffles.
//
// Between panels all four warps apply the finished panel to the next one
// (rank 16, in register tiles).  The columns beyond it are warp 2's, beside
// the next panel, since it runs out of panel rows first.  The inverse T =
// L^{-1} (diag64_factor_invert) is formed beside the panels as well, one
// column per lane, by the warps that have no panel rows (any more), block row
// by block row as the panels appear: T11 and T22 by substitution, -W = -L21
// T11 below T11, and at the end T21 = -T22 W by all four warps.
//
// Every element of L receives the multiply-adds of the textbook right-looking
// update, one by one in its order, so L does not depend on the blocking.
//
// What bounds it: the chain of 64 pivots (about 65 cycles each), then the
// three updates between panels (about 650 each).  Measured on B200, one CTA
// per SM, cycles: factor 7.6k, with the inverse 11.3k, and up to 1k more when
// its code is not in the instruction cache.  Before it (a pipeline of three
// warps over 32-wide halves, fully unrolled, one trip to another lane per
// pivot, and the inverse after the factor): 12.6k and 17.3k, and 18.9k and
// 27.8k with cold code, which is how a kernel that runs it once meets it.
//
// Rows and columns at or beyond the block's true width are identity
// padding, so a short last block (w < 64) runs the same code.
#pragma once

#include "tile_engine.cuh"

namespace b2p {

constexpr int kD64Ld = 68;   // row stride of S, T and the L^T view (floats)
constexpr int kD64Threads = 128;

// Barrier used between the engine's phases: the whole CTA, or a named
// barrier over the first N threads (when other warps of the CTA run a
// different role and must not be waited for).
struct CtaBarrier {
  __device__ __forceinline__ void operator()() const { __syncthreads(); }
};
template <int NTHREADS>
struct NamedBarrier1 {
  __device__ __forceinline__ void operator()() const {
    asm volatile("bar.sync 1, %0;" ::"n"(NTHREADS) : "memory");
  }
};

// The same over barrier 2 (a second group of warps that runs its own
// barrier 1 at the same time must not share the id).
template <int NTHREADS>
struct NamedBarrier2 {
  __device__ __forceinline__ void operator()() const {
    asm volatile("bar.sync 2, %0;" ::"n"(NTHREADS) : "memory");
  }
};

struct Diag64Smem {
  float S[64 * kD64Ld];   // block: A in, L out (lower part)
  float T[64 * kD64Ld];   // T^T, T = L^{-1} (T[c][j] = L^{-1}[j][c])
  float lt[64 * kD64Ld];  // L^T (diag64_lt): lt[m][j] = L[j][m]
  float invd[64];         // 1 / diag(L)
  int bad[4];             // first bad pivot within each panel, or -1
};

__device__ __forceinline__ float* diag64_lt(Diag64Smem& sm) { return sm.lt; }
__device__ __forceinline__ const float* diag64_lt(const Diag64Smem& sm) { return sm.lt; }

// ---- 16-wide pieces: one row (or one right-hand side) per lane ---------------
__device__ __forceinline__ void load_row16(float (&x)[16], const float* src) {
#pragma unroll
  for (int c4 = 0; c4 < 4; ++c4) {
    const float4 v = reinterpret_cast<const float4*>(src)[c4];
    x[4 * c4] = v.x, x[4 * c4 + 1] = v.y, x[4 * c4 + 2] = v.z, x[4 * c4 + 3] = v.w;
  }
}
__device__ __forceinline__ void store_row16(float* dst, const float (&x)[16]) {
#pragma unroll
  for (int c4 = 0; c4 < 4; ++c4)
    reinterpret_cast<float4*>(dst)[c4] = make_float4(x[4 * c4], x[4 * c4 + 1], x[4 * c4 + 2], x[4 * c4 + 3]);
}

// How an update subtracts a panel's 16 products: product by product, or in sums
// (the small orders), of all 16 or, for the matrix's first panel, of 2, 2, 4 and
// 8 (kFirstSumEnds: the last of each, as a mask).  A sum costs one rounding at
// the element's own size, and one at the sum's size per product.  On smooth
// covariances the first few products take nearly all of an element away, and
// what is rounded at the size of their sum is large against what remains; on
// Gram matrices the element keeps its size, and every subtraction costs.  Error
// of L against 64 bits over that of product-by-product 32-wide blocks with sums
// of 32 between them, which this replaced, at orders 33 to 128 on Gram matrices
// and squared-exponential covariances in the unit cube, two shifts each (a model
// of the roundings on the CPU): 0.45 to 1.00; 16 at a time throughout up to
// 1.36, product by product up to 1.71, 4 at a time up to 1.08.
enum Sums { kByProduct = 0, kSum16 = 1, kSumFirst = 2 };
constexpr uint32_t kFirstSumEnds = 1u << 1 | 1u << 3 | 1u << 7 | 1u << 15;

// The rank-16 update in register tiles of R rows by 4 columns, x[4r + c] -=
// sum_m a_rm lt[m][c0 + c], m = 0..15 ascending.  The columns' factors come
// from the L^T view, where a warp's reads of one m are contiguous; so do the
// rows' (a_rm = rows[m][r]) or they are rows of S or T^T (TROWS, a_rm =
// rows[r][m]).  Sums run in packed pairs.
template <int R, bool TROWS, int SUMS>
__device__ __forceinline__ void update_tile16(float (&x)[4 * R], const float* rows, const float* lt_c) {
  constexpr bool SUM = SUMS != kByProduct;
  constexpr uint32_t kEnds = SUMS == kSumFirst ? kFirstSumEnds : 1u << 15;
  float d[SUM ? 4 * R : 1];
  if (SUM) {
#pragma unroll
    for (int q = 0; q < 4 * R; ++q) d[q] = 0.0f;
  }
#pragma unroll (SUMS == kSumFirst ? 4 : 2)
  for (int m = 0; m < 16; m += 4) {
    float a[4][R];
    if (TROWS) {
#pragma unroll
      for (int r = 0; r < R; ++r) {
        const float4 v = *reinterpret_cast<const float4*>(rows + r * kD64Ld + m);
        a[0][r] = v.x, a[1][r] = v.y, a[2][r] = v.z, a[3][r] = v.w;
      }
    } else {
#pragma unroll
      for (int p = 0; p < 4; ++p) {
        if (R == 4) {
          const float4 v = *reinterpret_cast<const float4*>(rows + (m + p) * kD64Ld);
          a[p][0] = v.x, a[p][1] = v.y, a[p][R - 2] = v.z, a[p][R - 1] = v.w;
        } else {
          const float2 v = *reinterpret_cast<const float2*>(rows + (m + p) * kD64Ld);
          a[p][0] = v.x, a[p][1] = v.y;
        }
      }
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float4 b = *reinterpret_cast<const float4*>(lt_c + (m + p) * kD64Ld);
#pragma unroll
      for (int r = 0; r < R; ++r) {
        if (SUM) {
          fma2(d[4 * r + 0], d[4 * r + 1], a[p][r], b.x, b.y);
          fma2(d[4 * r + 2], d[4 * r + 3], a[p][r], b.z, b.w);
        } else {
          x[4 * r + 0] = fmaf(-a[p][r], b.x, x[4 * r + 0]);
          x[4 * r + 1] = fmaf(-a[p][r], b.y, x[4 * r + 1]);
          x[4 * r + 2] = fmaf(-a[p][r], b.z, x[4 * r + 2]);
          x[4 * r + 3] = fmaf(-a[p][r], b.w, x[4 * r + 3]);
        }
      }
      if (SUM && (SUMS == kSumFirst || p == 3) && (kEnds >> (m + p) & 1u) != 0) {
#pragma unroll
        for (int q = 0; q < 4 * R; ++q) {
          x[q] -= d[q];
          d[q] = 0.0f;
        }
      }
    }
  }
}

// The tile's R rows of four at `dst` (row stride kD64Ld), less panels
// k0 .. k1 - 1 of L (`rows`, `lt_c` as above, at panel 0): product by product,
// or with SUM in sums (`first`: panel 0 is the matrix's first).
template <int R, bool TROWS, bool SUM = false>
__device__ __forceinline__ void update_blocks(float* dst, const float* rows, const float* lt_c, int k0, int k1,
                                              bool first = false) {
  float x[4 * R];
#pragma unroll
  for (int r = 0; r < R; ++r) {
    const float4 v = *reinterpret_cast<const float4*>(dst + r * kD64Ld);
    x[4 * r] = v.x, x[4 * r + 1] = v.y, x[4 * r + 2] = v.z, x[4 * r + 3] = v.w;
  }
#pragma unroll 1
  for (int k = k0; k < k1; ++k) {
    const float* rk = rows + 16 * k * (TROWS ? 1 : kD64Ld);
    if (!SUM)
      update_tile16<R, TROWS, kByProduct>(x, rk, lt_c + 16 * k * kD64Ld);
    else if (first && k == 0)
      update_tile16<R, TROWS, kSumFirst>(x, rk, lt_c);
    else
      update_tile16<R, TROWS, kSum16>(x, rk, lt_c + 16 * k * kD64Ld);
  }
#pragma unroll
  for (int r = 0; r < R; ++r)
    *reinterpret_cast<float4*>(dst + r * kD64Ld) = make_float4(x[4 * r], x[4 * r + 1], x[4 * r + 2], x[4 * r + 3]);
}

// x <- L^{-1} x for the 16x16 lower L at lt (lt[m * kD64Ld + j] = L[j][m]) and
// invd, by right-looking forward substitution.
__device__ __forceinline__ void subst16(float (&x)[16], const float* lt, const float* invd) {
#pragma unroll
  for (int m = 0; m < 16; ++m) {
    x[m] *= invd[m];
#pragma unroll
    for (int j4 = (m + 1) / 4; j4 < 4; ++j4) {
      const float4 c = reinterpret_cast<const float4*>(lt + m * kD64Ld)[j4];
      const float cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int j = 4 * j4 + q;
        if (j > m) x[j] = fmaf(-x[m], cv[q], x[j]);
      }
    }
  }
}

// Factors the 16x16 block held by lanes 0..15 (row `lane`) and solves the
// rows of lanes 16..31 against it; 1/L[k][k] goes to invd.  A group of four
// columns updates the next four at once and the rest during the next group's
// chain.  NORMAL (see rsqrt_refined): returns 0, or a non-zero value if a
// pivot was not a normal positive number, and the caller starts again with
// the general form; that returns the first bad local pivot or -1.  The answer
// is the same on every lane.
template <bool NORMAL>
__device__ __forceinline__ int factor16(float (&x)[16], int lane, float* invd) {
  // A warp whose lanes come here apart (after a branch on the thread index)
  // would meet at every shuffle anew, at 30 times the cost.
  __syncwarp();
  int bad = NORMAL ? 0 : -1;
  float lp[4] = {0.f, 0.f, 0.f, 0.f};  // this lane's L of the previous group
#pragma unroll
  for (int k = 0; k < 16; k += 4) {
    float a[4][4], f[4][4], y[4], l[4];
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
      for (int r = c; r < 4; ++r) a[r][c] = __shfl_sync(kFullMask, x[k + c], k + r);
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      if (k >= 4) {
#pragma unroll
        for (int j = k + 4; j < 16; ++j) x[j] = fmaf(-lp[p], __shfl_sync(kFullMask, lp[p], j), x[j]);
      }
      const float d = a[p][p];
      if (NORMAL)
        bad |= pivot_normal(d) ? 0 : 1;
      else if (bad < 0 && pivot_bad(d))
        bad = k + p;
      y[p] = rsqrt_refined<NORMAL>(d);
#pragma unroll
      for (int r = p + 1; r < 4; ++r) a[r][p] *= y[p];
      l[p] = (lane == k + p) ? d * y[p] : x[k + p] * y[p];
#pragma unroll
      for (int c = p + 1; c < 4; ++c) {
#pragma unroll
        for (int r = c; r < 4; ++r) a[r][c] = fmaf(-a[r][p], a[c][p], a[r][c]);
        x[k + c] = fmaf(-l[p], a[c][p], x[k + c]);
      }
      if (k < 12) {
#pragma unroll
        for (int r = 0; r < 4; ++r) f[r][p] = __shfl_sync(kFullMask, l[p], k + 4 + r);
      }
      x[k + p] = l[p];
    }
    if (k < 12) {
#pragma unroll
      for (int p = 0; p < 4; ++p) {
#pragma unroll
        for (int r = 0; r < 4; ++r) x[k + 4 + r] = fmaf(-l[p], f[r][p], x[k + 4 + r]);
        lp[p] = l[p];
      }
    }
    if (threadIdx.x == 0) *reinterpret_cast<float4*>(invd + k) = make_float4(y[0], y[1], y[2], y[3]);
  }
  return bad;
}

// diag64_factor's result as every thread of the CTA can read it back once
// the factorization's last barrier has been passed by all of them.
__device__ __forceinline__ int diag64_status(const Diag64Smem& sm) {
#pragma unroll
  for (int p = 0; p < 4; ++p)
    if (sm.bad[p] >= 0) return 16 * p + sm.bad[p];
  return -1;
}

// T21^T = -W^T T22^T in place (T^T's rows 0..31, columns 32..63 hold -W^T; the
// four threads of a row are one warp's).  128 threads.
__device__ __forceinline__ void t21_product(float* TT) {
  const int tid = threadIdx.x;
  const int c = tid >> 2, i0 = 32 + (tid & 3) * 8;
  float acc[8];
#pragma unroll
  for (int q = 0; q < 8; ++q) acc[q] = 0.0f;
#pragma unroll 2
  for (int p = 0; p < 32; p += 4) {
    const float4 w4 = *reinterpret_cast<const float4*>(TT + c * kD64Ld + 32 + p);
    const float w[4] = {w4.x, w4.y, w4.z, w4.w};
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const float4 b0 = *reinterpret_cast<const float4*>(TT + (32 + p + e) * kD64Ld + i0);
      const float4 b1 = *reinterpret_cast<const float4*>(TT + (32 + p + e) * kD64Ld + i0 + 4);
      fma2(acc[0], acc[1], w[e], b0.x, b0.y);
      fma2(acc[2], acc[3], w[e], b0.z, b0.w);
      fma2(acc[4], acc[5], w[e], b1.x, b1.y);
      fma2(acc[6], acc[7], w[e], b1.z, b1.w);
    }
  }
  __syncwarp();
  float* o = TT + c * kD64Ld + i0;
  reinterpret_cast<float4*>(o)[0] = make_float4(acc[0], acc[1], acc[2], acc[3]);
  reinterpret_cast<float4*>(o)[1] = make_float4(acc[4], acc[5], acc[6], acc[7]);
}

// The engine's body, see the top of the file; INVERT adds T = L^{-1}.
// Phase ph (0 .. np - 1) factors panel ph; with INVERT a phase 4 ends the
// inverse.  np < 4 leaves out panels that are identity padding.  BELOW: S has
// 64 more rows (64 .. 127), which warps 4..7 solve along with the panels, 16
// rows each; their updates are left-looking, since these warps never run out
// of panel rows.  SUM: updates subtract sums of products (Sums; the small
// orders' form, `first` telling the matrix's first block; the n > 128 paths
// keep the product-by-product order).
template <bool INVERT, bool BELOW, bool SUM, class Bar>
__device__ __forceinline__ void diag64_panels(float* S, float* Lt, float* TT, float* invd, int* bad, int np, Bar bar,
                                              bool first = false) {
  const int tid = threadIdx.x;
  const int lane = tid & 31;
  const int warp = tid >> 5;
  if (tid == 0)
    for (int p = np; p < 4; ++p) bad[p] = -1;
#pragma unroll 1
  for (int ph = 0; ph < (INVERT ? 5 : np); ++ph) {
    if (ph > 0 && ph < 4) {
      // Panel ph - 1 applied to column block ph: rows 16 ph .. 63, two rows
      // and four columns a thread.
      const int r = 16 * ph + 2 * (tid >> 2), c = 16 * ph + 4 * (tid & 3);
      if (BELOW && tid >= kD64Threads) {
        const int rb = 2 * (tid >> 2);  // 64 ..
        update_blocks<2, true, SUM>(S + rb * kD64Ld + c, S + rb * kD64Ld, Lt + c, 0, ph, first);
      } else if (r < 64) {
        update_blocks<2, false, SUM>(S + r * kD64Ld + c, Lt + r, Lt + c, ph - 1, ph, first);
      }
      bar();
    }
    float x[16];
    float* row = nullptr;
    if (ph < 4 && ((warp < 3 && (warp + ph < 3 || warp == 0)) || (BELOW && warp >= 4))) {
      // The panel.  The last one has no rows of the block for lanes 16..31.
      const int r = 16 * (lane < 16 ? ph : (BELOW && warp >= 4) ? warp - 1 : ph + warp) + lane;
      const bool live = r < 64 || (BELOW && warp >= 4);
      row = S + (live ? r : 48) * kD64Ld + 16 * ph;
      load_row16(x, row);
      int b = factor16<true>(x, lane, invd + 16 * ph);
      if (b != 0) {
        load_row16(x, row);
        b = factor16<false>(x, lane, invd + 16 * ph);
      } else {
        b = -1;
      }
      if (tid == 0) bad[ph] = b;
      // The diagonal block is warp 0's to write, zero above its diagonal; into
      // S after the barrier, since every panel warp reads it there.
      if (live && (lane >= 16 || warp == 0)) {
        if (lane >= 16) store_row16(row, x);
        if (lane < 16) {
#pragma unroll
          for (int c = 0; c < 16; ++c) x[c] = c <= lane ? x[c] : 0.0f;
        }
        if (!BELOW || r < 64) {
          float* lc = Lt + 16 * ph * kD64Ld + r;
#pragma unroll
          for (int c = 0; c < 16; ++c) lc[c * kD64Ld] = x[c];
        }
      }
    } else if ((warp == 2 && ph < 3) || (!INVERT && warp == 3 && ph == 1)) {
      // Panels before ph applied to the columns beyond block ph: warp 2 one
      // block ahead; two blocks ahead it is warp 3's where that has no T.
      const int q = 32 + (lane & ~3), i = ph + (warp == 2 ? 1 : 2), c = 16 * i + 4 * (lane & 3);
      update_blocks<4, false, SUM>(S + q * kD64Ld + c, Lt + q, Lt + c, INVERT ? 0 : ph - 1, ph, first);
    } else if (INVERT && warp > 0 && warp < 4 && ph > 0) {
      // T, a row of T^T per column: warp 3 has columns 0..15, warp 1 16..31,
      // warp 2 32..63 (f: the first block row that is not zero).  Block row
      // ph - 1 is final once substituted against diagonal block ph - 1; below
      // row 32, columns 0..31 stop at -W.
      const int f = warp == 3 ? 0 : warp;
      const int own = warp == 2 ? lane : lane & 15;
      float* t = TT + 16 * f * kD64Ld;
      if (f == 2 || ph < 3) {
        float* trow = t + own * kD64Ld + 16 * (ph - 1);
        load_row16(x, trow);
        subst16(x, Lt + 16 * (ph - 1) * (kD64Ld + 1), invd + 16 * (ph - 1));
        if (own == lane) store_row16(trow, x);
        __syncwarp();
      }
      // What is final, applied to block row ph; warp 3 takes panel 0's part
      // of block row ph + 1 a phase early.
      const int q = 2 * (lane >> 2), g = 4 * (lane & 3);
      const int jobs = ph == 4 ? 0 : (f == 0 && ph < 3 ? 2 : 1);
#pragma unroll 1
      for (int j = 0; j < jobs; ++j) {
        const int c = 16 * (ph + j) + g;
        const int k = j == 1 ? 0 : (ph == 3 ? max(f, 1) : ph - 1);
        update_blocks<2, true>(t + q * kD64Ld + c, t + q * kD64Ld, Lt + c, k, k + 1);
      }
    } else if (INVERT && warp == 3) {
      // T^T starts as the identity.
#pragma unroll 4
      for (int e = lane; e < 64 * 16; e += 32) {
        const int r = e >> 4, c = (e & 15) * 4;
        *reinterpret_cast<float4*>(TT + r * kD64Ld + c) =
            make_float4(c == r ? 1.f : 0.f, c + 1 == r ? 1.f : 0.f, c + 2 == r ? 1.f : 0.f, c + 3 == r ? 1.f : 0.f);
      }
    }
    bar();
    if (warp == 0 && lane < 16 && ph < 4) store_row16(row, x);
  }
  if (INVERT && tid < kD64Threads) t21_product(TT);
  bar();
}

template <bool INVERT, class Bar>
__device__ __forceinline__ int diag64_run(Diag64Smem& sm, Bar bar) {
  diag64_panels<INVERT, false, false>(sm.S, diag64_lt(sm), sm.T, sm.invd, sm.bad, 4, bar);
  return diag64_status(sm);
}

// Factor the block in sm.S (lower triangle and diagonal read; the caller has
// filled it).  On return sm.S holds L in its lower triangle (what is above the
// diagonal is unspecified), the L^T view holds Lt[m][j] = L[j][m] for j >= m
// (other entries unspecified) and sm.invd 1/diag(L).  Returns the first bad
// pivot or -1.  Every thread of the CTA calls it; threads beyond the first
// four warps only take part in the barriers.
template <class Bar = CtaBarrier>
__device__ __forceinline__ int diag64_factor(Diag64Smem& sm, Bar bar = Bar()) {
  return diag64_run<false>(sm, bar);
}

// diag64_factor, and T = L^{-1} stored transposed in sm.T:
// sm.T[c * kD64Ld + j] = T[j][c] (0 for j < c).  Threads beyond the first four
// warps only take part in the barriers.
template <class Bar = CtaBarrier>
__device__ __forceinline__ int diag64_factor_invert(Diag64Smem& sm, Bar bar = Bar()) {
  return diag64_run<true>(sm, bar);
}

// Solve one panel row against the factored 64x64 block: x <- x L^{-T}
// (forward substitution, FP32, right-looking over the columns), with L^T as
// diag64_factor leaves it.  2080 multiply-adds per row, in pairs of columns;
// every shared-memory read is a warp-wide broadcast.
__device__ __forceinline__ void panel_solve64(float (&x)[64], const Diag64Smem& sm) {
  const float* Lt = diag64_lt(sm);
#pragma unroll
  for (int m = 0; m < 64; ++m) {
    x[m] *= sm.invd[m];
    const float nx = -x[m];
#pragma unroll
    for (int j4 = (m + 1) / 4; j4 < 16; ++j4) {
      const float4 c = reinterpret_cast<const float4*>(Lt + m * kD64Ld)[j4];
      const float cv[4] = {c.x, c.y, c.z, c.w};
#pragma unroll
      for (int q = 0; q < 4; q += 2) {
        const int j = 4 * j4 + q;
        if (j > m)
          fma2(x[j], x[j + 1], nx, cv[q], cv[q + 1]);
        else if (j + 1 > m)
          x[j + 1] = fmaf(nx, cv[q + 1], x[j + 1]);
      }
    }
  }
}

// Inverse only: T = L^{-1} stored transposed in sm.T like diag64_factor_invert,
// of the lower-triangular 64x64 block in sm.S (identity padding beyond the
// true width; zero above the diagonal), with L^T already in the L^T view.
// 128 threads.
__device__ __forceinline__ void diag64_invert_only(Diag64Smem& sm) {
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const float* Lt = diag64_lt(sm);
  float* TT = sm.T;
  if (tid < 64) sm.invd[tid] = 1.0f / sm.S[tid * kD64Ld + tid];
  for (int e = tid; e < 64 * 16; e += kD64Threads) {
    const int r = e >> 4, c = (e & 15) * 4;
    *reinterpret_cast<float4*>(TT + r * kD64Ld + c) =
        make_float4(c == r ? 1.f : 0.f, c + 1 == r ? 1.f : 0.f, c + 2 == r ? 1.f : 0.f, c + 3 == r ? 1.f : 0.f);
  }
  __syncthreads();
  // Warp w: columns 16w .. 16w + 15, T11 and T22.
  const int h = 2 * (warp >> 1);  // the half's first block row
  const int q = 2 * (lane >> 2), g = 4 * (lane & 3);
  float* t = TT + 16 * warp * kD64Ld;
  float* trow = t + (lane & 15) * kD64Ld;
  float x[16];
#pragma unroll 1
  for (int i = warp; i < h + 2; ++i) {
    load_row16(x, trow + 16 * i);
    subst16(x, Lt + 16 * i * (kD64Ld + 1), sm.invd + 16 * i);
    if (lane < 16) store_row16(trow + 16 * i, x);
    __syncwarp();
    if (i == h)
      update_blocks<2, true>(t + q * kD64Ld + 16 * (i + 1) + g, t + q * kD64Ld, Lt + 16 * (i + 1) + g, i, i + 1);
    __syncwarp();
  }
  __syncthreads();
  // -W (W = L21 T11): block row 2 on warps 0 and 1, 3 on 2 and 3.
  {
    const int c = 16 * (2 + (warp >> 1)) + g;
    float* tw = TT + (16 * (warp & 1) + q) * kD64Ld;
    update_blocks<2, true>(tw + c, tw, Lt + c, 0, 2);
  }
  __syncthreads();
  t21_product(TT);
  __syncthreads();
}

}  // namespace b2p
