// Plain FP32 factorization for n > 128: one launch of tile tasks.
//
// The matrix is cut into 64x64 tiles, and task (i, j) produces tile (i, j) of
// L whole, left-looking:
//
//   C = A_ij - sum_{k < j} L_ik L_jk^T        (one 64-wide panel at a time)
//   i == j:  factor C and invert the factor (diag64.cuh); L_jj and
//            T_j = L_jj^{-1} out
//   i >  j:  L_ij = C T_j^T; also clears the upper tile (j, i)
//
// CTAs draw tasks from a ticket counter, column by column, all rows of a
// column and all matrices of a group in turn; the next column's diagonal tile
// comes right after the one tile of this column that it needs, so that its
// factorization runs beside the rest of the column.  A task waits for the tiles it
// reads through per-row progress counters.  Every tile it can wait for has an
// earlier ticket, so it is finished or being worked on by a running CTA: no
// task waits for one that has not started, whatever the number of CTAs the
// GPU runs at a time.  All waits are bounded.  A CTA whose wait gives up takes
// the tickets away, so that the others leave, and the output is marked: info -1
// for the whole batch, and NaN on the diagonal of every L, since callers
// without info have nothing else to see it by.
//
// The order of the tickets is also the look-ahead: while column j's diagonal
// tile is being factored, the CTAs that drew the next columns' tasks
// subtract the panels that are final already.
//
// What bounds it: for few matrices the chain of a column (the last panel of
// the diagonal tile, its factorization, the multiply by T of the next row's
// tile, and the hand-over between CTAs through L2), otherwise the FP32 pipe.
// It replaces three launches and a side-stream update per block column
// (right-looking), whose chain ran through launch gaps and events and which
// read and wrote the trailing matrix once per column.  The arithmetic is the
// same, value for value: a panel's 64 products are summed in order and the sum
// subtracted from the tile, panels in order.
//
// Measured on B200, us per call against that form: 8x2048 1624 -> 775, 50x500
// 290 -> 158, 640x512 1958 -> 1212, 1x8192 10 291 -> 5084 (36 TFLOP/s).  The
// products run on packed multiply-adds (fma2); with fmaf 8x2048 was 884.  The
// chain is 14.6 us a column alone on the GPU (timestamps, 1x1024: diagonal
// engine 5.7, the two products 1.8 and 2.9 with their loads, the rest
// hand-overs) and about 22 us beside other tasks on the same SM.
//
// The reference reaches this schedule through cuSOLVER (submission.py:4268).
#include <algorithm>

#include "diag64.cuh"
#include "launch.h"

namespace b2p {

namespace {

constexpr int kTlB = 64;                  // tile edge
constexpr int kTlThreads = kD64Threads;   // 128: 8x4 outputs per thread
constexpr int kTlLd = kD64Ld;             // row stride of a whole tile
constexpr int kTlHalf = 32;               // panels are staged in halves of 32 columns
constexpr int kTlHalfLd = kTlHalf + 4;
constexpr int kTlRowHalf = kTlB * kTlHalfLd;  // row tile: [row][column]
constexpr int kTlColHalf = kTlHalf * kTlB;    // column tile: [column][row], swizzled
constexpr int kTlStage = kTlRowHalf + kTlColHalf;
constexpr size_t kTlSmem = ((sizeof(Diag64Smem) + 127) & ~(size_t)127) + 64;
constexpr int kTlCtasPerSm = 3;
constexpr uint32_t kTlPolls = 1u << 24;
constexpr int kTlGone = 0x60000000;  // above every ticket (tiles_fits)
static_assert(sizeof(Diag64Smem) >= 2 * kTlStage * sizeof(float), "the stages take the engine's place");
static_assert(sizeof(Diag64Smem) >= 2 * kTlB * kTlLd * sizeof(float), "P and T_j^T take the engine's place");

// Where T_j^T is, T^T[m][c] = T[c][m], 64 x 64 floats: two places in turn, so
// that a column's diagonal tile can be finished while the column before it is
// still being multiplied by its own.  One is the matrix's slot of the
// workspace, the other the upper tile (j, j + 1) of L itself, which the
// diagonal tile two columns on clears.  Column N - 2, whose upper tile may be
// narrower than 64, takes the slot.
__device__ __forceinline__ bool t_above(int j, int N) { return ((N - 2 - j) & 1) != 0; }
// Rows m >= 32 of columns c < 32 are zero in every T^T, so that quarter of the
// slot holds the counters instead (32 per row).
constexpr int kTlSlot = kTlB * kTlB;
constexpr int kTlTicket = 0;   // matrix 0 only: the next task, or from kTlGone on: a wait gave up
constexpr int kTlDone = 2;     // + j % 2: tiles below the diagonal finished in columns of that parity
constexpr int kTlRow = 4;      // + i: tiles of row i finished so far
constexpr int kTlMaxRows = 32 * 32 - kTlRow;

__device__ __forceinline__ int* tl_counter(float* slot, int f) {
  return reinterpret_cast<int*>(slot) + (32 + (f >> 5)) * kTlB + (f & 31);
}

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ int ld_relaxed(const int* p) {
  int v;
  asm volatile("ld.relaxed.gpu.global.b32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}

__device__ __forceinline__ void cp_async16(float* dst, const float* src, bool in) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(s), "l"(src), "r"(in ? 16 : 0) : "memory");
}
__device__ __forceinline__ void cp_async4(float* dst, const float* src, bool in) {
  const unsigned s = (unsigned)__cvta_generic_to_shared(dst);
  asm volatile("cp.async.ca.shared.global [%0], [%1], 4, %2;" ::"r"(s), "l"(src), "r"(in ? 4 : 0) : "memory");
}
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void cp_wait() {
  asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory");
}

// Zeros to rows row0 .. row0 + 63, columns col0 .. col0 + 63 (up to n).
__device__ __forceinline__ void clear_tile(float* mat, int n, int row0, int col0) {
  const int tid = threadIdx.x;
  const int cw = min(kTlB, n - col0);
  float* z = mat + (size_t)row0 * n + col0;
  if ((n & 3) == 0) {
    const int q4 = tid & 15;
    if (4 * q4 < cw)
#pragma unroll
      for (int r = tid >> 4; r < kTlB; r += kTlThreads / 16)
        reinterpret_cast<float4*>(z + (size_t)r * n)[q4] = make_float4(0.f, 0.f, 0.f, 0.f);
  } else {
    for (int e = tid; e < kTlB * kTlB; e += kTlThreads)
      if ((e & 63) < cw) z[(size_t)(e >> 6) * n + (e & 63)] = 0.0f;
  }
}

// Rows row0 .. row0 + 63 (zero from n on) of columns col0 .. col0 + 31.
__device__ __forceinline__ void stage_half(float* dst, const float* mat, int n, int row0, int col0) {
  const int tid = threadIdx.x;
  if ((n & 3) == 0) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int e = tid + kTlThreads * it, r = e >> 3, c = (e & 7) * 4;
      const bool in = row0 + r < n;
      cp_async16(dst + r * kTlHalfLd + c, mat + (size_t)(in ? row0 + r : 0) * n + col0 + c, in);
    }
  } else {
#pragma unroll 4
    for (int it = 0; it < 16; ++it) {
      const int e = tid + kTlThreads * it, r = e >> 5, c = e & 31;
      const bool in = row0 + r < n;
      cp_async4(dst + r * kTlHalfLd + c, mat + (size_t)(in ? row0 + r : 0) * n + col0 + c, in);
    }
  }
}

// The column tile's half goes to shared memory transposed, Bt[m][row], so that
// a thread's four columns of one m are one vector load (fma2).  Through
// registers: fetched a half ahead, stored when its place is free.  Row 4g + e
// of m sits at 4 (g ^ (m / 4 % 8)) + e: a warp's stores of four rows by eight
// m / 4 then meet 32 different banks.
__device__ __forceinline__ void fetch_cols(float (&v)[16], const float* mat, int n, int row0, int col0) {
  const int tid = threadIdx.x;
  if ((n & 3) == 0) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int e = tid + kTlThreads * it, row = row0 + (e >> 3);
      float4 x = make_float4(0.f, 0.f, 0.f, 0.f);
      if (row < n) x = __ldcg(reinterpret_cast<const float4*>(mat + (size_t)row * n + col0 + 4 * (e & 7)));
      v[4 * it] = x.x, v[4 * it + 1] = x.y, v[4 * it + 2] = x.z, v[4 * it + 3] = x.w;
    }
  } else {
#pragma unroll
    for (int it = 0; it < 16; ++it) {
      const int e = tid + kTlThreads * it, row = row0 + (e >> 5);
      v[it] = row < n ? __ldcg(mat + (size_t)row * n + col0 + (e & 31)) : 0.0f;
    }
  }
}
__device__ __forceinline__ int cols_at(int m, int row) { return m * kTlB + (row ^ (4 * ((m >> 2) & 7))); }
__device__ __forceinline__ void store_cols(float* Bt, const float (&v)[16], int n) {
  const int tid = threadIdx.x;
  if ((n & 3) == 0) {
#pragma unroll
    for (int it = 0; it < 4; ++it) {
      const int e = tid + kTlThreads * it;
#pragma unroll
      for (int q = 0; q < 4; ++q) Bt[cols_at(4 * (e & 7) + q, e >> 3)] = v[4 * it + q];
    }
  } else {
#pragma unroll
    for (int it = 0; it < 16; ++it) {
      const int e = tid + kTlThreads * it;
      Bt[cols_at(e & 31, e >> 5)] = v[it];
    }
  }
}

// acc[r][c] += sum_m A[ty + 8r][m] Bt[m][4 tx + c], m = 0 .. M - 1 ascending;
// HALF: a staged half panel (A of row stride kTlHalfLd, Bt as store_cols
// leaves it), else whole tiles of row stride kTlLd.  The half panel's is
// unrolled whole: 1140 cycles a 64x64x64 product per SM with three CTAs (90 %
// of the packed FP32 rate), 1580 unrolled by two.
template <bool HALF>
__device__ __forceinline__ void product(const float* A, const float* Bt, int ty, int tx, float (&acc)[8][4]) {
  constexpr int kLda = HALF ? kTlHalfLd : kTlLd;
#pragma unroll (HALF ? 8 : 2)
  for (int m = 0; m < (HALF ? kTlHalf : kTlB); m += 4) {
    float a[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float4 v = *reinterpret_cast<const float4*>(A + (ty + 8 * r) * kLda + m);
      a[r][0] = v.x, a[r][1] = v.y, a[r][2] = v.z, a[r][3] = v.w;
    }
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float4 b =
          *reinterpret_cast<const float4*>(Bt + (HALF ? cols_at(m, 4 * tx) + p * kTlB : (m + p) * kTlLd + 4 * tx));
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        fma2(acc[r][0], acc[r][1], a[r][p], b.x, b.y);
        fma2(acc[r][2], acc[r][3], a[r][p], b.z, b.w);
      }
    }
  }
}

}  // namespace

__global__ void __launch_bounds__(kTlThreads, kTlCtasPerSm)
    potrf_tiles_kernel(const float* __restrict__ a, float* l, int64_t batch, int n, int64_t group, int total,
                       float* tws, int32_t* info, uint32_t polls) {
  extern __shared__ __align__(16) unsigned char tl_raw[];
  float* const st0 = reinterpret_cast<float*>(tl_raw);  // two stages of (row tile, column tile)
  Diag64Smem& dg = *reinterpret_cast<Diag64Smem*>(tl_raw);
  volatile int* misc = reinterpret_cast<volatile int*>(tl_raw + kTlSmem - 64);
  const int tid = threadIdx.x;
  const int ty = tid >> 4, tx = tid & 15;
  const int N = (n + kTlB - 1) / kTlB;
  const int per = N * (N + 1) / 2;
  const bool vec = (n & 3) == 0;

  for (;;) {
    if (tid == 0) misc[0] = atomicAdd(tl_counter(tws, kTlTicket), 1);
    __syncthreads();
    const int ticket = misc[0];
    if (ticket >= kTlGone) break;
    if (ticket >= total) return;
    // Ticket -> (group of matrices, tile in column order, matrix of the group).
    const int64_t g0 = (int64_t)ticket / (group * per) * group;
    const int64_t gb = min(group, batch - g0);
    const int in_group = (int)(ticket - g0 * per);
    const int64_t b = g0 + in_group % gb;
    const int t = (int)(in_group / gb);
    // Tile 0 is (0, 0); then column q's N - q tiles, from tile 1 + q N -
    // q (q - 1) / 2 on: (q + 1, q), the diagonal tile (q + 1, q + 1), and the
    // rest of the column.
    int i = 0, j = 0;
    if (t > 0) {
      const float fn = 2.0f * N + 1.0f;
      int q = (int)((fn - sqrtf(fmaxf(fn * fn - 8.0f * (t - 1), 0.0f))) * 0.5f);
      q = max(0, min(q, N - 2));
      while (q > 0 && 1 + q * N - q * (q - 1) / 2 > t) --q;
      while (1 + (q + 1) * N - (q + 1) * q / 2 <= t) ++q;
      const int u = t - (1 + q * N - q * (q - 1) / 2);
      i = q + (u == 0 ? 1 : max(u, 1));
      j = u == 1 ? q + 1 : q;
    }

    float* slot = tws + (size_t)b * kTlSlot;
    const float* A = a + (size_t)b * n * n;
    float* L = l + (size_t)b * n * n;
    const int row0 = kTlB * i, col0 = kTlB * j;
    const int w = min(kTlB, n - col0);
    const bool diag = i == j;

    // C = A_ij: rows ty + 8r, columns 4 tx + q.
    float c[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int row = row0 + ty + 8 * r;
      const float* src = A + (size_t)min(row, n - 1) * n + col0 + 4 * tx;
      if (vec && !diag) {
        const float4 v = __ldg(reinterpret_cast<const float4*>(src));
        c[r][0] = v.x, c[r][1] = v.y, c[r][2] = v.z, c[r][3] = v.w;
      } else {
        // The lower part only of a diagonal tile.
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int cl = 4 * tx + q;
          c[r][q] = (row < n && cl < w && (!diag || col0 + cl <= row)) ? __ldg(src + q) : 0.0f;
        }
      }
    }

    // Diagonal tiles: all tiles of columns j - 2, j - 4, ... are finished (the
    // count that says so; whether it was reached when last looked at).
    const int done_want = (j >> 1) * (N - 1 - j) + (j >> 1) * ((j >> 1) + 1);
    bool column_free = false;
    // Number of leading panels known to be final in both rows; the whole CTA
    // calls it.  Waits for at least `need` of them; -1 when that gave up.
    auto panels_ready = [&](int need) -> int {
      if (tid == 0) {
        int got = -1;
        for (uint32_t p = 0; p < polls; ++p) {
          const int pi = ld_relaxed(tl_counter(slot, kTlRow + i));
          const int pj = ld_relaxed(tl_counter(slot, diag ? kTlDone + (j & 1) : kTlRow + j));
          const int both = diag ? pi : min(pi, pj);
          if (both >= need) {
            __threadfence();  // what the counters count was written before them
            got = min(both, j);
            if (diag) misc[4] = pj == done_want;
            break;
          }
          if ((p & 255) == 255 && ld_acquire(tl_counter(tws, kTlTicket)) >= kTlGone) break;
        }
        misc[1] = got;
      }
      __syncthreads();
      const int got = misc[1];
      if (diag) column_free = misc[4] != 0;
      __syncthreads();
      return got;
    };
    // Halves h of panels h / 2, two stages: half h + 1's row tile is copied and
    // its column tile fetched while half h is multiplied.
    auto rows_at = [&](int h) { return st0 + (h & 1) * kTlStage; };
    float cols[16];
    auto fetch = [&](int h) {
      stage_half(rows_at(h), L, n, row0, kTlHalf * h);
      cp_commit();
      fetch_cols(cols, L, n, col0, kTlHalf * h);
    };
    bool ok = true;
    int ready = 0;  // panels known final
    // The counters as thread 0 last read them, a half ago: the next look at
    // them costs nobody a wait.
    int seen_i = 0, seen_j = 0;
    float acc[8][4];
    bool next = false;  // half h has been fetched already
    for (int h = 0; h < 2 * j; ++h) {
      if (!next) {
        ready = panels_ready(h / 2 + 1);
        if (ready < 0) {
          ok = false;
          break;
        }
        fetch(h);
        store_cols(rows_at(h) + kTlRowHalf, cols, n);
      }
      const bool look = ready < j && (h & 1) != 0;
      if (look && tid == 0) {
        // What they count was written before them.
        __threadfence();
        misc[2 + ((h >> 1) & 1)] = min(min(seen_i, seen_j), j);
      }
      cp_wait<0>();
      // Half h has landed, and everyone is done with half h - 1's stage.
      __syncthreads();
      if (look) ready = max(ready, misc[2 + ((h >> 1) & 1)]);
      next = h + 1 < 2 * ready;
      if (next) fetch(h + 1);
      if (ready < j && (h & 1) == 0 && tid == 0) {
        seen_i = ld_relaxed(tl_counter(slot, kTlRow + i));
        seen_j = ld_relaxed(tl_counter(slot, kTlRow + j));
      }
      if ((h & 1) == 0) {
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
          for (int q = 0; q < 4; ++q) acc[r][q] = 0.0f;
      }
      product<true>(rows_at(h), rows_at(h) + kTlRowHalf, ty, tx, acc);
      if ((h & 1) != 0) {
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
          for (int q = 0; q < 4; ++q) c[r][q] -= acc[r][q];
      }
      if (next) store_cols(rows_at(h + 1) + kTlRowHalf, cols, n);
    }
    __syncthreads();

    if (ok && diag) {
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int rl = ty + 8 * r;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int cl = 4 * tx + q;
          dg.S[rl * kD64Ld + cl] = rl < w ? (cl <= rl ? c[r][q] : 0.0f) : (rl == cl ? 1.0f : 0.0f);
        }
      }
      __syncthreads();
      const int bad = diag64_factor_invert(dg);
      // T^T takes the place of column j - 2's, once nobody reads that any more:
      // when all of that column's tiles are finished (most often they were
      // when the last panel was waited for).
      const bool up = t_above(j, N);
      const bool wait = j > 1 && (up || j + 1 < N);
      if (wait && !column_free) {
        if (tid == 0) {
          int got = 0;
          for (uint32_t p = 0; p < polls; ++p) {
            if (ld_acquire(tl_counter(slot, kTlDone + (j & 1))) == done_want) {
              got = 1;
              break;
            }
            if ((p & 255) == 255 && ld_acquire(tl_counter(tws, kTlTicket)) >= kTlGone) break;
          }
          misc[1] = got;
        }
        __syncthreads();
        ok = misc[1] != 0;
      }
      if (ok && j + 1 < N) {
        float* dst = up ? L + (size_t)row0 * n + row0 + kTlB : slot;
        const int ld = up ? n : kTlB;
        if (vec || !up) {
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int e = tid + kTlThreads * it, r = e >> 4, cc = (e & 15) * 4;
            if (up || r < 32 || cc >= 32)
              *reinterpret_cast<float4*>(dst + (size_t)r * ld + cc) =
                  *reinterpret_cast<const float4*>(dg.T + r * kD64Ld + cc);
          }
        } else {
          for (int e = tid; e < kTlB * kTlB; e += kTlThreads)
            dst[(size_t)(e >> 6) * ld + (e & 63)] = dg.T[(e >> 6) * kD64Ld + (e & 63)];
        }
      }
      if (ok && info != nullptr && tid == 0) {
        // Only the last tile has padding, and only a pivot that is infinite makes it bad.
        if (j == 0)
          info[b] = bad >= 0 ? bad + 1 : 0;
        else if (bad >= 0 && col0 + bad < n && __ldcg(info + b) == 0)
          info[b] = col0 + bad + 1;
      }
      __syncthreads();
      if (ok) {
        // T_j is what the column waits for; L_jj itself is nobody's input.
        if (tid == 0) {
          __threadfence();
          atomicExch(tl_counter(slot, kTlRow + i), j + 1);
        }
        if (vec) {
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int e = tid + kTlThreads * it, r = e >> 4, cc = (e & 15) * 4;
            if (r < w && cc < w) {
              const float* sr = dg.S + r * kD64Ld + cc;
              *reinterpret_cast<float4*>(L + (size_t)(row0 + r) * n + col0 + cc) =
                  make_float4(cc <= r ? sr[0] : 0.f, cc + 1 <= r ? sr[1] : 0.f, cc + 2 <= r ? sr[2] : 0.f,
                              cc + 3 <= r ? sr[3] : 0.f);
            }
          }
        } else {
          for (int e = tid; e < kTlB * kTlB; e += kTlThreads) {
            const int r = e >> 6, cc = e & 63;
            if (r < w && cc < w) L[(size_t)(row0 + r) * n + col0 + cc] = cc <= r ? dg.S[r * kD64Ld + cc] : 0.0f;
          }
        }
        if (wait && up) clear_tile(L, n, col0 - 2 * kTlB, col0 - kTlB);
      }
    } else if (ok) {
      // P = C and T_j^T to shared memory, then L_ij = P T_j^T.
      float* P = st0;
      float* Tt = st0 + kTlB * kTlLd;
#pragma unroll
      for (int r = 0; r < 8; ++r)
        *reinterpret_cast<float4*>(P + (ty + 8 * r) * kTlLd + 4 * tx) = make_float4(c[r][0], c[r][1], c[r][2], c[r][3]);
      if (tid == 0) {
        int got = 0;
        for (uint32_t p = 0; p < polls; ++p) {
          if (ld_acquire(tl_counter(slot, kTlRow + j)) > j) {
            got = 1;
            break;
          }
          if ((p & 255) == 255 && ld_acquire(tl_counter(tws, kTlTicket)) >= kTlGone) break;
        }
        misc[1] = got;
      }
      __syncthreads();
      ok = misc[1] != 0;
      if (ok) {
        const bool up = t_above(j, N);
        const float* src = up ? L + (size_t)col0 * n + col0 + kTlB : slot;
        const int ld = up ? n : kTlB;
        if (vec || !up) {
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int e = tid + kTlThreads * it, r = e >> 4, cc = (e & 15) * 4;
            cp_async16(Tt + r * kTlLd + cc, src + (size_t)r * ld + cc, up || r < 32 || cc >= 32);
          }
        } else {
#pragma unroll 8
          for (int it = 0; it < 32; ++it) {
            const int e = tid + kTlThreads * it, r = e >> 6, cc = e & 63;
            cp_async4(Tt + r * kTlLd + cc, src + (size_t)r * ld + cc, true);
          }
        }
        cp_commit();
        cp_wait<0>();
        __syncthreads();
        float x[8][4];
#pragma unroll
        for (int r = 0; r < 8; ++r)
#pragma unroll
          for (int q = 0; q < 4; ++q) x[r][q] = 0.0f;
        product<false>(P, Tt, ty, tx, x);
#pragma unroll
        for (int r = 0; r < 8; ++r) {
          const int row = row0 + ty + 8 * r;
          if (row < n) {
            float* dst = L + (size_t)row * n + col0 + 4 * tx;
            if (vec) {
              *reinterpret_cast<float4*>(dst) = make_float4(x[r][0], x[r][1], x[r][2], x[r][3]);
            } else {
#pragma unroll
              for (int q = 0; q < 4; ++q) dst[q] = x[r][q];
            }
          }
        }
      }
    }
    __syncthreads();
    if (!ok) {
      // A wait gave up: nothing after it can be trusted.
      if (tid == 0) {
        atomicExch(tl_counter(tws, kTlTicket), kTlGone);
        __threadfence();
      }
      __syncthreads();
      break;
    }
    // L_jj and info come before this CTA's next ticket (see the end).
    if (diag && tid == 0) __threadfence();
    if (!diag && tid == 0) {
      __threadfence();
      atomicExch(tl_counter(slot, kTlRow + i), j + 1);
      atomicAdd(tl_counter(slot, kTlDone + (j & 1)), 1);
    }
    // The upper tile (j, i), unless T_j^T is there.
    if (!diag && !(i == j + 1 && t_above(j, N))) clear_tile(L, n, col0, row0);
  }
  // A wait gave up, here or elsewhere: mark the output.  Every store to a marked
  // place is followed by a mark: each CTA draws a ticket after its own stores, and
  // either that is past kTlGone and it marks them itself, or the marks of the CTA
  // that gave up come after its draw and so after them.
  if (info != nullptr)
    for (int64_t q = tid; q < batch; q += kTlThreads) info[q] = -1;
  const int64_t rows = batch * n;
  for (int64_t q = tid; q < rows; q += kTlThreads) {
    const int64_t b = q / n, r = q - b * n;
    l[(size_t)b * n * n + (size_t)r * (n + 1)] = __int_as_float(0x7fc00000);
  }
}

// Whether the tile kernel's counters and tickets cover (batch, n).
bool tiles_fits(int64_t batch, int64_t n) {
  const int64_t N = (n + kTlB - 1) / kTlB;
  return N <= kTlMaxRows && batch * (N * (N + 1) / 2) < (int64_t)1 << 30;
}

// `polls` bounds every wait.  stall (the diagnostic; -1: none): the matrix
// whose finished tiles of the even columns are never counted to the number
// that its diagonal tiles wait for.
static int launch_tiles(const float* a, float* l, int64_t batch, int n, float* tws, int32_t* info, uint32_t polls,
                        int64_t stall, cudaStream_t s) {
  const int N = (n + kTlB - 1) / kTlB;
  const int64_t total = batch * ((int64_t)N * (N + 1) / 2);
  const int64_t slots = (int64_t)device_sms() * kTlCtasPerSm;
  // Matrices taken side by side: enough that a column's tasks are several for
  // every CTA (fewer wait for their column's diagonal tile: 60x1024 874 us at
  // one task per CTA, 720 at four and more; 100x700 543 and 454, 640x512 1334
  // and 1171), and 64 MB of small ones, so that panels read back are in L2.
  const int64_t group = std::max<int64_t>({1, ((int64_t)64 << 20) / (4 * (int64_t)n * n), 8 * slots / N});
  if (int st = ensure_smem_attr((const void*)potrf_tiles_kernel, kTlSmem, kSlotTiles)) return st;
  // The counters (rows 32.. of each slot) start at zero.
  const size_t zero_rows = ((size_t)(kTlRow + N) + 31) / 32;
  const cudaError_t e = cudaMemset2DAsync(tws + 32 * kTlB, kTlSlot * sizeof(float), 0, zero_rows * kTlB * sizeof(float),
                                          (size_t)batch, s);
  if (e != cudaSuccess) return set_error(B2P_ERR_CUDA, "cudaMemset2DAsync(counters): %s", cudaGetErrorString(e));
  if (stall >= 0) {
    // kTlDone + 0 starts far below zero.
    const cudaError_t e2 = cudaMemsetAsync(tws + stall * kTlSlot + 32 * kTlB + kTlDone, 0x80, sizeof(int), s);
    if (e2 != cudaSuccess) return set_error(B2P_ERR_CUDA, "cudaMemsetAsync(counter): %s", cudaGetErrorString(e2));
  }
  {
    TraceScope ts(kKTiles, s, (double)batch * n * n * n / 3.0);
    potrf_tiles_kernel<<<(int)std::min<int64_t>(total, slots), kTlThreads, kTlSmem, s>>>(
        a, l, batch, n, std::min<int64_t>(group, batch), (int)total, tws, info, polls);
  }
  return check_launch("potrf_tiles_kernel");
}

int potrf_tiles(const float* a, float* l, int64_t batch, int n, float* tws, int32_t* info, cudaStream_t s) {
  return launch_tiles(a, l, batch, n, tws, info, kTlPolls, -1, s);
}

}  // namespace b2p

using namespace b2p;

extern "C" int b2p_debug_potrf_tiles_stall(const float* a, float* l, int64_t batch, int64_t n, int64_t matrix,
                                           uint32_t polls, void* workspace, size_t workspace_bytes, int32_t* info,
                                           void* stream) {
  set_error(B2P_OK, "%s", "");
  if (a == nullptr || l == nullptr || a == l || batch <= 0 || n <= 128 || n > (1 << 20) || !tiles_fits(batch, n) ||
      matrix < 0 || matrix >= batch || polls == 0 || polls > kTlPolls)
    return set_error(B2P_ERR_INVALID_ARG, "bad arguments to b2p_debug_potrf_tiles_stall");
  if ((reinterpret_cast<uintptr_t>(a) | reinterpret_cast<uintptr_t>(l) | reinterpret_cast<uintptr_t>(workspace)) & 15u)
    return set_error(B2P_ERR_INVALID_ARG, "buffers must be 16-byte aligned");
  const size_t need = blocked_workspace_bytes(batch, n, B2P_MODE_FP32);
  if (workspace == nullptr || workspace_bytes < need)
    return set_error(B2P_ERR_WORKSPACE, "workspace of %zu bytes required, %zu given", need, workspace_bytes);
  return launch_tiles(a, l, batch, (int)n, static_cast<float*>(workspace), info, polls, matrix,
                      static_cast<cudaStream_t>(stream));
}
