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
// column and all matrices of a group in turn.  A task waits for the tiles it
// reads through per-row progress counters.  Every tile it can wait for has an
// earlier ticket, so it is finished or being worked on by a running CTA: no
// task waits for one that has not started, whatever the number of CTAs the
// GPU runs at a time.  All waits are bounded.
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
// Measured on B200, us per call against that form: 8x2048 1624 -> 884, 50x500
// 290 -> 172, 640x512 1958 -> 1492 (19 TFLOP/s; ncu: issue slots 52 % busy,
// FMA pipe 38 %, three warps per scheduler).
//
// The reference reaches this schedule through cuSOLVER (submission.py:4268).
#include <algorithm>

#include "diag64.cuh"
#include "launch.h"

namespace b2p {

namespace {

constexpr int kTlB = 64;                  // tile edge
constexpr int kTlThreads = kD64Threads;   // 128: 8x4 outputs per thread
constexpr int kTlLd = kD64Ld;             // 68
constexpr int kTlTile = kTlB * kTlLd;     // floats per staged tile
constexpr size_t kTlSmem = 4 * kTlTile * sizeof(float) + 64;
constexpr int kTlCtasPerSm = 3;
constexpr uint32_t kTlPolls = 1u << 24;
static_assert(sizeof(Diag64Smem) <= 4 * kTlTile * sizeof(float), "the engine's state takes the staging's place");

// The workspace holds T_j^T of each matrix's current column, 64 x 64 floats,
// T^T[m][c] = T[c][m].  Rows m >= 32 of columns c < 32 are zero in every T^T,
// so that quarter of the slot holds the counters instead (32 per row).
constexpr int kTlSlot = kTlB * kTlB;
constexpr int kTlTicket = 0;   // matrix 0 only: the next task
constexpr int kTlAbort = 1;    // matrix 0 only: a wait gave up
constexpr int kTlDone = 2;     // tiles below the diagonal finished so far
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

// Rows row0 .. row0 + 63 (zero from n on) of columns col0 .. col0 + 63.
__device__ __forceinline__ void stage_tile(float* dst, const float* mat, int n, int row0, int col0) {
  const int tid = threadIdx.x;
  if ((n & 3) == 0) {
#pragma unroll
    for (int it = 0; it < 8; ++it) {
      const int e = tid + kTlThreads * it, r = e >> 4, c = (e & 15) * 4;
      const bool in = row0 + r < n;
      cp_async16(dst + r * kTlLd + c, mat + (size_t)(in ? row0 + r : 0) * n + col0 + c, in);
    }
  } else {
#pragma unroll 8
    for (int it = 0; it < 32; ++it) {
      const int e = tid + kTlThreads * it, r = e >> 6, c = e & 63;
      const bool in = row0 + r < n;
      cp_async4(dst + r * kTlLd + c, mat + (size_t)(in ? row0 + r : 0) * n + col0 + c, in);
    }
  }
}

// acc[r][q] = sum_m A[ty + 8r][m] B[tx + 16q][m], m ascending.
__device__ __forceinline__ void tile_abt(const float* A, const float* B, int ty, int tx, float (&acc)[8][4]) {
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[r][q] = 0.0f;
#pragma unroll 2
  for (int m = 0; m < kTlB; m += 4) {
    float b[4][4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
      const float4 v = *reinterpret_cast<const float4*>(B + (tx + 16 * q) * kTlLd + m);
      b[q][0] = v.x, b[q][1] = v.y, b[q][2] = v.z, b[q][3] = v.w;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float4 v = *reinterpret_cast<const float4*>(A + (ty + 8 * r) * kTlLd + m);
      const float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[r][q] = fmaf(a[p], b[q][p], acc[r][q]);
    }
  }
}

// acc[r][c] = sum_m A[ty + 8r][m] Bt[m][4 tx + c], m ascending.
__device__ __forceinline__ void tile_ab(const float* A, const float* Bt, int ty, int tx, float (&acc)[8][4]) {
#pragma unroll
  for (int r = 0; r < 8; ++r)
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[r][q] = 0.0f;
#pragma unroll 2
  for (int m = 0; m < kTlB; m += 4) {
    float b[4][4];
#pragma unroll
    for (int p = 0; p < 4; ++p) {
      const float4 v = *reinterpret_cast<const float4*>(Bt + (m + p) * kTlLd + 4 * tx);
      b[p][0] = v.x, b[p][1] = v.y, b[p][2] = v.z, b[p][3] = v.w;
    }
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const float4 v = *reinterpret_cast<const float4*>(A + (ty + 8 * r) * kTlLd + m);
      const float a[4] = {v.x, v.y, v.z, v.w};
#pragma unroll
      for (int p = 0; p < 4; ++p)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[r][q] = fmaf(a[p], b[p][q], acc[r][q]);
    }
  }
}

}  // namespace

__global__ void __launch_bounds__(kTlThreads, kTlCtasPerSm)
    potrf_tiles_kernel(const float* __restrict__ a, float* l, int64_t batch, int n, int64_t group, int total,
                       float* tws, int32_t* info) {
  extern __shared__ __align__(16) unsigned char tl_raw[];
  float* const st0 = reinterpret_cast<float*>(tl_raw);  // two stages of (row tile, column tile)
  Diag64Smem& dg = *reinterpret_cast<Diag64Smem*>(tl_raw);
  volatile int* misc = reinterpret_cast<volatile int*>(st0 + 4 * kTlTile);
  const int tid = threadIdx.x;
  const int ty = tid >> 4, tx = tid & 15;
  const int N = (n + kTlB - 1) / kTlB;
  const int per = N * (N + 1) / 2;
  const bool vec = (n & 3) == 0;

  for (;;) {
    if (tid == 0) misc[0] = atomicAdd(tl_counter(tws, kTlTicket), 1);
    __syncthreads();
    const int ticket = misc[0];
    if (ticket >= total) return;
    // Ticket -> (group of matrices, tile in column order, matrix of the group).
    const int64_t g0 = (int64_t)ticket / (group * per) * group;
    const int64_t gb = min(group, batch - g0);
    const int in_group = (int)(ticket - g0 * per);
    const int64_t b = g0 + in_group % gb;
    const int t = (int)(in_group / gb);
    // Column j starts at tile j N - j (j - 1) / 2.
    const float fn = 2.0f * N + 1.0f;
    int j = (int)((fn - sqrtf(fmaxf(fn * fn - 8.0f * t, 0.0f))) * 0.5f);
    j = max(0, min(j, N - 1));
    while (j > 0 && j * N - j * (j - 1) / 2 > t) --j;
    while ((j + 1) * N - (j + 1) * j / 2 <= t) ++j;
    const int i = j + t - (j * N - j * (j - 1) / 2);

    float* slot = tws + (size_t)b * kTlSlot;
    const float* A = a + (size_t)b * n * n;
    float* L = l + (size_t)b * n * n;
    const int row0 = kTlB * i, col0 = kTlB * j;
    const int w = min(kTlB, n - col0);
    const bool diag = i == j;

    // C = A_ij (lower part only of a diagonal tile).
    float c[8][4];
#pragma unroll
    for (int r = 0; r < 8; ++r) {
      const int row = row0 + ty + 8 * r;
      const float* src = A + (size_t)min(row, n - 1) * n + col0;
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const int cl = tx + 16 * q;
        c[r][q] = (row < n && cl < w && (!diag || col0 + cl <= row)) ? __ldg(src + cl) : 0.0f;
      }
    }

    // Number of leading panels known to be final in both rows; the whole CTA
    // calls it.  Waits for at least `need` of them; -1 when that gave up.
    auto panels_ready = [&](int need) -> int {
      if (tid == 0) {
        int got = -1;
        for (uint32_t p = 0; p < kTlPolls; ++p) {
          const int pi = ld_acquire(tl_counter(slot, kTlRow + i));
          const int pj = diag ? pi : ld_acquire(tl_counter(slot, kTlRow + j));
          if (min(pi, pj) >= need) {
            got = min(min(pi, pj), j);
            break;
          }
          if ((p & 255) == 255 && ld_acquire(tl_counter(tws, kTlAbort)) != 0) break;
        }
        misc[1] = got;
      }
      __syncthreads();
      const int got = misc[1];
      __syncthreads();
      return got;
    };
    auto stage = [&](int k) {
      float* dst = st0 + (k & 1) * 2 * kTlTile;
      stage_tile(dst, L, n, row0, kTlB * k);
      if (!diag) stage_tile(dst + kTlTile, L, n, col0, kTlB * k);
      cp_commit();
    };
    bool ok = true;
    int ready = 0, staged = 0;
    for (int k = 0; k < j; ++k) {
      // Panel k must be on its way, panel k + 1 should be.
      if (staged >= ready && staged < min(k + 2, j)) {
        const int got = panels_ready(staged > k ? 0 : k + 1);
        if (got < 0) {
          ok = false;
          break;
        }
        ready = got;
      }
      while (staged < min(k + 2, ready)) stage(staged++);
      if (staged > k + 1)
        cp_wait<1>();
      else
        cp_wait<0>();
      __syncthreads();
      const float* At = st0 + (k & 1) * 2 * kTlTile;
      float acc[8][4];
      tile_abt(At, diag ? At : At + kTlTile, ty, tx, acc);
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) c[r][q] -= acc[r][q];
      __syncthreads();
    }

    if (ok && diag) {
#pragma unroll
      for (int r = 0; r < 8; ++r) {
        const int rl = ty + 8 * r;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          const int cl = tx + 16 * q;
          dg.S[rl * kD64Ld + cl] = rl < w ? (cl <= rl ? c[r][q] : 0.0f) : (rl == cl ? 1.0f : 0.0f);
        }
      }
      __syncthreads();
      const int bad = diag64_factor_invert(dg);
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
      if (j + 1 < N) {
        // T^T takes the slot of column j - 1's, once nobody reads that any
        // more: when all of that column's tiles are finished.
        if (j > 0) {
          if (tid == 0) {
            const int want = j * N - j * (j + 1) / 2;
            int got = 0;
            for (uint32_t p = 0; p < kTlPolls; ++p) {
              if (ld_acquire(tl_counter(slot, kTlDone)) == want) {
                got = 1;
                break;
              }
              if ((p & 255) == 255 && ld_acquire(tl_counter(tws, kTlAbort)) != 0) break;
            }
            misc[1] = got;
          }
          __syncthreads();
          ok = misc[1] != 0;
        }
        if (ok) {
#pragma unroll
          for (int it = 0; it < 8; ++it) {
            const int e = tid + kTlThreads * it, r = e >> 4, cc = (e & 15) * 4;
            if (r < 32 || cc >= 32)
              *reinterpret_cast<float4*>(slot + r * kTlB + cc) =
                  *reinterpret_cast<const float4*>(dg.T + r * kD64Ld + cc);
          }
        }
      }
      if (info != nullptr && tid == 0) {
        if (j == 0)
          info[b] = bad >= 0 ? bad + 1 : 0;
        else if (bad >= 0 && __ldcg(info + b) == 0)
          info[b] = col0 + bad + 1;
      }
    } else if (ok) {
      // P = C and T_j^T to shared memory, then L_ij = P T_j^T.
      float* P = st0;
      float* Tt = st0 + kTlTile;
#pragma unroll
      for (int r = 0; r < 8; ++r)
#pragma unroll
        for (int q = 0; q < 4; ++q) P[(ty + 8 * r) * kTlLd + tx + 16 * q] = c[r][q];
      if (tid == 0) {
        int got = 0;
        for (uint32_t p = 0; p < kTlPolls; ++p) {
          if (ld_acquire(tl_counter(slot, kTlRow + j)) > j) {
            got = 1;
            break;
          }
          if ((p & 255) == 255 && ld_acquire(tl_counter(tws, kTlAbort)) != 0) break;
        }
        misc[1] = got;
      }
      __syncthreads();
      ok = misc[1] != 0;
      if (ok) {
#pragma unroll
        for (int it = 0; it < 8; ++it) {
          const int e = tid + kTlThreads * it, r = e >> 4, cc = (e & 15) * 4;
          cp_async16(Tt + r * kTlLd + cc, slot + r * kTlB + cc, r < 32 || cc >= 32);
        }
        cp_commit();
        cp_wait<0>();
        __syncthreads();
        float x[8][4];
        tile_ab(P, Tt, ty, tx, x);
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
      if (tid == 0) atomicExch(tl_counter(tws, kTlAbort), 1);
      if (info != nullptr)
        for (int64_t q = tid; q < batch; q += kTlThreads) info[q] = -1;
      return;
    }
    if (tid == 0) {
      __threadfence();
      if (!diag) atomicAdd(tl_counter(slot, kTlDone), 1);
      atomicExch(tl_counter(slot, kTlRow + i), j + 1);
    }
    if (!diag) {
      // The upper tile (j, i).
      const int cw = min(kTlB, n - row0);
      float* zb = L + (size_t)col0 * n + row0;
      if (vec) {
        const int q4 = tid & 15;
        if (4 * q4 < cw)
#pragma unroll
          for (int r = tid >> 4; r < kTlB; r += kTlThreads / 16)
            reinterpret_cast<float4*>(zb + (size_t)r * n)[q4] = make_float4(0.f, 0.f, 0.f, 0.f);
      } else {
        for (int e = tid; e < kTlB * kTlB; e += kTlThreads)
          if ((e & 63) < cw) zb[(size_t)(e >> 6) * n + (e & 63)] = 0.0f;
      }
    }
  }
}

// Whether the tile kernel's counters and tickets cover (batch, n).
bool tiles_fits(int64_t batch, int64_t n) {
  const int64_t N = (n + kTlB - 1) / kTlB;
  return N <= kTlMaxRows && batch * (N * (N + 1) / 2) < (int64_t)1 << 30;
}

int potrf_tiles(const float* a, float* l, int64_t batch, int n, float* tws, int32_t* info, cudaStream_t s) {
  const int N = (n + kTlB - 1) / kTlB;
  const int64_t total = batch * ((int64_t)N * (N + 1) / 2);
  const int64_t slots = (int64_t)device_sms() * kTlCtasPerSm;
  // Matrices taken side by side: about 64 MB of them, so that the panels read
  // back are in L2, but at least enough that a column has a task per CTA.
  const int64_t group = std::max<int64_t>({1, ((int64_t)64 << 20) / (4 * (int64_t)n * n), (slots + N - 1) / N});
  if (int st = ensure_smem_attr((const void*)potrf_tiles_kernel, kTlSmem, kSlotTiles)) return st;
  // The counters (rows 32.. of each slot) start at zero.
  const size_t zero_rows = ((size_t)(kTlRow + N) + 31) / 32;
  const cudaError_t e = cudaMemset2DAsync(tws + 32 * kTlB, kTlSlot * sizeof(float), 0, zero_rows * kTlB * sizeof(float),
                                          (size_t)batch, s);
  if (e != cudaSuccess) return set_error(B2P_ERR_CUDA, "cudaMemset2DAsync(counters): %s", cudaGetErrorString(e));
  {
    TraceScope ts(kKTiles, s, (double)batch * n * n * n / 3.0);
    potrf_tiles_kernel<<<(int)std::min<int64_t>(total, slots), kTlThreads, kTlSmem, s>>>(
        a, l, batch, n, std::min<int64_t>(group, batch), (int)total, tws, info);
  }
  return check_launch("potrf_tiles_kernel");
}

}  // namespace b2p
