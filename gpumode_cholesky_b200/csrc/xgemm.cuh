// Panel solve X = P T^T for one 128-row tile in shared memory (FP32 SIMT),
// skipping the zero half of T^T (T = L_kk^{-1} is lower triangular, so
// T^T[m][c] = 0 for m > c).
//
// Layout: PtT[m][r] = P[r][m] (64 x 128, row stride ld) and TT[m][c] = T[c][m]
// (64 x 64, row stride ldt).  Eight warps; lane -> rows 4*lane..4*lane+3;
// warp w -> the column groups {4w..4w+3} (m < 4w+4) and {60-4w..63-4w}
// (m < 64-4w), which balances the triangle at 68 K-steps per warp.  PtT is
// overwritten with X, row-major, once every warp has finished reading it;
// `bar` synchronises the 256 threads.  Rows go in pairs through packed
// multiply-adds (a lane's four rows of one m are one vector load).
//
// X keeps its 64-float rows whole so that what writes it out can take 16 (or,
// for the operand copy, 8) neighbouring lanes per row and store full lines; a
// lane per row, from X^T, stored 16 bytes in each of 32 lines at a time, and
// the output took 7.5k of a tile's 14.5k cycles (640 x 512, TF32: 946 -> 869
// us; 60 x 1024: 579 -> 542; 16 x 512: 144 -> 138).  The 16-byte chunks of row
// r are permuted by (r / 4) % 8, which keeps these stores free of bank
// conflicts and the reads at most two-way.
#pragma once

#include "common.cuh"

namespace b2p {

// Columns 4 chunk .. 4 chunk + 3 of row r of X.
__device__ __forceinline__ float4* x_chunk(float* X, int r, int chunk) {
  return reinterpret_cast<float4*>(X + r * 64 + 4 * (chunk ^ ((r >> 2) & 7)));
}

template <class Bar>
__device__ __forceinline__ void xgemm_tri(float* PtT, int ld, const float* TT, int ldt, Bar bar) {
  const int lane = threadIdx.x & 31, w = (threadIdx.x >> 5) & 7;
  const int cA = 4 * w, cB = 60 - 4 * w;
  const int mA = 4 * w + 4, mB = 64 - 4 * w;
  float accA[4][4], accB[4][4];  // [column][row]
#pragma unroll
  for (int i = 0; i < 4; ++i)
#pragma unroll
    for (int j = 0; j < 4; ++j) accA[i][j] = accB[i][j] = 0.0f;
#pragma unroll 4
  for (int m = 0; m < mA; ++m) {
    const float4 a = *reinterpret_cast<const float4*>(PtT + m * ld + 4 * lane);
    const float4 ba = *reinterpret_cast<const float4*>(TT + m * ldt + cA);
    const float4 bb = *reinterpret_cast<const float4*>(TT + m * ldt + cB);
    const float b4a[4] = {ba.x, ba.y, ba.z, ba.w};
    const float b4b[4] = {bb.x, bb.y, bb.z, bb.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      fma2(accA[j][0], accA[j][1], b4a[j], a.x, a.y);
      fma2(accA[j][2], accA[j][3], b4a[j], a.z, a.w);
      fma2(accB[j][0], accB[j][1], b4b[j], a.x, a.y);
      fma2(accB[j][2], accB[j][3], b4b[j], a.z, a.w);
    }
  }
#pragma unroll 4
  for (int m = mA; m < mB; ++m) {
    const float4 a = *reinterpret_cast<const float4*>(PtT + m * ld + 4 * lane);
    const float4 bb = *reinterpret_cast<const float4*>(TT + m * ldt + cB);
    const float b4b[4] = {bb.x, bb.y, bb.z, bb.w};
#pragma unroll
    for (int j = 0; j < 4; ++j) {
      fma2(accB[j][0], accB[j][1], b4b[j], a.x, a.y);
      fma2(accB[j][2], accB[j][3], b4b[j], a.z, a.w);
    }
  }
  bar();
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    *x_chunk(PtT, 4 * lane + i, w) = make_float4(accA[0][i], accA[1][i], accA[2][i], accA[3][i]);
    *x_chunk(PtT, 4 * lane + i, 15 - w) = make_float4(accB[0][i], accB[1][i], accB[2][i], accB[3][i]);
  }
  bar();
}

}  // namespace b2p
