// Inverses of the triangular factors of one 64 x 64 complex64 tile, by a CTA of
// kTileThreads threads: for the tile kernel of the tile-pivoting LU and the
// diagonal blocks of the triangular solves.
#pragma once
#include "common.cuh"

namespace mgt {

constexpr int kTileThreads = 512;
constexpr int kTileLD = 66;   // padded row stride of a tile in shared memory (even: pairs of entries load at once)

// UI = U^-1 (upper, diagonal reciprocals given) and LI = L^-1 (unit lower) of
// the 64 x 64 tile F by 16 x 16 blocks: the eight diagonal blocks by
// substitution, one per warp, then the block diagonals outwards:
// UI_ij = -UI_ii sum_k U_ik UI_kj by threads 0 .. 255 and likewise L by the
// others.  S: 6 x 256 scratch.  Only the triangles' blocks are written.
__device__ __forceinline__ void tile_inverses(const float2* F, float2* UI, float2* LI, float2* S, const float2* dinv,
                                              int tid) {
  const int warp = tid >> 5, lane = tid & 31;
  if (warp < 8 && lane < 16) {
    // Columns of the inverse, one per lane, right-looking.  L's blocks read from
    // the last row and column backwards are upper triangular with a unit
    // diagonal: one piece of code for both.
    const int b = (warp & 3) * 16;
    const bool up = warp < 4;
    const float2* f = up ? F + b * kTileLD + b : F + (b + 15) * kTileLD + b + 15;
    const int rs = up ? kTileLD : -kTileLD, cs = up ? 1 : -1;
    float2 x[16];
#pragma unroll
    for (int i = 0; i < 16; ++i) x[i] = make_float2(i == lane ? 1.f : 0.f, 0.f);
#pragma unroll
    for (int i = 15; i >= 0; --i) {
      if (up) x[i] = cmul(x[i], dinv[b + i]);
#pragma unroll
      for (int k = 0; k < i; ++k) cfms(x[k], f[k * rs + i * cs], x[i]);
    }
    float2* out = up ? UI + b * kTileLD + b + lane : LI + (b + 15) * kTileLD + b + 15 - lane;
#pragma unroll
    for (int i = 0; i < 16; ++i) out[i * rs] = x[i];
  }
  __syncthreads();
  const bool upper = tid < 256;
  const int t = tid & 255, r = t >> 4, c = t & 15;   // this thread's entry of every block
  float2* I = upper ? UI : LI;
  float2* Sq = S + (upper ? 0 : 3 * 256);
#pragma unroll 1
  for (int d = 1; d < 4; ++d) {
    const int np = 4 - d;
#pragma unroll 1
    for (int q = 0; q < np; ++q) {
      // U: row block i, column block i + 16 d; L: the mirror image
      const int i = 16 * q, j = 16 * (q + d);
      const float2* f = upper ? F + (i + r) * kTileLD + i + 16 : F + (j + r) * kTileLD + i;
      const float2* x = upper ? I + (i + 16) * kTileLD + j + c : I + i * kTileLD + i + c;
      float2 s0 = make_float2(0.f, 0.f), s1 = s0;
#pragma unroll 8
      for (int k = 0; k < 16 * d; k += 2) {
        const float4 v = *reinterpret_cast<const float4*>(f + k);
        cfms(s0, make_float2(v.x, v.y), x[k * kTileLD]);
        cfms(s1, make_float2(v.z, v.w), x[(k + 1) * kTileLD]);
      }
      Sq[q * 256 + t] = cadd(s0, s1);
    }
    __syncthreads();
#pragma unroll 1
    for (int q = 0; q < np; ++q) {
      const int i = 16 * q, j = 16 * (q + d);
      const float2* f = upper ? I + (i + r) * kTileLD + i : I + (j + r) * kTileLD + j;
      const float2* x = Sq + q * 256 + c;
      float2 s0 = make_float2(0.f, 0.f), s1 = s0;
#pragma unroll
      for (int k = 0; k < 16; k += 2) {
        const float4 v = *reinterpret_cast<const float4*>(f + k);
        cfma(s0, make_float2(v.x, v.y), x[k * 16]);
        cfma(s1, make_float2(v.z, v.w), x[(k + 1) * 16]);
      }
      (upper ? I[(i + r) * kTileLD + j + c] : I[(j + r) * kTileLD + i + c]) = cadd(s0, s1);
    }
    __syncthreads();
  }
}

}  // namespace mgt
