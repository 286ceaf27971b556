// Inverses of the triangular factors of one 64 x 64 complex64 tile, by a CTA of
// kTileThreads threads: for the tile kernel of the tile-pivoting LU and the
// diagonal blocks of the triangular solves.
#pragma once
#include "common.cuh"

namespace mgt {

constexpr int kTileThreads = 512;
constexpr int kTileLD = 66;   // padded row stride of a tile in shared memory (even: pairs of entries load at once)

// s = +- (rows f, f + ldf: K entries) (columns 0, 1 of x: K rows); K even, everything 16-byte aligned
template <bool NEG>
__device__ __forceinline__ void tile_product(float2 (&s)[2][2], const float2* f, int ldf, const float2* x, int ldx,
                                             int K) {
#pragma unroll
  for (int u = 0; u < 2; ++u) s[u][0] = s[u][1] = make_float2(0.f, 0.f);
#pragma unroll 4
  for (int k = 0; k < K; k += 2) {
    const float4 x0 = *reinterpret_cast<const float4*>(x + k * ldx);
    const float4 x1 = *reinterpret_cast<const float4*>(x + (k + 1) * ldx);
#pragma unroll
    for (int u = 0; u < 2; ++u) {
      const float4 a = *reinterpret_cast<const float4*>(f + u * ldf + k);
      const float2 a0 = make_float2(a.x, a.y), a1 = make_float2(a.z, a.w);
      if (NEG) {
        cfms(s[u][0], a0, make_float2(x0.x, x0.y));
        cfms(s[u][1], a0, make_float2(x0.z, x0.w));
        cfms(s[u][0], a1, make_float2(x1.x, x1.y));
        cfms(s[u][1], a1, make_float2(x1.z, x1.w));
      } else {
        cfma(s[u][0], a0, make_float2(x0.x, x0.y));
        cfma(s[u][1], a0, make_float2(x0.z, x0.w));
        cfma(s[u][0], a1, make_float2(x1.x, x1.y));
        cfma(s[u][1], a1, make_float2(x1.z, x1.w));
      }
    }
  }
}

// UI = U^-1 (upper, diagonal reciprocals given) and LI = L^-1 (unit lower) of
// the 64 x 64 tile F by 16 x 16 blocks: the eight diagonal blocks by
// substitution, one per warp, then the block diagonals outwards:
// UI_ij = -UI_ii sum_k U_ik UI_kj and likewise L.  S: 6 x 256 scratch.  Only the
// triangles' blocks are written.
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
  // block diagonals outwards, every block of one at once: 64 threads a block,
  // 2 x 2 entries a thread
  const int bi = tid >> 6, r = 2 * ((tid >> 3) & 7), c = 2 * (tid & 7);
#pragma unroll 1
  for (int d = 1; d < 4; ++d) {
    const int np = 4 - d;
    const bool on = bi < 2 * np, upper = bi < np;
    const int q = upper ? bi : bi - np, i = 16 * q, j = 16 * (q + d);
    float2* I = upper ? UI : LI;
    float2* Sq = S + bi * 256;
    float2 s[2][2];
    if (on) {
      // U: row block i, column block j; L: the mirror image
      tile_product<true>(s, upper ? F + (i + r) * kTileLD + i + 16 : F + (j + r) * kTileLD + i, kTileLD,
                         upper ? I + (i + 16) * kTileLD + j + c : I + i * kTileLD + i + c, kTileLD, 16 * d);
#pragma unroll
      for (int u = 0; u < 2; ++u)
        *reinterpret_cast<float4*>(Sq + (r + u) * 16 + c) = make_float4(s[u][0].x, s[u][0].y, s[u][1].x, s[u][1].y);
    }
    __syncthreads();
    if (on) {
      tile_product<false>(s, upper ? I + (i + r) * kTileLD + i : I + (j + r) * kTileLD + j, kTileLD, Sq + c, 16, 16);
#pragma unroll
      for (int u = 0; u < 2; ++u)
        *reinterpret_cast<float4*>(upper ? I + (i + r + u) * kTileLD + j + c : I + (j + r + u) * kTileLD + i + c) =
            make_float4(s[u][0].x, s[u][0].y, s[u][1].x, s[u][1].y);
    }
    __syncthreads();
  }
}

}  // namespace mgt
