// K3: complex64 multi-RHS triangular solves with the LU factors (the ?getrs
// half of torch.linalg.solve in solve(), Transmission2D.py:230 /
// Transmission3D.py:205).
//
// Block rows of 256, right-looking, one launch per block row: launch i
// subtracts T_ki X_i from every block row k that depends on it, and the
// cluster that holds the next block row goes on to X_k = T_kk^-1 B_k.  The
// inverses of the 256 x 256 diagonal blocks are made first: 64 x 64 blocks by
// substitution, doubled twice.
//
// What bounds a solve of few columns is the chain from block row to block row
// (n / 256 per triangle), then the factor's bytes; so a launch is one
// eight-CTA cluster per block row and 32 columns -- two halves of 128 rows,
// the K = 256 split over four CTAs, their sums exchanged through distributed
// shared memory -- and starts while its predecessor runs (programmatic
// dependent launch): barriers, tensor memory, the factor's block and its
// conversion are done before it waits for X_i.
//
// Products on the tensor cores: both operands scaled by a power of two (each
// row of the factor's tile, each right-hand side) to just below 2^15 and split
// into two fp16 parts, x = h + 2^-11 l, each rounded to nearest, so that h and
// l keep the full 22 bits down to 2^-28 of the largest value (2^-50 of it
// absolutely); the four part products accumulate in FP32 by weight
// (h h | h l + l h | l l).  Where the rows of the right-hand sides differ by more
// than 2^13 in their means, as they do for column-scaled factors, large values
// of one operand meet small ones of the other and that is not enough: such a
// product of 64 columns of K is made on the FP32 pipe (kTSpread).
//
// Measured, LU solve of 64 columns with the inverses made (ms): n = 2000 0.26,
// 6000 0.85, 12000 2.01; work items of 64-row blocks claimed by persistent CTAs,
// products on the FP32 pipe: 0.54, 1.66, 3.93.  A step takes 11 us on the chain
// (two products, each with its exchange of partial sums); from n = 6000 on the
// block rows beyond take as long or longer (12000: 20 us).
#include <cuda_fp16.h>

#include <algorithm>
#include <mutex>

#include "common.cuh"
#include "diag.cuh"
#include "tcgen05.cuh"
#include "tile_inverse.cuh"

namespace mgt {

constexpr int kTB = 64;       // order of the blocks inverted by substitution
constexpr int kTD = 256;      // block rows of the solve
constexpr int kTC = 32;       // right-hand sides per cluster
constexpr int kTK = 64;       // complex K per CTA
constexpr int kTThreads = 256;

// Row stride of the right-hand sides in lower_inverse_kernel: the four lanes
// of a column group read rows r..r+3, and a stride of 72 complex64 (an odd
// multiple of 64 bytes) puts those rows on different banks (with 64 they
// shared one: 4-way conflicts on every access).
constexpr int kInvLd = kTB + 8;
constexpr size_t kInvSmem = (size_t)(kTB * (kTB + 1) + kTB * kInvLd) * sizeof(float2);

// Inverses of the 64 x 64 diagonal blocks of a unit lower factor: one CTA per
// block, identity right-hand sides, substitution in shared memory.  Warp w owns
// columns 8w..8w+7 of the inverse, which is lower triangular: the steps above
// those columns multiply exact zeros and are skipped.
__global__ void __launch_bounds__(256)
lower_inverse_kernel(const float2* __restrict__ F, int64_t ldf, int n, float2* __restrict__ Inv) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  float2* Ts = reinterpret_cast<float2*>(smem_raw);   // [kTB][kTB + 1]
  float2* Xs = Ts + kTB * (kTB + 1);                    // [kTB][kInvLd]
  const int tid = threadIdx.x, r0 = blockIdx.x * kTB, rb = min(kTB, n - r0);
  for (int idx = tid; idx < kTB * kTB; idx += 256) {
    int r = idx >> 6, c = idx & 63;
    const bool ok = r < rb && c < rb;
    cp_async_elem<8>(Ts + r * (kTB + 1) + c, ok ? F + (int64_t)(r0 + r) * ldf + r0 + c : F, ok);
    Xs[r * kInvLd + c] = make_float2(r == c ? 1.f : 0.f, 0.f);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  const int warp = tid >> 5, lane = tid & 31;
  const int col = warp * 8 + (lane >> 2), t4 = lane & 3;   // 4 lanes per column, 64 columns
  for (int kk = warp * 8; kk < rb - 1; ++kk) {
    __syncwarp();
    const float2 xk = Xs[kk * kInvLd + col];
    for (int r = kk + 1 + t4; r < rb; r += 4) cfms(Xs[r * kInvLd + col], Ts[r * (kTB + 1) + kk], xk);
  }
  __syncthreads();
  float2* out = Inv + (int64_t)blockIdx.x * kTB * kTB;
  for (int idx = tid; idx < kTB * kTB; idx += 256) out[idx] = Xs[(idx >> 6) * kInvLd + (idx & 63)];
}

// The 64 x 64 diagonal blocks of the block rows' inverses, L's and U's, and
// zeros in the 64-column blocks beside each that lie outside the triangle; the
// sums of |entries| of the 256 x 256 diagonal blocks' rows.
constexpr size_t kInv64Smem = (3 * 64 * kTileLD + 6 * 256) * sizeof(float2);
__global__ void __launch_bounds__(kTileThreads)
tri_inverse64_kernel(const float2* __restrict__ F, int64_t ldf, int n, int nb, float2* __restrict__ Inv,
                     float* __restrict__ rowsum, float* __restrict__ cond) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  float2* Ts = reinterpret_cast<float2*>(smem_raw);   // [64][kTileLD]: the factors' block
  float2* UI = Ts + 64 * kTileLD;
  float2* LI = UI + 64 * kTileLD;
  float2* S = LI + 64 * kTileLD;                        // 6 x 256
  __shared__ float2 dinv[64];
  const int tid = threadIdx.x, q = blockIdx.x & 3, b = blockIdx.x >> 2;
  const int r0 = b * kTD + q * kTB, rb = max(0, min(kTB, n - r0));
  float2* lrows = Inv + (int64_t)b * kTD * kTD + q * kTB * kTD;
  float2* urows = lrows + (int64_t)nb * kTD * kTD;
  for (int idx = tid; idx < kTB * kTB; idx += kTileThreads) {
    const int r = idx >> 6, c = idx & 63;
    Ts[r * kTileLD + c] = r < rb && c < rb ? F[(int64_t)(r0 + r) * ldf + r0 + c] : make_float2(r == c ? 1.f : 0.f, 0.f);
  }
  for (int r = tid >> 5; r < kTB; r += kTileThreads / 32) {
    for (int c = (q + 1) * kTB + (tid & 31); c < kTD; c += 32) lrows[r * kTD + c] = make_float2(0.f, 0.f);
    for (int c = tid & 31; c < q * kTB; c += 32) urows[r * kTD + c] = make_float2(0.f, 0.f);
    float sl = 0.f, su = 0.f;
#pragma unroll
    for (int j = 0; j < kTD / 32; ++j) {
      const int c = (tid & 31) + 32 * j, rr = q * kTB + r;
      if (r < rb && b * kTD + c < n) {
        const float2 v = F[(int64_t)(r0 + r) * ldf + b * kTD + c];
        (c < rr ? sl : su) += fabsf(v.x) + fabsf(v.y);
      }
    }
    for (int o = 16; o; o >>= 1) {
      sl += __shfl_xor_sync(0xffffffffu, sl, o);
      su += __shfl_xor_sync(0xffffffffu, su, o);
    }
    if ((tid & 31) == 0) {
      rowsum[b * kTD + q * kTB + r] = sl + 1.f;
      rowsum[(nb + b) * kTD + q * kTB + r] = su;
    }
  }
  if (tid < 2 && q == 0) cond[tid * nb + b] = 0.f;
  __syncthreads();
  if (tid < kTB) dinv[tid] = crecip(Ts[tid * kTileLD + tid]);
  __syncthreads();
  tile_inverses(Ts, UI, LI, S, dinv, tid);
  for (int idx = tid; idx < kTB * kTB; idx += kTileThreads) {
    const int r = idx >> 6, c = idx & 63;
    urows[r * kTD + q * kTB + c] = c >= r ? UI[r * kTileLD + c] : make_float2(0.f, 0.f);
    lrows[r * kTD + q * kTB + c] = c < r ? LI[r * kTileLD + c] : make_float2(r == c ? 1.f : 0.f, 0.f);
  }
}

// acc (H x 16, this thread's rows rg + 32 a, columns 2 cg, 2 cg + 1) += A (H x H, row stride lda,
// rows < rn and columns < cn) * Bs (H x 16 in shared memory), K chunks of 32 from kb to ke.
// TRI 1 (2): A is lower (upper) triangular.  The next chunk loads during the products.
template <int H, int TRI>
__device__ __forceinline__ void strip_mm(float2 (&acc)[H / 32][2], const float2* __restrict__ A, int64_t lda, int rn,
                                         int cn, const float2* Bs, float2* As, int kb, int ke, int tid) {
  const int rg = tid >> 3, cg = tid & 7;
  auto load = [&](int kc) {
    float2* d = As + (kc & 1) * (H * 33);
    for (int idx = tid; idx < H * 32; idx += 256) {
      const int r = idx >> 5, c = 32 * kc + (idx & 31);
      const bool ok = r < rn && c < cn;
      cp_async_elem<8>(d + r * 33 + (idx & 31), ok ? A + (int64_t)r * lda + c : A, ok);
    }
    cp_async_commit();
  };
  __syncthreads();
  load(kb);
#pragma unroll
  for (int kc = 0; kc < H / 32; ++kc) {
    if (kc < kb || kc >= ke) continue;
    if (kc + 1 < ke) {
      load(kc + 1);
      cp_async_wait<1>();
    } else {
      cp_async_wait<0>();
    }
    __syncthreads();
    const float2* d = As + (kc & 1) * (H * 33);
#pragma unroll 8
    for (int k = 0; k < 32; ++k) {
      const float4 b = *reinterpret_cast<const float4*>(Bs + (32 * kc + k) * 16 + 2 * cg);
#pragma unroll
      for (int a = TRI == 1 ? kc : 0; a < (TRI == 2 ? kc + 1 : H / 32); ++a) {
        const float2 x = d[(rg + 32 * a) * 33 + k];
        cfma(acc[a][0], x, make_float2(b.x, b.y));
        cfma(acc[a][1], x, make_float2(b.z, b.w));
      }
    }
    __syncthreads();
  }
}

// One doubling of the inverses, H x H blocks to 2H x 2H: for L = [A 0; C B],
// -B^-1 (C A^-1); for U = [A C; 0 B], -A^-1 (C B^-1); 16 columns per CTA.
// Grid: x = (block row, pair, strip), y = L / U.
template <int H> constexpr size_t tri_double_smem() { return (size_t)H * (2 * 16 + 2 * 33) * sizeof(float2); }
template <int H>
__global__ void __launch_bounds__(256)
tri_double_kernel(const float2* __restrict__ F, int64_t ldf, int n, int nb, float2* __restrict__ Inv) {
  constexpr int PAIRS = kTD / (2 * H), STRIPS = H / 16, KC = H / 32;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  float2* Bs = reinterpret_cast<float2*>(smem_raw);   // [H][16]
  float2* Ss = Bs + H * 16;                             // [H][16]
  float2* As = Ss + H * 16;                             // 2 x [H][33]
  const int tid = threadIdx.x;
  const int strip = blockIdx.x % STRIPS, pair = (blockIdx.x / STRIPS) % PAIRS, b = blockIdx.x / (STRIPS * PAIRS);
  const bool upper = blockIdx.y != 0;
  const int o = pair * 2 * H, c0 = strip * 16;   // the pair's offset within the block row
  float2* I = Inv + ((int64_t)(upper ? nb : 0) + b) * kTD * kTD;
  // the right factor's diagonal block (A for L, B for U), the left one's, C
  const int ro = o + (upper ? H : 0), lo = o + (upper ? 0 : H);
  const int crow = b * kTD + lo, ccol = b * kTD + ro;
  for (int idx = tid; idx < H * 16; idx += 256) {
    const int r = idx >> 4, c = idx & 15;
    Bs[idx] = I[(int64_t)(ro + r) * kTD + ro + c0 + c];
  }
  const int rg = tid >> 3, cg = tid & 7;
  float2 acc[KC][2];
#pragma unroll
  for (int a = 0; a < KC; ++a) acc[a][0] = acc[a][1] = make_float2(0.f, 0.f);
  const int rn = max(0, min(H, n - crow)), cn = max(0, min(H, n - ccol));
  // columns c0 .. + 15 of a triangular inverse: rows from c0 on (L), to c0 + 15 (U)
  strip_mm<H, 0>(acc, rn > 0 && cn > 0 ? F + (int64_t)crow * ldf + ccol : F, ldf, rn, cn, Bs, As, upper ? 0 : c0 >> 5,
                 upper ? (c0 >> 5) + 1 : KC, tid);
#pragma unroll
  for (int a = 0; a < KC; ++a) {
    *reinterpret_cast<float4*>(Ss + (rg + 32 * a) * 16 + 2 * cg) =
        make_float4(acc[a][0].x, acc[a][0].y, acc[a][1].x, acc[a][1].y);
    acc[a][0] = acc[a][1] = make_float2(0.f, 0.f);
  }
  const float2* D = I + (int64_t)lo * kTD + lo;
  if (upper) strip_mm<H, 2>(acc, D, kTD, H, H, Ss, As, 0, KC, tid);
  else strip_mm<H, 1>(acc, D, kTD, H, H, Ss, As, 0, KC, tid);
#pragma unroll
  for (int a = 0; a < KC; ++a)
#pragma unroll
    for (int j = 0; j < 2; ++j)
      I[(int64_t)(lo + rg + 32 * a) * kTD + ro + c0 + 2 * cg + j] = make_float2(-acc[a][j].x, -acc[a][j].y);
}

// Skeel's condition number || |R| |T| e || of each diagonal block T with its
// inverse R, as the bits of a float (a NaN is the largest); grid x = (block row,
// quarter of its rows), y = L / U.
__global__ void __launch_bounds__(512)
tri_cond_kernel(int nb, const float2* __restrict__ Inv, const float* __restrict__ rowsum, unsigned* __restrict__ cond) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, b = blockIdx.x >> 2;
  const int64_t block = (blockIdx.y ? nb : 0) + b;
  const float2* I = Inv + block * kTD * kTD;
  float t[kTD / 32];
#pragma unroll
  for (int j = 0; j < kTD / 32; ++j) t[j] = rowsum[block * kTD + lane + 32 * j];
  unsigned mx = 0;
#pragma unroll
  for (int i = 0; i < 4; ++i) {
    const int r = (blockIdx.x & 3) * 64 + 16 * i + warp;
    float s = 0.f;
#pragma unroll
    for (int j = 0; j < kTD / 32; ++j) {
      const float2 v = I[r * kTD + lane + 32 * j];
      s = fmaf(fabsf(v.x) + fabsf(v.y), t[j], s);
    }
    for (int o = 16; o; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
    mx = max(mx, __float_as_uint(s) & 0x7FFFFFFFu);
  }
  if (lane == 0) atomicMax(cond + block, mx);
}

// (hi, lo) += a b: the product and the sum exactly, their errors into lo
__device__ __forceinline__ void df_fma(float& hi, float& lo, float a, float b) {
  const float p = a * b, e = fmaf(a, b, -p);
  const float s = hi + p, z = s - hi;
  lo += e + ((hi - (s - z)) + (p - z));
  hi = s;
}

// One Newton step R + R (I - T R) for the inverses R of ill-conditioned
// diagonal blocks, the residual in double-float.  Without it a solve with
// random factors (condition numbers of 5000 to 8000) has 2.5 times the residual
// that substitution in 64-row blocks leaves, with it a third; blocks of system
// matrices (10 to 400) solve to a half to a seventh of it as they are.
// 16 columns of a block per CTA; grid x = (block row, strip), y = L / U.
constexpr float kTCond = 500.f;
constexpr size_t kTNewtonSmem = (size_t)kTD * (16 + 16 + 17) * sizeof(float2);
__global__ void __launch_bounds__(512)
tri_newton_kernel(const float2* __restrict__ F, int64_t ldf, int n, int nb, const float2* __restrict__ Inv,
                  const float* __restrict__ cond, float2* __restrict__ Out) {
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  float2* Bs = reinterpret_cast<float2*>(smem_raw);   // [256][16]
  float2* Es = Bs + kTD * 16;                           // [256][16]
  float2* As = Es + kTD * 16;                           // [256][17]
  const int tid = threadIdx.x, b = blockIdx.x >> 4, c0 = (blockIdx.x & 15) * 16, d0 = b * kTD;
  const bool upper = blockIdx.y != 0;
  const int64_t block = (upper ? nb : 0) + b;
  const float2* I = Inv + block * kTD * kTD;
  float2* O = Out + block * kTD * kTD;
  if (cond[block] <= kTCond) return;   // (a NaN goes on)
  for (int idx = tid; idx < kTD * 16; idx += 512) Bs[idx] = I[(int64_t)(idx >> 4) * kTD + c0 + (idx & 15)];
  const int rg = tid >> 3, cg = tid & 7;   // rows rg + 64 a, columns 2 cg, 2 cg + 1
  float2 hi[4][2], lo[4][2];
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int j = 0; j < 2; ++j) hi[a][j] = lo[a][j] = make_float2(0.f, 0.f);
  // rows of a column of R: from its own on (L), up to its own (U)
  const int kb = upper ? 0 : c0, ke = upper ? c0 + 16 : kTD;
  for (int k0 = kb; k0 < ke; k0 += 16) {
    __syncthreads();
    for (int idx = tid; idx < kTD * 16; idx += 512) {
      const int r = idx >> 4, c = k0 + (idx & 15);
      float2 v = make_float2(r == c && (!upper || d0 + r >= n) ? 1.f : 0.f, 0.f);
      if (d0 + r < n && d0 + c < n && (upper ? c >= r : c < r)) v = F[(int64_t)(d0 + r) * ldf + d0 + c];
      As[r * 17 + (idx & 15)] = v;
    }
    __syncthreads();
#pragma unroll 1
    for (int k = 0; k < 16; ++k) {
      const float4 x = *reinterpret_cast<const float4*>(Bs + (k0 + k) * 16 + 2 * cg);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float2 t = As[(rg + 64 * a) * 17 + k];
        df_fma(hi[a][0].x, lo[a][0].x, t.x, x.x);
        df_fma(hi[a][0].x, lo[a][0].x, -t.y, x.y);
        df_fma(hi[a][0].y, lo[a][0].y, t.x, x.y);
        df_fma(hi[a][0].y, lo[a][0].y, t.y, x.x);
        df_fma(hi[a][1].x, lo[a][1].x, t.x, x.z);
        df_fma(hi[a][1].x, lo[a][1].x, -t.y, x.w);
        df_fma(hi[a][1].y, lo[a][1].y, t.x, x.w);
        df_fma(hi[a][1].y, lo[a][1].y, t.y, x.z);
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = rg + 64 * a, c = 2 * cg + j;
      Es[r * 16 + c] = make_float2(((r == c0 + c ? 1.f : 0.f) - hi[a][j].x) - lo[a][j].x, -hi[a][j].y - lo[a][j].y);
      hi[a][j] = make_float2(0.f, 0.f);
    }
  for (int k0 = kb; k0 < ke; k0 += 16) {
    __syncthreads();
    for (int idx = tid; idx < kTD * 16; idx += 512)
      As[(idx >> 4) * 17 + (idx & 15)] = I[(int64_t)(idx >> 4) * kTD + k0 + (idx & 15)];
    __syncthreads();
#pragma unroll 4
    for (int k = 0; k < 16; ++k) {
      const float4 x = *reinterpret_cast<const float4*>(Es + (k0 + k) * 16 + 2 * cg);
#pragma unroll
      for (int a = 0; a < 4; ++a) {
        const float2 t = As[(rg + 64 * a) * 17 + k];
        cfma(hi[a][0], t, make_float2(x.x, x.y));
        cfma(hi[a][1], t, make_float2(x.z, x.w));
      }
    }
  }
#pragma unroll
  for (int a = 0; a < 4; ++a)
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int r = rg + 64 * a, c = 2 * cg + j;
      O[(int64_t)r * kTD + c0 + c] = cadd(Bs[r * 16 + c], hi[a][j]);
    }
}

// ---------------------------------------------------------------- one block row

// Shared memory of tri_step_kernel: A operand [part][K slice][128 rows x 128 B],
// B operand [K slice][64 rows of h, 64 of l][128 B] (the same bytes hold the
// partial sums, 128 x 64 floats, once the products are done), the cluster's new
// block row (this CTA's 32 rows x 32 columns).
constexpr uint32_t kTSlice = 128 * 128;
constexpr size_t kTSmem = 1024 + 4 * kTSlice + 2 * kTSlice + kTC * kTC * sizeof(float2);

__device__ __forceinline__ uint32_t tri_mapa(uint32_t a, uint32_t rank) {
  uint32_t r;
  asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(a), "r"(rank));
  return r;
}
__device__ __forceinline__ float4 tri_ld4(uint32_t a) {
  float4 v;
  asm volatile("ld.shared::cluster.v4.f32 {%0, %1, %2, %3}, [%4];"
               : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
               : "r"(a)
               : "memory");
  return v;
}
__device__ __forceinline__ float2 tri_ld2(uint32_t a) {
  float2 v;
  asm volatile("ld.shared::cluster.v2.f32 {%0, %1}, [%2];" : "=f"(v.x), "=f"(v.y) : "r"(a) : "memory");
  return v;
}
__device__ __forceinline__ void tri_cluster_sync() {
  asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// byte offset of half `kr` (even) of row `row` in rows of 128 bytes, 16-byte chunks
// XOR-swizzled by the row (the K-major 128-byte-swizzle operand layout)
__device__ __forceinline__ uint32_t tri_swz(int row, int kr) {
  return (uint32_t)row * 128u + (uint32_t)((((kr >> 3) ^ (row & 7)) << 4) + (kr & 7) * 2);
}
// exponent e, |e| <= 126, with |x| 2^-e < 2^15 for every |x| up to the one with bits mx, which
// stays at 2^14 or above where e allows (0 for zero and non-finite maxima)
__device__ __forceinline__ int tri_exp(unsigned mx) {
  return mx == 0u || mx >= 0x7F800000u ? 0 : max((int)(mx >> 23) - 141, -126);
}
__device__ __forceinline__ float tri_pow2(int e) { return __int_as_float((127 + e) << 23); }   // |e| <= 126
// (x, y) times sc as h + 2^-11 l, two fp16 pairs: the difference is exact
__device__ __forceinline__ void tri_split(float2 v, float sc, uint32_t& h, uint32_t& l) {
  const float x = v.x * sc, y = v.y * sc;
  const __half2 hh = __floats2half2_rn(x, y);
  const float2 f = __half22float2(hh);
  const __half2 ll = __floats2half2_rn((x - f.x) * 2048.f, (y - f.y) * 2048.f);
  h = *reinterpret_cast<const uint32_t*>(&hh);
  l = *reinterpret_cast<const uint32_t*>(&ll);
}

// Rows warp, warp + 8, .. of a 128 x 64 tile, columns lane and lane + 32: into registers
__device__ __forceinline__ void tri_load_tile(float2 (&v)[16][2], const float2* __restrict__ A, int64_t lda, int rn,
                                              int cn, int warp, int lane) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int r = warp + 8 * i;
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const int c = lane + 32 * j;
      v[i][j] = r < rn && c < cn ? A[(int64_t)r * lda + c] : make_float2(0.f, 0.f);
    }
  }
}
// and from there to the A operand, each row with its own exponent
__device__ __forceinline__ void tri_store_tile(const float2 (&v)[16][2], unsigned char* abuf, int* rexp, int warp,
                                               int lane) {
#pragma unroll
  for (int i = 0; i < 16; ++i) {
    const int r = warp + 8 * i;
    unsigned mx = 0;
#pragma unroll
    for (int j = 0; j < 2; ++j)
      mx = max(mx, max(__float_as_uint(fabsf(v[i][j].x)), __float_as_uint(fabsf(v[i][j].y))));
    const int e = tri_exp(__reduce_max_sync(0xffffffffu, mx));
    if (lane == 0) rexp[r] = e;
    const float sc = tri_pow2(-e);
#pragma unroll
    for (int j = 0; j < 2; ++j) {
      const uint32_t at = (uint32_t)j * kTSlice + tri_swz(r, 2 * lane);
      tri_split(v[i][j], sc, *reinterpret_cast<uint32_t*>(abuf + at),
                *reinterpret_cast<uint32_t*>(abuf + 2 * kTSlice + at));
    }
  }
}

// The B operand from 64 x 32 values, this thread's rows 8 warp .. + 7 of column
// lane: rows 2c and 2c + 1 of B'^T hold (re, -im) and (im, re) of column c.
// rmean: the means of the rows' exponents over nonzero finite values (0: none).
__device__ __forceinline__ void tri_store_rhs(const float2 (&x)[8], unsigned char* bbuf, unsigned* cmax, int* cexp,
                                              int* rmean, int warp, int lane) {
  unsigned mx = 0;
  unsigned sum = 0;   // of row lane: exponents, and 2^16 for each
#pragma unroll
  for (int i = 0; i < 8; ++i) {
    const unsigned m = max(__float_as_uint(fabsf(x[i].x)), __float_as_uint(fabsf(x[i].y)));
    mx = max(mx, m);
    const unsigned si = __reduce_add_sync(0xffffffffu, m - 0x00800000u < 0x7F000000u ? 0x10000u + (m >> 23) : 0u);
    if (lane == i) sum = si;
  }
  if (lane < 8)
    rmean[8 * warp + lane] = sum ? __float2int_rn(__fdividef((float)(sum & 0xFFFFu), (float)(sum >> 16))) : 0;
  cmax[warp * 32 + lane] = mx;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) mx = max(mx, cmax[w * 32 + lane]);
  const int e = tri_exp(mx);
  if (warp == 0) cexp[lane] = e;
  const float sc = tri_pow2(-e);
  const int slice = warp >> 2, k0 = 16 * (warp & 3);   // 8 complex k: halves k0 .. k0 + 15 of the slice
  unsigned char* base = bbuf + slice * kTSlice;
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    uint32_t h0[4], h1[4], l0[4], l1[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      uint32_t h, l;
      tri_split(x[4 * g + i], sc, h, l);
      h0[i] = h ^ 0x80000000u;                      // re, -im
      h1[i] = __byte_perm(h, 0, 0x1032);            // im, re
      l0[i] = l ^ 0x80000000u;
      l1[i] = __byte_perm(l, 0, 0x1032);
    }
    const int kr = k0 + 8 * g;
    *reinterpret_cast<uint4*>(base + tri_swz(2 * lane, kr)) = make_uint4(h0[0], h0[1], h0[2], h0[3]);
    *reinterpret_cast<uint4*>(base + tri_swz(2 * lane + 1, kr)) = make_uint4(h1[0], h1[1], h1[2], h1[3]);
    *reinterpret_cast<uint4*>(base + tri_swz(64 + 2 * lane, kr)) = make_uint4(l0[0], l0[1], l0[2], l0[3]);
    *reinterpret_cast<uint4*>(base + tri_swz(64 + 2 * lane + 1, kr)) = make_uint4(l1[0], l1[1], l1[2], l1[3]);
  }
}
// Whether the FP32 pipe takes a product: the means differ by more than kTSpread
// (up to there the error of a product is at most 2^-50 2^13 of the sum of its
// terms' sizes, well within FP32's; a single large right-hand side leaves the
// means as they are), or a row of the factor is so near the ends of FP32's range
// that tri_read's sums of up to 2^38 would leave it on the way.
constexpr int kTSpread = 13;
__device__ __forceinline__ bool tri_rows_differ(const int* rmean, const int* rexp, int lane) {
  bool ends = false;
#pragma unroll
  for (int i = 0; i < 4; ++i) ends = ends || abs(rexp[lane + 32 * i]) > 88;
  const int m0 = rmean[lane], m1 = rmean[lane + 32];
  const int hi = __reduce_max_sync(0xffffffffu, max(m0, m1));
  const int lo = __reduce_min_sync(0xffffffffu, min(m0 ? m0 : 255, m1 ? m1 : 255));
  return hi - lo > kTSpread || __any_sync(0xffffffffu, ends);
}

// acc (laid out as tri_read's) += the 128 x 64 tile at A (rows < rn, columns < cn) times the 64 x 32 values
// xs, on the FP32 pipe
__device__ __noinline__ void tri_plain(float* acc, const float2* __restrict__ A, int64_t lda, int rn, int cn,
                                       const float2* xs, int warp, int lane) {
  const int row = 32 * (warp & 3) + lane, c0 = 16 * (warp >> 2);
  if (row >= rn) return;
  const float2* a = A + (int64_t)row * lda;
  float2 s[16];
#pragma unroll
  for (int c = 0; c < 16; ++c) s[c] = make_float2(0.f, 0.f);
  for (int k = 0; k < min(kTK, cn); ++k) {
    const float2 t = a[k];
#pragma unroll
    for (int c = 0; c < 16; ++c) cfma(s[c], t, xs[k * kTC + c0 + c]);
  }
#pragma unroll
  for (int c = 0; c < 16; ++c) {
    acc[2 * c] += s[c].x;
    acc[2 * c + 1] += s[c].y;
  }
}

// 128 x 64 real outputs over 128 real K: h parts of A into columns 0 .. 127 (h h | h l), l parts into
// 64 .. 191 (l h | l l); one thread
__device__ __forceinline__ void tri_issue(uint32_t tmem, const unsigned char* abuf, const unsigned char* bbuf) {
  using namespace tc;
#pragma unroll
  for (int s = 0; s < 2; ++s) {
    const uint64_t ah = kmajor_sw128_desc(smem_u32(abuf + s * kTSlice));
    const uint64_t al = kmajor_sw128_desc(smem_u32(abuf + (2 + s) * kTSlice));
    const uint64_t b = kmajor_sw128_desc(smem_u32(bbuf + s * kTSlice));
    const uint64_t bl = kmajor_sw128_desc(smem_u32(bbuf + s * kTSlice + 64 * 128));
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const bool first = s == 0 && ks == 0;
      const uint64_t o = (uint64_t)(2 * ks);
      mma_f16(tmem, ah + o, b + o, idesc_f16_m128(128), first ? 0u : 1u);
      if (first) {
        mma_f16(tmem + 64, al + o, b + o, idesc_f16_m128(64), 1u);
        mma_f16(tmem + 128, al + o, bl + o, idesc_f16_m128(64), 0u);
      } else {
        mma_f16(tmem + 64, al + o, b + o, idesc_f16_m128(128), 1u);
      }
    }
  }
}

// acc (row 32 (warp & 3) + lane, real columns 32 (warp >> 2) .. + 31) += the products in tensor memory
__device__ __forceinline__ void tri_read(float (&acc)[32], uint32_t tmem, const int* rexp, const int* cexp, int warp,
                                         int lane) {
  using namespace tc;
  const int half = warp >> 2;
  const uint32_t t = tmem + ((uint32_t)(32 * (warp & 3)) << 16) + (uint32_t)(32 * half);
  const int er = rexp[32 * (warp & 3) + lane];
#pragma unroll
  for (int p = 0; p < 4; ++p) {
    uint32_t hh[8], hl[8], ll[8];
    tmem_ld8(t + 8 * p, hh);
    tmem_ld8(t + 64 + 8 * p, hl);
    tmem_ld8(t + 128 + 8 * p, ll);
    tmem_wait_ld();
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      const float s0 = tri_pow2(er), s1 = tri_pow2(cexp[16 * half + 4 * p + c]);
#pragma unroll
      for (int q = 0; q < 2; ++q) {
        const int j = 2 * c + q;
        const float lo = fmaf(__uint_as_float(ll[j]), 0x1p-11f, __uint_as_float(hl[j]));
        acc[8 * p + j] += fmaf(lo, 0x1p-11f, __uint_as_float(hh[j])) * s0 * s1;
      }
    }
  }
}
// acc into P (128 rows of 16 float4, chunk c of row r at c ^ (r & 15))
__device__ __forceinline__ void tri_partials(const float (&acc)[32], float4* P, int warp, int lane) {
  const int row = 32 * (warp & 3) + lane;
#pragma unroll
  for (int p = 0; p < 8; ++p)
    P[row * 16 + ((8 * (warp >> 2) + p) ^ (row & 15))] =
        make_float4(acc[4 * p], acc[4 * p + 1], acc[4 * p + 2], acc[4 * p + 3]);
}

// This CTA's 32 rows of the cluster half's sum: row 32 kq + tid / 8, complex columns 4 (tid & 7) .. + 3
__device__ __forceinline__ void tri_gather(float2 (&s)[4], uint32_t paddr, int half, int kq, int tid) {
  const int row = 32 * kq + (tid >> 3), c4 = 2 * (tid & 7);
  float4 v[4][2];   // all on their way before the first is used
#pragma unroll
  for (int q = 0; q < 4; ++q) {
    const uint32_t base = tri_mapa(paddr, (uint32_t)(4 * half + q)) + (uint32_t)row * 256u;
#pragma unroll
    for (int j = 0; j < 2; ++j) v[q][j] = tri_ld4(base + (uint32_t)(((c4 + j) ^ (row & 15)) * 16));
  }
#pragma unroll
  for (int j = 0; j < 2; ++j) {
    s[2 * j].x = (v[0][j].x + v[1][j].x) + (v[2][j].x + v[3][j].x);
    s[2 * j].y = (v[0][j].y + v[1][j].y) + (v[2][j].y + v[3][j].y);
    s[2 * j + 1].x = (v[0][j].z + v[1][j].z) + (v[2][j].z + v[3][j].z);
    s[2 * j + 1].y = (v[0][j].w + v[1][j].w) + (v[2][j].w + v[3][j].w);
  }
}

// The inverses as A operands: tile (triangle, block row, half, K quarter) in the
// layout of abuf, and its 128 row exponents.
__global__ void __launch_bounds__(kTThreads)
tri_operand_kernel(const float2* __restrict__ Inv, const float2* __restrict__ refined, const float* __restrict__ cond,
                   unsigned char* __restrict__ ops, int* __restrict__ exps) {
  const int64_t tile = blockIdx.x, b = tile >> 3;
  const int half = (int)(tile >> 2) & 1, kq = (int)tile & 3, warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  float2 v[16][2];
  tri_load_tile(v, (cond[b] <= kTCond ? Inv : refined) + b * kTD * kTD + (int64_t)half * 128 * kTD + kq * kTK, kTD, 128, kTK, warp, lane);
  tri_store_tile(v, ops + tile * (4 * kTSlice), exps + tile * 128, warp, lane);
}

// One step of the solve in place on X.  src: the block row solved last (< 0:
// none, the first step).  The first cluster of grid x updates the next block
// row (src + 1 for L, src - 1 for U) with it and solves that.  The block rows
// beyond are updated by a cluster each (SPLIT), or by one CTA per 128 rows
// that takes the four quarters of K in turn.
template <bool UPPER, bool SPLIT>
__global__ void __launch_bounds__(kTThreads, 2)
tri_step_kernel(const float2* __restrict__ F, int64_t ldf, const unsigned char* __restrict__ ops,
                const int* __restrict__ exps, const float2* __restrict__ inv, const float2* __restrict__ refined,
                const float* __restrict__ cond, float2* X, int64_t ldx, int n, int ncols, int src, int first,
                int* status) {
  using namespace tc;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* abuf = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* bbuf = abuf + 4 * kTSlice;
  float2* fresh = reinterpret_cast<float2*>(bbuf + 2 * kTSlice);   // 32 rows x 32 columns
  __shared__ int rexp[128], cexp[kTC];
  __shared__ unsigned cmax[8 * 32];
  __shared__ int rmean[kTK];
  __shared__ uint64_t bar, bar_inv;
  __shared__ uint32_t tmem_slot;
  __shared__ int abort_flag;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int rank = (int)(blockIdx.x & 7), cl = (int)(blockIdx.x >> 3), cg = blockIdx.y * kTC;
  const bool alone = !SPLIT && cl > 0;   // no exchange with the cluster
  const int next = src < 0 ? first : UPPER ? src - 1 : src + 1;
  int half, kq, row0;
  if (alone) {
    half = 0;
    kq = 0;
    row0 = ((cl - 1) * 8 + rank) * 128 + (UPPER ? 0 : (next + 1) * kTD);
    if (row0 >= (UPPER ? next * kTD : n)) return;
  } else {
    half = rank >> 2;
    kq = rank & 3;
    row0 = (UPPER ? next - cl : next + cl) * kTD + half * 128;
  }
  if (tid == 0) {
    mbar_init(&bar, 1);
    mbar_init(&bar_inv, 1);
    abort_flag = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)), "r"(256)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  const int64_t tile = (int64_t)next * 8 + rank;   // of the inverse, for the first cluster
  float2 v[16][2];
  // the factor's (first) tile: nothing that a step writes
  if (src >= 0) {
    const int c0 = src * kTD + kq * kTK;
    tri_load_tile(v, F + (int64_t)row0 * ldf + c0, ldf, n - row0, n - c0, warp, lane);
    // the other three quarters on their way to L2: 12 lines of 128 bytes a row
    if (alone)
      for (int idx = tid; idx < 128 * 12; idx += kTThreads) {
        const int r = idx / 12, c = c0 + kTK + 16 * (idx % 12);
        if (row0 + r < n && c < n) asm volatile("prefetch.global.L2 [%0];" ::"l"(F + (int64_t)(row0 + r) * ldf + c));
      }
    tri_store_tile(v, abuf, rexp, warp, lane);
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = tmem_slot;
  asm volatile("griddepcontrol.launch_dependents;" ::: "memory");
  asm volatile("griddepcontrol.wait;" ::: "memory");

  // this CTA's share of a cluster's block row: 4 columns of one row per thread
  const int orow = row0 + 32 * kq + (tid >> 3), ocol = cg + 4 * (tid & 7);
  float2 b[4];
  if (!alone) {
#pragma unroll
    for (int j = 0; j < 4; ++j)
      b[j] = orow < n && ocol + j < ncols ? ldcg(X + (int64_t)orow * ldx + ocol + j) : make_float2(0.f, 0.f);
  }
  const uint32_t paddr = smem_u32(bbuf);
  float4* P = reinterpret_cast<float4*>(bbuf);
  uint32_t phase = 0;
  float2 x[8];
  float acc[32];
#pragma unroll
  for (int j = 0; j < 32; ++j) acc[j] = 0.f;
  // (the tile in abuf: the factor's columns from k0 on, or the inverse's) x (the right-hand sides in x), in tensor
  // memory; or true, and acc += it
  auto product = [&](bool inverse, int k0) -> bool {
    tri_store_rhs(x, bbuf, cmax, cexp, rmean, warp, lane);
    fence_async_smem();
    tc_fence_before();
    __syncthreads();
    if (tid == 0) {
      // a wait that runs out: noted, and once more, so that nothing is left in flight
      if (inverse && !mbar_wait(&bar_inv, 0, &abort_flag)) mbar_wait_plain(&bar_inv, 0);
      tc_fence_after();
      tri_issue(tmem, abuf, bbuf);
      mma_commit(&bar);
    }
    const bool differ = tri_rows_differ(rmean, rexp, lane);   // (beside the products)
    if (!mbar_wait(&bar, phase, &abort_flag)) mbar_wait_plain(&bar, phase);
    phase ^= 1;
    tc_fence_after();
    if (differ) {
      float2* xs = reinterpret_cast<float2*>(bbuf);
#pragma unroll
      for (int i = 0; i < 8; ++i) xs[(8 * warp + i) * kTC + lane] = x[i];
      __syncthreads();
      float part[32];
#pragma unroll
      for (int j = 0; j < 32; ++j) part[j] = acc[j];
      if (inverse)
        tri_plain(part,
                  (cond[next] <= kTCond ? inv : refined) + (int64_t)next * kTD * kTD + (int64_t)half * 128 * kTD + kq * kTK,
                  kTD, 128, kTK, xs, warp, lane);
      else
        tri_plain(part, F + (int64_t)row0 * ldf + k0, ldf, n - row0, n - k0, xs, warp, lane);
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[j] = part[j];
    }
    return differ;
  };
  // the products of a CTA whose wait ran out are NaN, and so are the block rows made of them
  auto poison = [&]() {
    if (*(volatile int*)&abort_flag) {
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[j] = __int_as_float(0x7FC00000);
    }
  };
  auto load_inverse = [&]() {
    if (tid == 0) {
      mbar_expect_tx(&bar_inv, 4 * kTSlice);
      bulk_load(abuf, ops + tile * (4 * kTSlice), 4 * kTSlice, &bar_inv);
    }
  };
  if (src >= 0) {
#pragma unroll 1
    for (int q = kq;; ++q) {
      const int k0 = src * kTD + q * kTK;
#pragma unroll
      for (int i = 0; i < 8; ++i) {
        const int k = k0 + 8 * warp + i;
        x[i] = k < n && cg + lane < ncols ? ldcg(X + (int64_t)k * ldx + cg + lane) : make_float2(0.f, 0.f);
      }
      const bool made = product(false, k0);
      if (!alone && cl == 0) load_inverse();   // the tile's products are done
      if (!made) tri_read(acc, tmem, rexp, cexp, warp, lane);
      poison();
      tc_fence_before();
      if (!alone || q == 3) break;
      __syncthreads();   // the exponents and tensor memory are read
      tri_load_tile(v, F + (int64_t)row0 * ldf + k0 + kTK, ldf, n - row0, n - k0 - kTK, warp, lane);
      tri_store_tile(v, abuf, rexp, warp, lane);
    }
    if (alone) {
      // rows of this thread, 16 columns each: through shared memory to whole rows
      __syncthreads();
      tri_partials(acc, P, warp, lane);
      __syncthreads();
      const bool in = cg + lane < ncols;
#pragma unroll 1
      for (int h = 0; h < 2; ++h) {
        float2* at = X + (int64_t)(row0 + 64 * h + warp) * ldx + cg + lane;   // rows 8 apart
        float2 o[8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
          if (in && row0 + 64 * h + warp + 8 * i < n) o[i] = ldcg(at + 8 * i * ldx);
#pragma unroll
        for (int i = 0; i < 8; ++i) {
          const int r = 64 * h + warp + 8 * i;
          const float2 p = reinterpret_cast<const float2*>(P + r * 16 + ((lane >> 1) ^ (r & 15)))[lane & 1];
          if (in && row0 + r < n) at[8 * i * ldx] = make_float2(o[i].x - p.x, o[i].y - p.y);
        }
      }
    } else {
      __syncthreads();
      tri_partials(acc, P, warp, lane);
      tri_cluster_sync();
      float2 s[4];
      tri_gather(s, paddr, half, kq, tid);
#pragma unroll
      for (int j = 0; j < 4; ++j) {
        b[j].x -= s[j].x;
        b[j].y -= s[j].y;
      }
    }
  } else {
    load_inverse();
  }
  if (!alone) {
    if (cl == 0) {
      // X = T^-1 B of this block row
#pragma unroll
      for (int j = 0; j < 4; j += 2)
        *reinterpret_cast<float4*>(fresh + (tid >> 3) * kTC + 4 * (tid & 7) + j) =
            make_float4(b[j].x, b[j].y, b[j + 1].x, b[j + 1].y);
      if (tid < 128) rexp[tid] = exps[tile * 128 + tid];
      tri_cluster_sync();   // the block row is complete, and the partial sums are read
      // rows 64 kq .. + 63 of the block row: 32 with each of two CTAs
      const uint32_t from = tri_mapa(smem_u32(fresh), (uint32_t)(2 * kq + (warp >> 2))) +
                            (uint32_t)((8 * (warp & 3) * kTC + lane) * 8);
#pragma unroll
      for (int i = 0; i < 8; ++i) x[i] = tri_ld2(from + (uint32_t)(i * kTC * 8));
#pragma unroll
      for (int j = 0; j < 32; ++j) acc[j] = 0.f;
      if (!product(true, 0)) tri_read(acc, tmem, rexp, cexp, warp, lane);
      poison();
      tc_fence_before();
      __syncthreads();
      tri_partials(acc, P, warp, lane);
      tri_cluster_sync();
      tri_gather(b, paddr, half, kq, tid);
    }
    // no CTA leaves while its partial sums are being read
    asm volatile("barrier.cluster.arrive.release.aligned;" ::: "memory");
#pragma unroll
    for (int j = 0; j < 4; ++j)
      if (orow < n && ocol + j < ncols) X[(int64_t)orow * ldx + ocol + j] = b[j];
    asm volatile("barrier.cluster.wait.acquire.aligned;" ::: "memory");
  } else {
    __syncthreads();
  }
  if (tid == 0 && *(volatile int*)&abort_flag) atomicExch(status, MGT_ERR_TIMEOUT);
  if (warp == 0) {
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(256) : "memory");
  }
}

// Workspace of a solve: the status words; the inverted diagonal
// blocks of L and of U; those of ill-conditioned blocks after the Newton step;
// the operands and their row exponents; the blocks' row sums and condition
// numbers.
struct TriWs {
  size_t inv = 256, refined, ops, exps, rowsum, cond, total;
  explicit TriWs(int64_t n) {
    const size_t blocks = 2 * (size_t)((n + kTD - 1) / kTD);
    refined = inv + blocks * kTD * kTD * sizeof(float2);
    ops = refined + blocks * kTD * kTD * sizeof(float2);
    exps = ops + blocks * 8 * 4 * kTSlice;
    rowsum = exps + blocks * 8 * 128 * sizeof(int);
    cond = rowsum + blocks * kTD * sizeof(float);
    total = cond + blocks * sizeof(float);
  }
};

size_t tri_solve_workspace_bytes(int64_t n) { return TriWs(n).total; }

template <bool UPPER>
static int tri_steps(const float2* F, int64_t ldf, const unsigned char* ops, const int* exps, const float2* inv,
                     const float2* refined, const float* cond, float2* X, int64_t ldx, int n, int nrhs, int* status,
                     cudaStream_t s) {
  const int nb = (n + kTD - 1) / kTD, ng = (nrhs + kTC - 1) / kTC, sms = device_sm_count();
  for (int i = 0; i < nb; ++i) {
    // step i solves block row i (from the end for U) after updating it and all that follow
    const int first = UPPER ? nb - 1 : 0, src = i == 0 ? -1 : UPPER ? nb - i : i - 1;
    const int rest = i == 0 ? 0 : nb - 1 - i;   // block rows beyond
    // K over the CTAs of a cluster while the launch is at most 1.75 rounds of
    // what is resident at once (two CTAs an SM, 3.5 in all); beyond, one CTA takes all of K
    // (34 K clocks for 128 rows, no sums to exchange, against 4 x 20 K).  Solves
    // of 64 columns with the line at 1.3, 2, 2.6, 3.4 and 4.6 CTAs an SM, ms:
    // n = 6000 0.98, 0.89, 0.86, 0.85, 0.85; 12000 2.23, 2.12, 2.06, 2.01, 2.07.
    const bool split = (int64_t)8 * (1 + rest) * ng <= 7 * sms / 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(8 * (1 + (split ? rest : (2 * rest + 7) / 8)), ng);
    cfg.blockDim = dim3(kTThreads);
    cfg.dynamicSmemBytes = kTSmem;
    cfg.stream = s;
    cudaLaunchAttribute at[2];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim = {8, 1, 1};
    // a step may start early when the launch before it is a step of this solve: the
    // factor and the inverses, which it reads before it waits, are complete
    at[1].id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at[1].val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = at;
    cfg.numAttrs = UPPER || i > 0 ? 2 : 1;
    count_launch();
    if (cudaLaunchKernelEx(&cfg, split ? tri_step_kernel<UPPER, true> : tri_step_kernel<UPPER, false>, F, ldf, ops, exps,
                           inv, refined, cond, X, ldx, n, nrhs, src, first, status) != cudaSuccess)
      return MGT_ERR_CUDA;
  }
  return MGT_OK;
}

// In-place X = U^-1 L^-1 X with the factors in F (unit lower and upper), nrhs
// columns.  inverses_ready: an earlier call with this workspace, n and F made
// the inverted diagonal blocks.
int tri_solve(const float2* F, int64_t ldf, float2* X, int64_t ldx, int n, int nrhs, void* work, bool inverses_ready,
              cudaStream_t s) {
  static OncePerDevice once;
  once([] {
    cudaFuncSetAttribute(tri_inverse64_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInv64Smem);
    cudaFuncSetAttribute(tri_double_kernel<64>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)tri_double_smem<64>());
    cudaFuncSetAttribute(tri_double_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                         (int)tri_double_smem<128>());
    cudaFuncSetAttribute(tri_newton_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTNewtonSmem);
    cudaFuncSetAttribute(tri_step_kernel<false, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTSmem);
    cudaFuncSetAttribute(tri_step_kernel<false, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTSmem);
    cudaFuncSetAttribute(tri_step_kernel<true, false>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTSmem);
    cudaFuncSetAttribute(tri_step_kernel<true, true>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTSmem);
  });
  int* status = (int*)((char*)work + kStatusOffset);
  if (cudaMemsetAsync(status, 0, 2 * sizeof(int), s) != cudaSuccess) return MGT_ERR_CUDA;
  const int nb = (n + kTD - 1) / kTD;
  const TriWs L(n);
  float2* inv = (float2*)((char*)work + L.inv);
  float2* refined = (float2*)((char*)work + L.refined);
  unsigned char* ops = (unsigned char*)work + L.ops;
  float* rowsum = (float*)((char*)work + L.rowsum);
  float* cond = (float*)((char*)work + L.cond);
  int* exps = (int*)((char*)work + L.exps);
  if (!inverses_ready) {
    count_launch(6);
    tri_inverse64_kernel<<<nb * (kTD / kTB), kTileThreads, kInv64Smem, s>>>(F, ldf, n, nb, inv, rowsum, cond);
    tri_double_kernel<64><<<dim3(nb * 8, 2), 256, tri_double_smem<64>(), s>>>(F, ldf, n, nb, inv);
    tri_double_kernel<128><<<dim3(nb * 8, 2), 256, tri_double_smem<128>(), s>>>(F, ldf, n, nb, inv);
    tri_cond_kernel<<<dim3(nb * 4, 2), 512, 0, s>>>(nb, inv, rowsum, (unsigned*)cond);
    tri_newton_kernel<<<dim3(nb * 16, 2), 512, kTNewtonSmem, s>>>(F, ldf, n, nb, inv, cond, refined);
    tri_operand_kernel<<<nb * 16, kTThreads, 0, s>>>(inv, refined, cond, ops, exps);
  }
  const size_t upper = (size_t)nb * kTD * kTD;
  int e = MGT_OK;
  constexpr int kCols = 65535 * kTC;   // columns of one launch
  for (int64_t c0 = 0; c0 < nrhs && e == MGT_OK; c0 += kCols) {
    const int nc = (int)std::min<int64_t>(kCols, nrhs - c0);
    e = tri_steps<false>(F, ldf, ops, exps, inv, refined, cond, X + c0, ldx, n, nc, status, s);
    if (e == MGT_OK)
      e = tri_steps<true>(F, ldf, ops + (size_t)nb * 8 * 4 * kTSlice, exps + (size_t)nb * 8 * 128, inv + upper,
                          refined + upper, cond + nb, X + c0, ldx, n, nc, status, s);
  }
  if (e != MGT_OK) return e;
  return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_ERR_CUDA;
}

// Inverses of the 64 x 64 diagonal blocks of a unit lower factor of order n
// (rows / columns at F), written to Inv[block][64][64]; the LU uses it for the
// two inner panels of a 128-wide block.
int lower_block_inverses(const float2* F, int64_t ldf, int n, float2* Inv, cudaStream_t s) {
  static OncePerDevice once;
  once([] { cudaFuncSetAttribute(lower_inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kInvSmem); });
  count_launch();
  lower_inverse_kernel<<<(n + kTB - 1) / kTB, 256, kInvSmem, s>>>(F, ldf, n, Inv);
  return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_ERR_CUDA;
}

}  // namespace mgt
