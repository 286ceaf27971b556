// complex128 products C (M x N) -= A (M x K) B (K x N), K <= 64, on the tensor
// cores: the trailing update of the complex128 LU.
//
// Why: the FP64 pipe of this part does about 1.7 fused multiply-adds per clock
// and SM (1.0-1.2 TFLOP/s in all), so a product of FP64 accuracy is made from
// exact FP16 products instead -- the Ozaki scheme of residual_tc.cu (Ozaki,
// Ogita, Oishi, Rump 2012; Mukunoki, Ozaki, Ogita, Imamura 2020):
//  * rows of A (as the real rows re, im, re, im, ...) and columns of B are
//    scaled by powers of two and written as 54-bit integers in seven balanced
//    base-256 digits, exact in FP16.  The largest entry of a row or column keeps
//    all its 53 bits.
//  * digit pairs (s, t) of equal weight s + t = l accumulate in one TMEM
//    accumulator per level l = 0 .. 7 (34 of the 49 pairs; the rest lie below
//    2^-60 of the scales).  128 real K at a time every level sum is an integer
//    below 2^24, exact in FP32.
//  * the levels are folded into one 64-bit integer per output in units of 2^-54
//    of the scales (levels 0 .. 5 exactly, 6 and 7 rounded to the unit), which
//    is rounded once to a double and subtracted from C: errors at the level of
//    one FP64 rounding of the product's scale, where a 128-term FP64 sum makes 128.
//
// zgemm_kernel: persistent, one CTA per SM walking tiles of 128 rows x 32
// complex columns (8 levels x 64 real columns fill TMEM):
//   warp 0     : TMEM allocation; bulk copies of B's digit blocks (56 KB per 32
//                complex K, 2 stages) and A's digit slices (8 KB, 6-slice ring)
//   warp 1     : MMA issuer: for digit s of A one MMA per 16-wide K step covers
//                up to four levels (B's digit slices are stacked along N)
//   warps 2-9  : epilogue: levels -> 64-bit integers -> C.  The integer is turned
//                into a double by integer instructions: one FP64 instruction per
//                output is left (an FP64 conversion costs as much as the subtraction)
//   warps 10-15: converters: byte digits -> FP16 operand slices
// The MMAs of the next tile run while the epilogue finishes the last one.
// Every wait is bounded; on expiry MGT_ERR_TIMEOUT is recorded, the CTA's tiles
// become NaN, the issued work is drained and TMEM freed.
#include <cuda_fp16.h>

#include <algorithm>
#include <climits>

#include "common.cuh"
#include "diag.cuh"
#include "tcgen05.cuh"
#include "zgemm_tc.cuh"

namespace mgt {
namespace zg {

constexpr int BM = 128;
constexpr int BNC = 32;
constexpr int BN = 2 * BNC;
constexpr int KCC = 32;                 // complex K per chunk
constexpr int NCH = kZK / KCC;          // chunk stride of the digit buffers
constexpr int DIG = 7, LEV = 8;
constexpr int ASLOTS = 4, DSLOTS = 4;
constexpr uint32_t A_SLICE = BM * 128, D_SLICE = BM * 64, B_SLICE = BN * 128, B_BLOCK = DIG * B_SLICE;
constexpr uint32_t TMEM_COLS = LEV * BN;
constexpr int NEPI = 8, NCONV = 6, EPI0 = 2;
constexpr int THREADS = (EPI0 + NEPI + NCONV) * 32;
constexpr int EPI_COLS = BN / (NEPI / 4);
constexpr long long BIAS = 0x0080808080808080LL;
constexpr int kNonFinite = 0x40000000;
constexpr int kPlainExp = 0x50000000;   // instead of row exponents: the product goes to the FP64 pipe
constexpr int FIX = 54;
static_assert(TMEM_COLS == 512, "all of TMEM");

constexpr uint32_t STAGE = 32 * 4 * 16;   // a warp's group of four columns on its way to whole row segments
constexpr size_t smem_bytes() {
  return 1024 + ASLOTS * A_SLICE + DSLOTS * D_SLICE + 2 * B_BLOCK + NEPI * STAGE + 256;
}

// polls (of some 50 clocks) without progress after which the producer gives up
constexpr uint32_t kProducerLimit = 1u << 27;

constexpr int kZeroExp = -100000;   // exponent of an exact zero
constexpr int kBadExp = 1000000;    // of an infinity or a NaN

// Exponent field (at least 1) of v 2^off.
__device__ __forceinline__ int expo(double v, int off) {
  const int hi = __double2hiint(v), ex = (hi >> 20) & 0x7ff;
  if (ex == 2047) return kBadExp;
  if (((hi & 0x7fffffff) | __double2loint(v)) == 0) return kZeroExp;
  return max(ex, 1) + off;
}

// Launched early only while every block is on the GPU at once, two an SM: beyond,
// the blocks that wait cost the kernel they wait for more than the launch saves
// (every launch early: n = 5997, 37 columns 59.7 -> 62.2 ms; n = 150, one column,
// 0.71 -> 0.65).
static bool early_fits(int64_t blocks) { return blocks <= 2 * device_sm_count(); }

// What to do with B's rows (ZRows); every lane of a warp calls it, every warp gets the same.
enum RowMode { kAsIs = 0, kShift = 1, kFp64 = 2 };
constexpr int kRowSpread = 4, kHalfSpread = 12, kShapeSpread = 6, kInvLimit = 1023 + 4;
__device__ __forceinline__ int row_mean(int4 s) {
  const int count = s.w + (int)((unsigned)s.z >> 31);   // a negative sum has borrowed from it
  return count ? 1023 + __float2int_rn(__fdividef((float)s.z, (float)count)) : 0;
}
// sh: the powers of two moved from rows lane and lane + 32 of B to A's columns.
template <int KIND>
__device__ __forceinline__ int row_mode(const ZRows& rows, int K, int lane, int (&sh)[2]) {
  sh[0] = sh[1] = 0;
  if (KIND == ZRows::NONE) return kAsIs;
  int4 st[2];   // every load on its way at once
  int inv = 0;
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    const int k = min(lane + 32 * i, K - 1);
    if (KIND == ZRows::MEAN) st[i] = __ldg(reinterpret_cast<const int4*>(rows.stats) + k);
    else st[i].x = __ldg(rows.stats + k);
  }
  if (KIND == ZRows::MAX && rows.inv) inv = __ldg(rows.inv);
  int lo = 1 << 20, hi = -1, slo = 1 << 20, shi = -1;   // of the sizes, and of largest less mean
#pragma unroll
  for (int i = 0; i < 2; ++i) {
    if (st[i].x <= 0) continue;   // zero (or not finite)
    const int e = KIND == ZRows::MEAN ? row_mean(st[i]) : st[i].x;
    lo = min(lo, e);
    hi = max(hi, e);
    slo = min(slo, st[i].x - e);
    shi = max(shi, st[i].x - e);
  }
  lo = __reduce_min_sync(0xffffffffu, lo);
  hi = __reduce_max_sync(0xffffffffu, hi);
  if (KIND == ZRows::MAX && inv >= kInvLimit) return kFp64;
  if (hi - lo <= kRowSpread) return kAsIs;
  if (KIND == ZRows::MAX) {
    if (hi - lo > kHalfSpread) return kFp64;
  } else {
    slo = __reduce_min_sync(0xffffffffu, slo);
    shi = __reduce_max_sync(0xffffffffu, shi);
    if (shi - slo > kShapeSpread) return kFp64;
  }
#pragma unroll
  for (int i = 0; i < 2; ++i)
    if (st[i].x > 0 && lane + 32 * i < K)
      sh[i] = KIND == ZRows::MEAN ? row_mean(st[i]) - 1023 : (st[i].x - 1023) >> 1;
  return kShift;
}

// Larger exponent field of both parts; 0 for zeros, infinities and NaN.
__device__ __forceinline__ int field(double2 v) {
  const int x = (__double2hiint(v.x) >> 20) & 0x7ff, y = (__double2hiint(v.y) >> 20) & 0x7ff;
  return max(x == 2047 ? 0 : x, y == 2047 ? 0 : y);
}

// v 2^(off + FIX - e) as an integer (round to nearest) for e = emax - 1022, emax >= expo(v, off):
// |result| < 2^54
__device__ __forceinline__ long long fixed54(double v, int off, int emax) {
  const long long b = __double_as_longlong(v);
  const int ex = (int)((b >> 52) & 0x7ff);
  long long m = b & 0xFFFFFFFFFFFFFll;
  if (ex) m |= 1ll << 52;
  const int sh = min(max(ex, 1) + off - emax + 1, 1);
  long long r;
  if (sh >= 0) r = m << sh;
  else if (sh > -54) r = (m + (1ll << (-sh - 1))) >> (-sh);
  else r = 0;
  return b < 0 ? -r : r;
}

__device__ __forceinline__ uint32_t pick4(long long a, long long b, long long c, long long d, int p) {
  const uint32_t x = p < 4 ? (uint32_t)a : (uint32_t)((unsigned long long)a >> 32);
  const uint32_t y = p < 4 ? (uint32_t)b : (uint32_t)((unsigned long long)b >> 32);
  const uint32_t z = p < 4 ? (uint32_t)c : (uint32_t)((unsigned long long)c >> 32);
  const uint32_t w = p < 4 ? (uint32_t)d : (uint32_t)((unsigned long long)d >> 32);
  const int k = p & 3;
  const uint32_t sel = (uint32_t)(k | ((4 + k) << 4));
  return __byte_perm(__byte_perm(x, y, sel), __byte_perm(z, w, sel), 0x5410);
}

// four biased digit bytes -> four FP16 values byte - 128 (exact)
__device__ __forceinline__ uint2 widen4(uint32_t x) {
  const uint32_t h0 = __byte_perm(x, 0x64646464u, 0x4140), h1 = __byte_perm(x, 0x64646464u, 0x4342);
  const __half2 c = __halves2half2(__ushort_as_half((unsigned short)0x6480), __ushort_as_half((unsigned short)0x6480));
  const __half2 d0 = __hsub2(*reinterpret_cast<const __half2*>(&h0), c);
  const __half2 d1 = __hsub2(*reinterpret_cast<const __half2*>(&h1), c);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&d0), *reinterpret_cast<const uint32_t*>(&d1));
}

// Distances between the slabs of a product over more than 64 columns of K: digit
// bytes, exponents, and elements of the output.
struct Slabs {
  size_t adig = 0, bdig = 0, aexp = 0, bexp = 0, c = 0;
  int tiles = 1 << 30;   // tiles per slab
};

// Operand digits, both operands in one launch: blocks [0, ablocks) take 32 rows
// of A each, the others 32 columns of B.  A: byte slices (row tile, chunk,
// digit) at half the width of the swizzled FP16 operand; B: the swizzled FP16
// operand itself (block (column tile, chunk): rows s 64 + 2 j, + 1).  Zeros
// beyond the operand.  K <= 64.  br: powers of two moved from B's rows to A's
// columns (ZRows; none where the product goes to the FP64 pipe).
template <int KIND>
__global__ void __launch_bounds__(256)
digits_kernel(const double2* __restrict__ A, int64_t lda, int M, int ablocks, const double2* __restrict__ B,
              int64_t ldb, int N, int K, ZRows br, unsigned char* __restrict__ adig,
              int* __restrict__ aexp, unsigned char* __restrict__ bdig, int* __restrict__ bexp, Slabs sl) {
  early_start();
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // slab blockIdx.y: columns 64 y .. of A, rows 64 y .. of B, its own digits and scales
  A += (int64_t)blockIdx.y * kZK;
  B += (int64_t)blockIdx.y * kZK * ldb;
  adig += blockIdx.y * sl.adig;
  aexp += blockIdx.y * sl.aexp;
  bdig += blockIdx.y * sl.bdig;
  bexp += blockIdx.y * sl.bexp;
  if (KIND == ZRows::MEAN) br.stats += (size_t)blockIdx.y * kZK * 4;
  K = min(kZK, K - (int)blockIdx.y * kZK);
  int sh[NCH];
  // (kFp64: the row exponents say so, and nothing made of the digits is used)
  const int mode = row_mode<KIND>(br, K, lane, sh);
  if ((int)blockIdx.x < ablocks) {
    for (int q = 0; q < 4; ++q) {
      const int row = blockIdx.x * 32 + warp * 4 + q;
      double2 v[NCH];
      int em = kZeroExp;
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        const int k = c * KCC + lane;
        v[c] = (row < M && k < K) ? A[(int64_t)row * lda + k] : make_double2(0.0, 0.0);
        em = max(em, max(expo(v[c].x, sh[c]), expo(v[c].y, sh[c])));
      }
      em = __reduce_max_sync(0xffffffffu, em);
      if (lane == 0 && row < M) aexp[row] = mode == kFp64 ? kPlainExp : em == kBadExp ? kNonFinite : em - 1022;
      const int rt = row / BM, rho = row % BM;
      const uint32_t at = (uint32_t)rho * 64u + ((uint32_t)((lane >> 2) ^ (rho & 7)) << 3) + (uint32_t)(lane & 3) * 2u;
#pragma unroll
      for (int c = 0; c < NCH; ++c) {
        const long long yr = fixed54(v[c].x, sh[c], em) + BIAS, yi = fixed54(v[c].y, sh[c], em) + BIAS;
        unsigned char* blk = adig + ((size_t)rt * NCH + c) * DIG * D_SLICE + at;
#pragma unroll
        for (int s = 0; s < DIG; ++s) {
          const int p = 8 * (DIG - 1 - s);
          const unsigned d = (unsigned)((yr >> p) & 255) | ((unsigned)((yi >> p) & 255) << 8);
          *reinterpret_cast<unsigned short*>(blk + s * D_SLICE) = (unsigned short)d;
        }
      }
    }
    return;
  }
  __shared__ int sm[8][32];
  const int ct = blockIdx.x - ablocks, j = ct * BNC + lane;
  double2 v[kZK / 8];
  int off[kZK / 8], em = kZeroExp;
#pragma unroll
  for (int i = 0; i < kZK / 8; ++i) {
    const int k = warp * (kZK / 8) + i;
    off[i] = KIND == ZRows::NONE ? 0 : -__shfl_sync(0xffffffffu, warp < 4 ? sh[0] : sh[1], k & 31);
    v[i] = (k < K && j < N) ? B[(int64_t)k * ldb + j] : make_double2(0.0, 0.0);
    em = max(em, max(expo(v[i].x, off[i]), expo(v[i].y, off[i])));
  }
  sm[warp][lane] = em;
  __syncthreads();
#pragma unroll
  for (int t = 0; t < 8; ++t) em = max(em, sm[t][lane]);
  if (warp == 0 && j < N) bexp[j] = em == kBadExp ? kNonFinite : em - 1022;
#pragma unroll
  for (int h = 0; h < 2; ++h) {
    const int k0 = warp * 8 + 4 * h, c = k0 / KCC, kk = k0 % KCC;
    long long yr[4], yi[4], yn[4];
#pragma unroll
    for (int i = 0; i < 4; ++i) {
      const int o = off[4 * h + i];
      const long long xr = fixed54(v[4 * h + i].x, o, em), xi = fixed54(v[4 * h + i].y, o, em);
      yr[i] = xr + BIAS;
      yi[i] = xi + BIAS;
      yn[i] = BIAS - xi;
    }
    unsigned char* blk = bdig + ((size_t)ct * NCH + c) * B_BLOCK;
#pragma unroll
    for (int s = 0; s < DIG; ++s) {
      const int p = DIG - 1 - s;
      const int rho = s * BN + 2 * lane;
      const uint2 a0 = widen4(pick4(yr[0], yn[0], yr[1], yn[1], p)), a1 = widen4(pick4(yr[2], yn[2], yr[3], yn[3], p));
      const uint2 b0 = widen4(pick4(yi[0], yr[0], yi[1], yr[1], p)), b1 = widen4(pick4(yi[2], yr[2], yi[3], yr[3], p));
      const int ch = kk >> 2;   // 16-byte chunk: real K 2 kk .. 2 kk + 7
      *reinterpret_cast<uint4*>(blk + (uint32_t)rho * 128u + ((uint32_t)(ch ^ (rho & 7)) << 4)) =
          make_uint4(a0.x, a0.y, a1.x, a1.y);
      *reinterpret_cast<uint4*>(blk + (uint32_t)(rho + 1) * 128u + ((uint32_t)(ch ^ ((rho + 1) & 7)) << 4)) =
          make_uint4(b0.x, b0.y, b1.x, b1.y);
    }
  }
}

// acc 2^sc rounded to nearest even, without FP64 arithmetic on the normal path
__device__ __forceinline__ double scaled_double(long long acc, int sc) {
  if (acc == 0) return 0.0;
  const unsigned long long u = acc < 0 ? 0ull - (unsigned long long)acc : (unsigned long long)acc;
  const int lz = __clzll((long long)u);
  const unsigned long long m = u << lz;
  unsigned long long keep = m >> 11;
  const unsigned rem = (unsigned)m & 0x7ffu;
  keep += (rem > 0x400u || (rem == 0x400u && (keep & 1ull))) ? 1ull : 0ull;
  const int be = 1023 + 63 - lz + sc;   // biased exponent
  if (be < 1 || be > 2045) return ldexp((double)acc, sc);
  const unsigned long long bits = ((unsigned long long)(be - 1) << 52) + keep;
  return __longlong_as_double((long long)(bits | (acc < 0 ? 0x8000000000000000ull : 0ull)));
}
// The same for |sc| <= 900, without branches: be0 = 1023 + 62 + sc.
__device__ __forceinline__ double scaled_plain(long long acc, int be0) {
  const unsigned long long u = acc < 0 ? 0ull - (unsigned long long)acc : (unsigned long long)acc;
  const int lz = __clzll((long long)u);
  const unsigned long long m = u << (lz & 63);
  unsigned long long keep = m >> 11;
  keep += ((unsigned)m & 0x7ffu) + ((unsigned)keep & 1u) > 0x400u ? 1ull : 0ull;
  const unsigned hi = (unsigned)(keep >> 32) + ((unsigned)(be0 - lz) << 20) + ((unsigned)(acc >> 32) & 0x80000000u);
  return u ? __hiloint2double((int)hi, (int)(unsigned)keep) : 0.0;
}

// a level sum, an integer of at most 2^22
__device__ __forceinline__ int level_int(uint32_t bits) {
  return __float_as_int(__uint_as_float(bits) + 12582912.f) - 0x4B400000;
}

// Digit slice s of A (descriptor ad) against B's slices (descriptor bb of the
// first): up to four levels per MMA, the K steps innermost.  s is a constant
// where this is inlined, so that an MMA costs its issuing thread no arithmetic
// but on the descriptors' low words (184 clocks each with the descriptors made
// on the way; 90 of tensor work).
__device__ __forceinline__ void issue_digit(uint32_t tmem, uint64_t ad, uint64_t bb, const int s, bool first) {
  using namespace tc;
  const int nt_all = DIG < LEV - s ? DIG : LEV - s;
#pragma unroll
  for (int t0 = 0; t0 < nt_all; t0 += 4) {
    const int nt = nt_all - t0 < 4 ? nt_all - t0 : 4;
#pragma unroll
    for (int ks = 0; ks < 4; ++ks) {
      const uint64_t a = ad + (uint64_t)(2 * ks), b = bb + (uint64_t)(t0 * (B_SLICE >> 4) + 2 * ks);
      const uint32_t d = tmem + (uint32_t)((s + t0) * BN);
      if (s == 1 && t0 == 4 && ks == 0) {
        // level 7 starts here (levels 0 .. 6 started with s = 0)
        mma_f16(d, a, b, idesc_f16_m128(2 * BN), 1u);
        mma_f16(d + 2 * BN, a, b + (uint64_t)(2 * (B_SLICE >> 4)), idesc_f16_m128(BN), first ? 0u : 1u);
      } else {
        mma_f16(d, a, b, idesc_f16_m128(nt * BN), s == 0 && ks == 0 && first ? 0u : 1u);
      }
    }
  }
}

// The same on the FP64 pipe (600 K clocks a tile of 128 x 32), by the whole CTA:
// thread = (column, every 16th row), K staged 16 at a time.  Calls, so that the
// kernel's registers are those of the way above.
struct Plain {
  const double2 *A, *B;
  int64_t lda, ldb;
  int K;
  ZOut out;
};
__device__ __noinline__ void plain_tiles(const Plain& p, unsigned char* smem, int M, int N, int ctiles,
                                         int total_tiles, double2* C, int64_t ldc, int* rowmax) {
  double2 (*As)[17] = reinterpret_cast<double2 (*)[17]>(smem);                                // [BM][16]
  double2 (*Bs)[BNC] = reinterpret_cast<double2 (*)[BNC]>(smem + BM * 17 * sizeof(double2));  // [16][BNC]
  const int tid = threadIdx.x, tx = tid & 31, ty = tid >> 5;
  for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) {
    const int row0 = (t / ctiles) * BM, col0 = (t % ctiles) * BNC;
    double2 acc[BM / 16];
#pragma unroll
    for (int i = 0; i < BM / 16; ++i) acc[i] = make_double2(0.0, 0.0);
    for (int k0 = 0; k0 < p.K; k0 += 16) {
      for (int i = tid; i < BM * 16; i += THREADS) {
        const int r = i >> 4, k = k0 + (i & 15);
        As[r][i & 15] = row0 + r < M && k < p.K ? p.A[(int64_t)(row0 + r) * p.lda + k] : make_double2(0.0, 0.0);
      }
      Bs[ty][tx] = k0 + ty < p.K && col0 + tx < N ? p.B[(int64_t)(k0 + ty) * p.ldb + col0 + tx] : make_double2(0.0, 0.0);
      __syncthreads();
#pragma unroll 4
      for (int k = 0; k < 16; ++k) {
        const double2 b = Bs[k][tx];
#pragma unroll
        for (int i = 0; i < BM / 16; ++i) cfma(acc[i], As[ty + 16 * i][k], b);
      }
      __syncthreads();
    }
#pragma unroll
    for (int i = 0; i < BM / 16; ++i) {
      const int row = row0 + ty + 16 * i;
      if (row < M && col0 + tx < N) {
        double2* c = C + (int64_t)row * ldc + col0 + tx;
        const double2 v = p.out == ZOut::SUB ? csub(*c, acc[i]) : acc[i];
        *c = v;
        if (rowmax) atomicMax(rowmax + row, field(v));
      }
    }
  }
}
// C = L^-1 C by substitution, 64 rows: two columns per warp, lane = rows lane and lane + 32
__device__ __noinline__ void plain_solve(const Plain& p, unsigned char* smem, int N, int total_tiles, double2* C,
                                         int64_t ldc, int* rowmax) {
  double2 (*L)[kZK + 1] = reinterpret_cast<double2 (*)[kZK + 1]>(smem);
  double2 (*X)[BNC + 1] = reinterpret_cast<double2 (*)[BNC + 1]>(smem + kZK * (kZK + 1) * sizeof(double2));
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  for (int i = tid; i < kZK * kZK; i += THREADS) {
    const int r = i / kZK, k = i % kZK;
    L[r][k] = k < r ? p.A[(int64_t)r * p.lda + k] : make_double2(0.0, 0.0);
  }
  for (int t = blockIdx.x; t < total_tiles; t += gridDim.x) {
    const int col0 = t * BNC;
    for (int i = tid; i < kZK * BNC; i += THREADS) {
      const int r = i / BNC, c = i % BNC;
      X[r][c] = col0 + c < N ? C[(int64_t)r * ldc + col0 + c] : make_double2(0.0, 0.0);
    }
    __syncthreads();
    for (int c = warp; c < BNC; c += THREADS / 32) {
      double2 x0 = X[lane][c], x1 = X[lane + 32][c];
      for (int k = 0; k < kZK - 1; ++k) {
        const double2 s = k < 32 ? x0 : x1;
        double2 xk;
        xk.x = __shfl_sync(0xffffffffu, s.x, k & 31);
        xk.y = __shfl_sync(0xffffffffu, s.y, k & 31);
        if (k < 31 && lane > k) cfms(x0, L[lane][k], xk);
        if (lane + 32 > k) cfms(x1, L[lane + 32][k], xk);
      }
      X[lane][c] = x0;
      X[lane + 32][c] = x1;
    }
    __syncthreads();
    for (int i = tid; i < kZK * BNC; i += THREADS) {
      const int r = i / BNC, c = i % BNC;   // a warp holds one row
      const bool in = col0 + c < N;
      if (in) C[(int64_t)r * ldc + col0 + c] = X[r][c];
      const int em = __reduce_max_sync(0xffffffffu, in ? field(X[r][c]) : 0);
      if (rowmax && c == 0 && em > 0) atomicMax(rowmax + r, em);
    }
    __syncthreads();
  }
}

// NaN in the place of the CTA's tiles, after a wait that ran out
__device__ __noinline__ void poison_tiles(int M, int N, int ctiles, int total_tiles, double2* C, int64_t ldc,
                                          const Slabs& sl) {
  const double nan = __longlong_as_double(0x7FF8000000000000LL);
  for (int tt = blockIdx.x; tt < total_tiles; tt += gridDim.x) {
    const int slab = tt / sl.tiles, t = tt - slab * sl.tiles;
    for (int i = threadIdx.x; i < BM * BNC; i += THREADS) {
      const int row = (t / ctiles) * BM + i / BNC, col = (t % ctiles) * BNC + i % BNC;
      if (row < M && col < N) C[slab * sl.c + (int64_t)row * ldc + col] = make_double2(nan, nan);
    }
  }
}

__global__ void __launch_bounds__(THREADS, 1)
zgemm_kernel(const unsigned char* __restrict__ adig, const int* __restrict__ aexp,
             const unsigned char* __restrict__ bdig, const int* __restrict__ bexp, int M, int N, int nch, int ctiles,
             int total_tiles, double2* C, int64_t ldc, Plain p64, int* __restrict__ rowmax, int* status,
             Slabs sl) {
  using namespace tc;
  const bool sub = p64.out == ZOut::SUB;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* aring = base;
  unsigned char* bring = aring + ASLOTS * A_SLICE;
  unsigned char* dring = bring + 2 * B_BLOCK;
  unsigned char* cstage = dring + DSLOTS * D_SLICE;
  uint64_t* full_a = reinterpret_cast<uint64_t*>(cstage + NEPI * STAGE);
  uint64_t* empty_a = full_a + ASLOTS;
  uint64_t* full_d = empty_a + ASLOTS;
  uint64_t* empty_d = full_d + DSLOTS;
  uint64_t* full_b = empty_d + DSLOTS;
  uint64_t* empty_b = full_b + 2;
  uint64_t* tfull = empty_b + 2;
  uint64_t* tempty = tfull + 1;
  uint64_t* done = tempty + 1;
  uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(done + 1);
  volatile int* abort = reinterpret_cast<volatile int*>(tmem_slot + 1);
  int* fp64 = reinterpret_cast<int*>(tmem_slot + 2);   // the digits' kernel marked the product

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int first = blockIdx.x, stride = gridDim.x;
  const int ntiles = total_tiles > first ? (total_tiles - first + stride - 1) / stride : 0;
  const int nblk = ntiles * nch;   // B blocks (and DIG times as many A slices) of this CTA

  if (threadIdx.x == 0) {
    for (int s = 0; s < ASLOTS; ++s) { mbar_init(&full_a[s], NCONV); mbar_init(&empty_a[s], 1); }
    for (int s = 0; s < DSLOTS; ++s) { mbar_init(&full_d[s], 1); mbar_init(&empty_d[s], NCONV); }
    for (int s = 0; s < 2; ++s) { mbar_init(&full_b[s], 1); mbar_init(&empty_b[s], 1); }
    mbar_init(tfull, 1);
    mbar_init(tempty, NEPI);
    mbar_init(done, 1);
    *abort = 0;
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == 0) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(tmem_slot)),
                 "r"(TMEM_COLS)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
  }
  tc_fence_before();
  __syncthreads();
  tc_fence_after();
  const uint32_t tmem = *tmem_slot;
  early_start();

  if (warp == 0 && lane == 0) {
    // ---------------- producer: whichever copy has a free slot
    const int nq = nblk * DIG;
    int ib = 0, q = 0;
    uint32_t idle = 0;
    while ((ib < nblk || q < nq) && !*abort) {
      bool progress = false;
      if (ib < nblk && (ib < 2 || mbar_test(&empty_b[ib & 1], ((ib >> 1) - 1) & 1))) {
        const int tt = first + (ib / nch) * stride, slab = tt / sl.tiles, ct = (tt - slab * sl.tiles) % ctiles;
        mbar_expect_tx(&full_b[ib & 1], B_BLOCK);
        bulk_load(bring + (ib & 1) * B_BLOCK, bdig + slab * sl.bdig + ((size_t)ct * NCH + ib % nch) * B_BLOCK, B_BLOCK,
                  &full_b[ib & 1]);
        ++ib;
        progress = true;
      }
      if (q < nq && (q < DSLOTS || mbar_test(&empty_d[q % DSLOTS], ((q / DSLOTS) - 1) & 1))) {
        const int blk = q / DIG, tt = first + (blk / nch) * stride, slab = tt / sl.tiles;
        const int rt = (tt - slab * sl.tiles) / ctiles;
        mbar_expect_tx(&full_d[q % DSLOTS], D_SLICE);
        bulk_load(dring + (q % DSLOTS) * D_SLICE,
                  adig + slab * sl.adig + (((size_t)rt * NCH + blk % nch) * DIG + q % DIG) * D_SLICE, D_SLICE, &full_d[q % DSLOTS]);
        ++q;
        progress = true;
      }
      if (progress) idle = 0;
      else if (++idle >= kProducerLimit) { *abort = 1; break; }
    }
    *fp64 = p64.A && *aexp == kPlainExp;   // (read here, where nothing waits for it)
    // copies in flight land before the CTA may exit
    for (int j = max(0, ib - 2); j < ib; ++j) mbar_wait_plain(&full_b[j & 1], (j >> 1) & 1);
    for (int j = max(0, q - DSLOTS); j < q; ++j) mbar_wait_plain(&full_d[j % DSLOTS], (j / DSLOTS) & 1);
  } else if (warp == 1 && lane == 0) {
    // ---------------- MMA issuer: one readout (at most 128 real K) per tile
    int q = 0, i = 0;
    bool ok = true;
    const uint64_t a0 = kmajor_sw128_desc(smem_u32(aring));
    for (int lt = 0; lt < ntiles && ok; ++lt) {
      if (lt > 0) {
        if (!mbar_wait(tempty, (lt - 1) & 1, abort)) { ok = false; break; }
        tc_fence_after();
      }
      for (int c = 0; c < nch && ok; ++c, ++i) {
        const int st = i & 1;
        if (!mbar_wait(&full_b[st], (i >> 1) & 1, abort)) { ok = false; break; }
        tc_fence_after();
        const uint64_t bb = kmajor_sw128_desc(smem_u32(bring + st * B_BLOCK));
#pragma unroll
        for (int s = 0; s < DIG; ++s, ++q) {
          if (!ok) continue;
          const int slot = q % ASLOTS;
          if (!mbar_wait(&full_a[slot], (q / ASLOTS) & 1, abort)) { ok = false; continue; }
          tc_fence_after();
          const uint64_t ad = a0 + (uint64_t)(slot * (A_SLICE >> 4));
          issue_digit(tmem, ad, bb, s, c == 0);
          mma_commit(&empty_a[slot]);
        }
        if (ok) mma_commit(&empty_b[st]);
      }
      if (ok) mma_commit(tfull);
    }
    mma_commit(done);   // arrives once every MMA issued above has completed
  } else if (warp >= EPI0 && warp < EPI0 + NEPI) {
    // ---------------- epilogue: thread = (row, half of the real columns)
    const int qd = warp & 3, part = (warp - EPI0) >> 2, r = qd * 32 + lane;
    const uint32_t tbase = tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(part * EPI_COLS);
    for (int lt = 0; lt < ntiles; ++lt) {
      const int tt = first + lt * stride, slab = tt / sl.tiles, t = tt - slab * sl.tiles;
      const int row = (t / ctiles) * BM + r, col0 = (t % ctiles) * BNC + part * (EPI_COLS / 2);
      double2* crow = C + slab * sl.c + (int64_t)row * ldc + col0;
      int ncol = row < M ? min(EPI_COLS / 2, N - col0) : 0;
      if (sub && ncol > 0) {
        asm volatile("prefetch.global.L2 [%0];" ::"l"(crow));
        asm volatile("prefetch.global.L2 [%0];" ::"l"(crow + (ncol - 1)));
      }
      if (!__all_sync(0xffffffffu, mbar_wait(tfull, lt & 1, abort))) break;   // (the warp leaves as one)
      tc_fence_after();
      long long acc[EPI_COLS];
#pragma unroll
      for (int p = 0; p < EPI_COLS / 4; ++p) {
        uint32_t v[LEV][4];
#pragma unroll
        for (int l = 0; l < LEV; ++l) tmem_ld4(tbase + (uint32_t)(l * BN + p * 4), v[l]);
        tmem_wait_ld();
        if (p == EPI_COLS / 4 - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(tempty)) : "memory");
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // level l weighs 2^(42 - 8 l) units of 2^-54; |L_0| <= 2^19, |L_1| <= 2^21, |L_2| <= 2^22,
          // |L_3| < 2^22.6: hi and mid are exact in 32 bits.  The conversions run at 16 lanes a clock
          // (4 K clocks a tile); up to 2^22 the sum with 1.5 2^23 has the integer in its low bits
          const int hi = (level_int(v[0][j]) << 8) + level_int(v[1][j]);
          const int mid = (level_int(v[2][j]) << 8) + __float2int_rz(__uint_as_float(v[3][j]));
          const int l4 = __float2int_rz(__uint_as_float(v[4][j])), l5 = __float2int_rz(__uint_as_float(v[5][j]));
          const int l67 = __float2int_rn(
              0.015625f * fmaf(__uint_as_float(v[7][j]), 0.00390625f, __uint_as_float(v[6][j])));
          acc[p * 4 + j] = ((long long)hi << 34) + ((long long)mid << 18) + ((long long)l4 << 10) +
                           (long long)((l5 << 2) + l67);
        }
      }
      const int ea = row < M ? aexp[slab * sl.aexp + row] : 0;
      const int ebl = lane < EPI_COLS / 2 && col0 + lane < N ? bexp[slab * sl.bexp + col0 + lane] : 0;
      // Where the whole warp has full rows, finite operands and results far from
      // overflow and underflow: no branch from entry to entry, and C in groups of
      // four columns that pass through shared memory, so that an access covers 64
      // bytes of 8 rows instead of 16 of 32 (entry by entry, 32 lines an access
      // and each load behind the store before it, a tile took 22 K clocks).
      constexpr int NC = EPI_COLS / 2, G = 4;
      int em = 0;
      const int ebmax = __reduce_max_sync(0xffffffffu, lane < NC ? ebl : INT_MIN);
      const int ebmin = __reduce_min_sync(0xffffffffu, lane < NC ? ebl : INT_MAX);
      if (ea == kPlainExp) ncol = 0;   // C stays as it is
      const bool plain = ncol == NC && ea != kNonFinite && ebmax < 1 << 20 && abs(ea + ebmax - FIX) <= 900 &&
                         abs(ea + ebmin - FIX) <= 900;
      if (__all_sync(0xffffffffu, plain)) {
        unsigned char* stage = cstage + (warp - EPI0) * STAGE;
        // this lane's place in the group: rows 8 i + lane / 4, column lane % 4
        const int r4 = lane >> 2, c4 = lane & 3;
        double2* cq = C + slab * sl.c + (int64_t)(row - lane + r4) * ldc + col0 + c4;
        int emr[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) emr[i] = 0;
#pragma unroll
        for (int g = 0; g < NC / G; ++g) {
          double2 o[4];
          if (sub) {
#pragma unroll
            for (int i = 0; i < 4; ++i) o[i] = cq[8 * i * ldc + G * g];
          }
#pragma unroll
          for (int j = 0; j < G; ++j) {
            const int be0 = ea + __shfl_sync(0xffffffffu, ebl, G * g + j) + (1023 + 62 - FIX);
            *reinterpret_cast<double2*>(stage + lane * 64 + ((j ^ ((lane >> 1) & 3)) << 4)) =
                make_double2(scaled_plain(acc[2 * (G * g + j)], be0), scaled_plain(acc[2 * (G * g + j) + 1], be0));
          }
          __syncwarp();
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            const int rr = 8 * i + r4;
            double2 v = *reinterpret_cast<const double2*>(stage + rr * 64 + ((c4 ^ ((rr >> 1) & 3)) << 4));
            if (sub) v = make_double2(o[i].x - v.x, o[i].y - v.y);
            cq[8 * i * ldc + G * g] = v;
            if (rowmax) emr[i] = max(emr[i], field(v));
          }
          __syncwarp();
        }
        if (rowmax) {
#pragma unroll
          for (int i = 0; i < 4; ++i) {
            emr[i] = max(emr[i], __shfl_xor_sync(0xffffffffu, emr[i], 1));
            emr[i] = max(emr[i], __shfl_xor_sync(0xffffffffu, emr[i], 2));
            if (c4 == 0 && emr[i] > 0) atomicMax(rowmax + row - lane + 8 * i + r4, emr[i]);
          }
        }
      } else {
#pragma unroll
        for (int j = 0; j < NC; ++j) {
          const int eb = __shfl_sync(0xffffffffu, ebl, j);
          if (j < ncol) {
            double2 v = sub ? crow[j] : make_double2(0.0, 0.0);
            if (ea == kNonFinite || eb == kNonFinite) {
              v.x = v.y = __longlong_as_double(0x7FF8000000000000LL);
            } else {
              const int sc = ea + eb - FIX;
              const double x = scaled_double(acc[2 * j], sc), y = scaled_double(acc[2 * j + 1], sc);
              v = sub ? make_double2(v.x - x, v.y - y) : make_double2(x, y);
            }
            crow[j] = v;
            em = max(em, field(v));
          }
        }
      }
      if (rowmax && em > 0) atomicMax(rowmax + row, em);
    }
  } else if (warp >= EPI0 + NEPI) {
    // ---------------- converters: staged byte slice -> FP16 operand slice
    const int ctid = threadIdx.x - (EPI0 + NEPI) * 32;
    const int nq = nblk * DIG;
    for (int q = 0; q < nq; ++q) {
      const int ds = q % DSLOTS, as = q % ASLOTS;
      const bool ok = mbar_wait(&full_d[ds], (q / DSLOTS) & 1, abort) &&
                      (q < ASLOTS || mbar_wait(&empty_a[as], ((q / ASLOTS) - 1) & 1, abort));
      const unsigned char* src = dring + ds * D_SLICE;
      unsigned char* dst = aring + as * A_SLICE;
      if (ok)
        for (int u = ctid; u < (int)(D_SLICE / 8); u += NCONV * 32) {
          const uint32_t off = (uint32_t)u * 8u;
          const uint2 v = *reinterpret_cast<const uint2*>(src + off);
          const uint2 w0 = widen4(v.x), w1 = widen4(v.y);
          *reinterpret_cast<uint4*>(dst + 2 * off) = make_uint4(w0.x, w0.y, w1.x, w1.y);
        }
      fence_async_smem();
      if (!__all_sync(0xffffffffu, ok)) break;   // (the warp leaves as one)
      if (lane == 0) {
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full_a[as])) : "memory");
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty_d[ds])) : "memory");
      }
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort) atomicExch(status, MGT_ERR_TIMEOUT);
  if (*abort) {
    poison_tiles(M, N, ctiles, total_tiles, C, ldc, sl);
  } else if (*fp64) {
    // every copy has landed, every product is done (the epilogue has waited for the last tile's)
    if (p64.out == ZOut::SOLVE) plain_solve(p64, base, N, total_tiles, C, ldc, rowmax);
    else plain_tiles(p64, base, M, N, ctiles, total_tiles, C, ldc, rowmax);
  }
  if (warp == 0) {
    if (lane == 0) mbar_wait_plain(done, 0);
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// ---------------------------------------------------------------- interchanges of the blocked LU

constexpr int SB = 32;       // panel width
constexpr int SLAB = 8;      // columns per CTA of zswap_kernel (one warp each in the solve)

// Forward substitution with a unit lower 32 x 32 factor, one column per warp, lane = row.
__device__ __forceinline__ double2 lower_solve32(const double2* L, int w, double2 x, int lane) {
  for (int k = 0; k < w - 1; ++k) {
    double2 xk;
    xk.x = __shfl_sync(0xffffffffu, x.x, k);
    xk.y = __shfl_sync(0xffffffffu, x.y, k);
    if (lane > k) cfms(x, L[lane * (SB + 1) + k], xk);
  }
  return x;
}

// Blocks: 8-column slabs of [lb, le), then of [rb, re), then (inv) four blocks of L11^-1's columns.
__global__ void __launch_bounds__(256)
zswap_kernel(double2* __restrict__ A, int64_t lda, int n, int j0, int w, ZSlots sl, int lb, int le, int rb, int re,
             int solve, double2* __restrict__ inv, int ldinv, int* __restrict__ invmax) {
  early_start();
  __shared__ __align__(16) double2 buf[2 * SB][SLAB];
  __shared__ __align__(16) double2 L[SB * (SB + 1)];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int nleft = le > lb ? (le - lb + SLAB - 1) / SLAB : 0, nright = re > rb ? (re - rb + SLAB - 1) / SLAB : 0;
  const int b = blockIdx.x;
  const bool is_inv = b >= nleft + nright, right = !is_inv && b >= nleft;
  if (is_inv || (right && solve))
    for (int i = tid; i < SB * SB; i += 256) {
      const int r = i / SB, k = i % SB;
      const bool ok = r < w && k < w;
      cp_async_elem<16>(L + r * (SB + 1) + k, ok ? A + (int64_t)(j0 + r) * lda + j0 + k : A, ok);
    }
  if (is_inv) {
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const int col = (b - nleft - nright) * 8 + warp;
    const double2 x = lower_solve32(L, w, make_double2(lane == col ? 1.0 : 0.0, 0.0), lane);
    inv[(int64_t)lane * ldinv + col] = x;
    const int em = __reduce_max_sync(0xffffffffu, field(x));
    if (lane == 0) atomicMax(invmax, em);
    return;
  }
  const int c0 = right ? rb + (b - nleft) * SLAB : lb + b * SLAB;
  const int ncols = min(SLAB, (right ? re : le) - c0);
  const int m = n - j0, ns = min(*sl.nslot, 2 * SB);
  const bool top_needed = right && solve;
  for (int i = tid; i < ns * SLAB; i += 256) {
    const int q = i / SLAB, cc = i % SLAB;
    const int2 v = sl.slots[q];
    const bool in = v.x >= 0 && v.x < m && v.y >= 0 && v.y < m;
    if (cc < ncols && in && (v.x != v.y || (top_needed && v.x < w)))
      cp_async_elem<16>(&buf[q][cc], A + (int64_t)(j0 + v.y) * lda + c0 + cc, true);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  if (top_needed && warp < ncols) {
    // the first 32 slots are the panel's own rows, in order
    double2 x = lane < w ? buf[lane][warp] : make_double2(0.0, 0.0);
    x = lower_solve32(L, w, x, lane);
    if (lane < w) buf[lane][warp] = x;
  }
  __syncthreads();
  for (int i = tid; i < ns * SLAB; i += 256) {
    const int q = i / SLAB, cc = i % SLAB;
    const int2 v = sl.slots[q];
    const bool in = v.x >= 0 && v.x < m && v.y >= 0 && v.y < m;
    if (cc < ncols && in && (v.x != v.y || (top_needed && v.x < w))) A[(int64_t)(j0 + v.x) * lda + c0 + cc] = buf[q][cc];
  }
}

// Both panels' interchanges on the columns left and right of a 64-wide block,
// 32 columns per CTA, one panel after the other; eight more CTAs (Inv) finish
// the block's inverse L^-1 = [[Ia, 0], [-Lb^-1 Lba Ia, Lb^-1]], a column per
// warp.  kexp (64 zeros) receives the largest exponent fields of the block's
// rows right of it.
__global__ void __launch_bounds__(256)
zswap_block_kernel(double2* __restrict__ A, int64_t lda, int n, int J0, int wa, int wb, ZSlots sa, ZSlots sb,
                   int nleft, int nright, double2* __restrict__ Inv, int* __restrict__ invmax, int* __restrict__ kexp) {
  early_start();
  // the moved rows (2 SB x 32), or the inverse's two 32 x 33 factors
  __shared__ __align__(16) unsigned char raw[2 * SB * (SB + 1) * sizeof(double2)];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
  const int b = blockIdx.x, j1 = J0 + wa, W = wa + wb;
  if (b >= nleft + nright) {
    // inverse CTAs: columns 0..31 are -Lb^-1 Lba Ia, columns 32..63 are Lb^-1
    double2* Lb = reinterpret_cast<double2*>(raw);
    double2* Lba = Lb + SB * (SB + 1);
    const int c8 = b - nleft - nright;
    for (int i = tid; i < SB * SB; i += 256) {
      const int r = i / SB, k = i % SB;
      const bool okb = r < wb && k < wb, oka = r < wb && k < wa;
      cp_async_elem<16>(Lb + r * (SB + 1) + k, okb ? A + (int64_t)(j1 + r) * lda + j1 + k : A, okb);
      cp_async_elem<16>(Lba + r * (SB + 1) + k, oka ? A + (int64_t)(j1 + r) * lda + J0 + k : A, oka);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    const int col = c8 * 8 + warp;
    double2 x;
    if (col < SB) {
      const double2 ia = Inv[(int64_t)lane * kZK + col];   // Ia[lane][col]
      x = make_double2(0.0, 0.0);
      for (int k = col; k < SB; ++k) {
        double2 v;
        v.x = __shfl_sync(0xffffffffu, ia.x, k);
        v.y = __shfl_sync(0xffffffffu, ia.y, k);
        cfms(x, Lba[lane * (SB + 1) + k], v);
      }
    } else {
      x = make_double2(lane == col - SB ? 1.0 : 0.0, 0.0);
    }
    x = lower_solve32(Lb, wb, x, lane);
    Inv[(int64_t)(SB + lane) * kZK + col] = x;
    if (col >= SB) Inv[(int64_t)lane * kZK + col] = make_double2(0.0, 0.0);
    const int em = __reduce_max_sync(0xffffffffu, field(x));
    if (lane == 0) atomicMax(invmax, em);
    return;
  }
  double2* buf = reinterpret_cast<double2*>(raw);   // [2 SB][32]
  const bool right = b >= nleft;
  const int c0 = right ? J0 + W + (b - nleft) * 32 : b * 32;
  const int ncols = min(32, (right ? n : J0) - c0);
  for (int set = 0; set < (wb > 0 ? 2 : 1); ++set) {
    const int jj = set ? j1 : J0, m = n - jj;
    const int2* slots = set ? sb.slots : sa.slots;
    const int ns = min(set ? *sb.nslot : *sa.nslot, 2 * SB);
    for (int i = tid; i < ns * 32; i += 256) {
      const int q = i >> 5, cc = i & 31;
      const int2 v = slots[q];
      const bool in = v.x >= 0 && v.x < m && v.y >= 0 && v.y < m && v.x != v.y;
      if (cc < ncols && in) cp_async_elem<16>(buf + i, A + (int64_t)(jj + v.y) * lda + c0 + cc, true);
    }
    cp_async_commit();
    cp_async_wait<0>();
    __syncthreads();
    for (int i = tid; i < ns * 32; i += 256) {
      const int q = i >> 5, cc = i & 31;
      const int2 v = slots[q];
      const bool in = v.x >= 0 && v.x < m && v.y >= 0 && v.y < m && v.x != v.y;
      if (cc < ncols && in) A[(int64_t)(jj + v.x) * lda + c0 + cc] = buf[i];
    }
    __syncthreads();
  }
  if (right && kexp)
    for (int k = warp; k < W; k += 8) {
      const double2 v = lane < ncols ? A[(int64_t)(J0 + k) * lda + c0 + lane] : make_double2(0.0, 0.0);
      const int em = __reduce_max_sync(0xffffffffu, field(v));
      if (lane == 0 && em > 0) atomicMax(kexp + k, em);
    }
}

static size_t up(size_t v, size_t a) { return (v + a - 1) / a * a; }

}  // namespace zg

static void set_attributes() {
  static OncePerDevice once;
  once([] {
    cudaFuncSetAttribute(zg::zgemm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)zg::smem_bytes());
  });
}

size_t zgemm_bytes(int64_t rows, int64_t cols) {
  using namespace zg;
  const size_t rt = (size_t)((rows + BM - 1) / BM), ct = (size_t)((cols + BNC - 1) / BNC);
  return 1024 + up(rt * NCH * DIG * D_SLICE, 1024) + up(ct * NCH * B_BLOCK, 1024) + up(rt * BM * sizeof(int), 256) +
         up(ct * BNC * sizeof(int), 256);
}

void ZGemmPlan::init(void* work, int64_t r, int64_t c) {
  using namespace zg;
  const size_t rt = (size_t)((r + BM - 1) / BM), ct = (size_t)((c + BNC - 1) / BNC);
  char* b = (char*)up((size_t)work, 1024);
  adig = (unsigned char*)b;
  b += up(rt * NCH * DIG * D_SLICE, 1024);
  bdig = (unsigned char*)b;
  b += up(ct * NCH * B_BLOCK, 1024);
  aexp = (int*)b;
  b += up(rt * BM * sizeof(int), 256);
  bexp = (int*)b;
  rows = r;
  cols = c;
}

int zgemm_digits(const ZGemmPlan& p, const double2* A, int64_t lda, int M, const double2* B, int64_t ldb, int N, int K,
                 const ZRows& rows, cudaStream_t s) {
  using namespace zg;
  if (!A) M = 0;
  if (!B) N = 0;
  if (K <= 0 || K > kZK || M > p.rows || N > p.cols || M < 0 || N < 0) return MGT_ERR_ARG;
  // whole 128-row tiles of A: rows beyond M are written as zeros
  const int ab = (M + BM - 1) / BM * (BM / 32), bb = (N + BNC - 1) / BNC;
  if (ab + bb == 0) return MGT_OK;
  count_launch();
  launch_early(early_fits(ab + bb),
               rows.kind == ZRows::MEAN  ? digits_kernel<ZRows::MEAN>
               : rows.kind == ZRows::MAX ? digits_kernel<ZRows::MAX>
                                         : digits_kernel<ZRows::NONE>,
               ab + bb, 256, 0, s, A, lda, M, ab, B, ldb, N, K, rows, p.adig, p.aexp,
               p.bdig, p.bexp, Slabs());
  return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_ERR_CUDA;
}

int zgemm_apply(const ZGemmPlan& p, const double2* A, int64_t lda, int M, const double2* B, int64_t ldb, int N, int K,
                double2* C, int64_t ldc, ZOut out, int* rowmax, int* status, cudaStream_t s) {
  using namespace zg;
  if (M <= 0 || N <= 0) return MGT_OK;
  if (K <= 0 || K > kZK || M > p.rows || N > p.cols || (out == ZOut::SOLVE && (M != kZK || K != kZK))) return MGT_ERR_ARG;
  set_attributes();
  const int rt = (M + BM - 1) / BM, ct = (N + BNC - 1) / BNC;
  const int64_t total = (int64_t)rt * ct;
  if (total > (1 << 30)) return MGT_ERR_UNSUPPORTED;
  const int ctas = (int)std::min<int64_t>(total, device_sm_count());
  count_launch();
  launch_early(total <= 8 * ctas, zgemm_kernel, ctas, THREADS, smem_bytes(), s, p.adig, p.aexp, p.bdig, p.bexp, M, N,
               (K + KCC - 1) / KCC, ct, (int)total, C, ldc, Plain{A, B, lda, ldb, K, out}, rowmax, status, Slabs());
  return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_ERR_CUDA;
}

// ---- products over any K: slabs of 64 columns, partial products summed in FP64

namespace zg {

// Sizes of B's rows (ZRows::MEAN), one warp per row.
__global__ void __launch_bounds__(256)
row_stats_kernel(const double2* __restrict__ B, int64_t ldb, int K, int N, int4* __restrict__ stats) {
  const int k = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (k >= K) return;
  int em = 0, sum = 0, count = 0;
  for (int c = lane; c < N; c += 32) {
    const int f = field(B[(int64_t)k * ldb + c]);
    em = max(em, f);
    sum += f ? f - 1023 : 0;
    count += f ? 1 : 0;
  }
  em = __reduce_max_sync(0xffffffffu, em);
  sum = __reduce_add_sync(0xffffffffu, sum);
  count = __reduce_add_sync(0xffffffffu, count);
  const long long both = ((long long)count << 32) + sum;
  if (lane == 0) stats[k] = make_int4(em, 0, (int)both, (int)(both >> 32));
}

// out = E0 - sum over slabs of part; a slab that the digits' kernel left to the
// FP64 pipe (its row exponents say so) is multiplied out here.
__global__ void slab_sum_kernel(const double2* __restrict__ part, int slabs, int M, int N,
                                const double2* __restrict__ E0, int64_t ld0, double2* __restrict__ out, int64_t ldo,
                                const int* __restrict__ aexp, size_t aexp_stride, const double2* __restrict__ A,
                                int64_t lda, const double2* __restrict__ B, int64_t ldb, int K) {
  early_start();
  const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (i >= (int64_t)M * N) return;
  const int64_t r = i / N, c = i - r * N;
  double2 s = make_double2(0.0, 0.0);
  for (int q = 0; q < slabs; ++q) {
    double2 p;
    if (__ldg(aexp + q * aexp_stride) == kPlainExp) {
      p = make_double2(0.0, 0.0);
      for (int k = q * kZK; k < min(K, (q + 1) * kZK); ++k) cfma(p, A[r * lda + k], B[k * ldb + c]);
    } else {
      p = part[(int64_t)q * M * N + i];
    }
    s = cadd(s, p);
  }
  const double2 e = E0 ? E0[r * ld0 + c] : make_double2(0.0, 0.0);
  out[r * ldo + c] = csub(e, s);
}

struct Wide {
  int slabs;
  size_t rt, ct, adig, bdig, aexp, bexp, stats, part, total;
  Wide(int64_t M, int64_t N, int64_t K) {
    slabs = (int)((K + kZK - 1) / kZK);
    rt = (size_t)((M + BM - 1) / BM);
    ct = (size_t)((N + BNC - 1) / BNC);
    adig = 0;
    bdig = adig + up(slabs * rt * NCH * DIG * D_SLICE, 1024);
    aexp = bdig + up(slabs * ct * NCH * B_BLOCK, 1024);
    bexp = aexp + up(slabs * rt * BM * sizeof(int), 256);
    stats = bexp + up(slabs * ct * BNC * sizeof(int), 256);
    part = stats + (size_t)slabs * kZK * sizeof(int4);
    total = part + (size_t)slabs * M * N * sizeof(double2) + 1024;
  }
};

}  // namespace zg

size_t zgemm_wide_bytes(int64_t M, int64_t N, int64_t K) { return zg::Wide(M, N, K).total; }

int zgemm_wide(const double2* A, int64_t lda, int M, const double2* B, int64_t ldb, int N, int K, const double2* E0,
               int64_t ld0, double2* out, int64_t ldo, void* work, int* status, cudaStream_t s) {
  using namespace zg;
  const Wide w(M, N, K);
  char* b = (char*)up((size_t)work, 1024);
  unsigned char* adig = (unsigned char*)b + w.adig;
  unsigned char* bdig = (unsigned char*)b + w.bdig;
  int* aexp = (int*)(b + w.aexp);
  int* bexp = (int*)(b + w.bexp);
  double2* part = (double2*)(b + w.part);
  const int64_t total = (int64_t)w.rt * w.ct * w.slabs;
  if (w.slabs > 65535 || total > (1 << 30)) return MGT_ERR_UNSUPPORTED;
  Slabs sl;
  sl.adig = w.rt * NCH * DIG * D_SLICE;
  sl.bdig = w.ct * NCH * B_BLOCK;
  sl.aexp = w.rt * BM;
  sl.bexp = w.ct * BNC;
  sl.c = (size_t)M * N;
  sl.tiles = (int)(w.rt * w.ct);
  set_attributes();
  const int ab = (int)w.rt * (BM / 32);
  int4* stats = (int4*)(b + w.stats);
  count_launch(4);
  launch_early(false, row_stats_kernel, (K + 7) / 8, 256, 0, s, B, ldb, K, N, stats);
  const ZRows rows{ZRows::MEAN, (const int*)stats, nullptr};
  launch_early(false, digits_kernel<ZRows::MEAN>, dim3(ab + (unsigned)w.ct, w.slabs), 256, 0, s, A, lda, M, ab, B, ldb, N, K, rows, adig, aexp,
                                                                  bdig, bexp, sl);
  launch_early(false, zgemm_kernel, (int)std::min<int64_t>(total, device_sm_count()), THREADS, smem_bytes(), s,
      adig, aexp, bdig, bexp, M, N, NCH, (int)w.ct, (int)total, part, N,
      Plain{nullptr, nullptr, 0, 0, 0, ZOut::SET}, nullptr, status, sl);
  launch_early(false, slab_sum_kernel, (unsigned)(((int64_t)M * N + 255) / 256), 256, 0, s, part, w.slabs, M, N, E0, ld0, out, ldo,
               aexp, sl.aexp, A, lda, B, ldb, K);
  return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_ERR_CUDA;
}

int zswap_panel(double2* A, int64_t lda, int n, int j0, int w, const ZSlots& sl, int lb, int le, int rb, int re,
                bool solve, double2* inv, int ldinv, int* invmax, cudaStream_t st) {
  using namespace zg;
  const int nl = le > lb ? (le - lb + SLAB - 1) / SLAB : 0, nr = re > rb ? (re - rb + SLAB - 1) / SLAB : 0;
  const int blocks = nl + nr + (inv ? 4 : 0);
  if (blocks == 0) return MGT_OK;
  count_launch();
  launch_early(early_fits(blocks), zswap_kernel, blocks, 256, 0, st, A, lda, n, j0, w, sl, lb, le, rb, re, solve ? 1 : 0, inv, ldinv, invmax);
  return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_ERR_CUDA;
}

int zswap_block(double2* A, int64_t lda, int n, int J0, int wa, int wb, const ZSlots& a, const ZSlots& b,
                double2* Inv, int* invmax, int* kexp, cudaStream_t st) {
  using namespace zg;
  const int nleft = (J0 + 31) / 32, nright = (n - J0 - wa - wb + 31) / 32;
  const int blocks = nleft + nright + (Inv ? 8 : 0);
  if (blocks == 0) return MGT_OK;
  count_launch();
  launch_early(early_fits(blocks), zswap_block_kernel, blocks, 256, 0, st, A, lda, n, J0, wa, wb, a, b, nleft, nright, Inv, invmax, kexp);
  return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_ERR_CUDA;
}

}  // namespace mgt
