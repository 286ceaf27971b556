// Tensor-core residual R = B - M X for iterative refinement: M in
// double-float form (MGT_CDF), X, B, R complex128.
//
// Method: an error-free splitting of both operands into small integers
// ("digits") that FP16 holds exactly, multiplied on the tensor cores with
// FP32 accumulation kept exact -- the Ozaki scheme (Ozaki, Ogita, Oishi and
// Rump, "Error-free transformations of matrix multiplication by using fast
// routines of matrix multiplication and its applications", Numer.
// Algorithms 2012), in its FP16 tensor-core form (Mukunoki, Ozaki, Ogita and
// Imamura, "DGEMM using Tensor Cores, and Its Accurate and Reproducible
// Versions", ISC 2020).
//  * The complex product is the real product A' B' of A' (rows x 2 kdim,
//    row i = Mr_i0, Mi_i0, Mr_i1, Mi_i1, ...) and B'^T (2 nrhs x 2 kdim: row
//    2j = Xr_0j, -Xi_0j, ...; row 2j+1 = Xi_0j, Xr_0j, ...).
//  * Row i of A' is scaled by 2^-e_i, 2^e_i bounding the row's largest
//    |re|, |im|, and every entry becomes the integer
//    X = round((hi + lo) 2^(54 - e_i)), |X| < 2^54, written with seven
//    balanced base-256 digits X = sum_{p=0..6} d_p 256^p: the bytes of
//    X + 128 (256^0 + ... + 256^6) minus 128, so d_0 .. d_5 lie in
//    [-128, 127] and the top digit d_6 in [-64, 64].  The columns of B' are
//    scaled by their own power of two the same way.
//  * A digit needs at most 8 bits and is exact in FP16; a product of two is
//    at most 2^14.  Counting digits from the top (s = 6 - p), the pairs
//    (s, t) with s + t = l share the weight 256^-l and accumulate in one
//    TMEM accumulator per level l = 0 .. 6; pairs with s + t > 6 lie below
//    2^-55 of the row and column scales and are not formed.  A level sums
//    256 products of each of its pairs before it is read out; levels 0 .. 4
//    then stay within 2^24 (the top digits are smaller), exact integers in
//    FP32, and 5 and 6 would round only beyond 2^24, by units that weigh
//    2^-4 and 2^-12.
//  * Every 256 real K the level sums are read out of TMEM and folded into
//    one 64-bit integer per output in units of 2^-48 of the row and column
//    scales: levels 0 .. 4 exactly, 5 and 6 rounded to within a unit.  A
//    64-bit accumulator per output sums them exactly (at most 2^15 real K per
//    CTA keeps it below 2^63); the result is scaled back once at the end.
// Accuracy (a numpy emulation of exactly this scheme on 2D / 3D systems of
// order 1400 / 2100): residual errors of 3e-14 / 1e-14 of ||B||, where six
// digits give 8e-12 / 2e-12.
//
// Two passes.  digitize_kernel turns M into its digits once per matrix
// (refinement reuses them for every residual): one byte per digit (the
// biased digit d + 128), seven digit slices of 128 rows x 64 real K per
// (row tile, 32-column chunk), 56 KB contiguous, each slice laid out as the
// MMA operand's 128-byte-swizzled K-major rows at half width, so that
// widening byte k of a slice to fp16 lands at byte 2k of the operand.
// residual_tc_kernel: one CTA per (32 complex right-hand sides) x (128 rows)
// x (a range of K in chunks), 448 threads:
//   warp 0      : TMEM allocation (7 levels x 64 columns); bulk copies: per chunk the right-hand sides' digit block
//                 (bdigits_kernel, 56 KB, 2 stages) and the seven 8 KB digit
//                 slices of M (10-slice ring), whichever has a free slot
//   warp 1      : MMA issuer, A' from TMEM.  Per chunk and digit s of A', one MMA per
//                 16-wide K step covers the levels s .. 6 at once: the seven
//                 digit slices of B' are stacked along N, so the levels
//                 s + t, t = 0 .. 6 - s, are adjacent TMEM columns (N <= 256
//                 per MMA: 10 MMAs per K step instead of 28)
//   warps 2-9   : epilogue: thread = (row, half of the 64 real columns);
//                 level sums -> 64-bit accumulators in registers
//   warps 10-13 : converters: a staged byte slice -> the fp16 operand slice in
//                 TMEM (32 columns, two slices; thread = row; one byte permute
//                 and one fp16 subtract per digit pair)
// Measured, n = 12000 and 64 right-hand sides, one residual: 2.4 ms with A' in
// shared memory and descriptors made as the MMAs were issued (issue bound, 184
// clocks an MMA), 1.4 ms now; n = 3750, 900: 3.46 -> 2.2 ms.
// Bound by the tensor pipe (3584 clocks a chunk; the digits are exact in fp16
// alone) and, next, by shared memory: with A' there too, written once and read
// ten times per K step, 670 KB a chunk went through it, 5200 clocks at 128 bytes
// a clock; with A' in TMEM 360 KB.  Slices in the order 0, 6, 1, 5, ..: a
// conversion overlaps the products of the slice before, and a slice's products
// shrink with s.
// Every wait is bounded; a CTA whose wait runs out writes NaN outputs, sets
// MGT_ERR_TIMEOUT in the status word, drains what it issued and returns.
#include <cuda_fp16.h>

#include <algorithm>

#include "common.cuh"
#include "diag.cuh"
#include "gemm_tc.cuh"
#include "residual_tc.cuh"
#include "tcgen05.cuh"

namespace mgt {
namespace rtc {

constexpr int BM = 128;                 // rows of M per tile
constexpr int BNC = 32;                 // complex right-hand sides per tile
constexpr int BN = 2 * BNC;             // real columns per tile (TMEM columns per level)
constexpr int KCC = 32;                 // complex K per chunk (64 real: one 128-byte fp16 row)
constexpr int DIG = 7;                  // digits per operand
constexpr int ASLOTS = 2;               // fp16 operand slices in TMEM
constexpr int DSLOTS = 10;              // byte-slice staging ring
constexpr uint32_t A_COLS = 32;                     // TMEM columns of one fp16 digit slice of A' (64 real K)
constexpr uint32_t D_SLICE = BM * 64;               // 8 KB: a digit slice of A', one byte per digit
constexpr uint32_t B_SLICE = BN * 128;              // 8 KB
constexpr uint32_t B_BLOCK = DIG * B_SLICE;         // 56 KB: one chunk of B', all digit slices
constexpr uint32_t TMEM_COLS = 512;
constexpr int NEPI = 8, NCONV = 4;
constexpr int EPI0 = 2;                             // first epilogue warp
constexpr int THREADS = (EPI0 + NEPI + NCONV) * 32;
constexpr int EPI_COLS = BN / (NEPI / 4);           // real columns per epilogue thread
// at most 512 chunks (32768 real K) per CTA: |sum| <= 2^15 * 2^48 = 2^63
// units of 2^-48, less the rounding of levels 5 and 6
constexpr int MAX_SPLIT_CHUNKS = 512;
constexpr int READ_CHUNKS = 4;          // chunks between readouts of the levels
constexpr long long BIAS = 0x0080808080808080LL;    // 128 in each of the seven digit positions
constexpr int FIX = 54;                             // |X| < 2^FIX

// polls (of some 50 clocks) without progress after which the producer gives up
constexpr uint32_t kProducerLimit = 1u << 27;

// the digit slice of A' taken j-th in a chunk: 0, 6, 1, 5, 2, 4, 3
__host__ __device__ constexpr int slice_at(int j) { return j & 1 ? DIG - 1 - (j >> 1) : j >> 1; }

constexpr size_t smem_bytes() {
  return 1024 + DSLOTS * D_SLICE + 2 * B_BLOCK + BM * sizeof(int) + 256;
}

// round(f * 2^sh) as a 64-bit integer (|f| * 2^sh < 2^54 by the row scale);
// zero and subnormal f (below 2^-126) give 0
__device__ __forceinline__ long long fixed_point(float f, int sh) {
  const uint32_t u = __float_as_uint(f);
  const int ex = (int)((u >> 23) & 0xFFu);
  if (ex == 0) return 0;
  const uint32_t m = (u & 0x7FFFFFu) | 0x800000u;   // |f| = m * 2^(ex - 150)
  const int s = ex - 150 + sh;
  long long r;
  if (s >= 0) r = (long long)m << min(s, 39);
  else if (s > -32) r = (long long)((m + (1u << (-s - 1))) >> (-s));
  else r = 0;
  return (u >> 31) ? -r : r;
}

// round(f * 2^sh) for the low part of a double-float entry (|f| * 2^sh < 2^30):
// one exact power-of-two multiply and one conversion
__device__ __forceinline__ long long fixed_low(float f, int sh) {
  if (sh > 127 || sh < -126) return fixed_point(f, sh);
  return (long long)__float2int_rn(f * __int_as_float((127 + sh) << 23));
}

// Digit at position p (0 = lowest) of y = X + BIAS, as an exact float.
__device__ __forceinline__ float digit_f(long long y, int p) {
  const uint32_t lo = (uint32_t)y, hi = (uint32_t)((unsigned long long)y >> 32);
  const uint32_t w = p < 4 ? lo : hi;
  const uint32_t byte = (w >> (8 * (p & 3))) & 255u;
  return __int_as_float(0x4B400000 | (int)byte) - 12583040.0f;   // byte - 128
}

// Four biased digit bytes b0..b3 -> two fp16 pairs (b0 - 128, b1 - 128),
// (b2 - 128, b3 - 128): a byte permute places each byte under 0x64 (the fp16
// encoding of 1024 + byte), and 1152 is subtracted (exact).
__device__ __forceinline__ uint2 widen4(uint32_t x) {
  const uint32_t h0 = __byte_perm(x, 0x64646464u, 0x4140), h1 = __byte_perm(x, 0x64646464u, 0x4342);
  const __half2 c = __halves2half2(__ushort_as_half((unsigned short)0x6480), __ushort_as_half((unsigned short)0x6480));
  const __half2 d0 = __hsub2(*reinterpret_cast<const __half2*>(&h0), c);
  const __half2 d1 = __hsub2(*reinterpret_cast<const __half2*>(&h1), c);
  return make_uint2(*reinterpret_cast<const uint32_t*>(&d0), *reinterpret_cast<const uint32_t*>(&d1));
}

// exponent of a row of M, or a column of X, holding a NaN or an infinity: its outputs are NaN
constexpr int kNonFinite = 0x40000000;

__device__ __forceinline__ int clamp_exp(int e) { return (e < -1200 || e > 1200) ? 0 : e; }

// (re, im) of an entry as integers round(v 2^(FIX - e)), 2^e above the row's largest part
__device__ __forceinline__ void entry_fixed(float4 v, int e, long long& re, long long& im) {
  re = fixed_point(v.x, FIX - e) + fixed_low(v.y, FIX - e);
  im = fixed_point(v.z, FIX - e) + fixed_low(v.w, FIX - e);
}
__device__ __forceinline__ long long fixed_double(double v, int e) {
  const long long b = __double_as_longlong(v);
  const int ex = (int)((b >> 52) & 0x7ff);
  long long m = b & 0xFFFFFFFFFFFFFll;
  if (ex) m |= 1ll << 52;
  const int sh = min(max(ex, 1) - 1075 + FIX - e, 1);
  const long long r = sh >= 0 ? m << sh : sh > -54 ? (m + (1ll << (-sh - 1))) >> (-sh) : 0ll;
  return b < 0 ? -r : r;
}
__device__ __forceinline__ void entry_fixed(double2 v, int e, long long& re, long long& im) {
  re = fixed_double(v.x, e);
  im = fixed_double(v.y, e);
}
// size of an entry as an ordered integer: the bits of its larger high part, or exponent field
__device__ __forceinline__ uint32_t entry_size(float4 v) {
  return max(__float_as_uint(fabsf(v.x)), __float_as_uint(fabsf(v.z)));
}
__device__ __forceinline__ uint32_t entry_size(double2 v) {
  return (uint32_t)max((__double2hiint(v.x) >> 20) & 0x7ff, (__double2hiint(v.y) >> 20) & 0x7ff);
}
// e with 2^e above every entry of at most that size
__device__ __forceinline__ int size_exponent(uint32_t m, float4) {
  int e = 0;
  if (m >= 0x7F800000u) return kNonFinite;
  if (m != 0u) frexpf(__uint_as_float(m), &e);
  return e;
}
__device__ __forceinline__ int size_exponent(uint32_t m, double2) {
  return m == 2047u ? kNonFinite : (int)max(m, 1u) - 1022;
}
__device__ __forceinline__ float4 zero_of(float4) { return make_float4(0.f, 0.f, 0.f, 0.f); }
__device__ __forceinline__ double2 zero_of(double2) { return make_double2(0.0, 0.0); }

// Byte offset of real K index kr (even) of row rho in a 128-row tile whose rows
// are 128-byte lines (64 fp16), 8-row groups 1024 B apart, 16-byte chunks
// XOR-swizzled by the row within its group: the K-major 128B-swizzle layout.
__device__ __forceinline__ uint32_t swz(int rho, int kr) {
  return (uint32_t)rho * 128u + ((uint32_t)(((kr >> 3) ^ (rho & 7)) << 4)) + (uint32_t)((kr & 7) * 2);
}

__global__ void __launch_bounds__(THREADS, 1)
residual_tc_kernel(const unsigned char* __restrict__ D, int rows, const int* __restrict__ row_exp,
                   const int* __restrict__ col_exp, const unsigned char* __restrict__ bdig, int nch_total, int ncols,
                   int chunks_per_split, const double2* __restrict__ B, int64_t ldb, double2* __restrict__ R,
                   int64_t ldr, double2* __restrict__ partial, int* status) {
  using namespace tc;
  extern __shared__ __align__(1024) unsigned char smem_raw[];
  unsigned char* base = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
  unsigned char* bring = base;
  unsigned char* dring = bring + 2 * B_BLOCK;
  int* rexp = reinterpret_cast<int*>(dring + DSLOTS * D_SLICE);
  uint64_t* full_a = reinterpret_cast<uint64_t*>(rexp + BM);
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

  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int ct = blockIdx.x, rt = blockIdx.y, sp = blockIdx.z, row0 = rt * BM;
  const int c_begin = sp * chunks_per_split;
  const int nchunk = max(0, min(nch_total, c_begin + chunks_per_split) - c_begin);
  const int nread = (nchunk + READ_CHUNKS - 1) / READ_CHUNKS;

  if (threadIdx.x < BM) rexp[threadIdx.x] = (row0 + (int)threadIdx.x < rows) ? clamp_exp(row_exp[row0 + threadIdx.x]) : 0;
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

  if (warp == 0 && lane == 0) {
    // ---------------- producer: digit blocks of B', digit slices of A'.
    // Whichever copy has a free slot is issued (B blocks first), so a B
    // block goes out as soon as the MMAs of the block two back have completed
    // rather than behind the slices of the current chunk.
    const unsigned char* dsrc = D + ((size_t)rt * nch_total + c_begin) * DIG * D_SLICE;
    const int nq = nchunk * DIG;
    int ib = 0, q = 0;
    uint32_t idle = 0;
    while ((ib < nchunk || q < nq) && !*abort) {
      bool progress = false;
      if (ib < nchunk && (ib < 2 || mbar_test(&empty_b[ib & 1], ((ib >> 1) - 1) & 1))) {
        mbar_expect_tx(&full_b[ib & 1], B_BLOCK);
        bulk_load(bring + (ib & 1) * B_BLOCK, bdig + ((size_t)ct * nch_total + c_begin + ib) * B_BLOCK, B_BLOCK,
                  &full_b[ib & 1]);
        ++ib;
        progress = true;
      }
      if (q < nq && (q < DSLOTS || mbar_test(&empty_d[q % DSLOTS], ((q / DSLOTS) - 1) & 1))) {
        mbar_expect_tx(&full_d[q % DSLOTS], D_SLICE);
        bulk_load(dring + (q % DSLOTS) * D_SLICE, dsrc + (size_t)(q / DIG * DIG + slice_at(q % DIG)) * D_SLICE, D_SLICE,
                  &full_d[q % DSLOTS]);
        ++q;
        progress = true;
      }
      if (progress) idle = 0;
      else if (++idle >= kProducerLimit) { *abort = 1; break; }
    }
    // copies in flight land before the CTA may exit
    for (int j = max(0, ib - 2); j < ib; ++j) mbar_wait_plain(&full_b[j & 1], (j >> 1) & 1);
    for (int j = max(0, q - DSLOTS); j < q; ++j) mbar_wait_plain(&full_d[j % DSLOTS], (j / DSLOTS) & 1);
  } else if (warp == 1 && lane == 0) {
    // ---------------- MMA issuer
    int q = 0;
    bool ok = true;
    const uint32_t atm = tmem + (uint32_t)(DIG * BN);
    for (int i = 0; i < nchunk && ok; ++i) {
      const bool first = i % READ_CHUNKS == 0;
      if (first && i > 0) {
        if (!mbar_wait(tempty, (i / READ_CHUNKS - 1) & 1, abort)) { ok = false; break; }
        tc_fence_after();
      }
      const int st = i & 1;
      if (!mbar_wait(&full_b[st], (i >> 1) & 1, abort)) { ok = false; break; }
      tc_fence_after();
      const uint64_t bb = kmajor_sw128_desc(smem_u32(bring + st * B_BLOCK));
#pragma unroll
      for (int j = 0; j < DIG; ++j, ++q) {
        if (!ok) continue;
        const int s = slice_at(j), slot = q & 1;
        if (!mbar_wait(&full_a[slot], (q / ASLOTS) & 1, abort)) { ok = false; continue; }
        tc_fence_after();
        const uint32_t ad = atm + (uint32_t)slot * A_COLS;
        // the K steps innermost: 3600 clocks a chunk, against 4500 with the two
        // ranges of levels innermost (the accumulator changes less often)
#pragma unroll
        for (int t0 = 0; t0 < DIG - s; t0 += 4) {
          const int nt = DIG - s - t0 < 4 ? DIG - s - t0 : 4;
#pragma unroll
          for (int ks = 0; ks < 4; ++ks)
            mma_f16_ta(tmem + (uint32_t)((s + t0) * BN), ad + (uint32_t)(8 * ks),
                       bb + (uint64_t)(t0 * (B_SLICE >> 4) + 2 * ks), idesc_f16_m128(nt * BN),
                       first && j == 0 && ks == 0 ? 0u : 1u);
        }
        mma_commit(&empty_a[slot]);
      }
      if (!ok) break;
      mma_commit(&empty_b[st]);
      if (i % READ_CHUNKS == READ_CHUNKS - 1 || i == nchunk - 1) mma_commit(tfull);
    }
    mma_commit(done);   // arrives once every MMA issued above has completed
  } else if (warp >= EPI0 && warp < EPI0 + NEPI) {
    // ---------------- epilogue: thread = (row, half of the real columns)
    // a warp reads the TMEM lanes of its rank modulo 4
    const int qd = warp & 3, part = (warp - EPI0) >> 2, r = qd * 32 + lane;
    long long acc[EPI_COLS];
#pragma unroll
    for (int j = 0; j < EPI_COLS; ++j) acc[j] = 0;
    const uint32_t tbase = tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(part * EPI_COLS);
    bool ok = true;
    for (int ro = 0; ro < nread; ++ro) {
      if (!__all_sync(0xffffffffu, mbar_wait(tfull, ro & 1, abort))) { ok = false; break; }
      tc_fence_after();
      // a fresh copy per readout keeps the 28 TMEM addresses from being
      // hoisted out of the loop into registers
      uint32_t tb;
      asm volatile("mov.b32 %0, %1;" : "=r"(tb) : "r"(tbase));
#pragma unroll
      for (int p = 0; p < EPI_COLS / 4; ++p) {
        uint32_t v[DIG][4];
#pragma unroll
        for (int l = 0; l < DIG; ++l) tmem_ld4(tb + (uint32_t)(l * BN + p * 4), v[l]);
        tmem_wait_ld();
        if (p == EPI_COLS / 4 - 1) {
          tc_fence_before();
          __syncwarp();
          if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(tempty)) : "memory");
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) {
          // level l weighs 2^(36 - 8 l) units of 2^-48.  With |L_0| <= 2^20,
          // |L_1| <= 2^22 (top digits at most 64), L_0 2^8 + L_1 is exact in 32
          // bits; levels 5 and 6 round to the nearest unit through one FMA
          // ((L_5 + L_6 / 256) / 16, its own rounding below 1/16 unit)
          const int hi = (__float2int_rz(__uint_as_float(v[0][j])) << 8) + __float2int_rz(__uint_as_float(v[1][j]));
          const int l4 = __float2int_rz(__uint_as_float(v[4][j]));
          const int l56 = __float2int_rn(
              0.0625f * fmaf(__uint_as_float(v[6][j]), 0.00390625f, __uint_as_float(v[5][j])));
          acc[p * 4 + j] += (long long)hi * (1 << 28) + (long long)__float2int_rz(__uint_as_float(v[2][j])) * (1 << 20) +
                            (long long)__float2int_rz(__uint_as_float(v[3][j])) * (1 << 12) +
                            (long long)((l4 << 4) + l56);
        }
      }
    }
    const int row = row0 + r;
    if (row < rows) {
      const bool good = ok && !*abort && row_exp[row] != kNonFinite;
      const int ea = rexp[r];
#pragma unroll
      for (int jc = 0; jc < EPI_COLS / 2; ++jc) {
        const int col = ct * BNC + part * (EPI_COLS / 2) + jc;
        if (col < ncols) {
          double2 val;
          if (good && col_exp[col] != kNonFinite) {
            const int e = ea + clamp_exp(col_exp[col]) - 48;
            val = make_double2((double)acc[2 * jc], (double)acc[2 * jc + 1]);
            if (e > -900 && e < 900) {
              const double sc = __longlong_as_double((long long)(e + 1023) << 52);
              val.x *= sc;
              val.y *= sc;
            } else {
              val.x = ldexp(val.x, e);
              val.y = ldexp(val.y, e);
            }
          } else {
            val = make_double2(__longlong_as_double(0x7FF8000000000000LL),
                               __longlong_as_double(0x7FF8000000000000LL));
          }
          if (partial) {
            partial[((int64_t)sp * rows + row) * ncols + col] = val;
          } else {
            const double2 b = B ? B[(int64_t)row * ldb + col] : make_double2(0.0, 0.0);
            R[(int64_t)row * ldr + col] = make_double2(b.x - val.x, b.y - val.y);
          }
        }
      }
    }
  } else if (warp >= EPI0 + NEPI) {
    // ---------------- converters: staged byte slice -> fp16 operand slice; thread = row
    const int qd = warp & 3, row = qd * 32 + lane;
    const uint32_t abase = tmem + ((uint32_t)(qd * 32) << 16) + (uint32_t)(DIG * BN);
    const int nq = nchunk * DIG;
    // the row's 64 digits, 16 bytes at a time: halves of two of the operand's swizzled 16-byte chunks
    uint4 raw[4];
    auto fetch = [&](int q) -> bool {
      const int ds = q % DSLOTS;
      if (!mbar_wait(&full_d[ds], (q / DSLOTS) & 1, abort)) return false;
      const unsigned char* src = dring + ds * D_SLICE + row * 64;
#pragma unroll
      for (int c = 0; c < 4; ++c) raw[c] = *reinterpret_cast<const uint4*>(src + ((c ^ ((row >> 1) & 3)) << 4));
      return true;
    };
    bool ok = nq > 0 && fetch(0);
    // (a warp leaves as one: its lanes wait for each other below)
    for (int q = 0; q < nq && __all_sync(0xffffffffu, ok); ++q) {
      uint32_t w[32];
#pragma unroll
      for (int c = 0; c < 4; ++c) {
        const bool odd = row & 1;   // the swizzle swaps the two halves of odd rows
        const uint2 w0 = widen4(odd ? raw[c].z : raw[c].x), w1 = widen4(odd ? raw[c].w : raw[c].y);
        const uint2 w2 = widen4(odd ? raw[c].x : raw[c].z), w3 = widen4(odd ? raw[c].y : raw[c].w);
        w[8 * c] = w0.x;
        w[8 * c + 1] = w0.y;
        w[8 * c + 2] = w1.x;
        w[8 * c + 3] = w1.y;
        w[8 * c + 4] = w2.x;
        w[8 * c + 5] = w2.y;
        w[8 * c + 6] = w3.x;
        w[8 * c + 7] = w3.y;
      }
      __syncwarp();
      if (lane == 0)
        asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&empty_d[q % DSLOTS])) : "memory");
      if (q + 1 < nq) ok = fetch(q + 1);   // on its way while this slice waits for its place
      const int as = q % ASLOTS;
      if (q >= ASLOTS) {
        if (!__all_sync(0xffffffffu, mbar_wait(&empty_a[as], ((q / ASLOTS) - 1) & 1, abort))) break;
        tc_fence_after();
      }
      tmem_st16(abase + (uint32_t)as * A_COLS, w);
      tmem_st16(abase + (uint32_t)as * A_COLS + 16, w + 16);
      tmem_wait_st();
      tc_fence_before();
      __syncwarp();
      if (lane == 0) asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(&full_a[as])) : "memory");
    }
  }
  tc_fence_before();
  __syncthreads();
  if (threadIdx.x == 0 && *abort) atomicExch(status, MGT_ERR_TIMEOUT);
  if (warp == 0) {
    // every issued MMA has completed before the accumulator columns are freed
    if (lane == 0) mbar_wait_plain(done, 0);
    __syncwarp();
    tc_fence_after();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(TMEM_COLS) : "memory");
  }
}

// e_i of each row: 2^e_i bounds the row's largest |re|, |im|; one warp per
// row.  Rows with a NaN or an infinity get kNonFinite.  V: float4 (double-float)
// or double2 (complex128).
template <typename V>
__global__ void rowexp_kernel(const V* __restrict__ M, int64_t ldm, int rows, int kdim, int* __restrict__ out) {
  const int row = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5), lane = threadIdx.x & 31;
  if (row >= rows) return;
  uint32_t m = 0;
  for (int k = lane; k < kdim; k += 32) m = max(m, entry_size(__ldg(&M[(int64_t)row * ldm + k])));
  m = __reduce_max_sync(0xffffffffu, m);
  if (lane == 0) out[row] = size_exponent(m, V());
}

// Byte p (0 = lowest) of each of four 64-bit words, packed low to high.
__device__ __forceinline__ uint32_t pick_bytes(const long long* y, int p) {
  const int b = p & 3;
  uint32_t w[4];
#pragma unroll
  for (int k = 0; k < 4; ++k) w[k] = p < 4 ? (uint32_t)y[k] : (uint32_t)((unsigned long long)y[k] >> 32);
  const uint32_t sel = (uint32_t)(b | ((4 + b) << 4));
  return __byte_perm(__byte_perm(w[0], w[1], sel), __byte_perm(w[2], w[3], sel), 0x5410);
}

// Digits of M (the A' operand) for every (row tile, chunk): block
// (rt, c) holds slices s = 0 .. 6 (digit p = 6 - s), 8 KB each, byte
// (rho, kr) of a slice at rho * 64 + (((kr >> 3) ^ (rho & 7)) << 3) + (kr & 7):
// the swizzled fp16 operand layout at half width.  Zeros beyond rows and kdim.
// Thread = (row, 8 real K = 4 complex entries), four per thread.
template <typename V>
__global__ void __launch_bounds__(256)
digitize_kernel(const V* __restrict__ M, int64_t ldm, int rows, int kdim, const int* __restrict__ row_exp,
                unsigned char* __restrict__ D, int nch) {
  const int c = blockIdx.x, rt = blockIdx.y;
  unsigned char* blk = D + ((size_t)rt * nch + c) * DIG * D_SLICE;
#pragma unroll 1
  for (int t = threadIdx.x; t < BM * 8; t += 256) {
    const int rho = t >> 3, grp = t & 7, row = rt * BM + rho;
    const bool rin = row < rows;
    const int ex = rin ? clamp_exp(row_exp[row]) : 0;
    long long y[8];
#pragma unroll
    for (int e = 0; e < 4; ++e) {
      const int kc = c * KCC + grp * 4 + e;
      const V v = (rin && kc < kdim) ? __ldg(&M[(int64_t)row * ldm + kc]) : zero_of(V());
      entry_fixed(v, ex, y[2 * e], y[2 * e + 1]);
      y[2 * e] += BIAS;
      y[2 * e + 1] += BIAS;
    }
    const uint32_t off = (uint32_t)rho * 64u + ((uint32_t)(grp ^ (rho & 7)) << 3);
#pragma unroll
    for (int s = 0; s < DIG; ++s) {
      const int p = DIG - 1 - s;
      *reinterpret_cast<uint2*>(blk + s * D_SLICE + off) = make_uint2(pick_bytes(y, p), pick_bytes(y + 4, p));
    }
  }
}

// f_j of each right-hand side: 2^f_j bounds the column's largest |re|, |im|.
// Block (32 columns x 8 row lanes) over a range of rows; atomicMax per column
// (the output starts at a large negative value).
__global__ void colexp_kernel(const double2* __restrict__ X, int64_t ldx, int kdim, int ncols, int* __restrict__ out) {
  const int j = blockIdx.x * 32 + (threadIdx.x & 31), ty = threadIdx.x >> 5;
  __shared__ uint32_t red[8][32];
  uint32_t m = 0;      // largest exponent field (no FP64 comparisons: their pipe is slow)
  bool any = false;
  if (j < ncols)
    for (int k = blockIdx.y * 8 + ty; k < kdim; k += gridDim.y * 8) {
      const double2 x = X[(int64_t)k * ldx + j];
      any |= ((__double_as_longlong(x.x) | __double_as_longlong(x.y)) << 1) != 0;
      m = max(m, entry_size(x));
    }
  red[ty][threadIdx.x & 31] = m | (any ? 0x8000u : 0u);
  __syncthreads();
  if (ty == 0 && j < ncols) {
    uint32_t a = any ? 0x8000u : 0u;
    for (int t = 1; t < 8; ++t) {
      m = max(m, red[t][threadIdx.x & 31] & 0x7fffu);
      a |= red[t][threadIdx.x & 31] & 0x8000u;
    }
    if (a) atomicMax(&out[j], size_exponent(m, double2()));
  }
}

// Digit blocks of B'^T: block (column tile ct, chunk c) holds the seven digit
// slices (top digit first) of its 64 rows x 64 real K, each slice in the
// swizzled layout the MMA reads; zeros beyond kdim and ncols.  One thread per
// (complex K index, complex column).
__global__ void bdigits_kernel(const double2* __restrict__ X, int64_t ldx, int kdim, int ncols,
                               const int* __restrict__ col_exp, unsigned char* __restrict__ out, int nch, int ctiles) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  const int cols = ctiles * BNC;
  if (idx >= (int64_t)nch * KCC * cols) return;
  const int j = (int)(idx % cols), k = (int)(idx / cols);
  double2 x = make_double2(0.0, 0.0);
  int e = 0;
  if (j < ncols) {
    e = clamp_exp(col_exp[j]);
    if (k < kdim) x = X[(int64_t)k * ldx + j];
  }
  const long long xr = fixed_double(x.x, e), xi = fixed_double(x.y, e);
  const long long yr = xr + BIAS, yi = xi + BIAS, yn = BIAS - xi;
  const int ctile = j / BNC, jj = j % BNC, c = k / KCC, kk = k % KCC;
  unsigned char* blk = out + ((size_t)ctile * nch + c) * B_BLOCK;
#pragma unroll
  for (int s = 0; s < DIG; ++s) {
    const int p = DIG - 1 - s;
    const int rho = s * BN + 2 * jj;
    // row 2jj (real part): Xr, -Xi; row 2jj + 1 (imaginary part): Xi, Xr
    *reinterpret_cast<__half2*>(blk + swz(rho, 2 * kk)) = __floats2half2_rn(digit_f(yr, p), digit_f(yn, p));
    *reinterpret_cast<__half2*>(blk + swz(rho + 1, 2 * kk)) = __floats2half2_rn(digit_f(yi, p), digit_f(yr, p));
  }
}

// R = B - sum of the split-K partials (FP64); partial is [split][row][col]
__global__ void tc_reduce_kernel(const double2* __restrict__ partial, int splits, int rows, int ncols,
                                 const double2* __restrict__ B, int64_t ldb, double2* __restrict__ R, int64_t ldr) {
  const int64_t idx = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
  if (idx >= (int64_t)rows * ncols) return;
  const int r = (int)(idx / ncols), c = (int)(idx - (int64_t)r * ncols);
  double2 acc = B ? B[(int64_t)r * ldb + c] : make_double2(0.0, 0.0);
  for (int q = 0; q < splits; ++q) {
    const double2 v = partial[(int64_t)q * rows * ncols + idx];
    acc.x -= v.x;
    acc.y -= v.y;
  }
  R[(int64_t)r * ldr + c] = acc;
}

// Split of the K range, an even number of chunks each, at least 8, at most 16
// splits and MAX_SPLIT_CHUNKS chunks: the one with the shortest estimate, in
// chunks of 3.4 us -- rounds of CTAs (one an SM) times a CTA's chunks and 2 more
// for its start and end, and the split sums written and read once at 6.7 TB/s.
// Against four rounds whatever their fill, 64 columns: n = 2000 116 -> 91 us a
// residual, 3750 237 -> 216, 6000 512 -> 470; 33 columns, 21000 5.19 -> 4.66 ms.
static void plan_splits(int rows, int kdim, int ncols, int* splits, int* cps) {
  const int nch = (kdim + KCC - 1) / KCC;
  const int ctiles = (ncols + BNC - 1) / BNC;   // the choice depends on whole column tiles only
  const int64_t tiles = (int64_t)((rows + BM - 1) / BM) * ctiles;
  const int sms = device_sm_count();
  const int lo = (nch + MAX_SPLIT_CHUNKS - 1) / MAX_SPLIT_CHUNKS, hi = std::max(lo, std::min(16, nch / 8));
  double best = 0.0;
  for (int sp = lo; sp <= hi; ++sp) {
    int c = (nch + sp - 1) / sp;
    if ((c & 1) && c < nch) ++c;
    const int n = (nch + c - 1) / c;
    const double rounds = (double)((tiles * n + sms - 1) / sms);
    const double cost = rounds * (c + 2) + (n > 1 ? 1.4e-6 * n * (double)rows * (ctiles * BNC) : 0.0);
    if (sp == lo || cost < best) {
      best = cost;
      *cps = c;
      *splits = n;
    }
  }
}

// workspace of one application (the digits of M are the caller's)
struct TcResWs {
  int* status;
  int* colexp;
  unsigned char* bdig;
  double2* partial;
  int splits, cps, nch, ctiles;
  size_t total;
  TcResWs(void* base, int rows, int kdim, int ncols) {
    char* b = (char*)base;
    size_t off = 0;
    auto take = [&](size_t bytes, size_t align) {
      off = (off + align - 1) / align * align;
      char* p = b ? b + off : nullptr;
      off += bytes;
      return p;
    };
    plan_splits(rows, kdim, ncols, &splits, &cps);
    nch = (kdim + KCC - 1) / KCC;
    ctiles = (ncols + BNC - 1) / BNC;
    status = (int*)take(256, 256);
    colexp = (int*)take((size_t)ncols * sizeof(int), 256);
    bdig = (unsigned char*)take((size_t)ctiles * nch * B_BLOCK, 1024);
    // room for as many columns or fewer (fewer may take more splits)
    size_t sums = 0;
    for (int c = BNC; c < ncols + BNC; c += BNC) {
      int sp, per;
      plan_splits(rows, kdim, std::min(c, ncols), &sp, &per);
      if (sp > 1) sums = std::max(sums, (size_t)sp * rows * std::min(c, ncols));
    }
    char* p = take(sums * sizeof(double2), 256);
    partial = splits > 1 ? (double2*)p : nullptr;
    total = off + 256;
  }
};

static size_t align_up(size_t v, size_t a) { return (v + a - 1) / a * a; }

}  // namespace rtc

bool residual_tc_supported(int64_t rows, int64_t kdim, int64_t ncols) {
  return tc_available() && rows > 0 && kdim > 0 && ncols > 0 && rows <= (1 << 24) && kdim <= (1 << 22) &&
         ncols <= (1 << 16);
}

size_t residual_tc_digits_bytes(int64_t rows, int64_t kdim) {
  using namespace rtc;
  return (size_t)((rows + BM - 1) / BM) * (size_t)((kdim + KCC - 1) / KCC) * DIG * D_SLICE;
}

size_t residual_tc_apply_bytes(int64_t rows, int64_t kdim, int64_t ncols) {
  if (!residual_tc_supported(rows, kdim, ncols)) return 0;
  return rtc::TcResWs(nullptr, (int)rows, (int)kdim, (int)ncols).total;
}

size_t residual_tc_workspace_bytes(int64_t rows, int64_t kdim, int64_t ncols) {
  using namespace rtc;
  if (!residual_tc_supported(rows, kdim, ncols)) return 0;
  return align_up((size_t)rows * sizeof(int), 1024) + align_up(residual_tc_digits_bytes(rows, kdim), 1024) +
         residual_tc_apply_bytes(rows, kdim, ncols);
}

template <typename V>
int residual_tc_prepare(const V* M, int64_t ldm, int rows, int kdim, int* rowexp, unsigned char* digits,
                        cudaStream_t s) {
  using namespace rtc;
  if (!residual_tc_supported(rows, kdim, 1)) return MGT_ERR_UNSUPPORTED;
  if (!M || !rowexp || !digits || ((uintptr_t)digits & 15)) return MGT_ERR_ARG;
  const int nch = (kdim + KCC - 1) / KCC;
  count_launch(2);
  rowexp_kernel<V><<<(rows + 7) / 8, 256, 0, s>>>(M, ldm, rows, kdim, rowexp);
  digitize_kernel<V><<<dim3(nch, (rows + BM - 1) / BM), 256, 0, s>>>(M, ldm, rows, kdim, rowexp, digits, nch);
  return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_ERR_CUDA;
}
template int residual_tc_prepare(const float4*, int64_t, int, int, int*, unsigned char*, cudaStream_t);
template int residual_tc_prepare(const double2*, int64_t, int, int, int*, unsigned char*, cudaStream_t);

int residual_tc_apply(const unsigned char* digits, const int* rowexp, int rows, int kdim, const double2* X,
                      int64_t ldx, int ncols, const double2* B, int64_t ldb, double2* R, int64_t ldr, void* work,
                      size_t work_bytes, cudaStream_t s) {
  using namespace rtc;
  if (!residual_tc_supported(rows, kdim, ncols)) return MGT_ERR_UNSUPPORTED;
  if (!digits || !rowexp || ((uintptr_t)digits & 15)) return MGT_ERR_ARG;
  TcResWs w(work, rows, kdim, ncols);
  if (!work || work_bytes < w.total) return MGT_ERR_WORKSPACE;
  static OncePerDevice once;
  once([] {
    cudaFuncSetAttribute(residual_tc_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem_bytes());
  });
  if (cudaMemsetAsync(w.status, 0, sizeof(int), s) != cudaSuccess) return MGT_ERR_CUDA;
  // column exponents start far below any real one (0x80808080)
  if (cudaMemsetAsync(w.colexp, 0x80, (size_t)ncols * sizeof(int), s) != cudaSuccess) return MGT_ERR_CUDA;
  count_launch(2);
  colexp_kernel<<<dim3((ncols + 31) / 32, std::min(64, (kdim + 7) / 8)), 256, 0, s>>>(X, ldx, kdim, ncols, w.colexp);
  const int64_t nb = (int64_t)w.nch * KCC * w.ctiles * BNC;
  bdigits_kernel<<<(unsigned)((nb + 255) / 256), 256, 0, s>>>(X, ldx, kdim, ncols, w.colexp, w.bdig, w.nch, w.ctiles);
  count_launch();
  // column tiles of one row tile are neighbours in the launch order, so the
  // second reads the row tile's digit slices from L2
  dim3 grid(w.ctiles, (rows + BM - 1) / BM, w.splits);
  residual_tc_kernel<<<grid, THREADS, smem_bytes(), s>>>(digits, rows, rowexp, w.colexp, w.bdig, w.nch, ncols,
                                                           w.cps, B, ldb, R, ldr, w.partial, w.status);
  if (w.splits > 1) {
    const int64_t tot = (int64_t)rows * ncols;
    count_launch();
    tc_reduce_kernel<<<(unsigned)((tot + 255) / 256), 256, 0, s>>>(w.partial, w.splits, rows, ncols, B, ldb, R, ldr);
  }
  return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_ERR_CUDA;
}

size_t residual_tc_split(void* work, int64_t rows, int64_t kdim, int** rowexp, unsigned char** digits, char** aw) {
  using namespace rtc;
  char* b = (char*)work;
  const size_t d_off = align_up((size_t)rows * sizeof(int), 1024);
  const size_t a_off = d_off + align_up(residual_tc_digits_bytes(rows, kdim), 1024);
  if (rowexp) *rowexp = (int*)b;
  if (digits) *digits = (unsigned char*)(b + d_off);
  if (aw) *aw = b + a_off;
  return a_off;
}

template <typename V>
int residual_tc(const V* M, int64_t ldm, int rows, int kdim, const double2* X, int64_t ldx, int ncols,
                const double2* B, int64_t ldb, double2* R, int64_t ldr, void* work, size_t work_bytes,
                cudaStream_t s) {
  if (!residual_tc_supported(rows, kdim, ncols)) return MGT_ERR_UNSUPPORTED;
  if (!work || work_bytes < residual_tc_workspace_bytes(rows, kdim, ncols)) return MGT_ERR_WORKSPACE;
  int* rowexp;
  unsigned char* digits;
  char* aw;
  const size_t a_off = residual_tc_split(work, rows, kdim, &rowexp, &digits, &aw);
  int e = residual_tc_prepare(M, ldm, rows, kdim, rowexp, digits, s);
  if (e != MGT_OK) return e;
  return residual_tc_apply(digits, rowexp, rows, kdim, X, ldx, ncols, B, ldb, R, ldr, aw, work_bytes - a_off, s);
}
template int residual_tc(const float4*, int64_t, int, int, const double2*, int64_t, int, const double2*, int64_t, double2*,
                         int64_t, void*, size_t, cudaStream_t);
template int residual_tc(const double2*, int64_t, int, int, const double2*, int64_t, int, const double2*, int64_t,
                         double2*, int64_t, void*, size_t, cudaStream_t);


}  // namespace mgt
