// tcgen05 (TF32x3) complex trailing update for the complex64 LU.
#pragma once
#include <cuda.h>
#include <cuda_fp16.h>

#include "common.cuh"

namespace mgt {

// Split operand buffers and their TMA descriptors, built once per
// factorisation for matrices of order <= nmax.
struct TcPlan {
  void* Ahi = nullptr;     // fp32 (TF32x3) or fp16 (F16x2) split operands
  void* Alo = nullptr;
  void* Bhi = nullptr;
  void* Blo = nullptr;
  float* invA = nullptr;   // F16x2: inverse row scales of A, inverse column scales of B
  float* invB = nullptr;
  int mode = 0;            // MGT_TC_TF32X3 or MGT_TC_F16X2, fixed when the plan is built
  int64_t nmax = 0;
  CUtensorMap mAhi, mAlo, mBhi, mBlo;
  int init(void* scratch, int64_t nmax);
};

size_t tc_scratch_bytes(int64_t n);
// split-product scheme of the tensor-core update (MGT_TC_TF32X3 / MGT_TC_F16X2)
int tc_set_mode(int mode);
int tc_get_mode();
bool tc_available();

// TMA map of a complex64 matrix C (rows x cols, leading dimension ldc even,
// 16-byte aligned base) viewed as fp32 (rows x 2 cols), 128 x 32 boxes.
int tc_make_cmap(CUtensorMap* map, float2* C, int64_t rows, int64_t cols, int64_t ldc);

// C -= A (M x K) * B (K x N), K <= 256, where C is the M x N block of the
// matrix described by cmap starting at fp32 column cx0 (= 2 * complex
// column) and row cy0; the block must extend to the matrix's last row and
// column (TMA stores are clipped there).  max_ctas <= 0: one CTA per SM.
int gemm_sub_tc(const TcPlan& plan, const CUtensorMap& cmap, int M, int N, int K, const float2* A, int64_t lda,
                const float2* B, int64_t ldb, int cx0, int cy0, int* status, cudaStream_t s, int max_ctas = 0);

// The same in its three steps: operand splits into the plan's buffers, then
// the tcgen05 kernel, which reads only the split buffers and the C block.
int tc_split_a(const TcPlan& plan, int M, int K, const float2* A, int64_t lda, cudaStream_t s);
int tc_split_b(const TcPlan& plan, int N, int K, const float2* B, int64_t ldb, cudaStream_t s);
// The F16x2 splits of K = 128 operands, for kernels that have the operands at hand:
// the plan's buffers (row stride `stride` halves) and inverse scales.
struct TcSplitOut {
  __half *ahi, *alo, *bhi, *blo;
  float *inva, *invb;
  int stride;
};
TcSplitOut tc_split_out(const TcPlan& plan);

// power-of-two exponent e with max 2^-e in [0.5, 1) (0 for zero or non-finite maxima); bits of max given
__device__ __forceinline__ int tc_scale_exp(unsigned mx) {
  int e = 0;
  if (mx != 0u && mx < 0x7F800000u) {
    frexpf(__uint_as_float(mx), &e);
    e = max(-120, min(120, e));
  }
  return e;
}
__device__ __forceinline__ void tc_split2(float x, __half& h, __half& l) {
  h = __float2half_rn(x);
  l = __float2half_rn(x - __half2float(h));
}
// row i of A: 128 complex values at a, by one warp
__device__ __forceinline__ void tc_split_row(const TcSplitOut& o, const float2* a, int i, int lane) {
  float2 v[4];
  unsigned mx = 0;
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    v[j] = a[lane + 32 * j];
    mx = max(mx, max(__float_as_uint(fabsf(v[j].x)), __float_as_uint(fabsf(v[j].y))));
  }
  const int e = tc_scale_exp(__reduce_max_sync(0xffffffffu, mx));
  const float sc = ldexpf(1.f, -e);
#pragma unroll
  for (int j = 0; j < 4; ++j) {
    __half2 h, l;
    tc_split2(v[j].x * sc, h.x, l.x);
    tc_split2(v[j].y * sc, h.y, l.y);
    const int64_t at = (int64_t)i * o.stride + 2 * (lane + 32 * j);
    *reinterpret_cast<__half2*>(o.ahi + at) = h;
    *reinterpret_cast<__half2*>(o.alo + at) = l;
  }
  if (lane == 0) o.inva[i] = ldexpf(1.f, e);
}
// columns col0, col0 + 1, ... of B, 128 complex values each at U[k * ld + c]: QN consecutive threads per column
template <int QN>
__device__ __forceinline__ void tc_split_cols(const TcSplitOut& o, const float2* U, int ld, int col0, int tid) {
  const int c = tid / QN, q = tid % QN;
  unsigned mx = 0;
#pragma unroll 8
  for (int k = q; k < 128; k += QN) {
    const float2 u = U[k * ld + c];
    mx = max(mx, max(__float_as_uint(fabsf(u.x)), __float_as_uint(fabsf(u.y))));
  }
#pragma unroll
  for (int off = QN / 2; off; off >>= 1) mx = max(mx, __shfl_xor_sync(0xffffffffu, mx, off));
  const int e = tc_scale_exp(mx);
  const float sc = ldexpf(1.f, -e);
  const int64_t row = (int64_t)2 * (col0 + c) * o.stride;
#pragma unroll 4
  for (int k = q; k < 128; k += QN) {
    const float2 u = U[k * ld + c];
    __half rh, rl, ih, il;
    tc_split2(u.x * sc, rh, rl);
    tc_split2(u.y * sc, ih, il);
    // row 2j: Br, -Bi; row 2j + 1: Bi, Br
    *reinterpret_cast<__half2*>(o.bhi + row + 2 * k) = __halves2half2(rh, __hneg(ih));
    *reinterpret_cast<__half2*>(o.blo + row + 2 * k) = __halves2half2(rl, __hneg(il));
    *reinterpret_cast<__half2*>(o.bhi + row + o.stride + 2 * k) = __halves2half2(ih, rh);
    *reinterpret_cast<__half2*>(o.blo + row + o.stride + 2 * k) = __halves2half2(il, rl);
  }
  if (q == 0) o.invb[col0 + c] = ldexpf(1.f, e);
}

// bcol: the first column of B (within the split) this launch uses.  early: the
// launch before it in the stream, nothing between, is one that ends the operands
// and calls early_start.
int tc_gemm(const TcPlan& plan, const CUtensorMap& cmap, int M, int N, int K, int cx0, int cy0, int* status,
            cudaStream_t s, int max_ctas = 0, int bcol = 0, bool early = false);

// The 128 x 128 tiles on and above the diagonal of the M x M block of C at row
// and column c0 (it ends at the matrix's last row and column); the operands
// from row / column off of the splits on.  Tiles tbegin .. tend (of
// tc_upper_tiles(M), row by row).
int tc_upper_tiles(int M);
int tc_gemm_upper(const TcPlan& plan, const CUtensorMap& cmap, int M, int K, int c0, int off, int tbegin, int tend,
                  int* status, cudaStream_t s, int max_ctas = 0);

}  // namespace mgt
