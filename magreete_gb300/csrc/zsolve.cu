// Triangular solves of the complex128 LU for several right-hand sides:
// X = U^-1 L^-1 X in place, block rows of 64.
//
// Per block row i: X_i = Inv_i X_i (the block's inverted diagonal, FP64), then
// every remaining row takes X_r -= F_(r, i) X_i as one tensor-core product of
// FP64 accuracy (zgemm_tc.cu).  Three launches per block row: the diagonal
// product (which also records the sizes of its rows, for the scaling of the
// product's K: ZRows), the digits of the factor's block column and of X_i, and the
// product.  The chain of block rows is what bounds a solve of few columns:
// about 23 us per block row, where block-to-block flags with FP64 products of
// 64 x 64 blocks (19 clocks per FP64 warp instruction and SM) took 130 us.
#include <algorithm>

#include "common.cuh"
#include "diag.cuh"
#include "zgemm_tc.cuh"

namespace mgt {
namespace zs {

constexpr int TB = 64;
constexpr int LD = TB + 1;

// Inverse of every 64 x 64 diagonal block of both factors, one column per
// warp, lane = rows lane and lane + 32: blocks (block row, 8-column group,
// 0: unit lower, 1: upper).  The lower inverses come first in Inv.
__global__ void __launch_bounds__(256)
inverse_kernel(const double2* __restrict__ F, int64_t ldf, int n, double2* __restrict__ Inv) {
  extern __shared__ __align__(16) unsigned char zs_smem[];
  double2* T = reinterpret_cast<double2*>(zs_smem);
  __shared__ double2 dinv[TB];
  const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, i = blockIdx.x;
  const bool upper = blockIdx.z != 0;
  const int r0 = i * TB, rb = min(TB, n - r0), col = blockIdx.y * 8 + warp;
  for (int e = tid; e < TB * TB; e += 256) {
    const int r = e / TB, c = e % TB;
    const bool ok = r < rb && c < rb;
    cp_async_elem<16>(T + r * LD + c, ok ? F + (int64_t)(r0 + r) * ldf + r0 + c : F, ok);
  }
  cp_async_commit();
  cp_async_wait<0>();
  __syncthreads();
  if (upper && tid < TB) dinv[tid] = tid < rb ? crecip(T[tid * LD + tid]) : make_double2(0.0, 0.0);
  __syncthreads();
  double2 x0 = make_double2(lane == col ? 1.0 : 0.0, 0.0), x1 = make_double2(lane + 32 == col ? 1.0 : 0.0, 0.0);
  if (col >= rb) x0.x = x1.x = 0.0;
  if (!upper) {
    for (int k = col; k < rb - 1; ++k) {
      const double2 s = k < 32 ? x0 : x1;
      double2 xk;
      xk.x = __shfl_sync(0xffffffffu, s.x, k & 31);
      xk.y = __shfl_sync(0xffffffffu, s.y, k & 31);
      if (k < 31 && lane > k) cfms(x0, T[lane * LD + k], xk);
      if (lane + 32 > k) cfms(x1, T[(lane + 32) * LD + k], xk);
    }
  } else if (col < rb) {
    for (int k = col; k >= 0; --k) {
      double2 s = k < 32 ? x0 : x1;
      double2 xk;
      xk.x = __shfl_sync(0xffffffffu, s.x, k & 31);
      xk.y = __shfl_sync(0xffffffffu, s.y, k & 31);
      xk = cmul(xk, dinv[k]);
      if (lane == (k & 31)) (k < 32 ? x0 : x1) = xk;
      if (lane < k) cfms(x0, T[lane * LD + k], xk);
      if (k > 32 && lane + 32 < k) cfms(x1, T[(lane + 32) * LD + k], xk);
    }
  }
  double2* out = Inv + ((int64_t)blockIdx.z * gridDim.x + i) * TB * TB;
  out[lane * TB + col] = x0;
  out[(lane + 32) * TB + col] = x1;
}

// X_i = Inv X_i on CW columns per CTA; thread = (row, a quarter of K), its part
// of Inv's row in registers.  stats: 16 bytes a row, as ZRows::MEAN reads them
// (nonzero finite entries).
template <int CW>
__global__ void __launch_bounds__(256)
diag_kernel(const double2* __restrict__ Inv, int upper, double2* __restrict__ X, int64_t ldx, int rb, int ncols,
            int* __restrict__ stats) {
  early_start();
  __shared__ double2 xs[CW][TB];
  const int tid = threadIdx.x, row = tid >> 2, q = tid & 3;
  const int c0 = blockIdx.x * CW, nc = min(CW, ncols - c0);
  for (int e = tid; e < CW * TB; e += 256) {
    const int r = e / CW, c = e % CW;
    xs[c][r] = (r < rb && c < nc) ? X[(int64_t)r * ldx + c0 + c] : make_double2(0.0, 0.0);
  }
  double2 inv[TB / 4];
#pragma unroll
  for (int t = 0; t < TB / 4; ++t) inv[t] = Inv[row * TB + q + 4 * t];
  __syncthreads();
  // only the triangle's part of K, by the warp's eight rows
  const int wr0 = (tid >> 5) * 8;
  const int tb = upper ? wr0 / 4 : 0, te = upper ? TB / 4 : wr0 / 4 + 2;
  int em = 0, sum = 0, count = 0;
  for (int c = 0; c < nc; ++c) {
    double2 acc = make_double2(0.0, 0.0);
#pragma unroll
    for (int t = 0; t < TB / 4; ++t)
      if (t >= tb && t < te) cfma(acc, inv[t], xs[c][q + 4 * t]);
#pragma unroll
    for (int o = 1; o < 4; o <<= 1) {
      acc.x += __shfl_xor_sync(0xffffffffu, acc.x, o);
      acc.y += __shfl_xor_sync(0xffffffffu, acc.y, o);
    }
    if (q == 0 && row < rb) {
      X[(int64_t)row * ldx + c0 + c] = acc;
      const int ex = (__double2hiint(acc.x) >> 20) & 0x7ff, ey = (__double2hiint(acc.y) >> 20) & 0x7ff;
      const int f = max(ex == 2047 ? 0 : ex, ey == 2047 ? 0 : ey);
      em = max(em, f);
      sum += f ? f - 1023 : 0;
      count += f ? 1 : 0;
    }
  }
  if (q == 0 && row < rb && count > 0) {
    atomicMax(stats + 4 * row, em);
    atomicAdd(reinterpret_cast<unsigned long long*>(stats + 4 * row + 2),
              (unsigned long long)(((long long)count << 32) + sum));
  }
}

// Columns solved together: the digits of a block row of right-hand sides take 3.5 KB a
// column, and from some thousand columns on the chain of block rows is no longer
// what a solve waits for.
constexpr int64_t kCols = 16384;

struct Ws {
  size_t status = kStatusOffset, stats = 256, inv, plan, total;   // stats: 4 TB ints per block row and triangle
  Ws(int64_t n, int64_t nrhs) {
    const int64_t nb = (n + TB - 1) / TB;
    inv = (stats + (size_t)(2 * nb * 4 * TB) * sizeof(int) + 255) & ~size_t(255);
    plan = inv + (size_t)(2 * nb) * TB * TB * sizeof(double2);
    total = plan + zgemm_bytes(n, std::min(nrhs, kCols));
  }
};

}  // namespace zs

size_t zsolve_workspace_bytes(int64_t n, int64_t nrhs) { return zs::Ws(n, nrhs).total; }

// X = U^-1 L^-1 X for at most kCols columns; stats: zeros
static int solve_columns(const double2* F, int64_t ldf, double2* X, int64_t ldx, int n, int nrhs, const double2* inv,
                         int* stats, int* status, const ZGemmPlan& plan, cudaStream_t s) {
  using namespace zs;
  const int nb = (n + TB - 1) / TB;
  for (int step = 0; step < 2 * nb; ++step) {
    const bool upper = step >= nb;
    const int i = upper ? 2 * nb - 1 - step : step, r0 = i * TB, rb = std::min(TB, n - r0);
    double2* Xi = X + (int64_t)r0 * ldx;
    const double2* iv = inv + (size_t)(upper ? nb + i : i) * TB * TB;
    int* st = stats + (size_t)step * 4 * TB;
    count_launch();
    if (nrhs <= 2 * device_sm_count())
      launch_early(true, diag_kernel<1>, nrhs, 256, 0, s, iv, upper, Xi, ldx, rb, nrhs, st);
    else
      launch_early(false, diag_kernel<4>, (nrhs + 3) / 4, 256, 0, s, iv, upper, Xi, ldx, rb, nrhs, st);
    const int q0 = upper ? 0 : r0 + rb, m = upper ? r0 : n - q0;
    if (m <= 0) continue;
    const ZRows rows{ZRows::MEAN, st, nullptr};
    const double2* Fi = F + (int64_t)q0 * ldf + r0;
    int e = zgemm_digits(plan, Fi, ldf, m, Xi, ldx, nrhs, rb, rows, s);
    if (e == MGT_OK)
      e = zgemm_apply(plan, Fi, ldf, m, Xi, ldx, nrhs, rb, X + (int64_t)q0 * ldx, ldx, ZOut::SUB, nullptr, status, s);
    if (e != MGT_OK) return e;
  }
  return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_ERR_CUDA;
}

int zsolve(const double2* F, int64_t ldf, double2* X, int64_t ldx, int n, int nrhs, void* work, cudaStream_t s) {
  using namespace zs;
  static OncePerDevice once;
  const size_t smem = (size_t)TB * LD * sizeof(double2);
  once([smem] { cudaFuncSetAttribute(inverse_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem); });
  const Ws L(n, nrhs);
  const int nb = (n + TB - 1) / TB;
  int* status = (int*)((char*)work + L.status);
  int* stats = (int*)((char*)work + L.stats);
  double2* inv = (double2*)((char*)work + L.inv);
  ZGemmPlan plan;
  plan.init((char*)work + L.plan, n, std::min<int64_t>(nrhs, kCols));
  if (cudaMemsetAsync(work, 0, L.inv, s) != cudaSuccess) return MGT_ERR_CUDA;   // status, sizes of rows
  count_launch();
  inverse_kernel<<<dim3(nb, 8, 2), 256, smem, s>>>(F, ldf, n, inv);
  for (int64_t c0 = 0; c0 < nrhs; c0 += kCols) {
    if (c0 > 0 && cudaMemsetAsync(stats, 0, L.inv - L.stats, s) != cudaSuccess) return MGT_ERR_CUDA;
    const int e = solve_columns(F, ldf, X + c0, ldx, n, (int)std::min<int64_t>(kCols, nrhs - c0), inv, stats, status, plan, s);
    if (e != MGT_OK) return e;
  }
  return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_ERR_CUDA;
}

}  // namespace mgt
