// SIMT complex GEMM update (FP64 pipe for complex128, FP32 pipe for
// complex64).  16 RT x 16 RT output tile per CTA of 256 threads, K staged
// through shared memory 16 at a time, RT x RT complex outputs per thread.
//
// complex128 is bound by the FP64 pipe (about 1.7 fused multiply-adds per
// clock and SM) whatever the tile, so the tile is chosen for balance: a 64-wide
// tile takes 142 us at K = 32, however few there are.  RT = 1 while 32-wide
// tiles would give fewer than four per SM, else RT = 2.  The sum over K runs in
// the same order for every RT: bit-identical results.  complex64 keeps RT = 4
// (its FP32 pipe is bound by shared-memory reads per product).
#include "gemm.cuh"
#include "diag.cuh"

namespace mgt {

constexpr int kGK = 16;

template <typename T, int RT>
__global__ void __launch_bounds__(256)
cgemm_sub_kernel(int M, int N, int K, const cplx<T>* __restrict__ A, int64_t lda,
                 const cplx<T>* __restrict__ B, int64_t ldb, cplx<T>* __restrict__ C, int64_t ldc) {
  early_start();
  using V = cplx<T>;
  constexpr int GT = 16 * RT;
  __shared__ V As[kGK][GT + 1];
  __shared__ V Bs[kGK][GT];
  const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
  const int row0 = blockIdx.y * GT, col0 = blockIdx.x * GT;
  V acc[RT][RT];
#pragma unroll
  for (int i = 0; i < RT; ++i)
#pragma unroll
    for (int j = 0; j < RT; ++j) acc[i][j] = czero<V>();
  for (int k0 = 0; k0 < K; k0 += kGK) {
#pragma unroll
    for (int q = 0; q < RT; ++q) {
      int idx = tid + 256 * q;
      int r = idx >> 4, kk = idx & 15;
      V v = czero<V>();
      if (row0 + r < M && k0 + kk < K) v = A[(int64_t)(row0 + r) * lda + k0 + kk];
      As[kk][r] = v;
      int kb = idx / GT, cc = idx % GT;
      V u = czero<V>();
      if (k0 + kb < K && col0 + cc < N) u = B[(int64_t)(k0 + kb) * ldb + col0 + cc];
      Bs[kb][cc] = u;
    }
    __syncthreads();
#pragma unroll
    for (int kk = 0; kk < kGK; ++kk) {
      V a[RT], b[RT];
#pragma unroll
      for (int i = 0; i < RT; ++i) a[i] = As[kk][ty + 16 * i];
#pragma unroll
      for (int j = 0; j < RT; ++j) b[j] = Bs[kk][tx + 16 * j];
#pragma unroll
      for (int i = 0; i < RT; ++i)
#pragma unroll
        for (int j = 0; j < RT; ++j) cfma(acc[i][j], a[i], b[j]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int i = 0; i < RT; ++i) {
    int r = row0 + ty + 16 * i;
    if (r >= M) continue;
#pragma unroll
    for (int j = 0; j < RT; ++j) {
      int c = col0 + tx + 16 * j;
      if (c < N) {
        V* p = C + (int64_t)r * ldc + c;
        *p = csub(*p, acc[i][j]);
      }
    }
  }
}

template <typename T, int RT>
static int gemm_sub_rt(int M, int N, int K, const cplx<T>* A, int64_t lda, const cplx<T>* B, int64_t ldb,
                       cplx<T>* C, int64_t ldc, cudaStream_t s) {
  constexpr int GT = 16 * RT;
  dim3 grid((N + GT - 1) / GT, (M + GT - 1) / GT);
  if (grid.y > 65535) return MGT_ERR_UNSUPPORTED;
  count_launch();
  // (complex64 updates run on side streams too, after waits for events: ordinary launches)
  launch_early(sizeof(T) == 8 && (int64_t)grid.x * grid.y <= 2 * device_sm_count(), cgemm_sub_kernel<T, RT>, grid, 256, 0, s, M, N, K, A, lda, B, ldb, C, ldc);
  return cudaGetLastError() == cudaSuccess ? MGT_OK : MGT_ERR_CUDA;
}

template <typename T>
int gemm_sub(int M, int N, int K, const cplx<T>* A, int64_t lda, const cplx<T>* B, int64_t ldb,
             cplx<T>* C, int64_t ldc, cudaStream_t s) {
  if (M <= 0 || N <= 0 || K <= 0) return MGT_OK;
  if constexpr (sizeof(T) == 8) {
    const int64_t tiles = (int64_t)((N + 31) / 32) * ((M + 31) / 32);
    if (tiles < 4 * device_sm_count()) return gemm_sub_rt<T, 1>(M, N, K, A, lda, B, ldb, C, ldc, s);
    if ((M + 31) / 32 <= 65535) return gemm_sub_rt<T, 2>(M, N, K, A, lda, B, ldb, C, ldc, s);
  }
  return gemm_sub_rt<T, 4>(M, N, K, A, lda, B, ldb, C, ldc, s);
}

template int gemm_sub<double>(int, int, int, const double2*, int64_t, const double2*, int64_t, double2*, int64_t, cudaStream_t);
template int gemm_sub<float>(int, int, int, const float2*, int64_t, const float2*, int64_t, float2*, int64_t, cudaStream_t);

}  // namespace mgt
