// complex128 products of up to 64 columns of K on the tensor cores (zgemm_tc.cu),
// and the row interchanges of the complex128 LU's blocked path.
#pragma once
#include "common.cuh"

namespace mgt {

constexpr int kZK = 64;          // largest complex K of one product

// Operand digits and scales, in a workspace of zgemm_bytes(rows, cols).
struct ZGemmPlan {
  unsigned char* adig = nullptr;   // digits of A (rows x kZK)
  unsigned char* bdig = nullptr;   // digits of B (kZK x cols)
  int* aexp = nullptr;             // row / column exponents
  int* bexp = nullptr;
  int64_t rows = 0, cols = 0;
  void init(void* work, int64_t rows, int64_t cols);
};
size_t zgemm_bytes(int64_t rows, int64_t cols);

// digits of A (M x K) and of B (K x N) into the plan (either may be null); K <= kZK.  kexp (device, K
// ints, or null): largest exponent field of each row of B, scaled out of B's rows into A's columns
int zgemm_digits(const ZGemmPlan& p, const double2* A, int64_t lda, int M, const double2* B, int64_t ldb, int N, int K,
                 const int* kexp, cudaStream_t s);
// C (M x N) -= A B (sub) or C = A B, from rows [arow, arow + M) (arow a multiple of 128) and
// columns [bcol, bcol + N) (bcol a multiple of 32) of the plan's digits; rowmax (M zeros, or null)
// receives the largest exponent fields of C's rows; max_ctas <= 0: one CTA per SM
int zgemm_apply(const ZGemmPlan& p, int arow, int M, int bcol, int N, int K, double2* C, int64_t ldc, bool sub,
                int* rowmax, int* status, cudaStream_t s, int max_ctas = 0);

// out (M x N) = E0 - A B for any K (E0 may be null: zero), in a workspace of zgemm_wide_bytes: every 64
// columns of K have their own scales, their products are summed in FP64.  The status word is the first int
// of the workspace's first 1024-byte boundary.
size_t zgemm_wide_bytes(int64_t M, int64_t N, int64_t K);
int zgemm_wide(const double2* A, int64_t lda, int M, const double2* B, int64_t ldb, int N, int K, const double2* E0,
               int64_t ld0, double2* out, int64_t ldo, void* work, cudaStream_t s);

// ---- blocked complex128 LU: interchanges and block inverses
struct ZSlots {
  const int2* slots;   // (position, source) pairs relative to the panel's first row
  const int* nslot;
};
// interchanges of the 32-column panel at j0 on columns [lb, le) and [rb, re); with solve the latter get
// U = L11^-1 A on the panel's rows; inv (or null) receives L11^-1 (32 x 32, leading dimension ldinv)
int zswap_panel(double2* A, int64_t lda, int n, int j0, int w, const ZSlots& s, int lb, int le, int rb, int re,
                bool solve, double2* inv, int ldinv, cudaStream_t st);
// interchanges of the two panels of the block at J0 (widths wa, wb) on columns [0, J0) and [J0 + wa + wb, n);
// with Inv (64 x 64, its upper left 32 x 32 made by zswap_panel) the rest of the block's L^-1; kexp (64
// zeros, or null) receives the largest exponent fields of the block's rows right of it
int zswap_block(double2* A, int64_t lda, int n, int J0, int wa, int wb, const ZSlots& a, const ZSlots& b,
                double2* Inv, int* kexp, cudaStream_t st);

// ---- triangular solves X = U^-1 L^-1 X in place (zsolve.cu); the status word is the first int of work
size_t zsolve_workspace_bytes(int64_t n, int64_t nrhs);
int zsolve(const double2* F, int64_t ldf, double2* X, int64_t ldx, int n, int nrhs, void* work, cudaStream_t s);

}  // namespace mgt
