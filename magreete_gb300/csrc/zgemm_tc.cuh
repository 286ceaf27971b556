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

// How the rows of B (K of them) may differ in size.  A product's error is one
// rounding of (largest entry of A's row) x (largest entry of B's column), which
// is the error of an FP64 sum only while neither is much larger than what meets
// it.  A power of two per k may be moved from B's row to A's column first; where
// none serves, the product is made on the FP64 pipe (the digits' kernel decides and
// marks the row exponents; no host involved).
//   MAX (the LU's updates; stats: the largest exponent field of each row of B).
//     Multipliers are at most sqrt 2, so no scaling keeps the errors of each
//     column small against that column, whatever the rows; equal scales of the
//     rows keep those of each row small.  Spreads of the rows' sizes up to 2^4:
//     as they are; up to 2^12: half the exponents moved, a loss of at most 2^6 =
//     K either way, the bound of an FP64 sum of K terms; beyond: FP64.  (Rows
//     of the engine's systems spread by 2^2 to 2^8, Poisson clouds at the upper
//     end; pairs of scatterers at 1e-4 of their wavelength by 2^30, where
//     moving whole exponents lost 1e9 of a column's accuracy.)
//   MEAN (the solves and the propagation; stats: 16 bytes a row -- the largest field, 4 unused
//     bytes, and in 64 bits the sum of the fields less 1023 plus 2^32 for each nonzero entry).  Right-hand sides may have single
//     large entries, so that a row's mean says what meets A's column: spreads of
//     the means up to 2^4: as they are; beyond, where the rows are alike but for
//     their means (largest less mean within 2^6): the means moved; else FP64.
struct ZRows {
  enum Kind { NONE = 0, MAX = 1, MEAN = 2 };
  int kind = NONE;
  const int* stats = nullptr;   // of kZK rows (MEAN: 16-byte aligned)
  const int* inv = nullptr;     // (or null) largest exponent field of A, an inverse: from 2^4 on FP64 too
};

// digits of A (M x K) and of B (K x N) into the plan (either may be null); K <= kZK
int zgemm_digits(const ZGemmPlan& p, const double2* A, int64_t lda, int M, const double2* B, int64_t ldb, int N, int K,
                 const ZRows& rows, cudaStream_t s);
// C (M x N) -= A B (SUB), C = A B (SET), or, for the LU's U12, C = L^-1 C (SOLVE: M = K = 64; the digits
// are those of L^-1 and of C, and A is the unit lower L), from the plan's digits.  A and B: the operands, for
// the FP64 pipe.  rowmax (M zeros, or null) receives the largest exponent fields of C's rows
enum class ZOut { SUB, SET, SOLVE };
int zgemm_apply(const ZGemmPlan& p, const double2* A, int64_t lda, int M, const double2* B, int64_t ldb, int N, int K,
                double2* C, int64_t ldc, ZOut out, int* rowmax, int* status, cudaStream_t s);

// out (M x N) = E0 - A B for any K (E0 may be null: zero), in a workspace of zgemm_wide_bytes: every 64
// columns of K have their own scales (and ZRows::MEAN of their own), their products are summed in FP64.
size_t zgemm_wide_bytes(int64_t M, int64_t N, int64_t K);
int zgemm_wide(const double2* A, int64_t lda, int M, const double2* B, int64_t ldb, int N, int K, const double2* E0,
               int64_t ld0, double2* out, int64_t ldo, void* work, int* status, cudaStream_t s);

// ---- blocked complex128 LU: interchanges and block inverses
struct ZSlots {
  const int2* slots;   // (position, source) pairs relative to the panel's first row
  const int* nslot;
};
// interchanges of the 32-column panel at j0 on columns [lb, le) and [rb, re); with solve the latter get
// U = L11^-1 A on the panel's rows; inv (or null) receives L11^-1 (32 x 32, leading dimension ldinv),
// invmax (zero) its largest exponent field
int zswap_panel(double2* A, int64_t lda, int n, int j0, int w, const ZSlots& s, int lb, int le, int rb, int re,
                bool solve, double2* inv, int ldinv, int* invmax, cudaStream_t st);
// interchanges of the two panels of the block at J0 (widths wa, wb) on columns [0, J0) and [J0 + wa + wb, n);
// with Inv (64 x 64, its upper left 32 x 32 made by zswap_panel) the rest of the block's L^-1 and its
// largest field; kexp (64 zeros, or null) receives the largest exponent fields of the block's rows right of it
int zswap_block(double2* A, int64_t lda, int n, int J0, int wa, int wb, const ZSlots& a, const ZSlots& b,
                double2* Inv, int* invmax, int* kexp, cudaStream_t st);

// ---- triangular solves X = U^-1 L^-1 X in place (zsolve.cu); status words where mgt_workspace_status reads them
size_t zsolve_workspace_bytes(int64_t n, int64_t nrhs);
int zsolve(const double2* F, int64_t ldf, double2* X, int64_t ldx, int n, int nrhs, void* work, cudaStream_t s);

}  // namespace mgt
