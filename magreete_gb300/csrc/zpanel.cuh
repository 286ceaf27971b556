// Panel factorisation of the complex128 LU (zpanel.cu).
#pragma once
#include "common.cuh"

namespace mgt {

constexpr int kZNB = 32;            // panel columns
// 64-bit words of the messages between at most `ctas` CTAs: two key tables, then two rows each
constexpr size_t zpanel_words(int ctas) { return (size_t)ctas * (4 + 2 * (3 * kZNB + 4)); }

// Scratch of one panel: interchange slots and candidate records of the LU workspace.
struct ZPanelWs {
  int* status;            // [0] error, [1] first zero pivot
  int* nslot;
  int2* slots;            // 2 kZNB (position, source) pairs
  unsigned long long* records;   // zpanel_words(max_ctas) words, zero when a factorisation starts
  int max_ctas;
};

// Whether a panel of m rows fits `max_ctas` CTAs of about rows_target, at most 128, rows.
inline bool zpanel_fits(int m, int rows_target, int max_ctas) {
  return rows_target <= 128 && m <= 128 * (max_ctas > 1 ? max_ctas : 1);
}

// Factors columns [0, w) (w <= 32) of the m-row panel at P in place, with partial pivoting
// (LAPACK's rule); MGT_ERR_UNSUPPORTED where the panel does not fit (nothing is launched).
// allow_cluster, allow_wide: as one cluster; as CTAs that exchange through global memory.
int zpanel_factor(double2* P, int64_t lda, int m, int w, int j0, int32_t* perm, const ZPanelWs& ws, int rows_target,
                  int max_ctas, bool cooperative, bool allow_cluster, bool allow_wide, cudaStream_t s);

}  // namespace mgt
