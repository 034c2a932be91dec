// Jacobi sweeps with a row per warp: complex128, and the entry points (kernel and entry points' reasons in yb_jacobi.cuh).
#include "yb_jacobi.cuh"

namespace yb {

int jacobi_c128(YB_JACOBI_ARGS) {
  YB_ROWS(double2, 8, 2, 4);
  YB_ROWS(double2, 8, 4, 4);
  YB_ROWS(double2, 8, 6, 4);
  YB_ROWS(double2, 8, 8, 4);
  YB_ROWS(double2, 8, 11, 4);
  YB_ROWS(double2, 8, 14, 4);
  YB_ROWS(double2, 8, 17, 4);
  YB_ROWS(double2, 8, 20, 4);
  return YB_ERR_TOO_LARGE;
}

}  // namespace yb

extern "C" {

int64_t yb_svd_row_aux(int64_t n_blocks, int64_t n_pairs) {
  return yb::aux_zeroed(n_blocks, n_pairs) + 3 * n_pairs;
}

int yb_svd_row_limit(int precision, int dtype) {
  if (precision == 32) return dtype == YB_F64 ? 82 * 32 : (dtype == YB_C128 ? 40 * 32 : 0);
  if (precision == 64) return dtype == YB_F64 ? 41 * 32 : (dtype == YB_C128 ? 20 * 32 : 0);
  return 0;
}

int yb_svd_row_sweeps(void* work, const int64_t* blocks, int n_blocks, const int32_t* pair_items, int n_pairs,
                      int precision, int dtype, int max_sweeps, double tol_stop, int lmax, int64_t* state,
                      int64_t* aux, int64_t aux_words, void* stream) {
  if (n_blocks == 0 || n_pairs == 0 || max_sweeps <= 0) return YB_OK;
  if (!work || !blocks || !pair_items || !state || !aux || n_blocks < 0 || n_pairs < 0) return YB_ERR_INVALID;
  if ((precision != 32 && precision != 64) || (dtype != YB_F64 && dtype != YB_C128)) return YB_ERR_INVALID;
  if (lmax <= 0 || aux_words < yb_svd_row_aux(n_blocks, n_pairs) || ((uintptr_t)aux & 15u)) return YB_ERR_INVALID;
  if (lmax > yb_svd_row_limit(precision, dtype)) return YB_ERR_TOO_LARGE;
  cudaStream_t s = (cudaStream_t)stream;
  if (precision == 32)
    return dtype == YB_F64 ? yb::jacobi_f32(work, blocks, n_blocks, pair_items, n_pairs, max_sweeps, tol_stop, lmax, state, aux, s)
                           : yb::jacobi_c64(work, blocks, n_blocks, pair_items, n_pairs, max_sweeps, tol_stop, lmax, state, aux, s);
  return dtype == YB_F64 ? yb::jacobi_f64(work, blocks, n_blocks, pair_items, n_pairs, max_sweeps, tol_stop, lmax, state, aux, s)
                         : yb::jacobi_c128(work, blocks, n_blocks, pair_items, n_pairs, max_sweeps, tol_stop, lmax, state, aux, s);
}

}  // extern "C"
