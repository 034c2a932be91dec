// Jacobi sweeps with a row per warp: FP64 (kernel and entry points' reasons in yb_jacobi.cuh).
#include "yb_jacobi.cuh"

namespace yb {

int jacobi_f64(YB_JACOBI_ARGS) {
  YB_ROWS(double, 8, 2, 4);
  YB_ROWS(double, 8, 4, 4);
  YB_ROWS(double, 8, 6, 4);
  YB_ROWS(double, 8, 8, 4);
  YB_ROWS(double, 8, 11, 4);
  YB_ROWS(double, 8, 14, 4);
  YB_ROWS(double, 8, 18, 4);
  YB_ROWS(double, 8, 23, 4);
  YB_ROWS(double, 8, 28, 4);
  YB_ROWS(double, 8, 34, 4);
  YB_ROWS(double, 8, 41, 4);
  return YB_ERR_TOO_LARGE;
}

}  // namespace yb
