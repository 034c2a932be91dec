// Jacobi sweeps with a row per warp: FP32 (kernel and entry points' reasons in yb_jacobi.cuh).
#include "yb_jacobi.cuh"

namespace yb {

int jacobi_f32(YB_JACOBI_ARGS) {
  YB_ROWS(float, 16, 2, 8);
  YB_ROWS(float, 16, 4, 8);
  YB_ROWS(float, 16, 6, 8);
  YB_ROWS(float, 16, 8, 8);
  YB_ROWS(float, 16, 11, 8);
  YB_ROWS(float, 16, 14, 8);
  YB_ROWS(float, 12, 18, 8);
  YB_ROWS(float, 12, 23, 8);
  YB_ROWS(float, 12, 28, 8);
  YB_ROWS(float, 12, 34, 8);
  YB_ROWS(float, 12, 41, 8);
  YB_ROWS(float, 8, 54, 8);
  YB_ROWS(float, 8, 68, 8);
  YB_ROWS(float, 8, 82, 8);
  return YB_ERR_TOO_LARGE;
}

}  // namespace yb
