// Jacobi sweeps with a row per warp: complex64 (kernel and entry points' reasons in yb_jacobi.cuh).
#include "yb_jacobi.cuh"

namespace yb {

int jacobi_c64(YB_JACOBI_ARGS) {
  YB_ROWS(float2, 16, 2, 8);
  YB_ROWS(float2, 16, 4, 8);
  YB_ROWS(float2, 16, 6, 8);
  YB_ROWS(float2, 12, 8, 8);
  YB_ROWS(float2, 12, 11, 8);
  YB_ROWS(float2, 12, 14, 8);
  YB_ROWS(float2, 12, 17, 8);
  YB_ROWS(float2, 12, 20, 8);
  YB_ROWS(float2, 8, 26, 8);
  YB_ROWS(float2, 8, 33, 8);
  YB_ROWS(float2, 8, 40, 8);
  return YB_ERR_TOO_LARGE;
}

}  // namespace yb
