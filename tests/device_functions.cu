// Kernels that call device functions of csrc/ on arrays, for the tests (built by them with nvcc).
#include "../yastn_gb300/csrc/yb_qr.cuh"

namespace yb {
void set_cuda_error(int) {}

namespace {
// n waits in turn for a flag that nobody sets
__global__ void qr_waits_kernel(const unsigned long long* flag, unsigned long long* err, int n) {
  for (int i = 1; i <= n; ++i) qr_wait(flag, (unsigned long long)i, err);
}
}  // namespace
}  // namespace yb

extern "C" int t_qr_waits(const void* flag, void* err, int n, void* stream) {
  yb::qr_waits_kernel<<<1, yb::kThreads, 0, (cudaStream_t)stream>>>((const unsigned long long*)flag,
                                                                    (unsigned long long*)err, n);
  return (int)cudaGetLastError();
}
