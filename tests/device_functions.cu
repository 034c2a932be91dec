// Kernels that call device functions of csrc/ on arrays, for the tests (built by them with nvcc).
#include "../yastn_gb300/csrc/yb_jacobi.cuh"
#include "../yastn_gb300/csrc/yb_qr.cuh"
#define warp_sum adjoint_warp_sum  // both have one
#include "../yastn_gb300/csrc/yb_adjoint.cu"
#undef warp_sum

namespace yb {
void set_cuda_error(int) {}

namespace {
// n waits in turn for a flag that nobody sets
__global__ void qr_waits_kernel(const unsigned long long* flag, unsigned long long* err, int n) {
  for (int i = 1; i <= n; ++i) qr_wait(flag, (unsigned long long)i, err);
}

__global__ void rsqrt_kernel(const double* u, double* out, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = rsqrt64(u[i]);
}

__global__ void div_kernel(const double* v, const double* d, double* out, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
    out[i] = trsm_div(v[i], d[i], 1.0 / d[i]);
}

// out: tau, 1 / (alpha - beta), beta, conj(tau / (alpha - beta)) (the last one real)
template <typename T>
__global__ void scalars_kernel(const T* alpha, const double* xn, T* out, int64_t n) {
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
    double ts;
    qr_scalars<T>(alpha[i], xn[i], out[4 * i], out[4 * i + 1], out[4 * i + 2], ts);
    if constexpr (Num<T>::cplx) out[4 * i + 3] = make_double2(ts, 0.0); else out[4 * i + 3] = ts;
  }
}
}  // namespace
}  // namespace yb

extern "C" int t_rsqrt(const void* u, void* out, int64_t n, void* stream) {
  yb::rsqrt_kernel<<<64, 256, 0, (cudaStream_t)stream>>>((const double*)u, (double*)out, n);
  return (int)cudaGetLastError();
}

extern "C" int t_div(const void* v, const void* d, void* out, int64_t n, void* stream) {
  yb::div_kernel<<<64, 256, 0, (cudaStream_t)stream>>>((const double*)v, (const double*)d, (double*)out, n);
  return (int)cudaGetLastError();
}

extern "C" int t_scalars(int cplx, const void* alpha, const void* xn, void* out, int64_t n, void* stream) {
  if (cplx)
    yb::scalars_kernel<double2><<<64, 256, 0, (cudaStream_t)stream>>>((const double2*)alpha, (const double*)xn,
                                                                      (double2*)out, n);
  else
    yb::scalars_kernel<double><<<64, 256, 0, (cudaStream_t)stream>>>((const double*)alpha, (const double*)xn,
                                                                     (double*)out, n);
  return (int)cudaGetLastError();
}

extern "C" int t_qr_waits(const void* flag, void* err, int n, void* stream) {
  yb::qr_waits_kernel<<<1, yb::kThreads, 0, (cudaStream_t)stream>>>((const unsigned long long*)flag,
                                                                    (unsigned long long*)err, n);
  return (int)cudaGetLastError();
}
