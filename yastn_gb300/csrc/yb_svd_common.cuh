// Shared by the block SVD / eigh / QR kernels (yb_svd.cu, yb_jacobi.cuh, yb_qr.cuh): the record
// layout of the blocks, the per-block state, numeric traits of the four working types, the Jacobi
// rotation of a row pair in the sweeps of yb_svd.cu and the bounded grid barrier of the cooperative
// launches.
#pragma once
#include <float.h>
#include "yb_common.cuh"

namespace yb {
namespace {

constexpr int kWarps = 8;
constexpr int kThreads = kWarps * 32;
constexpr long long kSpinLimit = 1ll << 22;

// record fields
enum { R_A = 0, R_M, R_N, R_U, R_S, R_V, R_X, R_W, R_P, R_K, R_L, R_NP, R_T, R_X32, R_W32, R_NSUP,
       R_QR, R_LQ, R_Z, R_VQ, R_TAU, R_RR, R_WS, R_NSUP64 };
// per-block state (int64): [0] max |cos| of the sweep in progress (double bits),
// [1] converged flag, [2] sweeps run in the current phase, [3] largest |cos| of the last sweep (until
// then the largest tangent of the sweep in progress, see stops),
// [4], [5] squared row norms (double bits) at or below which a row is rounding noise in the
// FP32 / FP64 phase: a pair with such a row is neither rotated nor counted for convergence,
// and the finalisation completes the vectors of those rows like those of zero values
enum { ST_MAXCOS = 0, ST_CONV = 1, ST_SWEEPS = 2, ST_LASTCOS = 3, ST_THR32 = 4, ST_THR64 = 5, ST_REC = 6 };
constexpr double kNoise32 = 1e-5;   // noise row norm relative to ||A||_F in the FP32 phase
constexpr double kNoise64 = 1e-14;  // idem in the FP64 phase (a few FP64 roundings of ||A||_F)
// control words after the per-block state: [0] barrier count [1] barrier generation
// [2] error flag [3] all-converged flag
enum { C_COUNT = 0, C_GEN = 1, C_ERR = 2, C_DONE = 3, C_REC = 4 };

template <typename T>
struct Eps;
template <>
struct Eps<float> {
  static constexpr double v = 5.9604644775390625e-08;  // 2^-24
};
template <>
struct Eps<double> {
  static constexpr double v = 1.1102230246251565e-16;  // 2^-53
};

// Numeric traits of the four working types: float, double, complex64 (float2) and
// complex128 (double2). R is the real type; fmac(x, y, acc) = acc + x conj(y).
template <typename T>
struct Num;
template <>
struct Num<float> {
  using R = float;
  static constexpr bool cplx = false;
  __device__ static float zero() { return 0.f; }
  __device__ static float one() { return 1.f; }
  __device__ static float abs2(float x) { return x * x; }
  __device__ static float fmac(float x, float y, float acc) { return fmaf(x, y, acc); }
  __device__ static float fma_(float a, float b, float acc) { return fmaf(a, b, acc); }
  __device__ static float mul(float a, float b) { return a * b; }
  __device__ static float scale(float s, float a) { return s * a; }
  __device__ static float conj(float a) { return a; }
  __device__ static float add(float a, float b) { return a + b; }
  __device__ static float sub(float a, float b) { return a - b; }
};
template <>
struct Num<double> {
  using R = double;
  static constexpr bool cplx = false;
  __device__ static double zero() { return 0.0; }
  __device__ static double one() { return 1.0; }
  __device__ static double abs2(double x) { return x * x; }
  __device__ static double fmac(double x, double y, double acc) { return fma(x, y, acc); }
  __device__ static double fma_(double a, double b, double acc) { return fma(a, b, acc); }
  __device__ static double mul(double a, double b) { return a * b; }
  __device__ static double scale(double s, double a) { return s * a; }
  __device__ static double conj(double a) { return a; }
  __device__ static double add(double a, double b) { return a + b; }
  __device__ static double sub(double a, double b) { return a - b; }
};
template <>
struct Num<float2> {
  using R = float;
  static constexpr bool cplx = true;
  __device__ static float2 zero() { return make_float2(0.f, 0.f); }
  __device__ static float2 one() { return make_float2(1.f, 0.f); }
  __device__ static float abs2(float2 x) { return fmaf(x.x, x.x, x.y * x.y); }
  __device__ static float2 fmac(float2 x, float2 y, float2 acc) {
    return make_float2(fmaf(x.x, y.x, fmaf(x.y, y.y, acc.x)), fmaf(x.y, y.x, fmaf(-x.x, y.y, acc.y)));
  }
  __device__ static float2 fma_(float2 a, float2 b, float2 acc) {
    return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, acc.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, acc.y)));
  }
  __device__ static float2 mul(float2 a, float2 b) { return fma_(a, b, zero()); }
  __device__ static float2 scale(float s, float2 a) { return make_float2(s * a.x, s * a.y); }
  __device__ static float2 conj(float2 a) { return make_float2(a.x, -a.y); }
  __device__ static float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
  __device__ static float2 sub(float2 a, float2 b) { return make_float2(a.x - b.x, a.y - b.y); }
};
template <>
struct Num<double2> {
  using R = double;
  static constexpr bool cplx = true;
  __device__ static double2 zero() { return make_double2(0.0, 0.0); }
  __device__ static double2 one() { return make_double2(1.0, 0.0); }
  __device__ static double abs2(double2 x) { return fma(x.x, x.x, x.y * x.y); }
  __device__ static double2 fmac(double2 x, double2 y, double2 acc) {
    return make_double2(fma(x.x, y.x, fma(x.y, y.y, acc.x)), fma(x.y, y.x, fma(-x.x, y.y, acc.y)));
  }
  __device__ static double2 fma_(double2 a, double2 b, double2 acc) {
    return make_double2(fma(a.x, b.x, fma(-a.y, b.y, acc.x)), fma(a.x, b.y, fma(a.y, b.x, acc.y)));
  }
  __device__ static double2 mul(double2 a, double2 b) { return fma_(a, b, zero()); }
  __device__ static double2 scale(double s, double2 a) { return make_double2(s * a.x, s * a.y); }
  __device__ static double2 conj(double2 a) { return make_double2(a.x, -a.y); }
  __device__ static double2 add(double2 a, double2 b) { return make_double2(a.x + b.x, a.y + b.y); }
  __device__ static double2 sub(double2 a, double2 b) { return make_double2(a.x - b.x, a.y - b.y); }
};

// conversions between the storage types
__device__ __forceinline__ float to32(double v) { return (float)v; }
__device__ __forceinline__ float2 to32(double2 v) { return make_float2((float)v.x, (float)v.y); }
__device__ __forceinline__ double to64(float v) { return (double)v; }
__device__ __forceinline__ double2 to64(float2 v) { return make_double2((double)v.x, (double)v.y); }
__device__ __forceinline__ double cabs2(double v) { return v * v; }
__device__ __forceinline__ double cabs2(double2 v) { return fma(v.x, v.x, v.y * v.y); }
__device__ __forceinline__ double cconj_(double v) { return v; }
__device__ __forceinline__ double2 cconj_(double2 v) { return make_double2(v.x, -v.y); }
__device__ __forceinline__ double add_real(double v, double c) { return v + c; }
__device__ __forceinline__ double2 add_real(double2 v, double c) { return make_double2(v.x + c, v.y); }
__device__ __forceinline__ double rscale(double v, double s) { return v * s; }
__device__ __forceinline__ double2 rscale(double2 v, double s) { return make_double2(v.x * s, v.y * s); }

__device__ __forceinline__ double warp_sum(double v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

__device__ __forceinline__ float warp_sum(float v) {
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
  return v;
}

// When a phase ends. A sweep whose largest |cos| is c leaves about c^2 where its rotations are small. One
// by a large tangent t, of two rows of nearly equal norm, moves their cosines with other rows, up to
// c, to where the sweep has already been: about t c is left. Equal singular values meet that: blocks
// of 3 to 20 such values stopped at c <= 1e-7 had vectors orthogonal to 4e-8 only. So an SVD's
// FP64 phase (mixed) ends after a sweep with c <= tol_stop and t c <= kMixed; eigh's stop is low enough by
// itself. Tangents below kTanMin cannot matter. After kMixedSweeps sweeps c alone decides.
constexpr double kMixed = 1e-12;
constexpr float kTanMin = 1e-6f;
constexpr int kMixedSweeps = 16;
template <typename R>
__host__ __device__ __forceinline__ bool mixed_stop(double tol_stop) { return sizeof(R) == 8 && tol_stop > 1e-9; }
__device__ __forceinline__ bool stops(double maxcos, double maxtan, double tol_stop, bool mixed, int64_t sweeps) {
  return maxcos <= tol_stop && (!mixed || maxcos * maxtan <= kMixed || sweeps >= kMixedSweeps);
}

// Jacobi rotation of a row pair from its warp-local partial sums al_ = |x_p|^2, be_ =
// |x_q|^2, ga_ = <x_p, x_q> (Rutishauser's formulas): returns true (every lane) if the pair
// is rotated, with (c, s) and the phase u (1 for real rows). |cos| of the pair goes to the
// block's running maximum. GB300 runs FP64 at 1/64 of the FP32 rate, so the FP32 phase
// keeps the whole computation in FP32, and the FP64 phase does the scalar part on lane 0
// only and broadcasts the result.
template <typename T>
__device__ __forceinline__ void warp_sum_t(T& v);
template <>
__device__ __forceinline__ void warp_sum_t<float>(float& v) { v = warp_sum(v); }
template <>
__device__ __forceinline__ void warp_sum_t<double>(double& v) { v = warp_sum(v); }
template <>
__device__ __forceinline__ void warp_sum_t<float2>(float2& v) { v.x = warp_sum(v.x); v.y = warp_sum(v.y); }
template <>
__device__ __forceinline__ void warp_sum_t<double2>(double2& v) { v.x = warp_sum(v.x); v.y = warp_sum(v.y); }

__device__ __forceinline__ float gabs(float g) { return fabsf(g); }
__device__ __forceinline__ double gabs(double g) { return fabs(g); }
__device__ __forceinline__ float gabs(float2 g) { return hypotf(g.x, g.y); }
__device__ __forceinline__ double gabs(double2 g) { return hypot(g.x, g.y); }

template <typename T>
struct Rotation {
  using R = typename Num<T>::R;
  // scalar part: from the summed (al, be, g) to (c, s, u); |cos| (st) and, with mixed, |tan| to the
  // running maxima
  __device__ static bool scalar(R al, R be, T ga, int64_t L, int64_t* st, R& c, R& s, T& u, R thr2, bool mixed) {
    if (!(al > thr2 && be > thr2 && al > R(0) && be > R(0))) return false;
    const R g = gabs(ga);
    const R cosv = g / (sqrt(al) * sqrt(be));
    atomicMax((unsigned long long*)st, (unsigned long long)__double_as_longlong((double)cosv));
    if (!(cosv > sqrt((R)L) * (R)Eps<R>::v)) return false;
    R zeta;
    if constexpr (Num<T>::cplx) {
      u.x = ga.x / g;
      u.y = ga.y / g;
      zeta = (be - al) / (R(2) * g);
    } else {
      u = R(1);
      zeta = (be - al) / (R(2) * ga);
    }
    const R t = copysign(R(1), zeta) / (fabs(zeta) + hypot(R(1), zeta));
    if (mixed && fabs(t) > R(kTanMin))
      atomicMax((unsigned long long*)st + (ST_LASTCOS - ST_MAXCOS), (unsigned long long)__double_as_longlong((double)fabs(t)));
    c = R(1) / sqrt(fma(t, t, R(1)));
    s = c * t;
    return true;
  }
  // thr2: squared noise norm of the phase; a pair with a row at or below it is left alone
  __device__ static bool get(R al_, R be_, T ga_, int64_t L, int lane, int64_t* st, R& c, R& s, T& u, R thr2,
                             bool mixed) {
    const R al = warp_sum(al_), be = warp_sum(be_);
    warp_sum_t<T>(ga_);
    if constexpr (sizeof(R) == 4) {
      // FP32: every lane computes the same (cheap) scalar part; one lane records |cos|
      if (!(al > thr2 && be > thr2 && al > R(0) && be > R(0))) return false;
      const R g = gabs(ga_);
      const R cosv = g / (sqrtf(al) * sqrtf(be));
      if (lane == 0) atomicMax((unsigned long long*)st, (unsigned long long)__double_as_longlong((double)cosv));
      if (!(cosv > sqrtf((float)L) * 5.9604645e-08f)) return false;
      R zeta;
      if constexpr (Num<T>::cplx) {
        u.x = ga_.x / g;
        u.y = ga_.y / g;
        zeta = (be - al) / (2.f * g);
      } else {
        u = 1.f;
        zeta = (be - al) / (2.f * ga_);
      }
      const R t = copysignf(1.f, zeta) / (fabsf(zeta) + hypotf(1.f, zeta));
      c = 1.f / sqrtf(fmaf(t, t, 1.f));
      s = c * t;
      return true;
    } else {
      int rot = 0;
      if (lane == 0) rot = scalar(al, be, ga_, L, st, c, s, u, thr2, mixed) ? 1 : 0;
      rot = __shfl_sync(0xffffffffu, rot, 0);
      if (!rot) return false;
      c = __shfl_sync(0xffffffffu, c, 0);
      s = __shfl_sync(0xffffffffu, s, 0);
      if constexpr (Num<T>::cplx) {
        u.x = __shfl_sync(0xffffffffu, u.x, 0);
        u.y = __shfl_sync(0xffffffffu, u.y, 0);
      } else {
        u = 1.0;
      }
      return true;
    }
  }
};

// (a, b) <- (c a - s u b, s a + c u b)
template <typename T>
__device__ __forceinline__ void rot2(T& a, T& b, typename Num<T>::R c, typename Num<T>::R s, T u) {
  T bu = b;
  if constexpr (Num<T>::cplx) bu = Num<T>::mul(u, b);
  const T na = Num<T>::sub(Num<T>::scale(c, a), Num<T>::scale(s, bu));
  const T nb = Num<T>::add(Num<T>::scale(s, a), Num<T>::scale(c, bu));
  a = na;
  b = nb;
}

// Grid barrier for a cooperative launch (all CTAs co-resident). The spin is bounded: on
// timeout the error flag is raised and false is returned, and the caller exits.
__device__ bool grid_barrier(unsigned long long* ctrl, unsigned nblocks) {
  __shared__ int ok;
  __syncthreads();
  if (threadIdx.x == 0) {
    ok = 1;
    volatile unsigned long long* gen = ctrl + C_GEN;
    const unsigned long long g = *gen;
    __threadfence();
    const unsigned long long arrived = atomicAdd(ctrl + C_COUNT, 1ull) + 1ull;
    if (arrived == nblocks) {
      ctrl[C_COUNT] = 0ull;
      __threadfence();
      atomicAdd(ctrl + C_GEN, 1ull);
    } else {
      long long spins = 0;
      while (*gen == g) {
        __nanosleep(32);
        if (++spins > kSpinLimit) {
          atomicExch(ctrl + C_ERR, 1ull);
          ok = 0;
          break;
        }
      }
    }
    __threadfence();
  }
  __syncthreads();
  return ok != 0;
}

}  // namespace
}  // namespace yb
