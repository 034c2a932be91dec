// Blocked Householder QR of all blocks in one cooperative launch (yb_svd_qr, yb_qr).
//
// Z holds the columns of M as rows. Groups of CTAs take a block at a time; panels of kPanel
// columns belong to the owners of a group in turn: an owner is a CTA, or for columns of more than
// kPairRows rows a cluster of two. When panel q is published, every CTA brings its V and T to shared
// memory and applies I - V T^H V^H to its own later panels; the owner of panel q + 1 takes that one
// first: its columns live in registers (256 threads a CTA, a row of the panel per thread and pass,
// V's entries of those rows straight from global memory), are updated by panel q, factored, and
// published through the block's ready counter. The waits are bounded (error word of the group). After
// the factorisation (a group barrier) R's rows and the FP32 start are written, and every warp forms
// its own columns of Q by the panels backwards.
//
// What bounds it: the path through the panels (each update and factorisation runs on one or two SMs,
// whose FP64 pipes issue a warp instruction every 19 cycles, 64 for a single warp: at k = 432 a panel
// takes 33 k cycles, a quarter each for its steps' inner products, their scalars, and the update
// before) and, for large blocks, the FP64 work of the updates. A panel of w columns costs that path a
// fixed part (publish, wait, V's load, w reductions and scalars) and FMAs that grow with w^2: w = 4 is
// the shortest per column by the count of instructions from L = 100 to 2000. A reflector's norm, its
// inner products with the panel's other columns and those that T needs are one reduction, and one warp
// does the scalars (done by all eight they cost more than the panel's FMAs at L = 100).
//
// Why kPairRows = 256: a second CTA helps where it has rows to take (the first 256 are the first
// CTA's), and its barriers cost what it saves around 432 rows: clusters against single CTAs, yb_svd_qr
// of two 432 x 432 blocks 2.37 / 2.36 ms, yb_qr of two 216 x 432 ones 1.34 / 1.40, two 540 x 432
// 2.64 / 2.73, yb_svd_qr of two 1296 x 1296 16.6 / 17.0, yb_qr of two 648 x 1296 6.9 / 7.9 (all with
// Q's panels still loaded in turn).
//
// Measured (GB300; before: a warp per column, one reflector at a time, published by itself): yb_qr
// of two 540 x 432 blocks 7.8 -> 2.5 ms; yb_svd_qr of two 432 x 432 blocks 6.2 -> 2.25 ms, two
// 1296 x 1296 62 -> 16.0 ms (10.6 ms at the DFMA rate), nine of 24..93 0.73 -> 0.39 ms, five complex
// ones of 31 x 24 .. 78 x 60 0.68 -> 0.47 ms; 595 blocks of 42..60 2.6 -> 1.4 ms.
#pragma once
#include <cooperative_groups.h>
#include "yb_svd_common.cuh"

namespace yb {
namespace {

constexpr int kPanel = 4;
constexpr int kMaxCl = 2;        // CTAs that factor a panel together
constexpr int64_t kPairRows = 256;  // columns longer than this are taken by kMaxCl CTAs

// The CL CTAs that share a panel are a cluster: barrier, and a store to the same place in all.
template <int CL>
__device__ __forceinline__ void qr_sync() {
  if constexpr (CL == 1) __syncthreads();
  else cooperative_groups::this_cluster().sync();
}
template <int CL, typename T>
__device__ __forceinline__ void qr_put(T* at, T v) {
  if constexpr (CL == 1) {
    *at = v;
  } else {
#pragma unroll
    for (int c = 0; c < CL; ++c) *cooperative_groups::this_cluster().map_shared_rank(at, c) = v;
  }
}
// Whether every CTA of the cluster got through a barrier of the group.
template <int CL>
__device__ __forceinline__ bool qr_all(bool ok) {
  if constexpr (CL > 1) {
    __shared__ int all[CL];
    if (threadIdx.x == 0) qr_put<CL>(all + cooperative_groups::this_cluster().block_rank(), (int)ok);
    qr_sync<CL>();
#pragma unroll
    for (int c = 0; c < CL; ++c) ok = ok && all[c];
    qr_sync<CL>();
  }
  return ok;
}

template <typename T>
__device__ __forceinline__ T ldcg_t(const T* p) { return __ldcg(p); }

template <typename T>
__device__ __forceinline__ T shfl_t(T v, int src) {
  if constexpr (Num<T>::cplx) {
    v.x = __shfl_sync(0xffffffffu, v.x, src);
    v.y = __shfl_sync(0xffffffffu, v.y, src);
    return v;
  } else {
    return __shfl_sync(0xffffffffu, v, src);
  }
}
template <typename T>
__device__ __forceinline__ T shfl_xor_t(T v, int o) {
  if constexpr (Num<T>::cplx) {
    v.x = __shfl_xor_sync(0xffffffffu, v.x, o);
    v.y = __shfl_xor_sync(0xffffffffu, v.y, o);
    return v;
  } else {
    return __shfl_xor_sync(0xffffffffu, v, o);
  }
}

// Sign and exponent of doubles by integer operations (an FP64 instruction takes a warp 64 cycles).
__device__ __forceinline__ double neg_if(double v, bool n) {
  return __longlong_as_double(__double_as_longlong(v) ^ (n ? (long long)(1ull << 63) : 0ll));
}
__device__ __forceinline__ double neg_t(double v) { return neg_if(v, true); }
__device__ __forceinline__ double2 neg_t(double2 v) { return make_double2(neg_if(v.x, true), neg_if(v.y, true)); }
__device__ __forceinline__ double times_pow2(double v, int e) {  // v normal and v 2^e normal, or v and the result 0
  const long long b = __double_as_longlong(v);
  const int x = (int)(b >> 52) & 0x7ff;
  return x == 0 || x + e <= 0 ? 0.0 : __longlong_as_double(b + ((long long)e << 52));
}
// a positive normal double within FP32's range to FP32 (truncated) and back
__device__ __forceinline__ float trunc32(double v) {
  return __int_as_float((int)((__double_as_longlong(v) - (896ll << 52)) >> 29));
}
__device__ __forceinline__ double widen64(float v) {
  return __longlong_as_double(((long long)__float_as_int(v) << 29) + (896ll << 52));
}

// Sums of N values over the warp, N = 4 or 16: the halves are exchanged while there is more than
// one value left (N + ... FP64 additions instead of 5 N). Lane l returns value (l >> 5 - log2 N).
template <typename T, int N>
__device__ __forceinline__ T warp_sums(T (&v)[N], int lane) {
  int o = 16;
#pragma unroll
  for (int n = N; n > 1; n >>= 1, o >>= 1) {
    const bool up = lane & o;
#pragma unroll
    for (int i = 0; i < n / 2; ++i) {
      const T give = up ? v[i] : v[i + n / 2], keep = up ? v[i + n / 2] : v[i];
      v[i] = Num<T>::add(keep, shfl_xor_t(give, o));
    }
  }
  T s = v[0];
#pragma unroll
  for (int r = 16 / N; r >= 1; r >>= 1) s = Num<T>::add(s, shfl_xor_t(s, r));
  return s;
}

// Waits (thread 0 polls, bounded) until *flag >= target; on timeout raises *err and returns (the
// caller carries on with whatever it reads: the host sees the error word and fails). Once *err is
// up, a wait lasts 64 polls: one timeout ends those of all later panels too.
__device__ __forceinline__ void qr_wait(const unsigned long long* flag, unsigned long long target,
                                        unsigned long long* err) {
  if (threadIdx.x == 0) {
    long long spins = 0;
    while (*(volatile const unsigned long long*)flag < target) {
      if (spins > 16) __nanosleep(32);
      if (++spins > kSpinLimit || ((spins & 63) == 0 && *(volatile const unsigned long long*)err != 0)) {
        atomicExch(err, 1ull);
        break;
      }
    }
    __threadfence();
  }
  __syncthreads();
}

// Shared memory of a CTA: V of a panel (kPanel rows of L - kPanel q elements; not when VS is
// false: V is then read from global memory), T, the partial sums of the reductions.
template <typename T>
struct QrShared {
  T Tm[kPanel][kPanel];          // T of the panel in Vs: Tm[j][i], j <= i, zero below
  T Tq[2][kPanel][kPanel];       // the same for the two panels at hand when Q is formed
  T part[2][kMaxCl * kWarps][kPanel * kPanel];
  T sum[kPanel * kPanel];        // V^H x of the update before a panel's factorisation
  T row[2][kPanel];              // the panel's row j
  T add[2][kPanel], f[2][kPanel];  // a step's updates: row j of the later columns += add, below x_c += f_c x_i
  T sc[2], diag[2], tau[2];
  T Tn[kPanel][kPanel];          // T of the panel being factored
};

template <typename T, bool VS>
struct QrPanel {  // panel q of a block: v(i, l) = entry of reflector i at row kPanel q + l
  const T* s;
  const T* g;  // V + kPanel q (L + 1)
  int64_t L;
  int len;
  __device__ __forceinline__ T v(int i, int l) const {
    if constexpr (VS) return s[i * len + l];
    if (l <= i) return l == i ? Num<T>::one() : Num<T>::zero();
    return __ldcg(g + i * L + l);
  }
};

// V and T of panel q (nb reflectors) for the CTA; V[c][l], l >= kPanel q, holds the reflectors
// below the diagonal and T (transposed) in the triangle of known entries.
template <typename T, bool VS>
__device__ __forceinline__ QrPanel<T, VS> qr_load_panel(const T* __restrict__ V, int64_t L, int64_t q, int nb, T* Vs,
                                                        QrShared<T>& sh) {
  const int64_t j0 = q * kPanel;
  QrPanel<T, VS> p = {Vs, V + j0 * L + j0, L, (int)(L - j0)};
  __syncthreads();  // the panel before is done with
  if (threadIdx.x < kPanel * kPanel) {
    const int i = threadIdx.x % kPanel, j = threadIdx.x / kPanel;
    sh.Tm[j][i] = (j <= i && i < nb) ? __ldcg(p.g + i * L + j) : Num<T>::zero();
  }
  if constexpr (VS) {
    for (int i = 0; i < kPanel; ++i) {
      const T* src = p.g + i * L;
      T* dst = Vs + i * p.len;
#pragma unroll 4
      for (int l = threadIdx.x; l < p.len; l += kThreads) {
        T v = Num<T>::zero();
        if (i < nb) v = l <= i ? (l == i ? Num<T>::one() : Num<T>::zero()) : __ldcg(src + l);
        dst[l] = v;
      }
    }
  }
  __syncthreads();
  return p;
}

// The same without waiting: V's copy to shared memory is left in flight, T in the returned entry
// (threads below kPanel^2).
template <typename T>
__device__ __forceinline__ T qr_fetch_panel(const T* __restrict__ V, int64_t L, int64_t q, int nb, T* Vs) {
  const int64_t j0 = q * kPanel;
  const T* g = V + j0 * L + j0;
  const int len = (int)(L - j0);
  for (int i = 0; i < kPanel; ++i) {
    const T* src = g + i * L;
    T* dst = Vs + i * len;
    for (int l = threadIdx.x; l < len; l += kThreads) {
      if (i < nb && l > i)
        asm volatile("cp.async.ca.shared.global [%0], [%1], %2;" ::"r"((unsigned)__cvta_generic_to_shared(dst + l)),
                     "l"(src + l), "n"(sizeof(T))
                     : "memory");
      else
        dst[l] = i < nb && l == i ? Num<T>::one() : Num<T>::zero();
    }
  }
  asm volatile("cp.async.commit_group;" ::: "memory");
  const int i = threadIdx.x % kPanel, j = threadIdx.x / kPanel;
  return j <= i && i < nb ? __ldcg(g + i * L + j) : Num<T>::zero();
}

// y = - op(T) w for the sums w of a warp's lanes; op(T) = T^H or T.
template <typename T, bool ADJ>
__device__ __forceinline__ void qr_apply_t(T (&w)[kPanel], T (&ny)[kPanel], const T (&Tm)[kPanel][kPanel], int lane) {
  const T mine = warp_sums<T, kPanel>(w, lane);  // lane l: value l >> 3
  const int i = lane >> 3;
  T y = Num<T>::zero();
#pragma unroll
  for (int j = 0; j < kPanel; ++j) {
    const T wj = shfl_t(mine, 8 * j);
    const T t = ADJ ? Num<T>::conj(Tm[j][i]) : Tm[i][j];
    y = Num<T>::fma_(t, wj, y);
  }
#pragma unroll
  for (int j = 0; j < kPanel; ++j) ny[j] = neg_t(shfl_t(y, 8 * j));
}

// x <- (I - V op(T) V^H) x on a row of Z from row kPanel q on; op(T) = T^H (factorisation) or T
// (forming Q). One warp; nb reflectors (the others are zero in Vs, skipped in global memory). xs: the
// warp's room for the row in shared memory, from which the update reads it again (null: not enough):
// read from global memory twice, the FP64 pipe waits twice (two 1296 x 1296 blocks 18.7 ms instead of
// 16.6); in registers, the variants by length spill and miss the instruction cache (20.8 ms).
template <typename T, bool VS, bool ADJ>
__device__ __forceinline__ void qr_apply_panel(T* __restrict__ x, const QrPanel<T, VS>& p, int nb,
                                               const T (&Tm)[kPanel][kPanel], int lane, T* __restrict__ xs) {
  T w[kPanel], ny[kPanel];
#pragma unroll
  for (int i = 0; i < kPanel; ++i) w[i] = Num<T>::zero();
#pragma unroll 4
  for (int l = lane; l < p.len; l += 32) {
    const T xv = ldcg_t(x + l);
    if (VS && xs) xs[l] = xv;
#pragma unroll
    for (int i = 0; i < kPanel; ++i)
      if (VS || i < nb) w[i] = Num<T>::fmac(xv, p.v(i, l), w[i]);
  }
  qr_apply_t<T, ADJ>(w, ny, Tm, lane);
#pragma unroll 4
  for (int l = lane; l < p.len; l += 32) {
    T xv = VS && xs ? xs[l] : ldcg_t(x + l);
#pragma unroll
    for (int j = 0; j < kPanel; ++j)
      if (VS || j < nb) xv = Num<T>::fma_(ny[j], p.v(j, l), xv);
    x[l] = xv;
  }
  __syncwarp();
}

// The reflector of a column from alpha (its entry on the diagonal) and xn = |x below|^2 (LAPACK
// larfg: beta real, tau = (beta - alpha) / beta, v = x / (alpha - beta) with v_0 = 1); a column
// that is already reduced gets tau = 0, sc = 0. With s = |beta|: tau = 1 + |Re alpha| / s (and
// sign(Re alpha) Im alpha / s), 1 / (alpha - beta) = conj(alpha - beta) / ((s + |Re alpha|)^2 + (Im alpha)^2);
// ts = conj(tau sc) = -1 / beta.
// All panels wait for this chain: 12 FP64 instructions of 64 cycles for a real column (the square
// root by a step of Householder's iteration of third order as in rsqrt64 of yb_jacobi.cuh, the reciprocal by
// one of the hyperpower iteration of third order, z (1 + e + e^2) with e = 1 - d z (M. Altman, Pacific J.
// Math. 10, 1960), both from an FP32 start with e below 5e-7: 1e-19 is left; scalings and signs by
// integers; results within 2^-50 of the exact ones for this alpha and xn) instead of 28; 2.7 k -> 1.6 k cycles a column with the updates' factors. Norms whose squares
// leave 2^+-900 take the library's functions.
template <typename T>
__device__ __forceinline__ void qr_scalars(T alpha, double xn, T& tau, T& sc, T& diag, double& ts) {
  double ar, ai;
  if constexpr (Num<T>::cplx) { ar = alpha.x; ai = alpha.y; } else { ar = alpha; ai = 0.0; }
  if (xn == 0.0 && ai == 0.0) {
    tau = Num<T>::zero();
    sc = Num<T>::zero();
    diag = alpha;
    ts = 0.0;
    return;
  }
  const double n2 = Num<T>::cplx ? fma(ar, ar, fma(ai, ai, xn)) : fma(ar, ar, xn);
  const bool ng = __double_as_longlong(ar) < 0;  // the sign of Re alpha, of -0 too
  // s = sqrt(n2), is = 1 / s, t1 = |ar| / s + 1, id = 1 / (s + |ar|); complex: id and fi = (s + |ar|, ai) / ((s + |ar|)^2 + ai^2)
  double s, is, t1, id, fi = 0.0;
  const int ex = (int)((__double_as_longlong(n2) >> 52) & 0x7ff) - 1023;
  if (ex > -900 && ex < 900) {
    const int h = ex >> 1;  // n2 = m 4^h, m in [1, 4)
    const double m = times_pow2(n2, -2 * h), a1 = times_pow2(neg_if(ar, ng), -h);
    const double y0 = widen64(rsqrtf(trunc32(m)));
    const double q0 = m * y0;
    const double e = fma(-q0, y0, 1.0);
    const double t = e * fma(e, 0.375, 0.5);
    const double y = fma(y0, t, y0), q = fma(q0, t, q0);  // 1 / sqrt(m), sqrt(m)
    const double d1 = q + a1;  // in [1, 4)
    t1 = fma(a1, y, 1.0);
    const double im = Num<T>::cplx ? times_pow2(ai, -h) : 0.0;
    const double d = Num<T>::cplx ? fma(d1, d1, im * im) : d1;
    double z = widen64(__frcp_rn(trunc32(d)));
    const double ez = fma(-d, z, 1.0);
    z = fma(z, fma(ez, ez, ez), z);
    s = times_pow2(q, h);
    is = times_pow2(y, -h);
    id = times_pow2(Num<T>::cplx ? z * d1 : z, -h);
    if constexpr (Num<T>::cplx) fi = times_pow2(im * z, -h);
  } else {
    s = sqrt(n2);
    is = 1.0 / s;
    t1 = fma(fabs(ar), is, 1.0);
    const double t = ai / (s + fabs(ar));
    id = 1.0 / ((s + fabs(ar)) * fma(t, t, 1.0));
    fi = t * id;
  }
  ts = neg_if(is, ng);
  if constexpr (Num<T>::cplx) {
    tau = make_double2(t1, ai * ts);
    sc = make_double2(neg_if(id, ng), neg_if(fi, true));
    diag = make_double2(neg_if(s, !ng), 0.0);
  } else {
    tau = t1;
    sc = neg_if(id, ng);
    diag = neg_if(s, !ng);
  }
}

__device__ __forceinline__ double qr_fma_re(double a, double x, double acc) { return fma(a, x, acc); }
__device__ __forceinline__ double2 qr_fma_re(double a, double2 x, double2 acc) {
  return make_double2(fma(a, x.x, acc.x), fma(a, x.y, acc.y));
}

// Column i of T from tau and S_ci = v_c^H v_i, c < i: T_ci = -tau sum_{c <= d < i} T_cd S_di.
template <typename T>
__device__ __forceinline__ void qr_t_column(T (&Tm)[kPanel][kPanel], const T (&S)[kPanel], T tau, int i) {
#pragma unroll
  for (int c = 0; c < kPanel; ++c) {
    if (c >= i) continue;
    T a = Num<T>::zero();
#pragma unroll
    for (int d = 0; d < kPanel; ++d)
      if (d >= c && d < i) a = Num<T>::fma_(Tm[c][d], S[d], a);
    Tm[c][i] = neg_t(Num<T>::mul(tau, a));
  }
  Tm[i][i] = tau;
}

// Updates panel `next` (nb columns) by panel next - 1, once that is published, and factors it; its
// rows from l0 on lie in registers: thread t holds rows l0 + t + 256 r, r < R (warps whose rows lie
// beyond the column do no arithmetic: the FP64 pipe is shared). Writes R's entries to Z and the
// reflectors and T to V. Warp 0 does a step's scalars, the last warp T's columns.
template <typename T, bool VS, int R, int CL>
__device__ __forceinline__ void qr_factor_panel(T* __restrict__ Z, T* __restrict__ V, int64_t L, int64_t next, int nb,
                                                QrPanel<T, VS>& p, T* Vs, QrShared<T>& sh,
                                                const unsigned long long* ready, unsigned long long* err) {
  constexpr int kT = CL * kThreads, kW = CL * kWarps;
  const int crank = CL == 1 ? 0 : (int)cooperative_groups::this_cluster().block_rank();
  const int t = threadIdx.x + crank * kThreads, lane = t & 31, gwarp = t >> 5, warp = threadIdx.x >> 5;
  const bool has_p = next > 0;
  const int64_t c0 = next * kPanel, l0 = has_p ? c0 - kPanel : 0;
  const int off = (int)(c0 - l0), len = (int)(L - l0);
  const int live = (len - 32 * gwarp + kT - 1) / kT;  // passes with rows of this warp (may be <= 0)
  qr_sync<CL>();  // the columns as the warps left them
  T x[R][kPanel];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < kPanel; ++c) {
      const int l = t + kT * r;
      x[r][c] = (l < len && c < nb) ? ldcg_t(Z + (c0 + c) * L + l0 + l) : Num<T>::zero();
    }
  if (has_p) {
    qr_wait(ready, (unsigned long long)next, err);
    // V's entries of the thread's rows in registers where they fit, else the panel in shared memory
    // (else the caller brings it there afterwards)
    constexpr bool kRegs = R * (int)sizeof(T) <= 48;
    const T* g = V + l0 * (L + 1);
    const int yi = (lane & 15) >> 2, yc = lane & 3;
    T v[kRegs ? R : 1][kPanel], tm[kPanel];
    if constexpr (kRegs) {
#pragma unroll
      for (int r = 0; r < R; ++r)
#pragma unroll
        for (int i = 0; i < kPanel; ++i) {
          const int l = t + kT * r;
          v[r][i] = l >= len || l < i ? Num<T>::zero() : l == i ? Num<T>::one() : __ldcg(g + i * L + l);
        }
    } else {
      p = qr_load_panel<T, VS>(V, L, next - 1, kPanel, Vs, sh);
    }
#pragma unroll
    for (int j = 0; j < kPanel; ++j) tm[j] = j <= yi ? __ldcg(g + yi * L + j) : Num<T>::zero();
    auto entry = [&](int r, int i) {
      if constexpr (kRegs) return v[r][i];
      const int l = t + kT * r;
      return l < len ? p.v(i, l) : Num<T>::zero();
    };
    T w[kPanel * kPanel];
#pragma unroll
    for (int e = 0; e < kPanel * kPanel; ++e) w[e] = Num<T>::zero();
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (r < live) {
#pragma unroll
        for (int i = 0; i < kPanel; ++i) {
          const T ve = entry(r, i);
#pragma unroll
          for (int c = 0; c < kPanel; ++c) w[i * kPanel + c] = Num<T>::fmac(x[r][c], ve, w[i * kPanel + c]);
        }
      }
    T mine = Num<T>::zero();
    if (live > 0) mine = warp_sums<T, kPanel * kPanel>(w, lane);  // lane l: value l >> 1
    if (!(lane & 1)) qr_put<CL>(&sh.part[0][gwarp][lane >> 1], mine);
    qr_sync<CL>();
    // the warps' sums: 32 / kW values a warp, then y_ic = sum_j conj(T_ji) w_jc at lane 4 i + c
    if (warp < kW / 2) {
      const int e = (lane + 32 * warp) / kW;
      T s = sh.part[0][lane % kW][e];
#pragma unroll
      for (int o = kW / 2; o >= 1; o >>= 1) s = Num<T>::add(s, shfl_xor_t(s, o));
      if (lane % kW == 0) sh.sum[e] = s;
    }
    __syncthreads();
    if (live > 0) {
      T y = Num<T>::zero();
#pragma unroll
      for (int j = 0; j < kPanel; ++j) y = Num<T>::fma_(Num<T>::conj(tm[j]), sh.sum[4 * j + yc], y);
      y = neg_t(y);
#pragma unroll
      for (int j = 0; j < kPanel; ++j) {
        T ny[kPanel];
#pragma unroll
        for (int cc = 0; cc < kPanel; ++cc) ny[cc] = shfl_t(y, 4 * j + cc);
#pragma unroll
        for (int r = 0; r < R; ++r)
          if (r < live) {
            const T ve = entry(r, j);
#pragma unroll
            for (int cc = 0; cc < kPanel; ++cc) x[r][cc] = Num<T>::fma_(ny[cc], ve, x[r][cc]);
          }
      }
    }
  }
  T Tm[kPanel][kPanel];  // kept by the last warp
#pragma unroll
  for (int i = 0; i < kPanel; ++i)
#pragma unroll
    for (int j = 0; j < kPanel; ++j) Tm[i][j] = Num<T>::zero();
#pragma unroll
  for (int i = 0; i < kPanel; ++i) {
    if (i >= nb) break;
    const int b = (i & 1) ^ 1;  // part[0] may still be read by the update above
    // below row j: |x_i|^2, x_i^H x_c (c > i), v_c^H x_i (c < i)
    T a[kPanel];
#pragma unroll
    for (int c = 0; c < kPanel; ++c) a[c] = Num<T>::zero();
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (r < live && (r > 0 || t > off + i)) {
#pragma unroll
        for (int c = 0; c < kPanel; ++c)
          a[c] = c >= i ? Num<T>::fmac(x[r][c], x[r][i], a[c]) : Num<T>::fmac(x[r][i], x[r][c], a[c]);
      }
    if (t == off + i) {
#pragma unroll
      for (int c = 0; c < kPanel; ++c) qr_put<CL>(&sh.row[b][c], x[0][c]);
    }
    T mine = Num<T>::zero();
    if (live > 0) mine = warp_sums<T, kPanel>(a, lane);  // lane l: value l >> 3
    if (!(lane & 7)) qr_put<CL>(&sh.part[b][gwarp][lane >> 3], mine);
    qr_sync<CL>();
    T s = Num<T>::zero();
    if (warp == 0 || warp == kWarps - 1) {
      s = sh.part[b][lane & 7][lane >> 3];
#pragma unroll
      for (int u = 1; u < CL; ++u) s = Num<T>::add(s, sh.part[b][(lane & 7) + u * kWarps][lane >> 3]);
#pragma unroll
      for (int o = 4; o >= 1; o >>= 1) s = Num<T>::add(s, shfl_xor_t(s, o));  // lane l: total l >> 3
    }
    if (warp == 0) {
      const T d = shfl_t(s, 8 * i);
      double xn;
      if constexpr (Num<T>::cplx) xn = d.x; else xn = d;
      T tau, sc, diag;
      double ts;
      qr_scalars<T>(sh.row[b][i], xn, tau, sc, diag, ts);
      // x_c -= conj(tau) (v^H x_c) v, v = sc x_i below row j; lane 8 c
      const T g = neg_t(qr_fma_re(ts, s, Num<T>::mul(Num<T>::conj(tau), sh.row[b][lane >> 3])));
      const T f = Num<T>::mul(g, sc);
      if (!(lane & 7)) {
        sh.add[b][lane >> 3] = g;
        sh.f[b][lane >> 3] = f;
      }
      if (lane == 0) { sh.sc[b] = sc; sh.diag[b] = diag; sh.tau[b] = tau; }
    }
    __syncthreads();
    if (warp == kWarps - 1) {
      // S_ci = v_c^H v_i = conj(v_c[j]) + sc sum below
      T S[kPanel];
#pragma unroll
      for (int c = 0; c < kPanel; ++c)
        S[c] = c < i ? Num<T>::fma_(sh.sc[b], shfl_t(s, 8 * c), Num<T>::conj(sh.row[b][c])) : Num<T>::zero();
      qr_t_column<T>(Tm, S, sh.tau[b], i);
    }
    const T sc = sh.sc[b];
#pragma unroll
    for (int r = 0; r < R; ++r)
      if (r < live && (r > 0 || t > off + i)) {
#pragma unroll
        for (int c = 0; c < kPanel; ++c)
          if (c > i) x[r][c] = Num<T>::fma_(sh.f[b][c], x[r][i], x[r][c]);
        x[r][i] = Num<T>::mul(sc, x[r][i]);
      }
    if (t == off + i) {
#pragma unroll
      for (int c = 0; c < kPanel; ++c) {
        if (c > i) x[0][c] = Num<T>::add(x[0][c], sh.add[b][c]);
        if (c == i) x[0][c] = sh.diag[b];
      }
    }
  }
  if (threadIdx.x == kThreads - 1) {
#pragma unroll
    for (int i = 0; i < kPanel; ++i)
#pragma unroll
      for (int j = 0; j < kPanel; ++j) sh.Tn[i][j] = Tm[i][j];
  }
  __syncthreads();
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < kPanel; ++c) {
      const int l = t + kT * r;
      if (l >= len || c >= nb) continue;
      const int64_t at = (c0 + c) * L + l0 + l;
      if (r == 0 && t <= off + c) {
        Z[at] = x[r][c];
        if (t >= off) V[at] = sh.Tn[t - off][c];
      } else {
        V[at] = x[r][c];
      }
    }
}

// The same for columns too long for registers: a warp per column, in global memory.
template <typename T, bool VS>
__device__ void qr_factor_panel_long(T* __restrict__ Z, T* __restrict__ V, int64_t L, int64_t next, int nb, bool has_p,
                                     const QrPanel<T, VS>& p, QrShared<T>& sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t c0 = next * kPanel;
  T* z = Z + (c0 + warp) * L;
  if (has_p && warp < nb) qr_apply_panel<T, VS, true>(z + c0 - kPanel, p, kPanel, sh.Tm, lane, (T*)nullptr);
  __syncthreads();
  T Tm[kPanel][kPanel];
#pragma unroll
  for (int i = 0; i < kPanel; ++i)
#pragma unroll
    for (int j = 0; j < kPanel; ++j) Tm[i][j] = Num<T>::zero();
#pragma unroll
  for (int i = 0; i < kPanel; ++i) {
    if (i >= nb) break;
    const int64_t j = c0 + i;
    const T* xi = Z + j * L;
    T* vi = V + j * L;
    const T* other = warp >= i ? z : V + (c0 + warp) * L;
    T a = Num<T>::zero();
    if (warp < nb)
      for (int64_t l = j + 1 + lane; l < L; l += 32) {
        const T u = ldcg_t(other + l), xv = ldcg_t(xi + l);
        a = warp >= i ? Num<T>::fmac(u, xv, a) : Num<T>::fmac(xv, u, a);
      }
    warp_sum_t<T>(a);
    if (lane == 0 && warp < nb) {
      sh.part[0][0][warp] = a;
      sh.row[0][warp] = ldcg_t(other + j);
    }
    __syncthreads();
    double xn;
    const T ti = sh.part[0][0][i];
    if constexpr (Num<T>::cplx) xn = ti.x; else xn = ti;
    T tau, sc, diag, S[kPanel];
    double ts;
    qr_scalars<T>(sh.row[0][i], xn, tau, sc, diag, ts);
#pragma unroll
    for (int c = 0; c < kPanel; ++c)
      S[c] = c < i ? Num<T>::fma_(sc, sh.part[0][0][c], Num<T>::conj(sh.row[0][c])) : Num<T>::zero();
    qr_t_column<T>(Tm, S, tau, i);
    if (warp > i && warp < nb) {
      const T g = neg_t(qr_fma_re(ts, sh.part[0][0][warp], Num<T>::mul(Num<T>::conj(tau), sh.row[0][warp])));
      const T f = Num<T>::mul(g, sc);
      for (int64_t l = j + 1 + lane; l < L; l += 32) z[l] = Num<T>::fma_(f, ldcg_t(xi + l), ldcg_t(z + l));
      if (lane == 0) z[j] = Num<T>::add(sh.row[0][warp], g);
    }
    if (warp == i)
      for (int64_t l = j + 1 + lane; l < L; l += 32) vi[l] = Num<T>::mul(sc, ldcg_t(xi + l));
    __syncthreads();
    if (warp == i && lane == 0) z[j] = diag;
  }
  if (warp < nb && lane <= warp) {
    T tv = Num<T>::zero();
#pragma unroll
    for (int j = 0; j < kPanel; ++j)
#pragma unroll
      for (int c = 0; c < kPanel; ++c)
        if (j == lane && c == warp) tv = Tm[j][c];
    V[(c0 + warp) * L + c0 + lane] = tv;
  }
  __syncthreads();
}

// All steps of block r for the CTAs of a group (VS: the panels' V fits in shared memory; MAXR:
// passes of 256 rows a panel may take in registers). False after a barrier timeout.
template <typename T, typename T32, int MAXR, bool VS, int CL>
__device__ bool qr_block(T* __restrict__ work, T32* __restrict__ work32, const int64_t* __restrict__ r, int group, int rank,
                         unsigned long long* ready, unsigned long long* ctrl, T* Vs,
                         int smem_elems, QrShared<T>& sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t gt = (int64_t)rank * kThreads + threadIdx.x, ngt = (int64_t)group * kThreads;
  const int64_t k = r[R_K], L = r[R_LQ];
  T* Z = work + r[R_Z];
  T* V = work + r[R_VQ];
  T* tau = work + r[R_TAU];
  T* RR = work + r[R_RR];
  const int64_t np = (k + kPanel - 1) / kPanel;
  T* xs = VS && (kPanel + kWarps) * L <= smem_elems ? Vs + (kPanel + warp) * L : nullptr;
  auto width = [&](int64_t q) { return (int)min((int64_t)kPanel, k - q * kPanel); };
  // factorisation: panel q applied to the later panels of this owner (a cluster of CL CTAs), panel
  // q + 1 factored by its owner
  const int owner = rank / CL, owners = group / CL, crank = rank % CL;
  for (int64_t q = -1; q + 1 < np; ++q) {
    const int64_t next = q + 1;
    const int64_t mine = next + ((owner - next) % owners + owners) % owners;  // first own panel from `next` on
    if (mine >= np) break;  // nothing of this owner's is left
    QrPanel<T, VS> p = {Vs, V, L, 0};
    if (mine == next) {
      const int64_t passes = (L - (q >= 0 ? q * kPanel : 0) + CL * kThreads - 1) / (CL * kThreads);
      const int nb = width(next);
#define YB_PANEL(R) qr_factor_panel<T, VS, (R <= MAXR ? R : 1), CL>(Z, V, L, next, nb, p, Vs, sh, ready, ctrl + C_ERR)
      if (passes <= 1) YB_PANEL(1);
      else if (MAXR >= 2 && passes <= 2) YB_PANEL(2);
      else if (CL > 1 && MAXR >= 3 && passes <= 3) YB_PANEL(3);
      else if (CL == 1 && MAXR >= 4 && passes <= 4) YB_PANEL(4);
      else if (MAXR >= 6 && passes <= 6) YB_PANEL(6);
      else if (MAXR >= 11 && passes <= 11) YB_PANEL(11);
      else {
        if (q >= 0) {
          qr_wait(ready, (unsigned long long)next, ctrl + C_ERR);
          p = qr_load_panel<T, VS>(V, L, q, kPanel, Vs, sh);
        }
        qr_sync<CL>();
        if (crank == 0) qr_factor_panel_long<T, VS>(Z, V, L, next, nb, q >= 0, p, sh);
      }
#undef YB_PANEL
      qr_sync<CL>();
      if (threadIdx.x == 0 && crank == 0) {
        __threadfence();
        atomicMax(ready, (unsigned long long)(next + 1));
      }
    } else if (q >= 0) {
      qr_wait(ready, (unsigned long long)next, ctrl + C_ERR);
      p = qr_load_panel<T, VS>(V, L, q, kPanel, Vs, sh);
    }
    if (q >= 0) {
      if (mine == next && next + owners < np) p = qr_load_panel<T, VS>(V, L, q, kPanel, Vs, sh);
      // this owner's later panels: a column per warp. In a cluster a column stays with its warp: CTA
      // j % CL takes column j of a panel.
      const int64_t first = mine == next ? mine + owners : mine;
      if constexpr (CL == 1) {
        for (int64_t e = warp;; e += kWarps) {
          const int64_t pan = first + (e / kPanel) * owners, c = pan * kPanel + e % kPanel;
          if (pan >= np) break;
          if (c < k) qr_apply_panel<T, VS, true>(Z + c * L + q * kPanel, p, kPanel, sh.Tm, lane, xs);
        }
      } else {
        constexpr int kCols = kPanel / CL, kTurn = kWarps / kCols;
        const int64_t o = (first - owner) / owners, turn = warp / kCols;
        const int j = crank + CL * (warp % kCols);
        for (int64_t pan = first + ((turn - o) % kTurn + kTurn) % kTurn * owners; pan < np; pan += kTurn * owners) {
          const int64_t c = pan * kPanel + j;
          if (c < k) qr_apply_panel<T, VS, true>(Z + c * L + q * kPanel, p, kPanel, sh.Tm, lane, xs);
        }
      }
    }
  }
  if (!qr_all<CL>(grid_barrier(ctrl, group))) return false;
  // R rows, tau, the FP32 start
  for (int64_t e = gt; e < k * k; e += ngt) {
    const int64_t i = e / k, c = e - i * k;
    const T v = (c >= i) ? ldcg_t(Z + c * L + i) : Num<T>::zero();
    RR[e] = v;
    if (work32) {  // no FP32 Jacobi start for yb_qr
      work32[r[R_X32] + e] = to32(v);
      work32[r[R_W32] + e] = (i == c) ? Num<T32>::one() : Num<T32>::zero();
    }
  }
  for (int64_t e = gt; e < k; e += ngt) tau[e] = ldcg_t(V + e * L + e);  // T's diagonal
  if (!qr_all<CL>(grid_barrier(ctrl, group))) return false;
  // Q's columns: row c of Z becomes (H_0 ... H_c e_c)^T, the panels backwards
  // Columns rank, rank + group, .. of a CTA, dealt to its warps in turn: every CTA has columns of all
  // panels (with 8 neighbouring columns a CTA, the last of 54 did all 108 panels of k = 432 alone).
  const int64_t top = rank < k ? rank + (k - 1 - rank) / group * group : -1;
  auto columns = [&](int64_t q, const QrPanel<T, VS>& p, const T(&Tm)[kPanel][kPanel]) {
    for (int64_t c = rank + (int64_t)group * warp; c < k; c += (int64_t)group * kWarps) {
      if (c < q * kPanel) continue;
      T* x = Z + c * L;
      if (c / kPanel == q) {
        for (int64_t l = lane; l < L; l += 32) x[l] = (l == c) ? Num<T>::one() : Num<T>::zero();
        __syncwarp();
      }
      qr_apply_panel<T, VS, false>(x + q * kPanel, p, width(q), Tm, lane, xs);
    }
  };
  const int64_t q0 = top < 0 ? -1 : top / kPanel;  // the first panel with columns of this CTA
  if (VS && (2 * kPanel + kWarps) * L <= smem_elems) {
    // two panels in shared memory, the next one's copy in flight (waited for in turn: yb_qr of two
    // 540 x 432 blocks 2.64 ms instead of 2.48, yb_svd_qr of two 1296 x 1296 16.6 instead of 16.0)
    T* buf[2] = {Vs, Vs + (kPanel + kWarps) * L};
    T tm = Num<T>::zero();
    if (q0 >= 0) tm = qr_fetch_panel<T>(V, L, q0, width(q0), buf[q0 & 1]);
    for (int64_t q = q0; q >= 0; --q) {
      const int h = (int)(q & 1);
      if (threadIdx.x < kPanel * kPanel) sh.Tq[h][threadIdx.x / kPanel][threadIdx.x % kPanel] = tm;
      asm volatile("cp.async.wait_group 0;" ::: "memory");
      __syncthreads();  // panel q is there; panel q + 1 is done with
      if (q > 0) tm = qr_fetch_panel<T>(V, L, q - 1, kPanel, buf[h ^ 1]);
      columns(q, QrPanel<T, VS>{buf[h], V + q * kPanel * (L + 1), L, (int)(L - q * kPanel)}, sh.Tq[h]);
    }
  } else {
    for (int64_t q = q0; q >= 0; --q)
      columns(q, qr_load_panel<T, VS>(V, L, q, width(q), Vs, sh), sh.Tm);
  }
  return qr_all<CL>(grid_barrier(ctrl, group));
}

template <typename T, typename T32, int MAXR, int CL>
__device__ __forceinline__ void
    qr_blocks(T* __restrict__ work, T32* __restrict__ work32, const int64_t* __restrict__ blocks, int n_blocks,
                  int group, unsigned long long* __restrict__ qctrl, int smem_elems) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Vs = reinterpret_cast<T*>(smem_raw);
  __shared__ QrShared<T> sh;
  const int g = blockIdx.x / group, rank = blockIdx.x % group;
  const int n_groups = gridDim.x / group;
  // qctrl: [n_blocks ready counters][C_REC words per group]
  unsigned long long* ctrl = qctrl + n_blocks + (int64_t)g * C_REC;
  if constexpr (CL > 1) {
    // launched without the clusters, a panel's owner would write to shared memory that is not there
    if (cooperative_groups::this_cluster().num_blocks() != CL) {
      if (threadIdx.x == 0) atomicExch(ctrl + C_ERR, 1ull);
      return;
    }
    qr_sync<CL>();  // every CTA of the cluster runs before its shared memory is written
  }
  for (int b = g; b < n_blocks; b += n_groups) {
    const int64_t* r = blocks + (int64_t)b * YB_SVD_REC;
    if (!r[R_QR]) continue;
    bool ok;
#define YB_BLOCK(MAX, VS, C) \
  qr_block<T, T32, MAX, VS, C>(work, work32, r, group, rank, qctrl + b, ctrl, Vs, smem_elems, sh)
    if constexpr (CL > 1) {
      ok = r[R_LQ] <= kPairRows ? YB_BLOCK(1, true, 1)
           : kPanel * r[R_LQ] <= smem_elems ? YB_BLOCK(MAXR, true, CL) : YB_BLOCK(MAXR, false, CL);
      ok = qr_all<CL>(ok);
    } else {
      ok = kPanel * r[R_LQ] <= smem_elems ? YB_BLOCK(MAXR, true, 1) : YB_BLOCK(MAXR, false, 1);
    }
#undef YB_BLOCK
    if (!ok) return;
  }
}

template <typename T, typename T32, int MAXR, int PER_SM>
__global__ void __launch_bounds__(kThreads, PER_SM)
    svd_qr_kernel(T* __restrict__ work, T32* __restrict__ work32, const int64_t* __restrict__ blocks, int n_blocks,
                  int group, unsigned long long* __restrict__ qctrl, int smem_elems) {
  qr_blocks<T, T32, MAXR, 1>(work, work32, blocks, n_blocks, group, qctrl, smem_elems);
}

template <typename T, typename T32, int MAXR>
__global__ void __cluster_dims__(kMaxCl, 1, 1) __launch_bounds__(kThreads, 1)
    svd_qr_cluster_kernel(T* __restrict__ work, T32* __restrict__ work32, const int64_t* __restrict__ blocks,
                          int n_blocks, int group, unsigned long long* __restrict__ qctrl, int smem_elems) {
  qr_blocks<T, T32, MAXR, kMaxCl>(work, work32, blocks, n_blocks, group, qctrl, smem_elems);
}

// Up to one block per eight SMs: clusters of CL CTAs, one CTA per SM, panels of up to 6 passes of
// CL x 256 rows in registers, 200 KB of shared memory. Up to one block per SM: the same without
// clusters, up to 11 (complex: 6) passes of 256 rows. More blocks than SMs, one CTA each: two CTAs
// per SM (the pipe of one is idle while the other waits) with fewer passes and half the shared
// memory. `launched` false: the clusters do not fit the device, nothing was launched.
template <typename T, typename T32, int MAXR, int PER_SM, int CL>
int qr_launch(void* work, void* work32, const int64_t* blocks, int n_blocks, int64_t* qctrl,
              int qctrl_words, int sms, cudaStream_t s, bool* launched) {
  void (*kernel)(T*, T32*, const int64_t*, int, int, unsigned long long*, int);
  if constexpr (CL > 1) kernel = svd_qr_cluster_kernel<T, T32, MAXR>;
  else kernel = svd_qr_kernel<T, T32, MAXR, PER_SM>;
  const int smem = 200 * 1024 / PER_SM;
  cudaLaunchAttribute attr[2] = {};
  attr[0].id = cudaLaunchAttributeCooperative;
  attr[0].val.cooperative = 1;
  attr[1].id = cudaLaunchAttributeClusterDimension;
  attr[1].val.clusterDim = {CL, 1, 1};
  cudaLaunchConfig_t cfg = {};
  cfg.gridDim = dim3((unsigned)(sms / CL * CL));
  cfg.blockDim = dim3(kThreads);
  cfg.dynamicSmemBytes = (size_t)smem;
  cfg.stream = s;
  cfg.attrs = attr;
  cfg.numAttrs = CL > 1 ? 2 : 1;
  *launched = false;
  int resident = 0;  // CTAs of the device, clusters when CL > 1
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) {
    if constexpr (CL > 1) e = cudaOccupancyMaxActiveClusters(&resident, kernel, &cfg);
    else e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&resident, kernel, kThreads, smem);
  }
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  const int capacity = CL > 1 ? CL * resident : sms * (resident < 1 ? 1 : resident);
  int group = capacity / n_blocks / CL * CL;
  if (CL > 1 && group * n_blocks * 8 < 7 * sms) return YB_OK;
  group = group < 1 ? 1 : group;
  int n_groups = capacity / group;
  if (n_groups > n_blocks) n_groups = n_blocks;
  if ((int64_t)n_groups * C_REC + n_blocks > qctrl_words) n_groups = (qctrl_words - n_blocks) / C_REC;
  if (n_groups < 1) return YB_ERR_INVALID;
  e = cudaMemsetAsync(qctrl, 0, sizeof(int64_t) * ((size_t)n_groups * C_REC + n_blocks), s);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  cfg.gridDim = dim3((unsigned)(n_groups * group));
  e = cudaLaunchKernelEx(&cfg, kernel, (T*)work, (T32*)work32, blocks, n_blocks, group, (unsigned long long*)qctrl,
                         smem / (int)sizeof(T));
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  *launched = true;
  return YB_OK;
}

template <typename T, typename T32>
int qr_factor(void* work, void* work32, const int64_t* blocks, int n_blocks, int64_t* qctrl,
              int qctrl_words, cudaStream_t s) {
  constexpr int kMany = Num<T>::cplx ? 2 : 4, kFew = Num<T>::cplx ? 6 : 11;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  bool launched = false;
  if (n_blocks * 8 <= sms) {
    const int st = qr_launch<T, T32, 6, 1, kMaxCl>(work, work32, blocks, n_blocks, qctrl, qctrl_words, sms, s,
                                                   &launched);
    if (st != YB_OK || launched) return st;
  }
  return n_blocks <= sms
             ? qr_launch<T, T32, kFew, 1, 1>(work, work32, blocks, n_blocks, qctrl, qctrl_words, sms, s, &launched)
             : qr_launch<T, T32, kMany, 2, 1>(work, work32, blocks, n_blocks, qctrl, qctrl_words, sms, s, &launched);
}

}  // namespace
}  // namespace yb
