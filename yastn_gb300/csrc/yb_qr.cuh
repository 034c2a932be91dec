// Blocked Householder QR of all blocks in one cooperative launch (yb_svd_qr, yb_qr).
//
// Z holds the columns of M as rows. Groups of CTAs take a block at a time; panels of kPanel
// columns belong to the CTAs of a group in turn. When panel q is published, every CTA brings its
// V and T to shared memory and applies I - V T^H V^H to its own later panels; the owner of panel
// q + 1 takes that one first: its columns live in registers (256 threads, a row of the panel per
// thread and pass), are updated by panel q, factored, and published through the block's ready
// counter. The waits are bounded (error word of the group). After the factorisation (a group
// barrier) R's rows and the FP32 start are written, and every warp forms its own columns of Q by
// the panels backwards.
//
// What bounds it: the path through the panels (each update and factorisation runs on one SM,
// whose FP64 pipe issues a warp instruction every 19 cycles, 64 for a single warp) and, for large
// blocks, the FP64 work of the updates. A panel of w columns costs that path a fixed part (publish,
// wait, V's load, w reductions and scalars) and FMAs that grow with w^2: w = 4 is the shortest per
// column by the count of instructions from L = 100 to 2000. A reflector's norm, its inner products
// with the panel's other columns and those that T needs are one reduction, and one warp does the
// scalars (done by all eight they cost more than the panel's FMAs at L = 100).
//
// Measured (GB300; before: a warp per column, one reflector at a time, published by itself): yb_qr
// of two 540 x 432 blocks 7.8 -> 3.1 ms; yb_svd_qr of two 432 x 432 blocks 6.2 -> 2.7 ms, two
// 1296 x 1296 62 -> 19 ms (10.6 ms at the DFMA rate), nine of 24..93 0.73 -> 0.47 ms, five complex
// ones of 31 x 24 .. 78 x 60 0.68 -> 0.54 ms; 595 blocks of 42..60 2.6 -> 1.4 ms.
#pragma once
#include "yb_svd_common.cuh"

namespace yb {
namespace {

constexpr int kPanel = 4;

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
// caller carries on with whatever it reads: the host sees the error word and fails).
__device__ __forceinline__ void qr_wait(const unsigned long long* flag, unsigned long long target,
                                        unsigned long long* err) {
  if (threadIdx.x == 0) {
    long long spins = 0;
    while (*(volatile const unsigned long long*)flag < target) {
      if (spins > 16) __nanosleep(32);
      if (++spins > kSpinLimit) {
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
  T part[2][kWarps][kPanel * kPanel];
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

// x <- (I - V op(T) V^H) x on a row of Z from row kPanel q on; op(T) = T^H (factorisation) or T
// (forming Q). One warp; nb reflectors (the others are zero in Vs, skipped in global memory).
template <typename T, bool VS, bool ADJ>
__device__ __forceinline__ void qr_apply_panel(T* __restrict__ x, const QrPanel<T, VS>& p, int nb, const QrShared<T>& sh,
                                               int lane) {
  T w[kPanel];
#pragma unroll
  for (int i = 0; i < kPanel; ++i) w[i] = Num<T>::zero();
#pragma unroll 4
  for (int l = lane; l < p.len; l += 32) {
    const T xv = ldcg_t(x + l);
#pragma unroll
    for (int i = 0; i < kPanel; ++i)
      if (VS || i < nb) w[i] = Num<T>::fmac(xv, p.v(i, l), w[i]);
  }
  const T mine = warp_sums<T, kPanel>(w, lane);  // lane l: value l >> 3
  const int i = lane >> 3;
  T y = Num<T>::zero();
#pragma unroll
  for (int j = 0; j < kPanel; ++j) {
    const T wj = shfl_t(mine, 8 * j);
    const T t = ADJ ? Num<T>::conj(sh.Tm[j][i]) : sh.Tm[i][j];
    y = Num<T>::fma_(t, wj, y);
  }
  T ny[kPanel];
#pragma unroll
  for (int j = 0; j < kPanel; ++j) ny[j] = Num<T>::scale(-1, shfl_t(y, 8 * j));
#pragma unroll 4
  for (int l = lane; l < p.len; l += 32) {
    T xv = ldcg_t(x + l);
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
// sign(Re alpha) Im alpha / s), 1 / (alpha - beta) = conj(alpha - beta) / ((s + |Re alpha|)^2 + (Im alpha)^2).
// The square root and the two reciprocals are refined from FP32 starts (about 20 FP64
// instructions instead of 60; the FP64 pipe issues one per 64 cycles and warp); norms whose
// squares leave 2^+-900 take the library's.
template <typename T>
__device__ __forceinline__ void qr_scalars(T alpha, double xn, T& tau, T& sc, T& diag) {
  double ar, ai;
  if constexpr (Num<T>::cplx) { ar = alpha.x; ai = alpha.y; } else { ar = alpha; ai = 0.0; }
  if (xn == 0.0 && ai == 0.0) {
    tau = Num<T>::zero();
    sc = Num<T>::zero();
    diag = alpha;
    return;
  }
  const double n2 = Num<T>::cplx ? fma(ar, ar, fma(ai, ai, xn)) : fma(ar, ar, xn);
  // s = sqrt(n2), 1 / s, 1 / (s + |ar|); complex: re and im = (s + |ar|, ai) / ((s + |ar|)^2 + ai^2)
  double s, is, id, fi = 0.0;
  const int ex = (int)((__double_as_longlong(n2) >> 52) & 0x7ff) - 1023;
  if (ex > -900 && ex < 900) {
    const int h = ex >> 1;  // n2 = m 4^h, m in [1, 4)
    const double dn = __longlong_as_double((long long)(1023 - h) << 52), up = __longlong_as_double((long long)(1023 + h) << 52);
    const double m = n2 * dn * dn;
    const double y0 = (double)rsqrtf((float)m);
    const double e = fma(-m * y0, y0, 1.0);
    const double y = fma(y0 * e, fma(e, 0.375, 0.5), y0);
    double q = m * y;
    q = fma(0.5 * y, fma(-q, q, m), q);
    const double d1 = fma(fabs(ar), dn, q);  // in [1, 4)
    const double im = ai * dn;
    const double d = Num<T>::cplx ? fma(d1, d1, im * im) : d1;
    double z = (double)(1.f / (float)d);
    z = fma(z, fma(-d, z, 1.0), z);
    z = fma(z, fma(-d, z, 1.0), z);
    s = q * up;
    is = y * dn;
    id = (Num<T>::cplx ? z * d1 : z) * dn;
    fi = im * z * dn;
  } else {
    s = sqrt(n2);
    is = 1.0 / s;
    const double t = ai / (s + fabs(ar));
    id = 1.0 / ((s + fabs(ar)) * fma(t, t, 1.0));
    fi = t * id;
  }
  const double sg = copysign(1.0, ar);
  if constexpr (Num<T>::cplx) {
    tau = make_double2(fma(fabs(ar), is, 1.0), sg * ai * is);
    sc = make_double2(sg * id, -fi);
    diag = make_double2(-sg * s, 0.0);
  } else {
    tau = fma(fabs(ar), is, 1.0);
    sc = sg * id;
    diag = -sg * s;
  }
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
    Tm[c][i] = Num<T>::scale(-1, Num<T>::mul(tau, a));
  }
  Tm[i][i] = tau;
}

// Updates panel `next` (nb columns) by panel next - 1, once that is published, and factors it; its
// rows from l0 on lie in registers: thread t holds rows l0 + t + 256 r, r < R (warps whose rows lie
// beyond the column do no arithmetic: the FP64 pipe is shared). Writes R's entries to Z and the
// reflectors and T to V. Warp 0 does a step's scalars, the last warp T's columns.
template <typename T, bool VS, int R>
__device__ __forceinline__ void qr_factor_panel(T* __restrict__ Z, T* __restrict__ V, int64_t L, int64_t next, int nb,
                                                QrPanel<T, VS>& p, T* Vs, QrShared<T>& sh,
                                                const unsigned long long* ready, unsigned long long* err) {
  const int t = threadIdx.x, lane = t & 31, warp = t >> 5;
  const bool has_p = next > 0;
  const int64_t c0 = next * kPanel, l0 = has_p ? c0 - kPanel : 0;
  const int off = (int)(c0 - l0), len = (int)(L - l0);
  const int live = (len - 32 * warp + kThreads - 1) / kThreads;  // passes with rows of this warp (may be <= 0)
  __syncthreads();  // the columns as this CTA's warps left them
  T x[R][kPanel];
#pragma unroll
  for (int r = 0; r < R; ++r)
#pragma unroll
    for (int c = 0; c < kPanel; ++c) {
      const int l = t + kThreads * r;
      x[r][c] = (l < len && c < nb) ? ldcg_t(Z + (c0 + c) * L + l0 + l) : Num<T>::zero();
    }
  if (has_p) {
    qr_wait(ready, (unsigned long long)next, err);
    p = qr_load_panel<T, VS>(V, L, next - 1, kPanel, Vs, sh);
    T w[kPanel * kPanel];
#pragma unroll
    for (int e = 0; e < kPanel * kPanel; ++e) w[e] = Num<T>::zero();
#pragma unroll
    for (int r = 0; r < R; ++r) {
      const int l = t + kThreads * r;
      if (r < live) {
#pragma unroll
        for (int i = 0; i < kPanel; ++i) {
          const T v = l < len ? p.v(i, l) : Num<T>::zero();
#pragma unroll
          for (int c = 0; c < kPanel; ++c) w[i * kPanel + c] = Num<T>::fmac(x[r][c], v, w[i * kPanel + c]);
        }
      }
    }
    T mine = Num<T>::zero();
    if (live > 0) mine = warp_sums<T, kPanel * kPanel>(w, lane);  // lane l: value l >> 1
    if (!(lane & 1)) sh.part[0][warp][lane >> 1] = mine;
    __syncthreads();
    if (live > 0) {
      // lane l < 16 (and l + 16): value l, warps 4 h .. 4 h + 3
      T s = Num<T>::zero();
#pragma unroll
      for (int u = 0; u < kWarps / 2; ++u) s = Num<T>::add(s, sh.part[0][(lane >> 4) * (kWarps / 2) + u][lane & 15]);
      s = Num<T>::add(s, shfl_xor_t(s, 16));
      // y_ic = sum_j conj(T_ji) w_jc at lane 4 i + c
      const int i = (lane & 15) >> 2, c = lane & 3;
      T y = Num<T>::zero();
#pragma unroll
      for (int j = 0; j < kPanel; ++j) y = Num<T>::fma_(Num<T>::conj(sh.Tm[j][i]), shfl_t(s, 4 * j + c), y);
      y = Num<T>::scale(-1, y);
#pragma unroll
      for (int j = 0; j < kPanel; ++j) {
        T ny[kPanel];
#pragma unroll
        for (int cc = 0; cc < kPanel; ++cc) ny[cc] = shfl_t(y, 4 * j + cc);
#pragma unroll
        for (int r = 0; r < R; ++r) {
          const int l = t + kThreads * r;
          if (r < live) {
            const T v = l < len ? p.v(j, l) : Num<T>::zero();
#pragma unroll
            for (int cc = 0; cc < kPanel; ++cc) x[r][cc] = Num<T>::fma_(ny[cc], v, x[r][cc]);
          }
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
      for (int c = 0; c < kPanel; ++c) sh.row[b][c] = x[0][c];
    }
    T mine = Num<T>::zero();
    if (live > 0) mine = warp_sums<T, kPanel>(a, lane);  // lane l: value l >> 3
    if (!(lane & 7)) sh.part[b][warp][lane >> 3] = mine;
    __syncthreads();
    T s = Num<T>::zero();
    if (warp == 0 || warp == kWarps - 1) {
      s = sh.part[b][lane & 7][lane >> 3];
#pragma unroll
      for (int o = 4; o >= 1; o >>= 1) s = Num<T>::add(s, shfl_xor_t(s, o));  // lane l: total l >> 3
    }
    if (warp == 0) {
      const T d = shfl_t(s, 8 * i);
      double xn;
      if constexpr (Num<T>::cplx) xn = d.x; else xn = d;
      T tau, sc, diag;
      qr_scalars<T>(sh.row[b][i], xn, tau, sc, diag);
      // x_c -= conj(tau) (v^H x_c) v, v = sc x_i below row j; lane 8 c
      const T w = Num<T>::fma_(Num<T>::conj(sc), s, sh.row[b][lane >> 3]);
      const T g = Num<T>::scale(-1, Num<T>::mul(Num<T>::conj(tau), w));
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
  if (t == kThreads - 1) {
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
      const int l = t + kThreads * r;
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
  if (has_p && warp < nb) qr_apply_panel<T, VS, true>(z + c0 - kPanel, p, kPanel, sh, lane);
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
    qr_scalars<T>(sh.row[0][i], xn, tau, sc, diag);
#pragma unroll
    for (int c = 0; c < kPanel; ++c)
      S[c] = c < i ? Num<T>::fma_(sc, sh.part[0][0][c], Num<T>::conj(sh.row[0][c])) : Num<T>::zero();
    qr_t_column<T>(Tm, S, tau, i);
    if (warp > i && warp < nb) {
      const T w = Num<T>::fma_(Num<T>::conj(sc), sh.part[0][0][warp], sh.row[0][warp]);
      const T g = Num<T>::scale(-1, Num<T>::mul(Num<T>::conj(tau), w)), f = Num<T>::mul(g, sc);
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
template <typename T, typename T32, int MAXR, bool VS>
__device__ bool qr_block(T* __restrict__ work, T32* __restrict__ work32, const int64_t* __restrict__ r, int group, int rank,
                         unsigned long long* ready, unsigned long long* ctrl, const double* scale_b, T* Vs,
                         QrShared<T>& sh) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int64_t gt = (int64_t)rank * kThreads + threadIdx.x, ngt = (int64_t)group * kThreads;
  const int64_t k = r[R_K], L = r[R_LQ];
  T* Z = work + r[R_Z];
  T* V = work + r[R_VQ];
  T* tau = work + r[R_TAU];
  T* RR = work + r[R_RR];
  const int64_t np = (k + kPanel - 1) / kPanel;
  auto width = [&](int64_t q) { return (int)min((int64_t)kPanel, k - q * kPanel); };
  // factorisation: panel q applied to this CTA's later panels, panel q + 1 factored by its owner
  for (int64_t q = -1; q + 1 < np; ++q) {
    const int64_t next = q + 1;
    const int64_t mine = next + ((rank - next) % group + group) % group;  // first own panel from `next` on
    if (mine >= np) break;  // nothing of this CTA's is left
    QrPanel<T, VS> p = {Vs, V, L, 0};
    if (mine == next) {
      const int64_t passes = (L - (q >= 0 ? q * kPanel : 0) + kThreads - 1) / kThreads;
      const int nb = width(next);
#define YB_PANEL(R) qr_factor_panel<T, VS, (R <= MAXR ? R : 1)>(Z, V, L, next, nb, p, Vs, sh, ready, ctrl + C_ERR)
      if (passes <= 1) YB_PANEL(1);
      else if (passes <= 2) YB_PANEL(2);
      else if (MAXR >= 4 && passes <= 4) YB_PANEL(4);
      else if (MAXR >= 6 && passes <= 6) YB_PANEL(6);
      else if (MAXR >= 11 && passes <= 11) YB_PANEL(11);
      else {
        if (q >= 0) {
          qr_wait(ready, (unsigned long long)next, ctrl + C_ERR);
          p = qr_load_panel<T, VS>(V, L, q, kPanel, Vs, sh);
        }
        qr_factor_panel_long<T, VS>(Z, V, L, next, nb, q >= 0, p, sh);
      }
#undef YB_PANEL
      __syncthreads();
      if (threadIdx.x == 0) {
        __threadfence();
        atomicMax(ready, (unsigned long long)(next + 1));
      }
    } else if (q >= 0) {
      qr_wait(ready, (unsigned long long)next, ctrl + C_ERR);
      p = qr_load_panel<T, VS>(V, L, q, kPanel, Vs, sh);
    }
    if (q >= 0) {
      // this CTA's later panels: a column per warp
      const int64_t first = mine == next ? mine + group : mine;
      for (int64_t e = warp;; e += kWarps) {
        const int64_t pan = first + (e / kPanel) * group, c = pan * kPanel + e % kPanel;
        if (pan >= np) break;
        if (c < k) qr_apply_panel<T, VS, true>(Z + c * L + q * kPanel, p, kPanel, sh, lane);
      }
    }
  }
  if (!grid_barrier(ctrl, group)) return false;
  // R rows, tau, the FP32 start
  const double sc = scale_b ? *scale_b : 0.0;  // no FP32 Jacobi start for yb_qr
  for (int64_t e = gt; e < k * k; e += ngt) {
    const int64_t i = e / k, c = e - i * k;
    const T v = (c >= i) ? ldcg_t(Z + c * L + i) : Num<T>::zero();
    RR[e] = v;
    if (scale_b) {
      work32[r[R_X32] + e] = to32(rscale(v, sc));
      work32[r[R_W32] + e] = (i == c) ? Num<T32>::one() : Num<T32>::zero();
    }
  }
  for (int64_t e = gt; e < k; e += ngt) tau[e] = ldcg_t(V + e * L + e);  // T's diagonal
  if (!grid_barrier(ctrl, group)) return false;
  // Q's columns: row c of Z becomes (H_0 ... H_c e_c)^T, the panels backwards
  // Columns rank, rank + group, .. of a CTA, dealt to its warps in turn: every CTA has columns of all
  // panels (with 8 neighbouring columns a CTA, the last of 54 did all 108 panels of k = 432 alone).
  const int64_t top = rank < k ? rank + (k - 1 - rank) / group * group : -1;
  for (int64_t q = np - 1; q >= 0; --q) {
    if (top < q * kPanel) continue;  // no column of this CTA from this panel on
    const QrPanel<T, VS> p = qr_load_panel<T, VS>(V, L, q, width(q), Vs, sh);
    for (int64_t c = rank + (int64_t)group * warp; c < k; c += (int64_t)group * kWarps) {
      if (c < q * kPanel) continue;
      T* x = Z + c * L;
      if (c / kPanel == q) {
        for (int64_t l = lane; l < L; l += 32) x[l] = (l == c) ? Num<T>::one() : Num<T>::zero();
        __syncwarp();
      }
      qr_apply_panel<T, VS, false>(x + q * kPanel, p, width(q), sh, lane);
    }
  }
  return grid_barrier(ctrl, group);
}

template <typename T, typename T32, int MAXR, int PER_SM>
__global__ void __launch_bounds__(kThreads, PER_SM)
    svd_qr_kernel(T* __restrict__ work, T32* __restrict__ work32, const int64_t* __restrict__ blocks, int n_blocks,
                  int group, unsigned long long* __restrict__ qctrl, const double* __restrict__ scale, int smem_elems) {
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Vs = reinterpret_cast<T*>(smem_raw);
  __shared__ QrShared<T> sh;
  const int g = blockIdx.x / group, rank = blockIdx.x % group;
  const int n_groups = gridDim.x / group;
  if (g >= n_groups) return;
  // qctrl: [n_blocks ready counters][C_REC words per group]
  unsigned long long* ctrl = qctrl + n_blocks + (int64_t)g * C_REC;
  for (int b = g; b < n_blocks; b += n_groups) {
    const int64_t* r = blocks + (int64_t)b * YB_SVD_REC;
    if (!r[R_QR]) continue;
    const double* sb = scale ? scale + b : nullptr;
    const bool ok = kPanel * r[R_LQ] <= smem_elems
                        ? qr_block<T, T32, MAXR, true>(work, work32, r, group, rank, qctrl + b, ctrl, sb, Vs, sh)
                        : qr_block<T, T32, MAXR, false>(work, work32, r, group, rank, qctrl + b, ctrl, sb, Vs, sh);
    if (!ok) return;
  }
}

// Up to one block per SM: one CTA per SM, panels of up to 11 (complex: 6) passes in registers,
// 200 KB of shared memory. More blocks than SMs, one CTA each: two CTAs per SM (the pipe of one is
// idle while the other waits) with fewer passes and half the shared memory.
template <typename T, typename T32, int MAXR, int PER_SM>
int qr_launch(void* work, void* work32, const int64_t* blocks, int n_blocks, double* scale, int64_t* qctrl,
              int qctrl_words, int sms, cudaStream_t s) {
  auto kernel = svd_qr_kernel<T, T32, MAXR, PER_SM>;
  const int smem = 200 * 1024 / PER_SM;
  int per_sm = 0;
  cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, smem);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, kThreads, smem);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  const int capacity = sms * (per_sm < 1 ? 1 : per_sm);
  int group = capacity / n_blocks;
  group = group < 1 ? 1 : group;
  int n_groups = capacity / group;
  if (n_groups > n_blocks) n_groups = n_blocks;
  if ((int64_t)n_groups * C_REC + n_blocks > qctrl_words) n_groups = (qctrl_words - n_blocks) / C_REC;
  if (n_groups < 1) return YB_ERR_INVALID;
  e = cudaMemsetAsync(qctrl, 0, sizeof(int64_t) * ((size_t)n_groups * C_REC + n_blocks), s);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  T* w = (T*)work;
  T32* w32 = (T32*)work32;
  unsigned long long* qc = (unsigned long long*)qctrl;
  int elems = smem / (int)sizeof(T);
  void* args[] = {&w, &w32, &blocks, &n_blocks, &group, &qc, &scale, &elems};
  e = cudaLaunchCooperativeKernel((const void*)kernel, dim3(n_groups * group), dim3(kThreads), args, smem, s);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  return YB_OK;
}

template <typename T, typename T32>
int qr_factor(void* work, void* work32, const int64_t* blocks, int n_blocks, double* scale, int64_t* qctrl,
              int qctrl_words, cudaStream_t s) {
  constexpr int kMany = Num<T>::cplx ? 2 : 4, kFew = Num<T>::cplx ? 6 : 11;
  int dev = 0, sms = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  return n_blocks <= sms
             ? qr_launch<T, T32, kFew, 1>(work, work32, blocks, n_blocks, scale, qctrl, qctrl_words, sms, s)
             : qr_launch<T, T32, kMany, 2>(work, work32, blocks, n_blocks, scale, qctrl, qctrl_words, sms, s);
}

}  // namespace
}  // namespace yb
