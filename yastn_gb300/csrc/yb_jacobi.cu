// Family (c), the sweeps: one-sided Jacobi on super-vectors of rows, each row kept by one warp.
//
// Rows are grouped into super-vectors of BR rows. A sweep rotates every pair of rows once: first
// the pairs inside each super-vector, then, in NS - 1 rounds of the circle method over the NS
// super-vectors, the BR x BR pairs across the two super-vectors P and Q of an item. One CTA of
// BR warps takes an item: warp w keeps row w of P (its X and its W part) in registers, Q's rows
// lie in shared memory, and in step i of BR warp w rotates its row with row (w + i) mod BR of Q.
// All blocks advance together; rounds are separated by the bounded grid barrier of one
// cooperative launch. W is rotated with X (a row is [x | w]), so nothing is accumulated apart.
//
// What bounds it. FP64: GB300 issues 2 DFMA per SM and cycle (64 cycles per warp instruction and
// scheduler), so the DFMAs of a pair are what counts. Per element: 1 for the inner product (the
// rows' squared norms are carried along and updated by the rotations; with a QR start they are
// kept in the block's scratch and recomputed once a sweep), and 2 for a rotation: rows carry a scale, so that
// c x - s y, s x + c y become two shears, x -= a y, y += b x (the scale is applied when the rows
// are written back). The angle needs no FP64 division or square root: its tangent is computed in
// FP32 from the exponents and leading bits of the norms and the inner product (an error of 1e-7
// in the angle leaves 1e-7 of a cosine that is itself small), and only 1 / sqrt(1 + t^2) is
// refined to FP64, which keeps the rotation orthogonal. FP32: latency and shared-memory traffic
// per step; a row of P stays in registers through all BR steps, so a step reads Q's row and
// writes it back.
//
// Measured (GB300; before: every pair of the 2 BR rows in every round, rows in shared memory,
// rotations accumulated and applied to W afterwards): two 432 x 432 blocks FP64 15.2 -> 6.7 ms,
// FP32 13.6 -> 6.7 ms; two 1296 x 1296 blocks FP64 195 -> 72 ms, FP32 103 -> 55 ms; nine
// blocks of 24..93 FP64 2.91 -> 0.81 ms, FP32 1.54 -> 0.82 ms.
#include "yb_svd_common.cuh"

namespace yb {
namespace {

template <typename T>
struct IsF32 {
  static constexpr bool v = sizeof(typename Num<T>::R) == 4;
};

// v = m 2^e with 1 <= |m| < 2 (m = 0 for zero and subnormal v; e = 1024 for Inf and NaN)
struct Split {
  float m;
  int e;
};

__device__ __forceinline__ Split split(double v) {
  const long long b = __double_as_longlong(v);
  const int e = (int)((b >> 52) & 0x7ff);
  Split r;
  r.m = e ? __int_as_float(0x3f800000 | (int)((b >> 29) & 0x7fffff)) : 0.f;
  if (b < 0) r.m = -r.m;
  r.e = e - 1023;
  return r;
}

__device__ __forceinline__ float pow2f(int e) {
  e = e < -126 ? -126 : (e > 126 ? 126 : e);
  return __int_as_float((e + 127) << 23);
}

// tan of the rotation angle from zeta = (be - al) / (2 g)
__device__ __forceinline__ float tan_from_zeta(float zeta) {
  const float z = fabsf(zeta);
  return copysignf(z > 1e9f ? 0.5f / z : 1.f / (z + sqrtf(fmaf(z, z, 1.f))), zeta);
}

// 1 / sqrt(u) in FP64 for u in [1, 8): FP32 start, one step of third order (error ~ 1e-20)
__device__ __forceinline__ double rsqrt64(double u) {
  const double y = (double)rsqrtf((float)u);
  const double e = fma(-u * y, y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

// A row of P in registers: its X and W parts, and (FP64) the squared norm of the true row and
// the scale d of the stored one (true row = d * stored row; i = 1 / d).
template <typename T, int NU>
struct Row {
  T x[NU], w[NU];
  double nrm, d, i;
};

// State of the rows in shared memory (FP64 phase).
struct RowState {
  double nrm, d, i;
};

// One pair: the warp's row P and the row q in shared memory ([x: 32 nu | w: 32 nw]).
// Returns true if it was rotated. FP32 (complex64) version: sums computed afresh, plain rotation.
template <typename T, int NU>
__device__ __forceinline__ bool pair32(Row<T, NU>& P, T* __restrict__ q, int nu, int nw, int lane, float thr2,
                                       float thr_cos, int& maxcos) {
  float al = 0.f, be = 0.f;
  T g = Num<T>::zero();
#pragma unroll
  for (int u = 0; u < NU; ++u) {
    if (u < nu) {
      const T y = q[u * 32 + lane];
      al += Num<T>::abs2(P.x[u]);
      be += Num<T>::abs2(y);
      g = Num<T>::fmac(P.x[u], y, g);
    }
  }
  al = warp_sum(al);
  be = warp_sum(be);
  warp_sum_t<T>(g);
  if (!(al > thr2 && be > thr2 && al > 0.f && be > 0.f)) return false;
  float ga;
  if constexpr (Num<T>::cplx) ga = hypotf(g.x, g.y); else ga = fabsf(g);
  const float cosv = ga * rsqrtf(al) * rsqrtf(be);
  maxcos = max(maxcos, __float_as_int(cosv));
  if (!(cosv > thr_cos)) return false;
  T u;
  float zeta;
  if constexpr (Num<T>::cplx) {
    u = make_float2(g.x / ga, g.y / ga);
    zeta = (be - al) / (2.f * ga);
  } else {
    u = 1.f;
    zeta = (be - al) / (2.f * g);
  }
  const float t = tan_from_zeta(zeta);
  const float c = 1.f / sqrtf(fmaf(t, t, 1.f)), s = c * t;
  // x <- c x - s u y, y <- s conj(u) x + c y
  auto rot = [&](T& x, T* yp) {
    const T y = *yp;
    T xn, yn;
    if constexpr (Num<T>::cplx) {
      const T su = make_float2(s * u.x, s * u.y);
      xn = make_float2(fmaf(c, x.x, -fmaf(su.x, y.x, -su.y * y.y)), fmaf(c, x.y, -fmaf(su.x, y.y, su.y * y.x)));
      yn = make_float2(fmaf(c, y.x, fmaf(su.x, x.x, su.y * x.y)), fmaf(c, y.y, fmaf(su.x, x.y, -su.y * x.x)));
    } else {
      xn = fmaf(c, x, -s * y);
      yn = fmaf(c, y, s * x);
    }
    x = xn;
    *yp = yn;
  };
#pragma unroll
  for (int v = 0; v < NU; ++v)
    if (v < nu) rot(P.x[v], q + v * 32 + lane);
  T* qw = q + nu * 32;
#pragma unroll
  for (int v = 0; v < NU; ++v)
    if (v < nw) rot(P.w[v], qw + v * 32 + lane);
  return true;
}

// FP64 (complex128) version: the squared norms are carried along, two shears per rotation.
template <typename T, int NU>
__device__ __forceinline__ bool pair64(Row<T, NU>& P, T* __restrict__ q, RowState* __restrict__ qs, int nu, int nw,
                                       int lane, double thr2, float thr_cos, int& maxcos) {
  const double al = P.nrm, be = qs->nrm;
  if (!(al > thr2 && be > thr2 && al > 0.0 && be > 0.0)) return false;
  T g0 = Num<T>::zero(), g1 = Num<T>::zero();  // two chains
#pragma unroll
  for (int u = 0; u < NU; u += 2) {
    if (u < nu) g0 = Num<T>::fmac(P.x[u], q[u * 32 + lane], g0);
    if (u + 1 < NU && u + 1 < nu) g1 = Num<T>::fmac(P.x[u + 1 < NU ? u + 1 : u], q[(u + 1) * 32 + lane], g1);
  }
  T g = Num<T>::add(g0, g1);
  warp_sum_t<T>(g);
  const double dy = qs->d, iy = qs->i;
  const double dd = P.d * dy;
  double ga;  // |g| (with the sign of a real g), and the phase of a complex one
  T ph;
  if constexpr (Num<T>::cplx) {
    const Split s0 = split(fmax(fabs(g.x), fabs(g.y)));
    const double sc = __longlong_as_double((long long)(1023 - (s0.e < -1000 ? -1000 : (s0.e > 1000 ? 1000 : s0.e))) << 52);
    const double gx = g.x * sc, gy = g.y * sc;
    const double n2 = fma(gx, gx, gy * gy);
    const double r = n2 > 0.0 ? rsqrt64(n2) : 0.0;
    ph = make_double2(gx * r, gy * r);
    ga = (g.x * ph.x + g.y * ph.y) * dd;
  } else {
    ph = 1.0;
    ga = g * dd;
  }
  const Split sa = split(al), sb = split(be), sg = split(ga);
  float mm = sa.m * sb.m;
  int es = sa.e + sb.e;
  if (es & 1) { mm *= 2.f; es -= 1; }
  float cosv = fabsf(sg.m) * rsqrtf(mm) * pow2f(sg.e - (es >> 1));
  if (sa.e == 1024 || sb.e == 1024 || sg.e == 1024) cosv = __int_as_float(0x7fffffff);
  maxcos = max(maxcos, __float_as_int(cosv));
  if (!(cosv > thr_cos)) return false;
  const Split sd = split(be - al);
  const float zeta = (sd.m / sg.m) * pow2f(sd.e - sg.e - 1);
  const double t = (double)tan_from_zeta(zeta);
  const double u1 = fma(t, t, 1.0);
  const double c = rsqrt64(u1), ci = u1 * c;  // 1 / sqrt(1 + t^2) and its inverse
  const double a = t * (dy * P.i), b = t * (c * c) * (P.d * iy);
  if constexpr (Num<T>::cplx) {
    const double2 au = make_double2(-a * ph.x, -a * ph.y), bu = make_double2(b * ph.x, -b * ph.y);
    auto rot = [&](double2& x, double2* yp) {
      double2 y = *yp;
      x = Num<T>::fma_(au, y, x);
      y = Num<T>::fma_(bu, x, y);
      *yp = y;
    };
#pragma unroll
    for (int v = 0; v < NU; ++v)
      if (v < nu) rot(P.x[v], q + v * 32 + lane);
    T* qw = q + nu * 32;
#pragma unroll
    for (int v = 0; v < NU; ++v)
      if (v < nw) rot(P.w[v], qw + v * 32 + lane);
  } else {
    auto rot = [&](double& x, double* yp) {
      double y = *yp;
      x = fma(-a, y, x);
      y = fma(b, x, y);
      *yp = y;
    };
#pragma unroll
    for (int v = 0; v < NU; ++v)
      if (v < nu) rot(P.x[v], q + v * 32 + lane);
    T* qw = q + nu * 32;
#pragma unroll
    for (int v = 0; v < NU; ++v)
      if (v < nw) rot(P.w[v], qw + v * 32 + lane);
  }
  double na = fma(-t, ga, al), nb = fma(t, ga, be);
  P.d *= c;
  P.i *= ci;
  const double ndy = dy * ci, niy = iy * c;
  if (!(na > 0.25 * al && nb > 0.25 * be)) {  // a large angle cancels: the norms from the rows
    double s0 = 0.0, s1 = 0.0;
#pragma unroll
    for (int v = 0; v < NU; ++v)
      if (v < nu) {
        s0 += Num<T>::abs2(P.x[v]);
        s1 += Num<T>::abs2(q[v * 32 + lane]);
      }
    na = warp_sum(s0) * (P.d * P.d);
    nb = warp_sum(s1) * (ndy * ndy);
  }
  P.nrm = na;
  __syncwarp();
  if (lane == 0) {
    qs->nrm = nb;
    qs->d = ndy;
    qs->i = niy;
  }
  return true;
}

template <typename T, int BR, int NU>
__global__ void __launch_bounds__(BR * 32) jacobi_rows_kernel(T* __restrict__ work, const int64_t* __restrict__ blocks,
                                                              int n_blocks, const int32_t* __restrict__ super_items,
                                                              int n_items, int max_rounds, int max_sweeps,
                                                              int inner_sweeps, double tol_stop,
                                                              int64_t* __restrict__ state) {
  constexpr bool f32 = IsF32<T>::v;
  using R = typename Num<T>::R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Qrows = reinterpret_cast<T*>(smem_raw);  // [BR][32 nu + 32 nw]
  __shared__ RowState qst[BR];
  __shared__ int s_cos, s_rot, any_active;
  unsigned long long* ctrl = reinterpret_cast<unsigned long long*>(state + (int64_t)n_blocks * ST_REC);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;

  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    for (int round = -1; round < max_rounds; ++round) {  // round -1: the pairs inside each super-vector
      for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
        const int b = super_items[2 * item];
        const int pi = super_items[2 * item + 1];
        int64_t* st = state + (int64_t)b * ST_REC;
        if (((volatile int64_t*)st)[ST_CONV]) continue;
        const int64_t* r = blocks + (int64_t)b * YB_SVD_REC;
        const int64_t k = r[R_K], L = r[R_L];
        const int NS = (int)r[f32 ? R_NSUP : R_NSUP64];
        if (round >= NS - 1) continue;
        T* X = work + r[f32 ? R_X32 : R_X];
        T* W = work + r[f32 ? R_W32 : R_W];
        // squared row norms between rounds: in the block's scratch for the sorted W (QR start); blocks
        // without one sum them again at every load
        double* norms = !f32 && r[R_QR] ? reinterpret_cast<double*>(work + r[R_WS]) : nullptr;
        const int nu = (int)((L + 31) >> 5), nw = (int)((k + 31) >> 5);
        const int stride = 32 * (nu + nw);
        const double thr2d = __longlong_as_double((long long)st[f32 ? ST_THR32 : ST_THR64]);
        const R thr2 = (R)thr2d;
        const float thr_cos = sqrtf((float)L) * (float)Eps<R>::v;
        Row<T, NU> P;
        int maxcos = 0;
        bool rotated = false;
        auto load_row = [&](int64_t g, auto store) {
#pragma unroll
          for (int u = 0; u < NU; ++u)
            if (u < nu) {
              const int64_t l = u * 32 + lane;
              store(u, true, (g < k && l < L) ? __ldcg(X + g * L + l) : Num<T>::zero());
            }
#pragma unroll
          for (int u = 0; u < NU; ++u)
            if (u < nw) {
              const int64_t l = u * 32 + lane;
              store(u, false, (g < k && l < k) ? __ldcg(W + g * k + l) : Num<T>::zero());
            }
        };
        auto pair = [&](int j) {
          T* q = Qrows + (size_t)j * stride;
          if constexpr (f32) return pair32<T, NU>(P, q, nu, nw, lane, thr2, thr_cos, maxcos);
          else return pair64<T, NU>(P, q, qst + j, nu, nw, lane, thr2, thr_cos, maxcos);
        };
        auto store_q = [&](int64_t g, int j) {  // row j of shared memory to row g
          if (g >= k) return;
          const T* q = Qrows + (size_t)j * stride;
          double d = 1.0;
          if constexpr (!f32) d = qst[j].d;
          for (int u = 0; u < nu; ++u) {
            const int64_t l = u * 32 + lane;
            T v = q[l];
            if constexpr (!f32) v = Num<T>::scale(d, v);
            if (l < L) X[g * L + l] = v;
          }
          for (int u = 0; u < nw; ++u) {
            const int64_t l = u * 32 + lane;
            T v = q[32 * nu + l];
            if constexpr (!f32) v = Num<T>::scale(d, v);
            if (l < k) W[g * k + l] = v;
          }
        };
        if (round < 0) {
          // inside super-vectors 2 pi and 2 pi + 1: halves against halves, BR/2 warps
          for (int sub = 0; sub < 2; ++sub) {
            const int64_t g = (int64_t)(2 * pi + sub) * BR + warp;
            __syncthreads();
            if (threadIdx.x == 0) { s_cos = 0; s_rot = 0; }
            {
              T* q = Qrows + (size_t)warp * stride;
              double acc = 0.0;
              load_row(g, [&](int u, bool is_x, T v) {
                q[(is_x ? 0 : 32 * nu) + u * 32 + lane] = v;
                if constexpr (!f32)
                  if (is_x) acc += Num<T>::abs2(v);
              });
              if constexpr (!f32) {
                acc = warp_sum(acc);
                if (lane == 0) { qst[warp].nrm = acc; qst[warp].d = 1.0; qst[warp].i = 1.0; }
              }
            }
            __syncthreads();
            maxcos = 0;
            rotated = false;
            for (int h = BR / 2; h >= 1; h >>= 1) {
              const bool act = warp < BR / 2;
              const int base = (warp / h) * 2 * h, p = base + warp % h;
              if (act) {
                const T* q = Qrows + (size_t)p * stride;
#pragma unroll
                for (int u = 0; u < NU; ++u)
                  if (u < nu) P.x[u] = q[u * 32 + lane];
#pragma unroll
                for (int u = 0; u < NU; ++u)
                  if (u < nw) P.w[u] = q[32 * nu + u * 32 + lane];
                P.nrm = qst[p].nrm; P.d = qst[p].d; P.i = qst[p].i;
              }
              for (int i = 0; i < h; ++i) {
                if (act) rotated |= pair(base + h + (warp + i) % h);
                __syncthreads();
              }
              if (act) {
                T* q = Qrows + (size_t)p * stride;
#pragma unroll
                for (int u = 0; u < NU; ++u)
                  if (u < nu) q[u * 32 + lane] = P.x[u];
#pragma unroll
                for (int u = 0; u < NU; ++u)
                  if (u < nw) q[32 * nu + u * 32 + lane] = P.w[u];
                if (lane == 0) { qst[p].nrm = P.nrm; qst[p].d = P.d; qst[p].i = P.i; }
              }
              __syncthreads();
            }
            if (lane == 0) {
              if (maxcos) atomicMax(&s_cos, maxcos);
              if (rotated) s_rot = 1;
            }
            __syncthreads();
            if (s_rot) store_q(g, warp);
            if constexpr (!f32)
              if (norms && lane == 0 && g < k) norms[g] = qst[warp].nrm;
            if (threadIdx.x == 0 && s_cos)
              atomicMax((unsigned long long*)st,
                        (unsigned long long)__double_as_longlong((double)__int_as_float(s_cos)));
          }
          continue;
        }
        int64_t SP, SQ;
        if (pi == 0) { SP = NS - 1; SQ = round; }
        else { SP = (round + pi) % (NS - 1); SQ = (round - pi + (NS - 1)) % (NS - 1); }
        const int64_t gp = SP * BR + warp, gq = SQ * BR + warp;
        __syncthreads();
        if (threadIdx.x == 0) { s_cos = 0; s_rot = 0; }
        double np = 0.0, nq = 0.0;
        load_row(gp, [&](int u, bool is_x, T v) {
          if (is_x) P.x[u] = v; else P.w[u] = v;
        });
        {
          T* q = Qrows + (size_t)warp * stride;
          load_row(gq, [&](int u, bool is_x, T v) {
            q[(is_x ? 0 : 32 * nu) + u * 32 + lane] = v;
          });
          if constexpr (!f32) {
            if (norms) {
              np = gp < k ? __ldcg(norms + gp) : 0.0;
              nq = gq < k ? __ldcg(norms + gq) : 0.0;
            } else {
              __syncwarp();
#pragma unroll
              for (int u = 0; u < NU; ++u)
                if (u < nu) {
                  np += Num<T>::abs2(P.x[u]);
                  nq += Num<T>::abs2(q[u * 32 + lane]);
                }
              np = warp_sum(np);
              nq = warp_sum(nq);
            }
            P.nrm = np;
            P.d = P.i = 1.0;
            if (lane == 0) {
              qst[warp].nrm = nq;
              qst[warp].d = qst[warp].i = 1.0;
            }
          }
        }
        __syncthreads();
        for (int rep = 0; rep < inner_sweeps; ++rep)
          for (int i = 0; i < BR; ++i) {
            rotated |= pair((warp + i) % BR);
            __syncthreads();
          }
        if (lane == 0) {
          if (maxcos) atomicMax(&s_cos, maxcos);
          if (rotated) s_rot = 1;
        }
        __syncthreads();
        if (s_rot) {
          if (gp < k) {
            double d = 1.0;
            if constexpr (!f32) d = P.d;
#pragma unroll
            for (int u = 0; u < NU; ++u)
              if (u < nu) {
                const int64_t l = u * 32 + lane;
                T v = P.x[u];
                if constexpr (!f32) v = Num<T>::scale(d, v);
                if (l < L) X[gp * L + l] = v;
              }
#pragma unroll
            for (int u = 0; u < NU; ++u)
              if (u < nw) {
                const int64_t l = u * 32 + lane;
                T v = P.w[u];
                if constexpr (!f32) v = Num<T>::scale(d, v);
                if (l < k) W[gp * k + l] = v;
              }
            if constexpr (!f32)
              if (norms && lane == 0) norms[gp] = P.nrm;
          }
          store_q(gq, warp);
          if constexpr (!f32)
            if (norms && lane == 0 && gq < k) norms[gq] = qst[warp].nrm;
        }
        if (threadIdx.x == 0 && s_cos)
          atomicMax((unsigned long long*)st, (unsigned long long)__double_as_longlong((double)__int_as_float(s_cos)));
      }
      if (!grid_barrier(ctrl, gridDim.x)) return;
    }
    // sweep end: a block whose largest |cos| in this sweep was <= tol_stop is converged
    if (blockIdx.x == 0) {
      if (threadIdx.x == 0) any_active = 0;
      __syncthreads();
      for (int b = threadIdx.x; b < n_blocks; b += blockDim.x) {
        int64_t* st = state + (int64_t)b * ST_REC;
        if (st[ST_CONV]) continue;
        const double mc = __longlong_as_double((long long)__ldcg((const long long*)st + ST_MAXCOS));
        st[ST_SWEEPS] += 1;
        st[ST_LASTCOS] = __double_as_longlong(mc);
        st[ST_MAXCOS] = 0;
        if (mc <= tol_stop) st[ST_CONV] = 1; else any_active = 1;
      }
      __syncthreads();
      if (threadIdx.x == 0) ctrl[C_DONE] = any_active ? 0ull : 1ull;
      __threadfence();
    }
    if (!grid_barrier(ctrl, gridDim.x)) return;
    if (((volatile unsigned long long*)ctrl)[C_DONE]) return;
  }
}

template <typename T, int BR, int NU>
int launch_rows(T* work, const int64_t* blocks, int n_blocks, const int32_t* items, int n_items, int max_rounds,
                int max_sweeps, int inner_sweeps, double tol_stop, int lmax, int64_t* state, cudaStream_t s) {
  // k <= L <= lmax for every block: a row takes at most 2 ceil(lmax / 32) units
  const size_t smem = (size_t)BR * 64 * ((lmax + 31) / 32) * sizeof(T);
  int dev = 0, sms = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(jacobi_rows_kernel<T, BR, NU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, jacobi_rows_kernel<T, BR, NU>, BR * 32, smem);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  if (per_sm < 1) return YB_ERR_TOO_LARGE;
  int grid = sms * per_sm;
  if (grid > n_items) grid = n_items;
  if (grid < 1) grid = 1;
  e = cudaMemsetAsync(state + (int64_t)n_blocks * ST_REC, 0, sizeof(int64_t) * C_REC, s);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  void* args[] = {&work, &blocks, &n_blocks, &items, &n_items, &max_rounds, &max_sweeps, &inner_sweeps, &tol_stop,
                  &state};
  e = cudaLaunchCooperativeKernel((const void*)jacobi_rows_kernel<T, BR, NU>, dim3(grid), dim3(BR * 32), args, smem,
                                  s);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  return YB_OK;
}

}  // namespace

// Row lengths (multiples of 32 elements) with a kernel: the row of P and its W part take
// 2 NU registers (4 NU for complex64 and FP64, 8 NU for complex128) of the 128 (16-row
// super-vectors) or 255 a thread has, and Q's rows BR * 64 NU elements of shared memory.
int jacobi_rows(void* work, const int64_t* blocks, int n_blocks, const int32_t* items, int n_items, int max_rounds,
                int rows_per_super, int precision, bool cplx, int max_sweeps, int inner_sweeps, double tol_stop,
                int lmax, int64_t* state, cudaStream_t s) {
  const int nu = (lmax + 31) / 32;
#define YB_ROWS(T, BR, NU)                                                                                       \
  if (rows_per_super == BR && nu <= NU)                                                                          \
    return launch_rows<T, BR, NU>((T*)work, blocks, n_blocks, items, n_items, max_rounds, max_sweeps,            \
                                  inner_sweeps, tol_stop, lmax, state, s)
  if (precision == 32 && !cplx) {
    YB_ROWS(float, 16, 4);
    YB_ROWS(float, 16, 14);
    YB_ROWS(float, 16, 28);
    YB_ROWS(float, 16, 41);
    YB_ROWS(float, 8, 14);
    YB_ROWS(float, 8, 41);
    YB_ROWS(float, 8, 82);
  } else if (precision == 32) {
    YB_ROWS(float2, 16, 4);
    YB_ROWS(float2, 16, 14);
    YB_ROWS(float2, 16, 20);
    YB_ROWS(float2, 8, 40);
  } else if (!cplx) {
    YB_ROWS(double, 4, 4);
    YB_ROWS(double, 4, 14);
    YB_ROWS(double, 4, 28);
    YB_ROWS(double, 4, 41);
  } else {
    YB_ROWS(double2, 4, 4);
    YB_ROWS(double2, 4, 14);
    YB_ROWS(double2, 4, 20);
  }
#undef YB_ROWS
  return YB_ERR_TOO_LARGE;
}

}  // namespace yb
