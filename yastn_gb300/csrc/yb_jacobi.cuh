// Family (c), the sweeps: one-sided Jacobi with a row per warp.
//
// The rows above the noise norm of a block form super-vectors of br rows. A sweep rotates every
// pair of rows once: the pairs inside each super-vector, then level by level the pairs between
// the two halves of a group of super-vectors (the halves are the next level's groups). One CTA
// takes a super-vector S of the smaller half and keeps it for the whole level, row w in the
// registers of warp w (its X and its W part); the super-vectors T of the larger half pass by,
// T's rows in shared memory, and in step i of br warp w rotates its row with row (w + i) mod br
// of T. W is rotated with X (a row is [x | w]), so nothing is accumulated apart.
//
// CTAs do not wait for each other at barriers: every super-vector has a counter of the items
// that it has been through in the sweep, and an item starts when its T (and, at the start of a
// level, its S) has the count that the schedule gives; a block's CTAs meet once a sweep, where
// the last one judges convergence. All CTAs are co-resident (cooperative launch) and every wait
// is bounded: on timeout the error word of the control block is set and the kernel ends.
// A first pass sums the rows' norms and lists the rows above the noise norm (rank-deficient
// blocks keep half of their rows out of all rounds); br follows from the number of listed rows:
// the smallest height with an SM for every item (below it the rounds' fixed cost grows, above it
// SMs stay idle).
//
// What bounds it. FP64: GB300 issues a DFMA of a warp every 64 cycles (19 cycles per SM with four
// warps and more), so the FP64 instructions of a pair are what counts. Per element: 1 for the inner
// product (the rows' squared norms are carried along, updated by the rotations and summed again
// once a sweep), and 2 for a rotation: rows carry a scale, so that c x - s y, s x + c y become
// two shears, x -= a y, y += b x (the scale is applied when the rows are written back). The
// angle needs no FP64 division or square root: its tangent is computed in FP32 from the
// exponents and leading bits of the norms and the inner product (an error of 1e-7 in the angle
// leaves 1e-7 of a cosine that is itself small), and only 1 / sqrt(1 + t^2) is refined to FP64,
// which keeps the rotation orthogonal. FP32: the latency of a step (inner product, reduction,
// angle) and its instructions; the same shears and carried norms.
//
// Measured (GB300; before: super-vectors in shared memory, all pairs of an item's rows in every
// round, a grid barrier per round, rotations accumulated and applied to W afterwards): two
// 432 x 432 blocks of rank 216: FP64 phase 15.2 -> 2.6 ms, FP32 13.6 -> 2.0 ms; two 1296 x 1296
// of rank 648: FP64 195 -> 18 ms, FP32 103 -> 9.9 ms; nine full-rank blocks of 24..93: FP64
// 2.91 -> 0.65 ms, FP32 1.54 -> 0.71 ms.
#pragma once
#include "yb_svd_common.cuh"

namespace yb {
namespace {

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

// 1 / sqrt(u) in FP64 for u in [1, 8): one step of Householder's iteration of third order (A. S.
// Householder, The Numerical Treatment of a Single Nonlinear Equation, 1970) for y^-2 = u,
// y (1 + e / 2 + 3 e^2 / 8) with e = 1 - u y^2, from FP32's 1 / sqrt (e up to 5e-7: what the step
// leaves, 5 e^3 / 16, is 4e-20); within 2^-52 of the root, not always correctly rounded
__device__ __forceinline__ double rsqrt64(double u) {
  const double y = (double)rsqrtf((float)u);
  const double e = fma(-u * y, y, 1.0);
  return fma(y * e, fma(e, 0.375, 0.5), y);
}

__device__ __forceinline__ float inv_sqrt(float u) { return rsqrtf(u); }
__device__ __forceinline__ double inv_sqrt(double u) { return rsqrt64(u); }

// cos and tan of a pair from its squared norms and |g| (real: g); FP32
__device__ __forceinline__ float pair_cos(float al, float be, float g) { return fabsf(g) * rsqrtf(al) * rsqrtf(be); }
__device__ __forceinline__ float pair_tan(float al, float be, float g) { return tan_from_zeta((be - al) / (2.f * g)); }
// the same from FP64 values by exponents and leading bits
__device__ __forceinline__ float pair_cos(double al, double be, double g) {
  const Split sa = split(al), sb = split(be), sg = split(g);
  float mm = sa.m * sb.m;
  int es = sa.e + sb.e;
  if (es & 1) { mm *= 2.f; es -= 1; }
  if (sa.e == 1024 || sb.e == 1024 || sg.e == 1024) return __int_as_float(0x7fffffff);
  return fabsf(sg.m) * rsqrtf(mm) * pow2f(sg.e - (es >> 1));
}
__device__ __forceinline__ float pair_tan(double al, double be, double g) {
  const Split sd = split(be - al), sg = split(g);
  return tan_from_zeta((sd.m / sg.m) * pow2f(sd.e - sg.e - 1));
}

__device__ __forceinline__ bool above(float v, float thr) { return v > thr && v > 0.f; }
// positive FP64 values compared on the integer pipe (NaN has the largest bits: not above)
__device__ __forceinline__ bool above(double v, double thr) {
  const long long a = __double_as_longlong(v), t = __double_as_longlong(thr);
  return a > t && a > 0 && a < 0x7ff0000000000001ll;
}

// Rows are stored scaled: true row = d * stored row, i = 1 / d; nrm = squared norm of the true row.
template <typename R>
struct RowState {
  R nrm, d, i;
};

template <typename T, int NU>
struct Row {
  T x[NU], w[NU];
  RowState<typename Num<T>::R> s;
};

// One pair: the warp's row P and the row q in shared memory ([x: 32 NU | w: 32 NU],
// zeros beyond the row) with state qs.
// Returns true if it was rotated. |cos| to maxcos; FP64: a tangent of kTanMin and more to *maxtan (shared memory).
template <typename T, int NU>
__device__ __forceinline__ bool rotate(Row<T, NU>& P, T* __restrict__ q, RowState<typename Num<T>::R>* __restrict__ qs,
                                       int lane, typename Num<T>::R thr2, float thr_cos, int& maxcos,
                                       int* __restrict__ maxtan) {
  using R = typename Num<T>::R;
  const R al = P.s.nrm, be = qs->nrm;
  if (!(above(al, thr2) && above(be, thr2))) return false;
  T g0 = Num<T>::zero(), g1 = Num<T>::zero();  // two chains
#pragma unroll
  for (int u = 0; u < NU; u += 2) {
    g0 = Num<T>::fmac(P.x[u], q[u * 32 + lane], g0);
    if (u + 1 < NU) g1 = Num<T>::fmac(P.x[u + 1 < NU ? u + 1 : u], q[(u + 1) * 32 + lane], g1);
  }
  T g = Num<T>::add(g0, g1);
  warp_sum_t<T>(g);
  const R dy = qs->d, iy = qs->i;
  const R dd = P.s.d * dy;
  R ga;  // |g| (a real g keeps its sign), and the phase of a complex one
  T ph;
  if constexpr (Num<T>::cplx) {
    if constexpr (sizeof(R) == 8) {
      const int e = split(fmax(fabs(g.x), fabs(g.y))).e;
      const double sc = __longlong_as_double((long long)(1023 - (e < -1000 ? -1000 : (e > 1000 ? 1000 : e))) << 52);
      const double gx = g.x * sc, gy = g.y * sc;
      const double n2 = fma(gx, gx, gy * gy);
      const double r = n2 > 0.0 ? rsqrt64(n2) : 0.0;
      ph = make_double2(gx * r, gy * r);
      ga = (g.x * ph.x + g.y * ph.y) * dd;
    } else {
      const float a = hypotf(g.x, g.y), r = a > 0.f ? 1.f / a : 0.f;
      ph = make_float2(g.x * r, g.y * r);
      ga = a * dd;
    }
  } else {
    ph = R(1);
    ga = g * dd;
  }
  const float cosv = pair_cos(al, be, ga);
  maxcos = max(maxcos, __float_as_int(cosv));
  if (!(cosv > thr_cos)) return false;
  const float tf = pair_tan(al, be, ga);
  const R t = (R)tf;
  const R u1 = t * t + R(1);
  const R c = inv_sqrt(u1), ci = u1 * c;  // 1 / sqrt(1 + t^2) and its inverse
  const R a = t * (dy * P.s.i), b = t * (c * c) * (P.s.d * iy);
  T au, bu;
  if constexpr (Num<T>::cplx) {
    au.x = -a * ph.x; au.y = -a * ph.y;
    bu.x = b * ph.x; bu.y = -b * ph.y;
  } else {
    au = -a;
    bu = b;
  }
  auto rot = [&](T& x, T* yp) {
    T y = *yp;
    x = Num<T>::fma_(au, y, x);
    y = Num<T>::fma_(bu, x, y);
    *yp = y;
  };
#pragma unroll
  for (int v = 0; v < NU; ++v) rot(P.x[v], q + v * 32 + lane);
#pragma unroll
  for (int v = 0; v < NU; ++v) rot(P.w[v], q + (NU + v) * 32 + lane);
  R na = al - t * ga, nb = be + t * ga;
  P.s.d *= c;
  P.s.i *= ci;
  const R ndy = dy * ci, niy = iy * c;
  if (fabsf(tf) > 0.25f) {  // a large angle may cancel: the norms from the rows
    R s0 = 0, s1 = 0;
#pragma unroll
    for (int v = 0; v < NU; ++v) {
      s0 += Num<T>::abs2(P.x[v]);
      s1 += Num<T>::abs2(q[v * 32 + lane]);
    }
    na = warp_sum(s0) * (P.s.d * P.s.d);
    nb = warp_sum(s1) * (ndy * ndy);
  }
  P.s.nrm = na;
  __syncwarp();
  if (lane == 0) {
    qs->nrm = nb;
    qs->d = ndy;
    qs->i = niy;
    if (sizeof(R) == 8 && fabsf(tf) > kTanMin) atomicMax(maxtan, __float_as_int(fabsf(tf)));
  }
  return true;
}

// ---- the schedule
// aux (int64 words, the first four parts zeroed by the launch):
//   [block words 4 n_blocks: arrivals of the sweep, sweeps published * 2 + stop, rows listed,
//    first item] [global words 4: first-pass arrivals, published flag, br, items]
//   [item states 2 (n_pairs + n_blocks) words: int4 (sweep, level, round, done)]
//   [counters n_pairs words: uint32 per super-vector] [norms 2 n_pairs doubles]
//   [row lists n_pairs words: int32 per row]
// The rows of block b start at 2 * (first pair item of b) in the per-row arrays.
enum { B_ARR = 0, B_PUB = 1, B_ROWS = 2, B_ITEM0 = 3, G_ARR = 0, G_PUB = 1, G_BR = 2, G_ITEMS = 3 };
constexpr unsigned kSweepCount = 8192;  // counter values per sweep (a super-vector is in fewer items)

struct Aux {
  unsigned long long *blk, *glob;
  int4* item;
  unsigned* ver;
  double* norms;
  int* act;
};

__host__ __device__ inline int64_t aux_zeroed(int64_t n_blocks, int64_t n_pairs) {
  return 4 * n_blocks + 4 + 2 * (n_pairs + n_blocks) + n_pairs;
}

__device__ __forceinline__ Aux aux_of(int64_t* aux, int n_blocks, int64_t n_pairs) {
  Aux a;
  a.blk = reinterpret_cast<unsigned long long*>(aux);
  a.glob = a.blk + 4 * (int64_t)n_blocks;
  a.item = reinterpret_cast<int4*>(a.glob + 4);
  a.ver = reinterpret_cast<unsigned*>(a.glob + 4 + 2 * (n_pairs + n_blocks));
  a.norms = reinterpret_cast<double*>(aux + aux_zeroed(n_blocks, n_pairs));
  a.act = reinterpret_cast<int*>(a.norms + 2 * n_pairs);
  return a;
}

__device__ __forceinline__ unsigned ld_acquire(const unsigned* p) {
  unsigned v;
  asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ unsigned long long ld_acquire(const unsigned long long* p) {
  unsigned long long v;
  asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(v) : "l"(p) : "memory");
  return v;
}
__device__ __forceinline__ void st_release(unsigned* p, unsigned v) {
  asm volatile("st.release.gpu.global.u32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void st_release(unsigned long long* p, unsigned long long v) {
  asm volatile("st.release.gpu.global.u64 [%0], %1;" ::"l"(p), "l"(v) : "memory");
}

// Where item pi of a block with ns super-vectors works in a level: the level's groups come from
// halving [0, ns) (smaller half first: ns / 2 supers of S, the rest T); item pi takes the pi-th S
// over the groups. n = 0: no S in this level. cnt: items each super-vector of the group has been
// through in the sweep before this level.
struct Place {
  int first, n, i;  // the group's first super-vector and size, the S index
  unsigned cnt;
};

__device__ inline Place place_of(int ns, int level, int pi) {
  Place p = {0, 0, 0, 0};
  for (int g = 0; g < (1 << level); ++g) {
    int first = 0, n = ns;
    unsigned cnt = 1;  // the pairs inside the super-vectors
    for (int bit = level - 1; bit >= 0; --bit) {
      const int h2 = n >> 1, h1 = n - h2;
      if ((g >> bit) & 1) {
        cnt += h2;  // T half: through every S
        first += h2;
        n = h1;
      } else {
        cnt += h2 ? h1 : 0;  // S half: through every T
        n = h2;
      }
    }
    if (pi < (n >> 1)) {
      p.first = first;
      p.n = n;
      p.i = pi;
      p.cnt = cnt;
      return p;
    }
    pi -= n >> 1;
  }
  return p;
}

template <typename T, int BRM, int NU>
__global__ void __launch_bounds__(BRM * 32) jacobi_rows_kernel(T* __restrict__ work, const int64_t* __restrict__ blocks,
                                                               int n_blocks, const int32_t* __restrict__ pair_items,
                                                               int n_pairs, int br_min, int n_sms, int max_sweeps,
                                                               double tol_stop, int64_t* __restrict__ state,
                                                               int64_t* __restrict__ aux_words) {
  using R = typename Num<T>::R;
  constexpr bool f32 = sizeof(R) == 4;
  constexpr int stride = 64 * NU;  // a row of T: X part, W part
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Trows = reinterpret_cast<T*>(smem_raw);  // [br][64 NU]
  __shared__ RowState<R> tst[BRM];
  __shared__ int s_flag, s_last, s_tan;
  __shared__ Place s_place;
  const Aux aux = aux_of(aux_words, n_blocks, n_pairs);
  unsigned long long* err = reinterpret_cast<unsigned long long*>(state + (int64_t)n_blocks * ST_REC) + C_ERR;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if (threadIdx.x == 0) s_tan = 0;

  // Waits (thread 0, bounded) until ready() holds; returns false on timeout. Ends with a barrier.
  auto wait = [&](auto ready) {
    if (threadIdx.x == 0) {
      int ok = 1;
      for (long long spins = 0; !ready(); ++spins) {
        if (spins > 64) __nanosleep(64);
        if (spins > kSpinLimit || (spins & 1023) == 1023 && ld_acquire(err)) {
          atomicExch(err, 1ull);
          ok = 0;
          break;
        }
      }
      s_flag = ok;
    }
    __syncthreads();
    const int ok = s_flag;
    __syncthreads();
    return ok != 0;
  };

  // ---- first pass: squared norms of all rows; the last CTA lists the rows above the noise norm
  for (int64_t it = (int64_t)blockIdx.x * BRM + warp; it < n_pairs; it += (int64_t)gridDim.x * BRM) {
    const int b = pair_items[2 * it];
    const int64_t* r = blocks + (int64_t)b * YB_SVD_REC;
    const int64_t k = r[R_K], L = r[R_L], row0 = 2 * (int64_t)pair_items[2 * it + 1];
    const T* X = work + r[f32 ? R_X32 : R_X];
    for (int64_t g = row0; g < row0 + 2 && g < k; ++g) {
      R s = 0;
      for (int64_t l = lane; l < L; l += 32) s += Num<T>::abs2(__ldcg(X + g * L + l));
      s = warp_sum(s);
      if (lane == 0) aux.norms[2 * r[R_P] + g] = (double)s;
    }
  }
  __syncthreads();
  if (threadIdx.x == 0) {
    __threadfence();
    s_last = atomicAdd(aux.glob + G_ARR, 1ull) + 1ull == gridDim.x;
    __threadfence();
  }
  __syncthreads();
  if (s_last) {
    for (int b = warp; b < n_blocks; b += BRM) {
      const int64_t* r = blocks + (int64_t)b * YB_SVD_REC;
      const int64_t* st = state + (int64_t)b * ST_REC;
      const int k = (int)r[R_K];
      const R thr2 = (R)__longlong_as_double((long long)st[f32 ? ST_THR32 : ST_THR64]);
      const int64_t base = 2 * r[R_P];
      int n = 0;
      for (int g0 = 0; g0 < k; g0 += 32) {
        const int g = g0 + lane;
        const bool on = g < k && above((R)__ldcg(aux.norms + base + g), thr2);
        const unsigned m = __ballot_sync(0xffffffffu, on);
        if (on) aux.act[base + n + __popc(m & ((1u << lane) - 1))] = g;
        n += __popc(m);
      }
      if (lane == 0) aux.blk[4 * b + B_ROWS] = (unsigned long long)n;
    }
    __syncthreads();
    if (warp == 0) {
      int br = br_min, total = 0;
      for (;; ++br) {
        total = 0;
        for (int b = lane; b < n_blocks; b += 32) {
          const int ka = (int)__ldcg(aux.blk + 4 * b + B_ROWS);
          total += ((ka + br - 1) / br + 1) / 2;
        }
        total = (int)__reduce_add_sync(0xffffffffu, total);
        if (br == BRM || total <= n_sms) break;
      }
      if (lane == 0) {
        unsigned long long first = 0;
        for (int b = 0; b < n_blocks; ++b) {
          const int ka = (int)__ldcg(aux.blk + 4 * b + B_ROWS);
          aux.blk[4 * b + B_ITEM0] = first;
          first += ((ka + br - 1) / br + 1) / 2;
          if (ka == 0) {  // nothing to rotate
            int64_t* st = state + (int64_t)b * ST_REC;
            st[ST_SWEEPS] += 1;
            st[ST_CONV] = 1;
          }
        }
        aux.glob[G_BR] = (unsigned long long)br;
        aux.glob[G_ITEMS] = first;
        __threadfence();
        st_release(aux.glob + G_PUB, 1ull);
      }
    }
  }
  if (!wait([&] { return ld_acquire(aux.glob + G_PUB) != 0ull; })) return;
  const int br = (int)__ldcg(aux.glob + G_BR), n_items = (int)__ldcg(aux.glob + G_ITEMS);
  const bool single = n_items <= (int)gridDim.x;  // one item per CTA: S stays in registers

  Row<T, NU> P;
  long long idle = 0;  // polls without an item that could start (CTAs of several items)
  for (int todo = 1; todo;) {
    todo = 0;
    bool moved = false;
    for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
      int4 is = make_int4(0, -1, 0, 0);  // sweep, level (-1: inside super-vectors), round, done
      if (!single) {
        is = __ldcg(aux.item + item);
        if (is.y == 0 && is.x == 0 && is.z == 0 && !(is.w & 2)) is.y = -1;  // untouched
        if (is.w & 1) continue;
      }
      // the block of the item: the last one that starts at or before it
      int b;
      {
        int lo = 0, hi = n_blocks - 1;
        while (lo < hi) {
          const int mid = (lo + hi + 1) >> 1;
          if ((int)__ldcg(aux.blk + 4 * mid + B_ITEM0) <= item) lo = mid; else hi = mid - 1;
        }
        b = lo;
        // blocks without items share the start of the next one that has some
        while ((int)__ldcg(aux.blk + 4 * b + B_ROWS) == 0) --b;
      }
      const int pi = item - (int)__ldcg(aux.blk + 4 * b + B_ITEM0);
      const int ka = (int)__ldcg(aux.blk + 4 * b + B_ROWS);
      const int ns = (ka + br - 1) / br, n_it = (ns + 1) / 2;
      unsigned long long* blk = aux.blk + 4 * b;
      int64_t* st = state + (int64_t)b * ST_REC;
      const int64_t* r = blocks + (int64_t)b * YB_SVD_REC;
      const int k = (int)r[R_K], L = (int)r[R_L];
      T* X = work + r[f32 ? R_X32 : R_X];
      T* W = work + r[f32 ? R_W32 : R_W];
      const int64_t base = 2 * r[R_P];
      const int* act = aux.act + base;
      double* norms = aux.norms + base;
      unsigned* ver = aux.ver + base;
      const R thr2 = (R)__longlong_as_double((long long)st[f32 ? ST_THR32 : ST_THR64]);
      const float thr_cos = sqrtf((float)L) * (float)Eps<R>::v;
      int levels = 0;
      while ((1 << levels) < ns) ++levels;
      int maxcos = 0;

      auto row_of = [&](int sup) { const int i = sup * br + warp; return warp < br && i < ka ? __ldcg(act + i) : -1; };
      // row g of X and W through out(u, is_x, value); zeros beyond the row and for g < 0
      auto load_row = [&](int g, auto out) {
        const T* xr = X + (int64_t)(g < 0 ? 0 : g) * L + lane;
        const T* wr = W + (int64_t)(g < 0 ? 0 : g) * k + lane;
        const int lx = g < 0 ? 0 : L - lane, lw = g < 0 ? 0 : k - lane;
#pragma unroll
        for (int u = 0; u < NU; ++u)
          out(u, true, 32 * u < lx ? __ldcg(xr + 32 * u) : Num<T>::zero());
#pragma unroll
        for (int u = 0; u < NU; ++u)
          out(u, false, 32 * u < lw ? __ldcg(wr + 32 * u) : Num<T>::zero());
      };
      auto store_row = [&](int g, R d, auto in) {
        if (g < 0) return;
        T* xr = X + (int64_t)g * L + lane;
        T* wr = W + (int64_t)g * k + lane;
        const int lx = L - lane, lw = k - lane;
#pragma unroll
        for (int u = 0; u < NU; ++u)
          if (32 * u < lx) xr[32 * u] = Num<T>::scale(d, in(u, true));
#pragma unroll
        for (int u = 0; u < NU; ++u)
          if (32 * u < lw) wr[32 * u] = Num<T>::scale(d, in(u, false));
      };
      T* my = Trows + (size_t)warp * stride;  // this warp's row of T
      auto load_t = [&](int g, bool sum) {
        R s = 0;
        load_row(g, [&](int u, bool is_x, T v) {
          my[(is_x ? u : NU + u) * 32 + lane] = v;
          if (sum && is_x) s += Num<T>::abs2(v);
        });
        if (sum) s = warp_sum(s); else s = g < 0 ? R(0) : (R)__ldcg(norms + g);
        if (lane == 0) { tst[warp].nrm = s; tst[warp].d = tst[warp].i = R(1); }
      };
      auto store_t = [&](int g) {
        store_row(g, tst[warp].d, [&](int u, bool is_x) { return my[(is_x ? u : NU + u) * 32 + lane]; });
        if (lane == 0 && g >= 0) norms[g] = (double)tst[warp].nrm;
      };
      auto load_s = [&](int g) {
        load_row(g, [&](int u, bool is_x, T v) { if (is_x) P.x[u] = v; else P.w[u] = v; });
        P.s.nrm = g < 0 ? R(0) : (R)__ldcg(norms + g);
        P.s.d = P.s.i = R(1);
      };
      auto store_s = [&](int g) {
        store_row(g, P.s.d, [&](int u, bool is_x) { return is_x ? P.x[u] : P.w[u]; });
        if (lane == 0 && g >= 0) norms[g] = (double)P.s.nrm;
      };
      // the rows written by this CTA are published: counter of super-vector s = value
      auto publish = [&](int s, unsigned value) {
        __syncthreads();
        if (threadIdx.x == 0) {
          __threadfence();
          st_release(ver + s, value);
        }
      };
      // largest |cos| and tangent of the item's pairs to the block's running maxima (a barrier lies between
      // the last rotation and this, and between this and the next one)
      auto report = [&] {
        if (!f32 && threadIdx.x == 0 && s_tan) {
          atomicMax((unsigned long long*)st + ST_LASTCOS, (unsigned long long)__double_as_longlong((double)__int_as_float(s_tan)));
          s_tan = 0;
        }
        if (lane == 0 && maxcos)
          atomicMax((unsigned long long*)st, (unsigned long long)__double_as_longlong((double)__int_as_float(maxcos)));
        maxcos = 0;
      };
      // multi-item CTAs only poll: an item that cannot start leaves the CTA to the next one
      auto can_start = [&](auto ready) -> int {  // 1 go, 0 not yet, -1 failed
        if (single) return wait(ready) ? 1 : -1;
        if (threadIdx.x == 0) s_flag = ready() ? 1 : 0;
        __syncthreads();
        const int v = s_flag;
        __syncthreads();
        return v;
      };

      for (;;) {  // single: all of the item; otherwise one step
        const unsigned vb = (unsigned)is.x * kSweepCount;
        if (is.y < 0) {
          if (is.x > 0) {  // the block's verdict on the sweep before
            const int go = can_start([&] { return ld_acquire(blk + B_PUB) >= 2ull * is.x; });
            if (go < 0) return;
            if (!go) break;
            if (__ldcg(blk + B_PUB) & 1ull) { is.w = 3; moved = true; break; }
          }
          for (int sub = 0; sub < 2; ++sub) {
            const int sup = 2 * pi + sub;
            if (sup >= ns) break;
            const int g = row_of(sup);
            __syncthreads();
            if (warp < br) load_t(g, true);
            __syncthreads();
            const int n = br + (br & 1);
            for (int i = 0; i < n - 1; ++i) {  // circle method over the br rows
              int p = warp == 0 ? n - 1 : (i + warp) % (n - 1);
              int q = warp == 0 ? i : (i - warp + n - 1) % (n - 1);
              if (p > q) { const int t = p; p = q; q = t; }
              if (warp < n / 2 && q < br) {
                T* pr = Trows + (size_t)p * stride;
#pragma unroll
                for (int u = 0; u < NU; ++u) {
                  P.x[u] = pr[u * 32 + lane];
                  P.w[u] = pr[(NU + u) * 32 + lane];
                }
                P.s = tst[p];
                if (rotate<T, NU>(P, Trows + (size_t)q * stride, tst + q, lane, thr2, thr_cos, maxcos, &s_tan)) {
#pragma unroll
                  for (int u = 0; u < NU; ++u) {
                    pr[u * 32 + lane] = P.x[u];
                    pr[(NU + u) * 32 + lane] = P.w[u];
                  }
                  if (lane == 0) tst[p] = P.s;
                }
              }
              __syncthreads();
            }
            if (warp < br) store_t(g);
            publish(sup, vb + 1u);
          }
          report();
          is.y = 0;
          is.z = 0;
          is.w |= 2;
          moved = true;
          if (!single) break;
          continue;
        }
        if (is.y >= levels) {  // sweep end: the last item of the block judges convergence
          __syncthreads();
          if (threadIdx.x == 0) {
            __threadfence();
            if (atomicAdd(blk + B_ARR, 1ull) + 1ull == (unsigned long long)n_it) {
              __threadfence();
              const double mc = __longlong_as_double((long long)__ldcg((const long long*)st + ST_MAXCOS));
              const double mt = __longlong_as_double((long long)__ldcg((const long long*)st + ST_LASTCOS));
              const bool conv = stops(mc, mt, tol_stop, mixed_stop<R>(tol_stop), is.x + 1);
              st[ST_SWEEPS] = is.x + 1;
              st[ST_LASTCOS] = conv || is.x + 1 >= max_sweeps ? __double_as_longlong(mc) : 0;
              st[ST_MAXCOS] = 0;
              if (conv) st[ST_CONV] = 1;
              blk[B_ARR] = 0ull;
              __threadfence();
              st_release(blk + B_PUB, 2ull * (is.x + 1) + (conv || is.x + 1 >= max_sweeps ? 1ull : 0ull));
            }
          }
          is.x += 1;
          is.y = -1;
          is.z = 0;
          moved = true;
          if (!single) break;
          continue;
        }
        // between the halves of a group
        __syncthreads();
        if (threadIdx.x == 0) s_place = place_of(ns, is.y, pi);
        __syncthreads();
        const Place pl = s_place;
        if (pl.n < 2) {
          is.y += 1;
          is.z = 0;
          moved = true;
          if (!single) break;
          continue;
        }
        const int h2 = pl.n >> 1, h1 = pl.n - h2;
        const int S = pl.first + pl.i;
        int gs = 0;
        bool stop = false;
        for (;;) {
          const int round = is.z;
          const int j = (pl.i + round) % h1;
          // items T has been through in this level: S index j, j - 1, .., 0, then h2 - 1, .., j + 1
          const int seen = pl.i <= j ? (j < h2 ? j : h2 - 1) - pl.i : j + 1 + h2 - 1 - pl.i;
          const int Tn = pl.first + h2 + j;
          const unsigned need = vb + pl.cnt + (unsigned)seen;
          const int go = can_start([&] {
            return ld_acquire(ver + Tn) >= need && (round > 0 || ld_acquire(ver + S) >= vb + pl.cnt);
          });
          if (go < 0) return;
          if (!go) { stop = true; break; }
          const int gt = row_of(Tn);
          if (round == 0 || !single) {
            gs = row_of(S);
            if (warp < br) load_s(gs);
          }
          if (warp < br) load_t(gt, false);
          if (single && !(P.s.d > R(1e-3) && P.s.d < R(1e3))) {  // S's scale after many rounds
#pragma unroll
            for (int u = 0; u < NU; ++u) {
              P.x[u] = Num<T>::scale(P.s.d, P.x[u]);
              P.w[u] = Num<T>::scale(P.s.d, P.w[u]);
            }
            P.s.d = P.s.i = R(1);
          }
          __syncthreads();
          for (int i = 0; i < br; ++i) {
            if (warp < br) {
              int q = warp + i;
              q -= q >= br ? br : 0;
              rotate<T, NU>(P, Trows + (size_t)q * stride, tst + q, lane, thr2, thr_cos, maxcos, &s_tan);
            }
            __syncthreads();
          }
          if (warp < br) {
            store_t(gt);
            if (round == h1 - 1 || !single) store_s(gs);
          }
          __syncthreads();
          if (threadIdx.x == 0) {
            __threadfence();
            st_release(ver + Tn, need + 1u);
            if (round == h1 - 1) st_release(ver + S, vb + pl.cnt + (unsigned)h1);
          }
          moved = true;
          is.z += 1;
          if (is.z == h1) break;
          if (!single) { stop = true; break; }
        }
        report();
        if (is.z == h1) {
          is.y += 1;
          is.z = 0;
        }
        if (stop || !single) break;
      }
      if (!single) {
        report();
        __syncthreads();
        if (threadIdx.x == 0) aux.item[item] = is;
        __syncthreads();
        if (!(is.w & 1)) todo = 1;
      }
    }
    if (moved) {
      idle = 0;
    } else if (!single && todo) {  // every item waits for another CTA
      if (threadIdx.x == 0) {
        __nanosleep(64);
        s_flag = 1;
        if (++idle > kSpinLimit || ((idle & 255) == 255 && ld_acquire(err))) {
          atomicExch(err, 1ull);
          s_flag = 0;
        }
      }
      __syncthreads();
      const int ok = s_flag;
      __syncthreads();
      if (!ok) return;
    }
  }
}

template <typename T, int BRM, int NU>
int launch_rows(T* work, const int64_t* blocks, int n_blocks, const int32_t* pairs, int n_pairs, int br_min,
                int max_sweeps, double tol_stop, int64_t* state, int64_t* aux, cudaStream_t s) {
  const size_t smem = (size_t)BRM * 64 * NU * sizeof(T);
  int dev = 0, sms = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess)
    e = cudaFuncSetAttribute(jacobi_rows_kernel<T, BRM, NU>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, jacobi_rows_kernel<T, BRM, NU>, BRM * 32, smem);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  if (per_sm < 1) return YB_ERR_TOO_LARGE;
  int grid = sms * per_sm;
  const int need = (n_pairs + br_min - 1) / br_min + n_blocks;  // items of the smallest super-vectors, at most
  if (grid > need) grid = need;
  e = cudaMemsetAsync(state + (int64_t)n_blocks * ST_REC, 0, sizeof(int64_t) * C_REC, s);
  if (e == cudaSuccess) e = cudaMemsetAsync(aux, 0, sizeof(int64_t) * aux_zeroed(n_blocks, n_pairs), s);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  void* args[] = {&work, &blocks, &n_blocks, &pairs, &n_pairs, &br_min, &sms, &max_sweeps, &tol_stop, &state, &aux};
  e = cudaLaunchCooperativeKernel((const void*)jacobi_rows_kernel<T, BRM, NU>, dim3(grid), dim3(BRM * 32), args, smem,
                                  s);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  return YB_OK;
}

#define YB_ROWS(T, BRM, NU, BR_MIN)                                                                             \
  if (lmax <= 32 * NU)                                                                                          \
    return launch_rows<T, BRM, NU>((T*)work, blocks, n_blocks, pairs, n_pairs, BR_MIN, max_sweeps, tol_stop, state, \
                                   aux, s)

}  // namespace

// One translation unit per working type; YB_ERR_TOO_LARGE above its longest rows. Variants by row
// length: a row of S and its W part take 2 NU registers (4 NU for complex64 and FP64, 8 NU for
// complex128) of the 65536 / (32 BRM), at most 255, of a thread, and T's rows BRM * 64 NU elements
// of shared memory; the units are unrolled without guards (behind a guard each the loads, FMAs
// and stores of a unit wait for each other: 5.2 instead of 2.6 ms for the FP64 phase of two
// 432 x 432 blocks), so a variant lies within a third of any length above 64. Super-vectors of at least 8 rows in FP32
// and 4 in FP64: below that a round's loads, stores and counters outweigh its steps.
#define YB_JACOBI_ARGS                                                                                          \
  void *work, const int64_t *blocks, int n_blocks, const int32_t *pairs, int n_pairs, int max_sweeps,           \
      double tol_stop, int lmax, int64_t *state, int64_t *aux, cudaStream_t s
int jacobi_f32(YB_JACOBI_ARGS);
int jacobi_c64(YB_JACOBI_ARGS);
int jacobi_f64(YB_JACOBI_ARGS);
int jacobi_c128(YB_JACOBI_ARGS);

}  // namespace yb
