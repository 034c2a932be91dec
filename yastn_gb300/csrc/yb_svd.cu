// Family (c): batched one-sided (Hestenes) Jacobi SVD / Hermitian eigendecomposition of
// all charge-sector blocks, mixed precision, real (FP64) or complex (complex128) data.
//
// Each block A (m x n, row-major) is handled in its "wide" orientation: the k=min(m,n)
// vectors to orthogonalise are the rows of A (m <= n) or of A^H (m > n), each of length
// L=max(m,n), held in a workspace X (an SVD with a QR start: the rows of R, of length k);
// rotations are accumulated in W (k x k), so that X = W X_0 at every step.
//
// GB300 has ~60x more FP32 than FP64 throughput, so the sweeps run in two phases:
//   1. FP32 sweeps on (X32, W32) (float or complex64) until the rows are orthogonal to
//      about 1e-4;
//   2. the host orthonormalises W = widen(W32) with Newton-Schulz steps and forms
//      X = W X_0 (emulated products on the tensor cores, the native FP64 ones for blocks that
//      svd_graded_flags_kernel names); then FP64 sweeps polish (X, W) until a
//      sweep whose largest |cos| was below tol_stop (typically 2-3 sweeps).
// The sweeps of rows that fit a warp's registers are those of yb_jacobi.cuh. This file holds the
// start, the products' scalings, the finalisation and the sweeps of longer rows (more than 2624
// elements in FP32, 1312 in FP64, half of each for complex data): super-vectors of rows in shared
// memory or one pair per warp, paired by a round-robin ordering (circle method over
// N = k rounded up to even, N-1 rounds of N/2 disjoint pairs; all blocks advance together). One
// persistent cooperative launch runs all the sweeps of a phase; rounds are separated
// by a grid barrier whose spin is bounded (an error flag is raised and the kernel exits
// if it ever times out). Finally S = row norms (descending), the normalised rows give Vh
// (wide) or U (tall, conjugated), and W^H gives the other factor (with a QR start the other way
// round, see below).
//
// A rotation is applied when |<x_p, x_q>| > sqrt(L) eps ||x_p|| ||x_q|| (the threshold of
// LAPACK's one-sided Jacobi); the angle of the sweeps here follows Rutishauser's formula with hypot
// (yb_jacobi.cuh: its tangent in FP32). For
// complex rows the phase u = g/|g| of g = <x_p, x_q> = sum_l x_p[l] conj(x_q[l]) is first
// moved onto x_q, which makes the pair's inner product real, and the real rotation of
// (|x_p|^2, |x_q|^2, |g|) follows: x_p <- c x_p - s u x_q, x_q <- s x_p + c u x_q (unitary).
#include <cooperative_groups.h>
#include "yb_svd_common.cuh"

namespace yb {
namespace {

// Per-block Frobenius norm -> shift[b] (eigh: makes a symmetric block positive definite)
// and scale[b], a power of two that brings the FP32 copy of the block (shift included)
// below 1 in magnitude, so that FP32 squares and dot products neither overflow nor lose
// the block to underflow. The rotations, and so W, do not depend on the scale. An SVD's FP64
// phase works on the scaled block too (S is scaled back at the end): squared norms and inner
// products of a block of norm 1e-140 would be subnormal there.
// A cluster of kFroCtas CTAs per block (one SM's FP64 pipe needs 0.5 ms for the 1.7 M squares of a
// 1296 x 1296 block); the partial sums are added in CTA order.
constexpr int kFroCtas = 8;

template <typename TI>
__global__ void __cluster_dims__(kFroCtas, 1, 1)
    block_fro_kernel(const TI* __restrict__ A, const int64_t* __restrict__ blocks, double* __restrict__ shift,
                     double* __restrict__ scale, int64_t* __restrict__ state) {
  // QR-preconditioned blocks start the FP32 phase from the rows of R, where small singular
  // values are explicit row norms rather than cancellations: its noise norm is FP64's
  __shared__ double red[32];
  __shared__ double part;
  const cooperative_groups::cluster_group cluster = cooperative_groups::this_cluster();
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  const int64_t cnt = r[R_M] * r[R_N];
  const TI* a = A + r[R_A];
  double acc = 0.0;
#pragma unroll 4
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < cnt; e += (int64_t)kFroCtas * blockDim.x)
    acc += cabs2(a[e]);
  acc = warp_sum(acc);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = acc;
  __syncthreads();
  if (threadIdx.x == 0) {
    double tot = 0.0;
    for (int w = 0; w < (int)(blockDim.x >> 5); ++w) tot += red[w];
    part = tot;
  }
  cluster.sync();
  if (blockIdx.x == 0 && threadIdx.x == 0) {
    double tot = 0.0;
    for (int c = 0; c < kFroCtas; ++c) tot += *cluster.map_shared_rank(&part, c);
    // ||A||_2 <= ||A||_F: A + shift I is positive definite; +1 keeps an all-zero block regular
    const double fro = sqrt(tot);
    double bound = fro;
    if (shift != nullptr) {
      shift[blockIdx.y] = fro + 1.0;
      bound = 2.0 * fro + 1.0;
    }
    int e = 0;
    if (bound > 0.0 && bound <= 1.0e300) frexp(bound, &e);
    scale[blockIdx.y] = ldexp(1.0, -e);
    // the FP32 phase works on scale * A, the FP64 phase too (eigh: on A + shift itself)
    const double sf = fro * ldexp(1.0, -e);
    const double t32 = (r[R_QR] ? kNoise64 : kNoise32) * sf, t64 = kNoise64 * (shift != nullptr ? fro : sf);
    state[(int64_t)blockIdx.y * ST_REC + ST_THR32] = __double_as_longlong(t32 * t32);
    state[(int64_t)blockIdx.y * ST_REC + ST_THR64] = __double_as_longlong(t64 * t64);
  }
  cluster.sync();  // every CTA's shared memory stays until it has been read
}

// X32 = scale_b (A or A^H) (+ shift on the diagonal) in FP32, W32 = I; resets the state.
template <typename TI, typename T32>
__global__ void svd_init_kernel(const TI* __restrict__ A, T32* __restrict__ work32,
                                const int64_t* __restrict__ blocks, int64_t* __restrict__ state,
                                const double* __restrict__ shift, const double* __restrict__ scale) {
  const double sc = scale[blockIdx.y];
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  const int64_t m = r[R_M], n = r[R_N], k = r[R_K], L = r[R_L];
  const bool tall = m > n;
  const int64_t xs = k * L, ws = k * k;
  T32* X = work32 + r[R_X32];
  T32* W = work32 + r[R_W32];
  const TI* a = A + r[R_A];
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < xs + ws;
       e += (int64_t)gridDim.x * blockDim.x) {
    if (e < xs) {
      const int64_t i = e / L, l = e - i * L;
      TI v = tall ? cconj_(a[l * n + i]) : a[e];
      if (shift != nullptr && i == l) v = add_real(v, shift[blockIdx.y]);
      X[e] = to32(rscale(v, sc));
    } else {
      const int64_t f = e - xs;
      const int64_t i = f / k, j = f - i * k;
      W[f] = (i == j) ? Num<T32>::one() : Num<T32>::zero();
    }
  }
  if (blockIdx.x == 0 && threadIdx.x < ST_THR32) state[blockIdx.y * ST_REC + threadIdx.x] = 0;
}

// Resets the sweep words (0..3) of each block's state (the noise norms stay).
__global__ void svd_state_reset_kernel(int64_t* __restrict__ state) {
  if (threadIdx.x < ST_THR32) state[blockIdx.x * ST_REC + threadIdx.x] = 0;
}

// W64 = widen(W32) (the host orthonormalises it next); resets the per-block state.
template <typename T32, typename T64>
__global__ void svd_widen_kernel(const T32* __restrict__ work32, T64* __restrict__ work64,
                                 const int64_t* __restrict__ blocks, int64_t* __restrict__ state) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  const int64_t k = r[R_K];
  const T32* W32 = work32 + r[R_W32];
  T64* W = work64 + r[R_W];
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < k * k; e += (int64_t)gridDim.x * blockDim.x)
    W[e] = to64(W32[e]);
  if (blockIdx.x == 0 && threadIdx.x < ST_THR32) state[blockIdx.y * ST_REC + threadIdx.x] = 0;
}

// T <- 1.5 I - 0.5 T for every block, T = W^H W at t_delta elements after W: the right factor of a
// Newton-Schulz step W' = W (1.5 I - 0.5 W^H W).
template <typename T64>
__global__ void svd_ns_prep_kernel(T64* __restrict__ work64, const int64_t* __restrict__ blocks, int64_t t_delta) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  const int64_t k = r[R_K];
  T64* T = work64 + r[R_W] + t_delta;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < k * k; e += (int64_t)gridDim.x * blockDim.x) {
    const T64 v = rscale(T[e], -0.5);
    T[e] = e / k == e % k ? add_real(v, 1.5) : v;
  }
}

// Operands of X = W R scaled along the contracted index: T = W D, Wn = D^-1 R, D the powers of two
// of a two-sided equilibration of R: with c_j the exponent of the largest entry of column j, row l
// gets the exponent max_j (exponent of R_lj - c_j), in [-200, 0]. The small rows of a graded R go
// with entries of W that are small for the large ones, so the entries of a row of T and of a column
// of Wn have one size each, and digits scaled per row of T and per column of Wn keep the relative
// accuracy that an FP64 sum of the products has, for R graded by rows, by columns or both.
// X's storage holds c (k values) and D (the next k) meanwhile (k = 1: no scaling).
__device__ __forceinline__ int top_exponent(double v) {  // -2000 for zero
  const int e = (int)((__double_as_longlong(v) >> 52) & 0x7ff);
  return e ? e - 1023 : -2000;
}
__device__ __forceinline__ int top_exponent(double2 v) { return max(top_exponent(v.x), top_exponent(v.y)); }
__device__ __forceinline__ double real_of(double v) { return v; }
__device__ __forceinline__ double real_of(double2 v) { return v.x; }
__device__ __forceinline__ void set_real(double& d, double v) { d = v; }
__device__ __forceinline__ void set_real(double2& d, double v) { d = make_double2(v, 0.0); }

// A non-finite R (exponent 1024) marks its block, if that has products from digits (k >= k_min): its FP64
// noise norm becomes NaN (it is NaN or Inf already unless the block's norm overflowed), see
// svd_poison_kernel.
template <typename T64>
__global__ void svd_col_exponents_kernel(T64* __restrict__ work64, const int64_t* __restrict__ blocks, int k_min,
                                         int64_t* __restrict__ state) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  if (!r[R_QR]) return;
  const int64_t k = r[R_K];
  const T64* R = work64 + r[R_RR];
  __shared__ int red[8][32];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int64_t j0 = (int64_t)blockIdx.x * 32; j0 < k; j0 += (int64_t)gridDim.x * 32) {
    const int64_t j = j0 + lane;
    int e = -2000;
    for (int64_t l = warp; l < k && l < j0 + 32; l += 8)
      if (j < k && l <= j) e = max(e, top_exponent(R[l * k + j]));
    red[warp][lane] = e;
    __syncthreads();
    if (warp == 0 && j < k) {
      for (int w = 1; w < 8; ++w) e = max(e, red[w][lane]);
      if (e == 1024 && k >= k_min) state[(int64_t)blockIdx.y * ST_REC + ST_THR64] = 0x7ff8000000000000ll;
      set_real(work64[r[R_X] + j], (double)e);
    }
    __syncthreads();
  }
}

// The digits of an emulated product hold no NaN or Inf: what a native product would make NaN is made
// NaN here, for the blocks that svd_col_exponents_kernel marked. which 0: X (U = the workspace); 1: the
// factor that comes from Q (U of tall blocks, Vh of the others).
template <typename T64>
__global__ void svd_poison_kernel(T64* __restrict__ U, T64* __restrict__ V, const int64_t* __restrict__ blocks,
                                  const int64_t* __restrict__ state, int k_min, int which) {
  const double thr = __longlong_as_double((long long)state[(int64_t)blockIdx.y * ST_REC + ST_THR64]);
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  const int64_t k = r[R_K];
  if (thr == thr || k < k_min) return;
  const bool tall = r[R_M] > r[R_N];
  T64* p = which == 0 ? U + r[R_X] : (tall ? U + r[R_U] : V + r[R_V]);
  const int64_t n = which == 0 ? k * r[R_L] : (tall ? r[R_M] * k : k * r[R_N]);
  const double nan = __longlong_as_double(0x7ff8000000000000ll);
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x) {
    if constexpr (Num<T64>::cplx) p[e] = make_double2(nan, nan); else p[e] = nan;
  }
}

template <typename T64>
__global__ void svd_row_scales_kernel(T64* __restrict__ work64, const int64_t* __restrict__ blocks) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  const int64_t k = r[R_K];
  if (!r[R_QR] || k < 2) return;
  const T64* R = work64 + r[R_RR];
  T64* c = work64 + r[R_X];
  const int lane = threadIdx.x & 31, nw = (int)(gridDim.x * blockDim.x) >> 5;
  for (int64_t l = (blockIdx.x * blockDim.x + threadIdx.x) >> 5; l < k; l += nw) {
    int e = -200;
    for (int64_t j = l + lane; j < k; j += 32) {
      const int v = top_exponent(R[l * k + j]);
      if (v > -2000) e = max(e, v - (int)real_of(c[j]));
    }
    e = __reduce_max_sync(0xffffffffu, e);
    if (lane == 0) set_real(c[k + l], __longlong_as_double((long long)(1023 + e) << 52));
  }
}

template <typename T64>
__global__ void svd_scale_wr_kernel(T64* __restrict__ work64, const int64_t* __restrict__ blocks, int64_t t_delta) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  if (!r[R_QR]) return;
  const int64_t k = r[R_K];
  const T64* W = work64 + r[R_W];
  const T64* R = work64 + r[R_RR];
  const T64* d = work64 + r[R_X] + k;
  T64* Ws = work64 + r[R_W] + t_delta;
  T64* Rs = work64 + r[R_W] + 2 * t_delta;
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < k * k; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e / k, j = e - i * k;
    Ws[e] = k < 2 ? W[e] : rscale(W[e], real_of(d[j]));
    // the inverse of a power of two: its exponent negated
    Rs[e] = k < 2 ? R[e]
                  : rscale(R[e], __longlong_as_double(((long long)2046 << 52) - __double_as_longlong(real_of(d[i]))));
  }
}

// Which blocks take their products with W from the FP64 kernel. Digits hold 57 bits below the largest
// element of a row of W and of a component of Q (a column of Q^T): an output V_ij = sum_l W_il Q_jl
// whose terms are all small against (max_l |W_il|) (max_l |Q_jl|) loses its relative accuracy,
// which an FP64 sum keeps. Such outputs are where A is graded by columns (rows of 24 columns over 12
// decades: V to 8e-5 in the smallest entries, A - U S V to 4e-6 of the column; FP64 5e-12 and 4e-14);
// no scaling of l repairs both triangles of V. A pair (i, j) counts as such unless some l has both
// elements within 2^-kGradedBits of their maxima (the output then holds 47 bits, what the sweeps leave
// of an entry of a graded block), or no l has both nonzero. In a block that is not graded pairs count by
// chance, up to 8 % where a row of W has one large element; the block is flagged where a row or
// a component has more than a quarter of its pairs. Rows of R at noise level were not rotated (W's
// row is a unit vector, its vector in V arbitrary) and are left out. The masks are bits: a word has 32
// terms of a pair. Bound: latency; the three launches take 23 us for nine blocks of 24..93, 44 for two
// 432 x 432, 264 for two 1296 x 1296 (of 2.1, 9.0 and 55 ms of the call's device time), the five
// flagged launches that find no flag 31 to 44 us.
constexpr int kGradedBits = 5;

struct GradedAt {  // a block's masks: [A big][A nonzero][B big][B nonzero][fails of A][fails of B]
  uint32_t *a, *b;
  int *na, *nb;
  int k, L, nw;
};
__device__ __forceinline__ GradedAt graded_at(const int64_t* r, const int64_t* at, int32_t* masks) {
  GradedAt g;
  g.k = (int)r[R_K];
  g.L = (int)r[R_LQ];
  g.nw = (g.k + 31) / 32;
  g.a = reinterpret_cast<uint32_t*>(masks + at[blockIdx.y]);
  g.b = g.a + 2 * (int64_t)g.k * g.nw;
  g.na = reinterpret_cast<int*>(g.b + 2 * (int64_t)g.L * g.nw);
  g.nb = g.na + g.k;
  return g;
}

// The masks: rows of W by a warp each (R's row tells noise), components of Q 32 to a CTA.
template <typename T64>
__global__ void __launch_bounds__(256) svd_graded_masks_kernel(const T64* __restrict__ work64,
                                                               const int64_t* __restrict__ blocks, int k_min,
                                                               const int64_t* __restrict__ state,
                                                               const int64_t* __restrict__ at, int32_t* __restrict__ masks) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  if (!r[R_QR] || r[R_K] < k_min) return;
  const GradedAt g = graded_at(r, at, masks);
  const double thr = __longlong_as_double((long long)state[(int64_t)blockIdx.y * ST_REC + ST_THR64]);
  const T64 *W = work64 + r[R_W], *R = work64 + r[R_RR], *Z = work64 + r[R_Z];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  __shared__ int red[8][32];
  for (int i = blockIdx.x * 8 + warp; i < g.k; i += gridDim.x * 8) {
    const T64* w = W + (int64_t)i * g.k;
    double n2 = 0.0;
    int top = -2000;
    for (int l = lane; l < g.k; l += 32) {
      n2 += cabs2(R[(int64_t)i * g.k + l]);
      top = max(top, top_exponent(w[l]));
    }
    n2 = warp_sum(n2);
    top = __reduce_max_sync(0xffffffffu, top);
    const bool noise = !(n2 > thr);
    for (int u = 0; u < g.nw; ++u) {
      const int l = 32 * u + lane, e = l < g.k ? top_exponent(w[l]) : -2000;
      const uint32_t big = __ballot_sync(0xffffffffu, l < g.k && (noise || (e > -2000 && e >= top - kGradedBits)));
      const uint32_t nz = __ballot_sync(0xffffffffu, e > -2000);
      if (lane == 0) {
        g.a[(int64_t)i * g.nw + u] = big;
        g.a[((int64_t)g.k + i) * g.nw + u] = nz;
      }
    }
    if (lane == 0) g.na[i] = 0;
  }
  for (int j0 = blockIdx.x * 32; j0 < g.L; j0 += gridDim.x * 32) {
    const int j = j0 + lane;
    int top = -2000;
#pragma unroll 4
    for (int l = warp; l < g.k; l += 8)
      if (j < g.L) top = max(top, top_exponent(Z[(int64_t)l * g.L + j]));
    red[warp][lane] = top;
    __syncthreads();
    for (int v = 0; v < 8; ++v) top = max(top, red[v][lane]);
    for (int u = warp; u < g.nw; u += 8) {
      uint32_t big = 0, nz = 0;
#pragma unroll 4
      for (int t = 0; t < 32; ++t) {
        const int l = 32 * u + t;
        const int e = l < g.k && j < g.L ? top_exponent(Z[(int64_t)l * g.L + j]) : -2000;
        if (e > -2000) {
          nz |= 1u << t;
          big |= (e >= top - kGradedBits ? 1u : 0u) << t;
        }
      }
      if (j < g.L) {
        g.b[(int64_t)j * g.nw + u] = big;
        g.b[((int64_t)g.L + j) * g.nw + u] = nz;
      }
    }
    if (warp == 0 && j < g.L) g.nb[j] = 0;
    __syncthreads();
  }
}

// The pairs, 32 x 32 to a CTA: a thread has one row of W and four components of Q.
__global__ void __launch_bounds__(256) svd_graded_pairs_kernel(const int64_t* __restrict__ blocks, int k_min,
                                                               const int64_t* __restrict__ at, int32_t* __restrict__ masks) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  if (!r[R_QR] || r[R_K] < k_min) return;
  const GradedAt g = graded_at(r, at, masks);
  __shared__ uint32_t sa[2][32][33], sb[2][32][33];
  const int ti = (g.k + 31) / 32, tj = (g.L + 31) / 32;
  const int i = threadIdx.x >> 3, jq = (threadIdx.x & 7) * 4;
  for (int64_t tile = blockIdx.x; tile < (int64_t)ti * tj; tile += gridDim.x) {
    const int i0 = (int)(tile / tj) * 32, j0 = (int)(tile % tj) * 32;
    uint32_t any[4] = {0, 0, 0, 0}, both[4] = {0, 0, 0, 0};
    bool done = false;
    for (int u0 = 0; u0 < g.nw && !done; u0 += 32) {
      const int nu = min(32, g.nw - u0);
      __syncthreads();
      for (int e = threadIdx.x; e < 2 * 32 * nu; e += 256) {
        const int half = e / (32 * nu), v = e / nu % 32, u = e % nu;
        sa[half][v][u] = i0 + v < g.k ? g.a[((int64_t)half * g.k + i0 + v) * g.nw + u0 + u] : 0u;
        sb[half][v][u] = j0 + v < g.L ? g.b[((int64_t)half * g.L + j0 + v) * g.nw + u0 + u] : 0u;
      }
      __syncthreads();
      for (int u = 0; u < nu; ++u)
#pragma unroll
        for (int q = 0; q < 4; ++q) {
          any[q] |= sa[0][i][u] & sb[0][jq + q][u];
          both[q] |= sa[1][i][u] & sb[1][jq + q][u];
        }
      done = __syncthreads_and(any[0] && any[1] && any[2] && any[3]);
    }
    int fails = 0;
#pragma unroll
    for (int q = 0; q < 4; ++q)  // beyond the edges nothing is nonzero
      if (any[q] == 0 && both[q] != 0) {
        ++fails;
        atomicAdd(g.nb + j0 + jq + q, 1);
      }
    if (fails) atomicAdd(g.na + i0 + i, fails);
  }
}

__global__ void svd_graded_flags_kernel(const int64_t* __restrict__ blocks, int k_min, const int64_t* __restrict__ at,
                                        int32_t* __restrict__ masks, int64_t* __restrict__ flags) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  if (!r[R_QR] || r[R_K] < k_min) return;
  const GradedAt g = graded_at(r, at, masks);
  bool on = false;
  for (int i = threadIdx.x; i < g.k; i += blockDim.x) on = on || 4 * (int64_t)g.na[i] > g.L;
  for (int j = threadIdx.x; j < g.L; j += blockDim.x) on = on || 4 * (int64_t)g.nb[j] > g.k;
  if (on) flags[blockIdx.y] = 1;
}

// X = scale_b X, for an SVD whose X was formed from A itself.
template <typename T64>
__global__ void svd_scale_x_kernel(T64* __restrict__ work64, const int64_t* __restrict__ blocks,
                                   const double* __restrict__ scale) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  const int64_t n = r[R_K] * r[R_L];
  const double c = scale[blockIdx.y];
  T64* X = work64 + r[R_X];
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
    X[e] = rscale(X[e], c);
}

// X = shift_b * W (eigh: the FP64 phase then adds W A with the grouped GEMM, X = W (A + shift I)).
template <typename T64>
__global__ void svd_shift_prefill_kernel(T64* __restrict__ work64, const int64_t* __restrict__ blocks,
                                         const double* __restrict__ shift) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  const int64_t k = r[R_K];
  const double c = shift[blockIdx.y];
  const T64* W = work64 + r[R_W];
  T64* X = work64 + r[R_X];
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < k * k; e += (int64_t)gridDim.x * blockDim.x)
    X[e] = rscale(W[e], c);
}

constexpr int kChunk = 8;  // elements per lane per row kept in flight
constexpr int kLoadBatch = 8;  // independent loads per thread when a CTA stages rows
constexpr int kRowRegs = 16;   // row elements per lane kept in registers in a blocked inner round

// Rotates rows (p, q) of X and W by one Jacobi rotation. Loads are issued a chunk at a
// time (kChunk per lane and row, all before any store of the chunk) so that the L2
// latency is paid once per chunk rather than once per element. Rows are rewritten by
// other SMs between rounds, so loads bypass L1 (ld.global.cg).
template <typename T>
__device__ __forceinline__ void rotate_rows(T* __restrict__ a, T* __restrict__ b, int64_t len, int lane,
                                            typename Num<T>::R c, typename Num<T>::R s, T u) {
  for (int64_t base = 0; base < len; base += 32 * kChunk) {
    T x[kChunk], y[kChunk];
#pragma unroll
    for (int j = 0; j < kChunk; ++j) {
      const int64_t i = base + j * 32 + lane;
      x[j] = (i < len) ? __ldcg(a + i) : Num<T>::zero();
      y[j] = (i < len) ? __ldcg(b + i) : Num<T>::zero();
    }
#pragma unroll
    for (int j = 0; j < kChunk; ++j) {
      const int64_t i = base + j * 32 + lane;
      if (i < len) {
        rot2<T>(x[j], y[j], c, s, u);
        a[i] = x[j];
        b[i] = y[j];
      }
    }
  }
}

template <typename T>
__device__ __forceinline__ void rotate_pair(T* __restrict__ X, T* __restrict__ W, int64_t k, int64_t L, int64_t p,
                                            int64_t q, int lane, int64_t* st, bool mixed) {
  using R = typename Num<T>::R;
  T* xp = X + p * L;
  T* xq = X + q * L;
  // partial sums in the working precision (FP32 in the FP32 phase keeps the FP64 pipe free)
  R al_ = 0, be_ = 0;
  T ga_ = Num<T>::zero();
  for (int64_t base = 0; base < L; base += 32 * kChunk) {
    T x[kChunk], y[kChunk];
#pragma unroll
    for (int j = 0; j < kChunk; ++j) {
      const int64_t i = base + j * 32 + lane;
      x[j] = (i < L) ? __ldcg(xp + i) : Num<T>::zero();
      y[j] = (i < L) ? __ldcg(xq + i) : Num<T>::zero();
    }
#pragma unroll
    for (int j = 0; j < kChunk; ++j) {
      al_ += Num<T>::abs2(x[j]);
      be_ += Num<T>::abs2(y[j]);
      ga_ = Num<T>::fmac(x[j], y[j], ga_);
    }
  }
  R c = 0, s = 0;
  T u = Num<T>::one();
  const R thr2 = (R)__longlong_as_double((long long)st[sizeof(R) == 4 ? ST_THR32 : ST_THR64]);
  if (!Rotation<T>::get(al_, be_, ga_, L, lane, st + ST_MAXCOS, c, s, u, thr2, mixed)) return;
  rotate_rows<T>(xp, xq, L, lane, c, s, u);
  rotate_rows<T>(W + p * k, W + q * k, k, lane, c, s, u);
}

// All sweeps of one precision phase in one cooperative launch.
template <typename T>
__global__ void __launch_bounds__(kThreads) svd_sweeps_kernel(T* __restrict__ work, const int64_t* __restrict__ blocks,
                                                              int n_blocks, const int32_t* __restrict__ pair_items,
                                                              int n_items, int max_rounds, int max_sweeps,
                                                              double tol_stop, int64_t* __restrict__ state) {
  unsigned long long* ctrl = reinterpret_cast<unsigned long long*>(state + (int64_t)n_blocks * ST_REC);
  __shared__ int any_active;
  const int lane = threadIdx.x & 31;
  const int64_t gwarp = (int64_t)blockIdx.x * kWarps + (threadIdx.x >> 5);
  const int64_t nwarps = (int64_t)gridDim.x * kWarps;
  const int rx = sizeof(typename Num<T>::R) == 4 ? R_X32 : R_X;
  const int rw = sizeof(typename Num<T>::R) == 4 ? R_W32 : R_W;
  const bool mixed = mixed_stop<typename Num<T>::R>(tol_stop);
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    for (int round = 0; round < max_rounds; ++round) {
      for (int64_t item = gwarp; item < n_items; item += nwarps) {
        const int b = pair_items[2 * item];
        const int pi = pair_items[2 * item + 1];
        int64_t* st = state + (int64_t)b * ST_REC;
        if (((volatile int64_t*)st)[ST_CONV]) continue;
        const int64_t* r = blocks + (int64_t)b * YB_SVD_REC;
        const int64_t k = r[R_K], L = r[R_L], N = r[R_NP];
        if (round >= N - 1) continue;
        int64_t p, q;
        if (pi == 0) {
          p = N - 1;
          q = round;
        } else {
          p = (round + pi) % (N - 1);
          q = (round - pi + (N - 1)) % (N - 1);
        }
        if (p >= k || q >= k) continue;  // the dummy vector of an odd count
        if (p > q) { const int64_t tq = p; p = q; q = tq; }
        rotate_pair<T>(work + r[rx], work + r[rw], k, L, p, q, lane, st, mixed);
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
        const double mc = __longlong_as_double((long long)st[ST_MAXCOS]);
        const bool conv = stops(mc, __longlong_as_double((long long)st[ST_LASTCOS]), tol_stop, mixed, st[ST_SWEEPS] += 1);
        st[ST_LASTCOS] = conv || sweep + 1 == max_sweeps ? st[ST_MAXCOS] : 0;
        st[ST_MAXCOS] = 0;
        if (conv) st[ST_CONV] = 1; else any_active = 1;
      }
      __syncthreads();
      if (threadIdx.x == 0) ctrl[C_DONE] = any_active ? 0ull : 1ull;
      __threadfence();
    }
    if (!grid_barrier(ctrl, gridDim.x)) return;
    if (((volatile unsigned long long*)ctrl)[C_DONE]) return;
  }
}

// ---------------------------------------------------------------------------------------
// Blocked variant for the FP32 phase: rows are grouped into super-vectors of BR rows; the
// circle method pairs super-vectors (R_NSUP of them, even), and one CTA per pair loads the
// 2*BR rows into shared memory, runs up to inner_sweeps one-sided Jacobi sweeps among them
// (circle method over the 2*BR rows, one warp per pair, rotations accumulated in a
// 2BR x 2BR matrix Q), writes the rows back and applies Q to the matching rows of W
// (column by column, in place). Outer rounds are separated by the grid barrier.
template <typename T, int BR>
__global__ void __launch_bounds__(BR * 32) svd_block_sweeps_kernel(T* __restrict__ work,
                                                                   const int64_t* __restrict__ blocks, int n_blocks,
                                                                   const int32_t* __restrict__ super_items,
                                                                   int n_items, int max_rounds, int max_sweeps,
                                                                   int inner_sweeps, double tol_stop, int lmax,
                                                                   int64_t* __restrict__ state) {
  constexpr int R2 = 2 * BR;
  using R = typename Num<T>::R;
  extern __shared__ __align__(16) unsigned char smem_raw[];
  T* Xs = reinterpret_cast<T*>(smem_raw);   // [R2][lmax]
  T* Qs = Xs + (size_t)R2 * lmax;           // [R2][R2]
  __shared__ int any_rot, any_active;
  __shared__ int64_t grow[R2];              // global row of each local row (-1: absent)
  unsigned long long* ctrl = reinterpret_cast<unsigned long long*>(state + (int64_t)n_blocks * ST_REC);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int rx = sizeof(typename Num<T>::R) == 4 ? R_X32 : R_X;
  const int rw = sizeof(typename Num<T>::R) == 4 ? R_W32 : R_W;
  const bool mixed = mixed_stop<typename Num<T>::R>(tol_stop);
  for (int sweep = 0; sweep < max_sweeps; ++sweep) {
    for (int round = 0; round < max_rounds; ++round) {
      for (int item = blockIdx.x; item < n_items; item += gridDim.x) {
        const int b = super_items[2 * item];
        const int pi = super_items[2 * item + 1];
        int64_t* st = state + (int64_t)b * ST_REC;
        if (((volatile int64_t*)st)[ST_CONV]) continue;
        const int64_t* r = blocks + (int64_t)b * YB_SVD_REC;
        const int64_t k = r[R_K], L = r[R_L], NS = r[sizeof(R) == 4 ? R_NSUP : R_NSUP64];
        if (round >= NS - 1) continue;
        int64_t P, Q;
        if (pi == 0) { P = NS - 1; Q = round; }
        else { P = (round + pi) % (NS - 1); Q = (round - pi + (NS - 1)) % (NS - 1); }
        T* X = work + r[rx];
        T* W = work + r[rw];
        __syncthreads();
        if (threadIdx.x < R2) {
          const int sv = threadIdx.x < BR ? (int)P : (int)Q;
          const int64_t g = (int64_t)sv * BR + (threadIdx.x % BR);
          grow[threadIdx.x] = (g < k) ? g : -1;
        }
        for (int e = threadIdx.x; e < R2 * R2; e += blockDim.x)
          Qs[e] = (e / R2 == e % R2) ? Num<T>::one() : Num<T>::zero();
        if (threadIdx.x == 0) any_rot = 0;
        __syncthreads();
        {
          // the rows of the pair: kLoadBatch independent L2 loads in flight per thread
          const unsigned tot = (unsigned)(R2 * L), Lu = (unsigned)L;
          for (unsigned e0 = threadIdx.x; e0 < tot; e0 += blockDim.x * kLoadBatch) {
            T v[kLoadBatch];
#pragma unroll
            for (int u = 0; u < kLoadBatch; ++u) {
              const unsigned e = e0 + u * blockDim.x;
              v[u] = Num<T>::zero();
              if (e < tot) {
                const unsigned i = e / Lu, l = e - i * Lu;
                const int64_t g = grow[i];
                if (g >= 0) v[u] = __ldcg(X + g * L + l);
              }
            }
#pragma unroll
            for (int u = 0; u < kLoadBatch; ++u) {
              const unsigned e = e0 + u * blockDim.x;
              if (e < tot) {
                const unsigned i = e / Lu, l = e - i * Lu;
                Xs[(size_t)i * lmax + l] = v[u];
              }
            }
          }
        }
        __syncthreads();
        for (int inner = 0; inner < inner_sweeps; ++inner) {
          __shared__ int rot_this;
          if (threadIdx.x == 0) rot_this = 0;
          __syncthreads();
          for (int ir = 0; ir < R2 - 1; ++ir) {
            int p, q;
            if (warp == 0) { p = R2 - 1; q = ir; }
            else { p = (ir + warp) % (R2 - 1); q = (ir - warp + (R2 - 1)) % (R2 - 1); }
            if (p > q) { const int t = p; p = q; q = t; }
            if (grow[p] >= 0 && grow[q] >= 0) {
              T* xp = Xs + (size_t)p * lmax;
              T* xq = Xs + (size_t)q * lmax;
              R al_ = 0, be_ = 0;
              T ga_ = Num<T>::zero();
              // rows of at most 32 kRowRegs elements stay in registers between the inner
              // products and the rotation (one shared-memory read and write per element)
              // (only for CTAs of up to 256 threads: wider ones have 128 registers per thread)
              constexpr int RR = (BR <= 8 && sizeof(T) * BR <= 64) ? kRowRegs : 1;
              const bool in_regs = RR == kRowRegs && L <= 32 * kRowRegs;
              T ra[RR], rb[RR];
              if (in_regs) {
#pragma unroll
                for (int u = 0; u < RR; ++u) {
                  const int l = lane + 32 * u;
                  ra[u] = (l < L) ? xp[l] : Num<T>::zero();
                  rb[u] = (l < L) ? xq[l] : Num<T>::zero();
                  al_ += Num<T>::abs2(ra[u]);
                  be_ += Num<T>::abs2(rb[u]);
                  ga_ = Num<T>::fmac(ra[u], rb[u], ga_);
                }
              } else {
                for (int64_t l = lane; l < L; l += 32) {
                  const T a = xp[l], b = xq[l];
                  al_ += Num<T>::abs2(a);
                  be_ += Num<T>::abs2(b);
                  ga_ = Num<T>::fmac(a, b, ga_);
                }
              }
              R c = 0, s = 0;
              T u = Num<T>::one();
              const R thr2 = (R)__longlong_as_double((long long)st[sizeof(R) == 4 ? ST_THR32 : ST_THR64]);
              if (Rotation<T>::get(al_, be_, ga_, L, lane, st + ST_MAXCOS, c, s, u, thr2, mixed)) {
                if (in_regs) {
#pragma unroll
                  for (int v = 0; v < RR; ++v) {
                    const int l = lane + 32 * v;
                    if (l < L) {
                      rot2<T>(ra[v], rb[v], c, s, u);
                      xp[l] = ra[v];
                      xq[l] = rb[v];
                    }
                  }
                } else {
                  for (int64_t l = lane; l < L; l += 32) {
                    T a = xp[l], b = xq[l];
                    rot2<T>(a, b, c, s, u);
                    xp[l] = a;
                    xq[l] = b;
                  }
                }
                for (int l = lane; l < R2; l += 32) {
                  T a = Qs[p * R2 + l], b = Qs[q * R2 + l];
                  rot2<T>(a, b, c, s, u);
                  Qs[p * R2 + l] = a;
                  Qs[q * R2 + l] = b;
                }
                if (lane == 0) { rot_this = 1; any_rot = 1; }
              }
            }
            __syncthreads();
          }
          const int rotated = rot_this;
          __syncthreads();  // every thread has read rot_this before the next sweep resets it
          if (!rotated) break;
        }
        if (any_rot) {
          const unsigned tot = (unsigned)(R2 * L), Lu = (unsigned)L;
          for (unsigned e = threadIdx.x; e < tot; e += blockDim.x) {
            const unsigned i = e / Lu, l = e - i * Lu;
            const int64_t g = grow[i];
            if (g >= 0) X[g * L + l] = Xs[(size_t)i * lmax + l];
          }
          // W rows: W_new = Q W_old for the 2*BR rows, one column per thread at a time
          for (int64_t c = threadIdx.x; c < k; c += blockDim.x) {
            T old[R2];
#pragma unroll
            for (int j = 0; j < R2; ++j) old[j] = (grow[j] >= 0) ? __ldcg(W + grow[j] * k + c) : Num<T>::zero();
#pragma unroll
            for (int i = 0; i < R2; ++i) {
              if (grow[i] < 0) continue;
              T acc = Num<T>::zero();
#pragma unroll
              for (int j = 0; j < R2; ++j) acc = Num<T>::fma_(Qs[i * R2 + j], old[j], acc);
              W[grow[i] * k + c] = acc;
            }
          }
        }
      }
      if (!grid_barrier(ctrl, gridDim.x)) return;
    }
    if (blockIdx.x == 0) {
      if (threadIdx.x == 0) any_active = 0;
      __syncthreads();
      for (int b = threadIdx.x; b < n_blocks; b += blockDim.x) {
        int64_t* st = state + (int64_t)b * ST_REC;
        if (st[ST_CONV]) continue;
        const double mc = __longlong_as_double((long long)st[ST_MAXCOS]);
        const bool conv = stops(mc, __longlong_as_double((long long)st[ST_LASTCOS]), tol_stop, mixed, st[ST_SWEEPS] += 1);
        st[ST_LASTCOS] = conv || sweep + 1 == max_sweeps ? st[ST_MAXCOS] : 0;
        st[ST_MAXCOS] = 0;
        if (conv) st[ST_CONV] = 1; else any_active = 1;
      }
      __syncthreads();
      if (threadIdx.x == 0) ctrl[C_DONE] = any_active ? 0ull : 1ull;
      __threadfence();
    }
    if (!grid_barrier(ctrl, gridDim.x)) return;
    if (((volatile unsigned long long*)ctrl)[C_DONE]) return;
  }
}

template <typename T, int BR>
int launch_block_sweeps(T* work, const int64_t* blocks, int n_blocks, const int32_t* items, int n_items,
                        int max_rounds, int max_sweeps, int inner_sweeps, double tol_stop, int lmax, int64_t* state,
                        cudaStream_t s) {
  const size_t smem = ((size_t)2 * BR * lmax + (size_t)4 * BR * BR) * sizeof(T);
  int dev = 0, sms = 0, per_sm = 0, optin = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&optin, cudaDevAttrMaxSharedMemoryPerBlockOptin, dev);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  if (smem > (size_t)optin) return YB_ERR_TOO_LARGE;
  e = cudaFuncSetAttribute(svd_block_sweeps_kernel<T, BR>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e == cudaSuccess)
    e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, svd_block_sweeps_kernel<T, BR>, BR * 32, smem);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  if (per_sm < 1) return YB_ERR_TOO_LARGE;
  int grid = sms * per_sm;
  if (grid > n_items) grid = n_items;
  if (grid < 1) grid = 1;
  e = cudaMemsetAsync(state + (int64_t)n_blocks * ST_REC, 0, sizeof(int64_t) * C_REC, s);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  void* args[] = {&work, &blocks, &n_blocks, &items, &n_items, &max_rounds, &max_sweeps, &inner_sweeps, &tol_stop,
                  &lmax, &state};
  e = cudaLaunchCooperativeKernel((const void*)svd_block_sweeps_kernel<T, BR>, dim3(grid), dim3(BR * 32), args, smem,
                                  s);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  return YB_OK;
}

// ---------------------------------------------------------------- QR preconditioning
// A block whose spectrum is graded (singular values spread over many decades, as in the
// projector blocks of a corner transfer matrix step) keeps one-sided Jacobi busy for tens of
// FP64 sweeps when started from the rows of A, where the small singular values are hidden
// in cancellations. Started from the rows of the triangular factor R of a Householder QR,
// they are explicit (graded row norms): the FP32 phase then resolves the whole spectrum and
// FP64 needs a few sweeps. With M = X_0^T (A^T for wide/square blocks, conj(A) for tall
// ones; M's columns are the rows of X_0) and M = Q R:
//   wide:  A = R^T Q^T;      W R = S Y  =>  U = Y^T,  Vh = conj(W) Q^T
//   tall:  A = conj(Q R);                 =>  U = conj(Q) W^T,  Vh = conj(Y)
// (Y: rows of X = W R normalised, W: the accumulated rotations). Z holds M's columns as
// rows (Z = X_0, k rows of length L); the factorisation leaves R in Z's upper part and the
// Householder vectors in V (yb_qr.cuh); Q^T is then formed in place (backward accumulation).

// Z = X_0 in FP64 (A, or A^H for tall blocks), scaled by scale[b], a power of two, where it is given
// (see block_fro_kernel). Records with [16] = 2 (yb_qr, M = A): Z's rows are the first k columns of
// A (length L = m).
template <typename T>
__global__ void svd_qr_load_kernel(const T* __restrict__ A, T* __restrict__ work, const int64_t* __restrict__ blocks,
                                   const double* __restrict__ scale) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  if (!r[R_QR]) return;
  const int64_t m = r[R_M], n = r[R_N], k = r[R_K], L = r[R_LQ];
  const bool tall = m > n, plain = r[R_QR] == 2;
  const double sc = scale != nullptr ? scale[blockIdx.y] : 1.0;
  const T* a = A + r[R_A];
  T* Z = work + r[R_Z];
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < k * L; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e / L, l = e - i * L;
    Z[e] = rscale(plain ? a[l * n + i] : (tall ? cconj_(a[l * n + i]) : a[e]), sc);
  }
}

// Candidate vectors of the blocked completion: G (L x nz, row-major per record) filled with
// values uniform in [-1, 1) from a counter-based hash of (record, element) (deterministic;
// any full-rank draw works: the candidates are projected and orthonormalised afterwards).
// recs: int64 pairs (offset, count) per record.
template <typename T>
__global__ void fill_candidates_kernel(T* __restrict__ G, const int64_t* __restrict__ recs) {
  const int64_t off = recs[2 * blockIdx.y], cnt = recs[2 * blockIdx.y + 1];
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < cnt; e += (int64_t)gridDim.x * blockDim.x) {
    uint64_t h = (uint64_t)(off + e) * 0x9E3779B97F4A7C15ull + (uint64_t)blockIdx.y * 0xD1B54A32D192ED03ull;
    h ^= h >> 31; h *= 0xBF58476D1CE4E5B9ull; h ^= h >> 29; h *= 0x94D049BB133111EBull; h ^= h >> 32;
    const double u = (double)(h >> 11) * 0x1.0p-52 - 1.0;
    if constexpr (Num<T>::cplx) {
      const uint64_t h2 = h * 0x2545F4914F6CDD1Dull;
      G[off + e] = make_double2(u, (double)(h2 >> 11) * 0x1.0p-52 - 1.0);
    } else {
      G[off + e] = u;
    }
  }
}

// yb_qr output: Q (m x k, row-major) from Z = Q^T and the square part of R (k x k of the
// k x n rows) from R's rows, both with the signs that make R's diagonal positive (LAPACK's
// diagonal is beta = -sign(Re alpha) |x|: s_c = -1 where it is negative, as the reference's
// sign(diag(R)) fix; a zero diagonal keeps +1). R's entries below the diagonal are zero.
template <typename T>
__global__ void qr_finalize_kernel(const T* __restrict__ work, T* __restrict__ Q, T* __restrict__ Rout,
                                   const int64_t* __restrict__ blocks) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  const int64_t n = r[R_N], k = r[R_K], L = r[R_LQ];
  const T* Z = work + r[R_Z];
  const T* RR = work + r[R_RR];
  T* q = Q + r[R_U];
  T* rr = Rout + r[R_V];
  auto sgn = [&](int64_t c) -> double {
    const T d = RR[c * k + c];
    double re;
    if constexpr (Num<T>::cplx) re = d.x; else re = d;
    return re < 0.0 ? -1.0 : 1.0;
  };
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < L * k; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t l = e / k, c = e - l * k;
    q[e] = rscale(Z[c * L + l], sgn(c));
  }
  for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < k * k; e += (int64_t)gridDim.x * blockDim.x) {
    const int64_t i = e / k, c = e - i * k;
    rr[i * n + c] = (c >= i) ? rscale(RR[e], sgn(i)) : Num<T>::zero();
  }
}

// Finalisation: singular values = row norms, sorted descending (index tie-break), U, S, Vh
// written; vectors of values at noise level are completed to an orthonormal set.
// mode 0: SVD. mode 1/2: Hermitian eigendecomposition of a block shifted by shift[b]
// (lambda = sigma - shift), eigenvectors = columns of W^H, ordered ascending (1) or by
// |lambda| descending (2); Vh is not written.
// It takes three launches: the rows' norms (a warp per row, all SMs) into S, unsorted;
// the vectors, each CTA gathering 32 positions of the descending order through shared memory (both
// the reads of X's and W's rows and the writes of U's columns coalesce); S sorted in place and the
// rows at noise level counted, with their completion, by one CTA per block. Positions are ranks,
// counted on integer keys (FP64 compares would take the FP64 pipe). As one CTA per block it took
// 5.3 ms for two 1296 x 1296 blocks.

// Sort key of a value of S (larger keys first): singular values as they are, eigenvalues ascending
// (mode 1) or by magnitude (mode 2).
__device__ __forceinline__ unsigned long long final_key(double v, int mode) {
  const double x = mode == 1 ? 0.0 - v : (mode == 2 ? fabs(v) : v + 0.0);
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return (long long)b < 0 ? ~b : b | 0x8000000000000000ull;
}

// Position of key i among the k keys: descending, ties by index.
__device__ __forceinline__ int final_rank(const unsigned long long* __restrict__ key, int k, int i) {
  const unsigned long long v = key[i];
  int rank = 0;
#pragma unroll 8
  for (int j = 0; j < i; ++j) rank += key[j] >= v;
#pragma unroll 8
  for (int j = i + 1; j < k; ++j) rank += key[j] > v;
  return rank;
}

template <typename T>
__global__ void svd_norms_kernel(const T* __restrict__ work, double* __restrict__ S, const int64_t* __restrict__ blocks,
                                 int mode, const double* __restrict__ shift) {
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  const int64_t k = r[R_K], L = r[R_L];
  const T* X = work + r[R_X];
  const int lane = threadIdx.x & 31;
  const int64_t nw = (int64_t)gridDim.x * blockDim.x >> 5;
  for (int64_t i = (blockIdx.x * (int64_t)blockDim.x + threadIdx.x) >> 5; i < k; i += nw) {
    double acc = 0.0;
#pragma unroll 4
    for (int64_t l = lane; l < L; l += 32) acc += cabs2(X[i * L + l]);
    acc = warp_sum(acc);
    if (lane == 0) S[r[R_S] + i] = mode == 0 ? sqrt(acc) : sqrt(acc) - shift[blockIdx.y];
  }
}

template <typename T>
__global__ void __launch_bounds__(256) svd_vectors_kernel(T* __restrict__ work, T* __restrict__ U,
                                                          const double* __restrict__ S, T* __restrict__ Vh,
                                                          const int64_t* __restrict__ blocks, int mode,
                                                          const int64_t* __restrict__ state) {
  extern __shared__ unsigned char smem_raw[];
  unsigned long long* key = reinterpret_cast<unsigned long long*>(smem_raw);  // [k]
  __shared__ int row[32];
  __shared__ double inv[32];
  __shared__ T tile[32][33];
  const int64_t* r = blocks + (int64_t)blockIdx.y * YB_SVD_REC;
  const int64_t m = r[R_M], n = r[R_N], k = r[R_K], L = r[R_L];
  const bool tall = m > n, qr = r[R_QR] != 0;
  const T* X = work + r[R_X];
  const T* W = work + r[R_W];
  T* WS = work + r[R_WS];
  T* Ub = U + r[R_U];
  T* Vb = mode == 0 ? Vh + r[R_V] : nullptr;
  const double* Sb = S + r[R_S];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  if ((int64_t)blockIdx.x * 32 >= k) return;
  const double zthr = mode == 0 && state ? sqrt(__longlong_as_double((long long)state[(int64_t)blockIdx.y * ST_REC + ST_THR64])) : 0.0;
  for (int i = threadIdx.x; i < k; i += 256) key[i] = final_key(Sb[i], mode);
  __syncthreads();
  const int j0 = (int)blockIdx.x * 32, nj = min(32, (int)k - j0);
  for (int i = threadIdx.x; i < k; i += 256) {
    const int p = final_rank(key, (int)k, i);
    if (p >= j0 && p < j0 + 32) {
      const double sv = Sb[i];
      row[p - j0] = i;
      inv[p - j0] = (sv > zthr && sv > 0.0) ? 1.0 / sv : 0.0;
    }
  }
  __syncthreads();
  // 32 rows (positions) x 32 entries of a k x len matrix M through the tile: row jj of the tile by
  // load(jj, l); store(jj, l, v) coalesced along jj (by_column) or along l
  auto pass = [&](int64_t len, bool by_column, auto load, auto store) {
    for (int64_t l0 = 0; l0 < len; l0 += 32) {
      __syncthreads();
      for (int jj = warp; jj < nj; jj += 8)
        if (l0 + lane < len) tile[jj][lane] = load(jj, l0 + lane);
      __syncthreads();
      for (int a = warp; a < 32; a += 8) {
        const int jj = by_column ? lane : a;
        const int64_t l = l0 + (by_column ? a : lane);
        if (jj < nj && l < len) store(jj, l, tile[jj][l - l0]);
      }
    }
  };
  if (mode != 0) {  // eigenvectors: columns of W^H
    pass(k, true, [&](int jj, int64_t l) { return cconj_(W[(int64_t)row[jj] * k + l]); },
         [&](int jj, int64_t l, T v) { Ub[l * k + j0 + jj] = v; });
    return;
  }
  // wide (X_0 = A): Vh rows = x_j / s_j, U = W^H; tall (X_0 = A^H): U columns = conj(x_j) / s_j,
  // Vh = W. QR-preconditioned (X_0 = R): wide: U columns = x_j / s_j, and the sorted conj(W)
  // goes to WS for Vh = conj(W) Q^T; tall: Vh rows = conj(x_j) / s_j, WS = sorted W for
  // U = conj(Q) W^T (both products follow as GEMMs). Rows at the rounding-noise level were not
  // rotated: their vectors are zero here and completed like those of zero values.
  const bool to_u = tall != qr;  // the factor built from the rows of X
  pass(L, to_u,
       [&](int jj, int64_t l) {
         const T v = rscale(X[(int64_t)row[jj] * L + l], inv[jj]);
         return tall ? cconj_(v) : v;
       },
       [&](int jj, int64_t l, T v) {
         if (to_u) Ub[l * k + j0 + jj] = v; else Vb[(int64_t)(j0 + jj) * n + l] = v;
       });
  pass(k, !qr && !tall,
       [&](int jj, int64_t l) {
         const T w = W[(int64_t)row[jj] * k + l];
         return tall ? w : cconj_(w);
       },
       [&](int jj, int64_t l, T v) {
         if (qr) WS[(int64_t)(j0 + jj) * k + l] = v;
         else if (tall) Vb[(int64_t)(j0 + jj) * n + l] = v;
         else Ub[l * k + j0 + jj] = v;
       });
}

// S sorted in place (mode 0: and divided by scale[b], where that is given); for an SVD the rows at
// noise level counted and small completions done here.
template <typename T>
__global__ void __launch_bounds__(1024) svd_finalize_kernel(T* __restrict__ U, double* __restrict__ S,
                                                            T* __restrict__ Vh, const int64_t* __restrict__ blocks,
                                                            int mode, const double* __restrict__ scale,
                                                            const int64_t* __restrict__ state,
                                                            int64_t* __restrict__ n_small) {
  extern __shared__ unsigned char smem_raw[];
  const int64_t* r = blocks + (int64_t)blockIdx.x * YB_SVD_REC;
  const int64_t m = r[R_M], n = r[R_N], k = r[R_K], L = r[R_L];
  // [key / real coefficients: k words][values / imaginary coefficients: k doubles]
  unsigned long long* key = reinterpret_cast<unsigned long long*>(smem_raw);
  double* sig = reinterpret_cast<double*>(smem_raw);
  double* cim = sig + k;
  __shared__ int n_zero;
  const bool tall = m > n;
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
  double* Sb = S + r[R_S];
  T* Ub = U + r[R_U];
  T* Vb = Vh + r[R_V];
  if (threadIdx.x == 0) n_zero = 0;
  for (int i = threadIdx.x; i < k; i += blockDim.x) {
    const double v = Sb[i];
    cim[i] = v;
    key[i] = final_key(v, mode);
  }
  __syncthreads();
  const double zthr = mode == 0 && state ? sqrt(__longlong_as_double((long long)state[(int64_t)blockIdx.x * ST_REC + ST_THR64]))
                                         : 0.0;
  const double unscale = mode == 0 && scale ? 1.0 / scale[blockIdx.x] : 1.0;  // a power of two
  for (int i = threadIdx.x; i < k; i += blockDim.x) {
    const double v = cim[i];
    Sb[final_rank(key, (int)k, i)] = v * unscale;
    if (!(v > zthr && v > 0.0)) atomicAdd(&n_zero, 1);
  }
  __syncthreads();
  if (mode != 0 || n_zero == 0) return;
  const bool to_u = tall != (r[R_QR] != 0);  // the factor built from the rows of X
  // large completions (n_zero k L above 2^22) are left to the host's blocked completion
  // (random candidates projected with GEMMs and orthonormalised by yb_qr): the count
  // goes to n_small[b] and the vectors stay as written
  if (n_small != nullptr && (double)n_zero * (double)k * (double)L > 4194304.0) {
    if (threadIdx.x == 0) n_small[blockIdx.x] = n_zero;
    return;
  }
  // completion: the small values sit at the end (positions k - n_zero .. k-1); each of their
  // vectors becomes a unit vector e_c orthogonalised against all earlier vectors by two passes
  // of classical Gram-Schmidt (all coefficients of a pass at once). The candidate is the
  // coordinate least covered by the earlier (orthonormal) vectors, c = argmin_l
  // sum_{i<j} |v_i[l]|^2: its residual norm^2 is 1 minus that sum, at least (L - j) / L since
  // the sums over l add up to j. The coefficients of a pass live in shared memory: real parts
  // in the sig array (no longer needed), imaginary parts in the complex area.
  const int64_t stride_v = to_u ? k : 1;  // distance between consecutive entries of one vector
  const int64_t stride_j = to_u ? 1 : n;  // distance between vectors
  T* base = to_u ? Ub : Vb;
  __shared__ double red[32];
  __shared__ int64_t redi[32];
  __shared__ double nrm_s;
  __shared__ int64_t cand_s;
  double* cre = sig;
  for (int64_t j = k - n_zero; j < k; ++j) {
    T* vj = base + j * stride_j;
    {
      // coverage of each coordinate by v_0..v_{j-1}; block argmin (ties: the smaller l)
      double bv = 3.0e300;
      int64_t bl = L;
      if (to_u) {
        for (int64_t l = warp; l < L; l += nw) {
          double acc = 0.0;
          for (int64_t i = lane; i < j; i += 32) acc += cabs2(base[l * stride_v + i]);
          acc = warp_sum(acc);
          if (acc < bv) { bv = acc; bl = l; }
        }
      } else {
        for (int64_t l = threadIdx.x; l < L; l += blockDim.x) {
          double acc = 0.0;
          for (int64_t i = 0; i < j; ++i) acc += cabs2(base[i * stride_j + l]);
          if (acc < bv) { bv = acc; bl = l; }
        }
      }
      for (int o = 16; o > 0; o >>= 1) {
        const double ov = __shfl_xor_sync(0xffffffffu, bv, o);
        const long long ol = __shfl_xor_sync(0xffffffffu, (long long)bl, o);
        if (ov < bv || (ov == bv && ol < bl)) { bv = ov; bl = ol; }
      }
      if (lane == 0) { red[warp] = bv; redi[warp] = bl; }
      __syncthreads();
      if (threadIdx.x == 0) {
        double v = red[0];
        int64_t c = redi[0];
        for (int w = 1; w < nw; ++w)
          if (red[w] < v || (red[w] == v && redi[w] < c)) { v = red[w]; c = redi[w]; }
        cand_s = c < L ? c : 0;
      }
      __syncthreads();
    }
    const int64_t cand = cand_s;
    {
      for (int64_t l = threadIdx.x; l < L; l += blockDim.x)
        vj[l * stride_v] = (l == cand) ? Num<T>::one() : Num<T>::zero();
      __syncthreads();
      for (int pass = 0; pass < 2; ++pass) {
        // coefficients c_i = <v_i, v_j> = sum_l conj(v_i[l]) v_j[l], i < j
        if (to_u) {
          // vectors are contiguous across i for a fixed l: one thread per i
          for (int64_t i = threadIdx.x; i < j; i += blockDim.x) {
            T acc = Num<T>::zero();
            for (int64_t l = 0; l < L; ++l) acc = Num<T>::fmac(vj[l * stride_v], base[l * stride_v + i], acc);
            if constexpr (Num<T>::cplx) {
              cre[i] = acc.x;
              cim[i] = acc.y;
            } else {
              cre[i] = acc;
            }
          }
        } else {
          // vectors are contiguous along l: one warp per i
          for (int64_t i = warp; i < j; i += nw) {
            T acc = Num<T>::zero();
            for (int64_t l = lane; l < L; l += 32) acc = Num<T>::fmac(vj[l], base[i * stride_j + l], acc);
            warp_sum_t<T>(acc);
            if (lane == 0) {
              if constexpr (Num<T>::cplx) {
                cre[i] = acc.x;
                cim[i] = acc.y;
              } else {
                cre[i] = acc;
              }
            }
          }
        }
        __syncthreads();
        // v_j -= sum_i c_i v_i
        if (to_u) {
          // row l of U holds entry l of every vector: one warp per l
          for (int64_t l = warp; l < L; l += nw) {
            T acc = Num<T>::zero();
            for (int64_t i = lane; i < j; i += 32) {
              T cf;
              if constexpr (Num<T>::cplx) cf = make_double2(cre[i], cim[i]);
              else cf = cre[i];
              acc = Num<T>::add(acc, Num<T>::mul(cf, base[l * stride_v + i]));
            }
            warp_sum_t<T>(acc);
            if (lane == 0) vj[l * stride_v] = Num<T>::sub(vj[l * stride_v], acc);
          }
        } else {
          for (int64_t l = threadIdx.x; l < L; l += blockDim.x) {
            T v = vj[l];
            for (int64_t i = 0; i < j; ++i) {
              T cf;
              if constexpr (Num<T>::cplx) cf = make_double2(cre[i], cim[i]);
              else cf = cre[i];
              v = Num<T>::sub(v, Num<T>::mul(cf, base[i * stride_j + l]));
            }
            vj[l] = v;
          }
        }
        __syncthreads();
      }
      double acc = 0.0;
      for (int64_t l = threadIdx.x; l < L; l += blockDim.x) acc += cabs2(vj[l * stride_v]);
      acc = warp_sum(acc);
      if (lane == 0) red[warp] = acc;
      __syncthreads();
      if (threadIdx.x == 0) {
        double tot = 0.0;
        for (int w = 0; w < nw; ++w) tot += red[w];
        nrm_s = sqrt(tot);
      }
      __syncthreads();
      const double nrm = nrm_s;
      for (int64_t l = threadIdx.x; l < L; l += blockDim.x)
        vj[l * stride_v] = nrm > 0.0 ? rscale(vj[l * stride_v], 1.0 / nrm) : Num<T>::zero();
      __syncthreads();
    }
  }
}

template <typename T>
int launch_sweeps(T* work, const int64_t* blocks, int n_blocks, const int32_t* pair_items, int n_items,
                  int max_rounds, int max_sweeps, double tol_stop, int64_t* state, cudaStream_t s) {
  int dev = 0, sms = 0, per_sm = 0;
  cudaError_t e = cudaGetDevice(&dev);
  if (e == cudaSuccess) e = cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  if (e == cudaSuccess) e = cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, svd_sweeps_kernel<T>, kThreads, 0);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  const int need = (n_items + kWarps - 1) / kWarps;
  int grid = sms * per_sm;
  if (grid > need) grid = need;
  if (grid < 1) grid = 1;
  // zero the barrier/control words (stream-ordered)
  e = cudaMemsetAsync(state + (int64_t)n_blocks * ST_REC, 0, sizeof(int64_t) * C_REC, s);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  void* args[] = {&work, &blocks, &n_blocks, &pair_items, &n_items, &max_rounds, &max_sweeps, &tol_stop, &state};
  e = cudaLaunchCooperativeKernel((const void*)svd_sweeps_kernel<T>, dim3(grid), dim3(kThreads), args, 0, s);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  return YB_OK;
}

}  // namespace

// yb_qr_f64.cu, yb_qr_c128.cu: the factorisation of every block (yb_qr.cuh)
int qr_factor_f64(void* work, void* work32, const int64_t* blocks, int n_blocks, int64_t* qctrl,
                  int qctrl_words, cudaStream_t s);
int qr_factor_c128(void* work, void* work32, const int64_t* blocks, int n_blocks, int64_t* qctrl,
                   int qctrl_words, cudaStream_t s);

template <typename T>
int block_sweeps_t(T* w, const int64_t* blocks, int n_blocks, const int32_t* super_items, int n_items,
                          int max_rounds, int rows_per_super, int max_sweeps, int inner_sweeps, double tol_stop,
                          int lmax, int64_t* state, cudaStream_t s) {
  constexpr bool fp64 = sizeof(typename Num<T>::R) == 8;
  switch (rows_per_super) {
    case 16:
      if constexpr (fp64) return YB_ERR_INVALID;
      else return yb::launch_block_sweeps<T, 16>(w, blocks, n_blocks, super_items, n_items, max_rounds, max_sweeps,
                                                 inner_sweeps, tol_stop, lmax, state, s);
    case 8: return yb::launch_block_sweeps<T, 8>(w, blocks, n_blocks, super_items, n_items, max_rounds, max_sweeps,
                                                inner_sweeps, tol_stop, lmax, state, s);
    case 4: return yb::launch_block_sweeps<T, 4>(w, blocks, n_blocks, super_items, n_items, max_rounds, max_sweeps,
                                                inner_sweeps, tol_stop, lmax, state, s);
    default: return YB_ERR_INVALID;
  }
}

template <typename T>
int qr_t(const void* a, void* work, void* work32, const int64_t* blocks, int n_blocks, int64_t* state, double* scale,
         int64_t* qctrl, int qctrl_words, cudaStream_t s) {
  if (state) block_fro_kernel<T><<<dim3(kFroCtas, (unsigned)n_blocks), 256, 0, s>>>((const T*)a, blocks, nullptr, scale, state);
  svd_qr_load_kernel<T><<<dim3(64, (unsigned)n_blocks), 256, 0, s>>>((const T*)a, (T*)work, blocks, scale);
  const int st = Num<T>::cplx ? qr_factor_c128(work, work32, blocks, n_blocks, qctrl, qctrl_words, s)
                              : qr_factor_f64(work, work32, blocks, n_blocks, qctrl, qctrl_words, s);
  if (st != YB_OK) return st;
  if (state) svd_state_reset_kernel<<<n_blocks, 32, 0, s>>>(state);
  return check_launch();
}

template <typename T>
int finalize_t(void* work, void* U, double* S, void* Vh, const int64_t* blocks, int n_blocks, int max_k,
                      int mode, const double* shift, const int64_t* state, int64_t* n_small, cudaStream_t s) {
  const size_t keys = (size_t)max_k * sizeof(double), smem = 2 * keys;
  auto vec = svd_vectors_kernel<T>;
  auto fin = svd_finalize_kernel<T>;
  cudaError_t e = cudaSuccess;
  // dynamic and static shared memory together may pass 48 KB: up to 17.5 KB static in the vectors'
  // kernel, half a KB in the last one
  if (keys > 24 * 1024) e = cudaFuncSetAttribute(vec, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)keys);
  if (e == cudaSuccess && smem > 32 * 1024)
    e = cudaFuncSetAttribute(fin, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
  if (e != cudaSuccess) { set_cuda_error((int)e); return YB_ERR_CUDA; }
  const unsigned tiles = (unsigned)((max_k + 31) / 32), nb = (unsigned)n_blocks;
  svd_norms_kernel<T><<<dim3(tiles * 4 < 128 ? tiles * 4 : 128, nb), 256, 0, s>>>((const T*)work, S, blocks, mode, shift);
  vec<<<dim3(tiles, nb), 256, keys, s>>>((T*)work, (T*)U, S, (T*)Vh, blocks, mode, state);
  fin<<<nb, 1024, smem, s>>>((T*)U, S, (T*)Vh, blocks, mode, shift, state, n_small);
  return check_launch();
}

}  // namespace yb

extern "C" {

int yb_svd_init(const void* a, void* work32, const int64_t* blocks, int n_blocks, int dtype, int64_t* state,
                double* shift, double* scale, void* stream) {
  if (n_blocks == 0) return YB_OK;
  if (dtype != YB_F64 && dtype != YB_C128) return YB_ERR_INVALID;
  if (!a || !work32 || !blocks || !state || !scale) return YB_ERR_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  dim3 grid(64, (unsigned)n_blocks);
  if (dtype == YB_F64) {
    yb::block_fro_kernel<double><<<dim3(yb::kFroCtas, (unsigned)n_blocks), 256, 0, s>>>((const double*)a, blocks, shift, scale, state);
    yb::svd_init_kernel<double, float><<<grid, 256, 0, s>>>((const double*)a, (float*)work32, blocks, state, shift,
                                                            scale);
  } else {
    yb::block_fro_kernel<double2><<<dim3(yb::kFroCtas, (unsigned)n_blocks), 256, 0, s>>>((const double2*)a, blocks, shift, scale, state);
    yb::svd_init_kernel<double2, float2><<<grid, 256, 0, s>>>((const double2*)a, (float2*)work32, blocks, state,
                                                              shift, scale);
  }
  return yb::check_launch();
}

int yb_svd_qr(const void* a, void* work64, void* work32, const int64_t* blocks, int n_blocks, int dtype,
              int64_t* state, double* scale, int64_t* qctrl, int qctrl_words, void* stream) {
  if (n_blocks == 0) return YB_OK;
  if (dtype != YB_F64 && dtype != YB_C128) return YB_ERR_INVALID;
  if (!a || !work64 || !work32 || !blocks || !state || !scale || !qctrl) return YB_ERR_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == YB_F64)
    return yb::qr_t<double>(a, work64, work32, blocks, n_blocks, state, scale, qctrl, qctrl_words, s);
  return yb::qr_t<double2>(a, work64, work32, blocks, n_blocks, state, scale, qctrl, qctrl_words, s);
}

int yb_fill_candidates(void* G, const int64_t* recs, int n_recs, int dtype, void* stream) {
  if (n_recs == 0) return YB_OK;
  if (!G || !recs) return YB_ERR_INVALID;
  const dim3 grid(32, (unsigned)n_recs);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == YB_F64) yb::fill_candidates_kernel<double><<<grid, 256, 0, s>>>((double*)G, recs);
  else if (dtype == YB_C128) yb::fill_candidates_kernel<double2><<<grid, 256, 0, s>>>((double2*)G, recs);
  else return YB_ERR_INVALID;
  return yb::check_launch();
}

int yb_qr(const void* a, void* Q, void* R, void* work64, const int64_t* blocks, int n_blocks, int dtype,
          int64_t* qctrl, int qctrl_words, void* stream) {
  if (n_blocks == 0) return YB_OK;
  if (dtype != YB_F64 && dtype != YB_C128) return YB_ERR_INVALID;
  if (!a || !Q || !R || !work64 || !blocks || !qctrl) return YB_ERR_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  const dim3 grid(64, (unsigned)n_blocks);
  int st;
  if (dtype == YB_F64) {
    st = yb::qr_t<double>(a, work64, nullptr, blocks, n_blocks, nullptr, nullptr, qctrl, qctrl_words, s);
    if (st != YB_OK) return st;
    yb::qr_finalize_kernel<double><<<grid, 256, 0, s>>>((const double*)work64, (double*)Q, (double*)R, blocks);
  } else {
    st = yb::qr_t<double2>(a, work64, nullptr, blocks, n_blocks, nullptr, nullptr, qctrl, qctrl_words, s);
    if (st != YB_OK) return st;
    yb::qr_finalize_kernel<double2><<<grid, 256, 0, s>>>((const double2*)work64, (double2*)Q, (double2*)R, blocks);
  }
  return yb::check_launch();
}

int yb_svd_sweeps(void* work, const int64_t* blocks, int n_blocks, const int32_t* pair_items, int n_pair_items,
                  int max_rounds, int precision, int dtype, int max_sweeps, double tol_stop, int64_t* state,
                  void* stream) {
  if (n_blocks == 0 || n_pair_items == 0 || max_sweeps <= 0) return YB_OK;
  if (!work || !blocks || !pair_items || !state) return YB_ERR_INVALID;
  if (dtype != YB_F64 && dtype != YB_C128) return YB_ERR_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  const bool c = dtype == YB_C128;
  if (precision == 32 && !c)
    return yb::launch_sweeps<float>((float*)work, blocks, n_blocks, pair_items, n_pair_items, max_rounds, max_sweeps,
                                    tol_stop, state, s);
  if (precision == 32 && c)
    return yb::launch_sweeps<float2>((float2*)work, blocks, n_blocks, pair_items, n_pair_items, max_rounds,
                                     max_sweeps, tol_stop, state, s);
  if (precision == 64 && !c)
    return yb::launch_sweeps<double>((double*)work, blocks, n_blocks, pair_items, n_pair_items, max_rounds,
                                     max_sweeps, tol_stop, state, s);
  if (precision == 64 && c)
    return yb::launch_sweeps<double2>((double2*)work, blocks, n_blocks, pair_items, n_pair_items, max_rounds,
                                      max_sweeps, tol_stop, state, s);
  return YB_ERR_INVALID;
}

int yb_svd_block_sweeps(void* work32, const int64_t* blocks, int n_blocks, const int32_t* super_items,
                        int n_items, int max_rounds, int rows_per_super, int precision, int dtype, int max_sweeps,
                        int inner_sweeps, double tol_stop, int lmax, int64_t* state, void* stream) {
  if (n_blocks == 0 || n_items == 0 || max_sweeps <= 0) return YB_OK;
  if (!work32 || !blocks || !super_items || !state || lmax <= 0 || inner_sweeps <= 0) return YB_ERR_INVALID;
  if (precision != 32 && precision != 64) return YB_ERR_INVALID;
  cudaStream_t s = (cudaStream_t)stream;
  if (precision == 64) {
    if (rows_per_super != 4 && rows_per_super != 8) return YB_ERR_INVALID;
    if (dtype == YB_F64)
      return yb::block_sweeps_t<double>((double*)work32, blocks, n_blocks, super_items, n_items, max_rounds,
                                        rows_per_super, max_sweeps, inner_sweeps, tol_stop, lmax, state, s);
    if (dtype == YB_C128)
      return yb::block_sweeps_t<double2>((double2*)work32, blocks, n_blocks, super_items, n_items, max_rounds,
                                         rows_per_super, max_sweeps, inner_sweeps, tol_stop, lmax, state, s);
    return YB_ERR_INVALID;
  }
  if (dtype == YB_F64)
    return yb::block_sweeps_t<float>((float*)work32, blocks, n_blocks, super_items, n_items, max_rounds, rows_per_super,
                                 max_sweeps, inner_sweeps, tol_stop, lmax, state, s);
  if (dtype == YB_C128)
    return yb::block_sweeps_t<float2>((float2*)work32, blocks, n_blocks, super_items, n_items, max_rounds,
                                  rows_per_super, max_sweeps, inner_sweeps, tol_stop, lmax, state, s);
  return YB_ERR_INVALID;
}

int yb_svd_widen(const void* work32, void* work64, const int64_t* blocks, int n_blocks, int dtype, int64_t* state,
                 void* stream) {
  if (n_blocks == 0) return YB_OK;
  if (!work32 || !work64 || !blocks || !state) return YB_ERR_INVALID;
  dim3 grid(64, (unsigned)n_blocks);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == YB_F64)
    yb::svd_widen_kernel<float, double><<<grid, 256, 0, s>>>((const float*)work32, (double*)work64, blocks, state);
  else if (dtype == YB_C128)
    yb::svd_widen_kernel<float2, double2><<<grid, 256, 0, s>>>((const float2*)work32, (double2*)work64, blocks,
                                                               state);
  else
    return YB_ERR_INVALID;
  return yb::check_launch();
}

int yb_svd_ns_prep(void* work64, const int64_t* blocks, int n_blocks, int dtype, int64_t t_delta, void* stream) {
  if (n_blocks == 0) return YB_OK;
  if (!work64 || !blocks || t_delta <= 0) return YB_ERR_INVALID;
  const dim3 grid(64, (unsigned)n_blocks);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == YB_F64) yb::svd_ns_prep_kernel<double><<<grid, 256, 0, s>>>((double*)work64, blocks, t_delta);
  else if (dtype == YB_C128) yb::svd_ns_prep_kernel<double2><<<grid, 256, 0, s>>>((double2*)work64, blocks, t_delta);
  else return YB_ERR_INVALID;
  return yb::check_launch();
}

int yb_svd_scale_wr(void* work64, const int64_t* blocks, int n_blocks, int dtype, int64_t t_delta, int k_min,
                    int64_t* state, void* stream) {
  if (n_blocks == 0) return YB_OK;
  if (!work64 || !blocks || !state || t_delta <= 0) return YB_ERR_INVALID;
  const dim3 grid(64, (unsigned)n_blocks);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == YB_F64) {
    yb::svd_col_exponents_kernel<double><<<grid, 256, 0, s>>>((double*)work64, blocks, k_min, state);
    yb::svd_row_scales_kernel<double><<<grid, 256, 0, s>>>((double*)work64, blocks);
    yb::svd_scale_wr_kernel<double><<<grid, 256, 0, s>>>((double*)work64, blocks, t_delta);
  } else if (dtype == YB_C128) {
    yb::svd_col_exponents_kernel<double2><<<grid, 256, 0, s>>>((double2*)work64, blocks, k_min, state);
    yb::svd_row_scales_kernel<double2><<<grid, 256, 0, s>>>((double2*)work64, blocks);
    yb::svd_scale_wr_kernel<double2><<<grid, 256, 0, s>>>((double2*)work64, blocks, t_delta);
  } else {
    return YB_ERR_INVALID;
  }
  return yb::check_launch();
}

int yb_svd_poison(void* U, void* V, const int64_t* blocks, int n_blocks, int dtype, const int64_t* state, int k_min,
                  int which, void* stream) {
  if (n_blocks == 0) return YB_OK;
  if (!U || !blocks || !state || which < 0 || which > 1 || (which == 1 && !V)) return YB_ERR_INVALID;
  const dim3 grid(8, (unsigned)n_blocks);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == YB_F64)
    yb::svd_poison_kernel<double><<<grid, 256, 0, s>>>((double*)U, (double*)V, blocks, state, k_min, which);
  else if (dtype == YB_C128)
    yb::svd_poison_kernel<double2><<<grid, 256, 0, s>>>((double2*)U, (double2*)V, blocks, state, k_min, which);
  else
    return YB_ERR_INVALID;
  return yb::check_launch();
}

int yb_svd_shift_prefill(void* work64, const int64_t* blocks, int n_blocks, int dtype, const double* shift,
                         void* stream) {
  if (n_blocks == 0) return YB_OK;
  if (!work64 || !blocks || !shift) return YB_ERR_INVALID;
  dim3 grid(64, (unsigned)n_blocks);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == YB_F64)
    yb::svd_shift_prefill_kernel<double><<<grid, 256, 0, s>>>((double*)work64, blocks, shift);
  else if (dtype == YB_C128)
    yb::svd_shift_prefill_kernel<double2><<<grid, 256, 0, s>>>((double2*)work64, blocks, shift);
  else
    return YB_ERR_INVALID;
  return yb::check_launch();
}

int yb_svd_graded(const void* work64, const int64_t* blocks, int n_blocks, int dtype, int k_min, const int64_t* state,
                  const int64_t* at_masks, int32_t* masks, int64_t* flags, void* stream) {
  if (n_blocks == 0) return YB_OK;
  if (!work64 || !blocks || !state || !at_masks || !masks || !flags) return YB_ERR_INVALID;
  const dim3 grid(64, (unsigned)n_blocks);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == YB_F64)
    yb::svd_graded_masks_kernel<double><<<grid, 256, 0, s>>>((const double*)work64, blocks, k_min, state, at_masks, masks);
  else if (dtype == YB_C128)
    yb::svd_graded_masks_kernel<double2><<<grid, 256, 0, s>>>((const double2*)work64, blocks, k_min, state, at_masks, masks);
  else
    return YB_ERR_INVALID;
  yb::svd_graded_pairs_kernel<<<dim3(152, (unsigned)n_blocks), 256, 0, s>>>(blocks, k_min, at_masks, masks);
  yb::svd_graded_flags_kernel<<<dim3(1, (unsigned)n_blocks), 256, 0, s>>>(blocks, k_min, at_masks, masks, flags);
  return yb::check_launch();
}

int yb_svd_scale_x(void* work64, const int64_t* blocks, int n_blocks, int dtype, const double* scale, void* stream) {
  if (n_blocks == 0) return YB_OK;
  if (!work64 || !blocks || !scale) return YB_ERR_INVALID;
  const dim3 grid(64, (unsigned)n_blocks);
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == YB_F64) yb::svd_scale_x_kernel<double><<<grid, 256, 0, s>>>((double*)work64, blocks, scale);
  else if (dtype == YB_C128) yb::svd_scale_x_kernel<double2><<<grid, 256, 0, s>>>((double2*)work64, blocks, scale);
  else return YB_ERR_INVALID;
  return yb::check_launch();
}

int yb_svd_finalize(void* work, void* U, double* S, void* Vh, const int64_t* blocks, int n_blocks, int dtype,
                    int max_k, int mode, const double* shift, const int64_t* state, int64_t* n_small,
                    void* stream) {
  if (n_blocks == 0) return YB_OK;
  if (dtype != YB_F64 && dtype != YB_C128) return YB_ERR_INVALID;
  if (mode < 0 || mode > 2 || (mode != 0 && shift == nullptr)) return YB_ERR_INVALID;
  if (max_k > 8192) return YB_ERR_TOO_LARGE;
  if (max_k <= 0) return YB_OK;
  cudaStream_t s = (cudaStream_t)stream;
  if (dtype == YB_F64)
    return yb::finalize_t<double>(work, U, S, Vh, blocks, n_blocks, max_k, mode, shift, state, n_small, s);
  return yb::finalize_t<double2>(work, U, S, Vh, blocks, n_blocks, max_k, mode, shift, state, n_small, s);
}

}  // extern "C"
