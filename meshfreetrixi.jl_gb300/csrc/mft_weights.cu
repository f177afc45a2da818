// K2: batched FP64 polyharmonic-spline + polynomial RBF-FD weights.
//
// Restates the per-node loop of compute_flux_operator
// (src/solvers/pointcloudsolver/compute_operators.jl:409-453 and :549-594):
//   shift_stencil (:225-246)  X^_j = (X_j - X_centre) * s,  s_d = 1/max_j |dX_jd|
//   M = [R P; P' 0] upper (interpolation_block :265-267), R_ij = |X^_i - X^_j|^p,
//   P_im = monomial_m(X^_i)
//   RHS: d^k/dx_d^k of |x - X^_j|^p at the centre (mirror_stencil :248-263 with the
//   centre entry at (eps,...,eps)), monomial derivatives at the origin
//   w = M \ rhs by Bunch-Kaufman (LAPACK dsytf2 + dsytrs, upper), weights s_d^k w.
//
// One warp per system (several for the large ones), the system in shared memory, one
// persistent launch over all nodes with a work counter; systems are taken largest first so
// that uneven stencil sizes (interior vs boundary, 2D vs 3D) balance across warps.  Every
// matrix element sees the same sequence of separately rounded operations as in the CPU
// restatement (updates are element-independent and the solve's dot products use a fixed
// 32-way strided partial-sum order), so the weights are bit-identical to it.
//
// What bounds it: the FP64 pipe, which takes one warp instruction per ~17 cycles and SM
// whatever the number of active lanes (85 % busy, 65,536 systems of n = 45).  So the design
// minimises FP64 warp instructions, not operations: magnitudes are compared as integers, the
// forward solve runs inside the factorisation (one division per pivot for both), divisions
// with one divisor and tree sums of several right-hand sides share instructions, pivot tests
// are decided in FP32 where they are clear.  262,144 systems of n = 45: 71.2 -> 33 ms (5800 ->
// 2150 FP64 instructions per system; 475 of them are the factorisation's multiply-adds).
#include <cuda_runtime.h>
#include <math.h>

#include <string.h>

#include <algorithm>
#include <mutex>
#include <numeric>
#include <string>
#include <vector>

#include "mft_ctx.h"
#include "mft_fpbits.h"

namespace mft {

namespace {

constexpr int kWarpsPerBlock = 2;  // systems per block with one warp per system
// Larger systems share several warps: their packed matrices limit an SM to a few systems, and
// one warp each leaves the FP64 pipe idle behind shared-memory and reduction latencies, while
// every column step of several warps costs block barriers.  Measured on 32,768 stencils (2D k
// 35 / 40-60, 3D k 60-90), per bucket of n = k + monomials: n > 80: 2.21 ms with two warps,
// 2.05 with three, 2.06 with four; 64 < n <= 80: 1.02 / 0.88 / 0.95 with one / two / three;
// 48 < n <= 64: 0.565 / 0.514 with one / two; n <= 48: 3.37 / 4.33 (one warp).
__host__ __device__ constexpr int system_warps(int n) { return n > 80 ? 3 : n > 48 ? 2 : 1; }
constexpr unsigned kFull = 0xffffffffu;

// One batch of stencils sharing dimension, basis and derivative order.
constexpr int kMaxMono = 84;  // monomials of total degree <= 6 in 3D
struct WGroup {
  int dim, npoly, rbf_pow, order;
  int periodic;
  double period[3];
  const int64_t* rowptr;
  const int32_t* cols;
  const double* xyz;
  double* w_out;  // nnz x dim (stencil order)
  double* resid;  // optional per node
  int mono[kMaxMono][3];
  // monomial m of a row as a product of two earlier ones (msrc, indices), of one
  // coordinate (msrc[m][0] = -2 - axis) or 1 (msrc[m][0] = -1): the products
  // pow_int(x, a) pow_int(y, b) pow_int(z, c) take, in the same order
  int16_t msrc[kMaxMono][2];
  // the terms of phs_deriv (cc pow(2 x_d, ex)) cm pow(r, er), j ascending, and order!
  int nterm;
  double term_cc[5], term_cm[5];
  int term_ex[5], term_er[5];
  double fact_order;
};

constexpr int kMaxGroups = 2;
// Work item codes: group << kGroupShift | node.
constexpr int kGroupShift = 48;

struct WArgs {
  int nmax, kmax, dmax;
  int64_t nsys;
  const int64_t* order_list;  // work item codes, largest stencil first
  int* bad;                   // smallest node index with a zero pivot, or INT_MAX
  unsigned long long* next;
  WGroup g[kMaxGroups];
};

__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ddiv(double a, double b) { return __ddiv_rn(a, b); }

// x^k by repeated multiplication from the left (1 x = x exactly); 1 / x^-k for k < 0
__device__ __forceinline__ double pow_int(double x, int k) {
  if (k == 0) return 1.0;
  double r = x;
  for (int i = 1; i < (k < 0 ? -k : k); ++i) r = dmul(r, x);
  return k < 0 ? ddiv(1.0, r) : r;
}

// d^k/dx_d^k of r^p (Faa di Bruno on s^(p/2), s = |x|^2) with the group's constants; same
// operation order as the CPU restatement.
__device__ __forceinline__ double phs_deriv(const WGroup& g, double xd, double r) {
  double sum = 0.0;
  for (int j = 0; j < g.nterm; ++j)
    sum = dadd(sum, dmul(dmul(dmul(g.term_cc[j], pow_int(dmul(2.0, xd), g.term_ex[j])),
                              g.term_cm[j]),
                         pow_int(r, g.term_er[j])));
  return sum;
}

__device__ __forceinline__ double min_image(double d, double L) {
  if (d > 0.5 * L) return dsub(d, L);
  if (d < -0.5 * L) return dadd(d, L);
  return d;
}

// Magnitudes are compared on their bit patterns (for values >= 0 the order of the patterns
// is the order of the values), because an FP64 comparison takes a slot of the FP64 pipe,
// which bounds these kernels: one warp instruction per ~17 cycles and SM, whatever the
// number of active lanes (measured), against four integer ones per cycle.
// The patterns are handled as two 32-bit words: the compiler turns tests for NaN or zero on a
// 64-bit pattern back into FP64 comparisons.
struct Words { unsigned hi, lo; };
__device__ __forceinline__ Words mag_words(double x) {
  return {(unsigned)__double2hiint(x) & 0x7FFFFFFFu, (unsigned)__double2loint(x)};
}
__device__ __forceinline__ bool words_nan(Words w) {
  return w.hi > 0x7FF00000u || (w.hi == 0x7FF00000u && w.lo != 0);
}
__device__ __forceinline__ bool nonzero(double x) {
  const Words w = mag_words(x);
  return (w.hi | w.lo) != 0;
}
// Search key of |x|: its pattern + 1, and 0 for NaN (which never wins a search) and for
// "no candidate".
__device__ __forceinline__ unsigned long long mag_key(double x) {
  const Words w = mag_words(x);
  const unsigned long long k = (((unsigned long long)w.hi << 32) | w.lo) + 1;
  return words_nan(w) ? 0ull : k;
}
__device__ __forceinline__ double key_value(unsigned long long key) {
  const unsigned long long b = key ? key - 1 : 0x7FF8000000000000ull;
  return __hiloint2double((int)(b >> 32), (int)b);
}
// a >= b for a, b >= 0 (false when either is NaN)
__device__ __forceinline__ bool mag_ge(double a, double b) {
  const unsigned long long ka = mag_key(a), kb = mag_key(b);
  return ka >= kb && kb != 0;
}

// Largest key of a warp: the high words' maximum, then the low words' among its holders.
__device__ __forceinline__ unsigned long long warp_max_key(unsigned long long k) {
  const unsigned hi = (unsigned)(k >> 32);
  const unsigned mh = __reduce_max_sync(kFull, hi);
  const unsigned ml = __reduce_max_sync(kFull, hi == mh ? (unsigned)k : 0u);
  return ((unsigned long long)mh << 32) | ml;
}

// Synchronisation of the threads that share one system: the warp (W == 1) or the block.
template <int W>
__device__ __forceinline__ void gsync() {
  if (W == 1) __syncwarp();
  else __syncthreads();
}

// Largest key over the threads that share a system, and the smallest index that holds it
// (i: the thread's candidate, 1 << 30 for none; red_k, red_i: W-entry shared scratch).
// Every thread of the block must call it when W > 1.  Without any candidate (all NaN) the
// index is `lo`, so that every later access stays inside the system.
template <int W>
__device__ __forceinline__ void group_argmax(unsigned long long& k, int& i, int lo,
                                             unsigned long long* red_k, int* red_i) {
  const unsigned long long m = warp_max_key(k);
  i = __reduce_min_sync(kFull, k == m ? i : (1 << 30));
  k = m;
  if (W > 1) {
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) { red_k[w] = k; red_i[w] = i; }
    __syncthreads();
    k = red_k[0];
    i = red_i[0];
    for (int q = 1; q < W; ++q) {
      const unsigned long long k2 = red_k[q];
      const int i2 = red_i[q];
      if (k2 > k || (k2 == k && i2 < i)) { k = k2; i = i2; }
    }
    __syncthreads();
  }
  if (k == 0) i = lo;
}

template <int W>
__device__ __forceinline__ unsigned long long group_max_key(unsigned long long k,
                                                            unsigned long long* red_k) {
  k = warp_max_key(k);
  if (W > 1) {
    const int w = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0) red_k[w] = k;
    __syncthreads();
    k = red_k[0];
    for (int q = 1; q < W; ++q) k = red_k[q] > k ? red_k[q] : k;
    __syncthreads();
  }
  return k;
}

__device__ __forceinline__ double warp_max(double v) {
  for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(kFull, v, o));
  return v;
}

// The tree sum over a warp of ND values per lane, each in the order of a
// __shfl_down tree (lane l adds lane l + 16, then + 8, ...).  While several values are
// left, a level's two halves of the lanes reduce different ones: lanes with bit `o` clear
// keep the first of a pair, the others the second (an FP64 addition serves both; addition
// commutes, so the sums keep their bits).  The total of value d lands in the lane whose
// low bits fold_lane gives.
template <int ND>
__device__ __forceinline__ double fold_sums(double (&v)[ND], int lane) {
  int nd = ND;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    const bool up = (lane & o) != 0;
    if (nd > 1) {
#pragma unroll
      for (int d = 0; d < ND; d += 2) {
        if (d >= nd) continue;
        const double a = v[d], b = d + 1 < nd ? v[(d + 1) % ND] : v[d];
        const double got = __shfl_xor_sync(kFull, up ? a : b, o);
        v[d / 2] = dadd(up ? b : a, got);
      }
      nd = (nd + 1) / 2;
    } else {
      v[0] = dadd(v[0], __shfl_xor_sync(kFull, v[0], o));
    }
  }
  return v[0];
}
// Lane that holds value d of fold_sums<ND>: bit 16 >> q of the lane is bit q of d (the
// remaining bits are zero).
__host__ __device__ constexpr int fold_lane(int d) {
  return ((d & 1) << 4) | ((d & 2) << 2) | (d & 4);
}

// Row i and column j (0 <= i <= j) of element t of the upper triangle packed by columns
// (t = j(j+1)/2 + i): j = floor((sqrt(8t + 1) - 1) / 2) from an FP32 square root, off by at
// most one for t < 2^20, then corrected.  No loop over columns: stepping from element to
// element with one made the lanes of a warp diverge (an update of 475 full-warp
// multiply-adds took 722 warp instructions at n = 45).
__device__ __forceinline__ void tri_rc(int t, int& i, int& j) {
  float q;
  asm("sqrt.approx.f32 %0, %1;" : "=f"(q) : "f"((float)(8 * t + 1)));
  int c = (int)((q - 1.0f) * 0.5f);
  if (((c * (c + 1)) >> 1) > t) --c;
  if ((((c + 1) * (c + 2)) >> 1) <= t) ++c;
  j = c;
  i = t - ((c * (c + 1)) >> 1);
}

// num / den; a zero numerator (common: the zero block, the right-hand sides) over a nonzero
// number is formed directly, off the division's slow path.
__device__ __forceinline__ double div0(double num, double den) {
  const bool zero = !nonzero(num) && mag_key(den) > 1;
  const double q = ddiv(zero ? 1.0 : num, den);
  const int sign = (__double2hiint(num) ^ __double2hiint(den)) & (int)0x80000000;
  return zero ? __hiloint2double(sign, 0) : q;
}

// dsytf2's tests, for a, b, c >= 0: a >= alpha b, and a >= (alpha b) (b / c), decided in FP32
// when the two sides differ by more than the FP32 evaluation's error (three conversions, a
// division and two multiplications: < 1e-6 relative); the FP64 expression otherwise.
__device__ __forceinline__ bool fp32_range(float x) { return x >= 1e-9f && x <= 1e9f; }
__device__ __forceinline__ bool ge_scaled(double a, double alpha, double b) {
  const float fa = fpconv::d2f(a), fb = fpconv::d2f(b);
  if (fp32_range(fa) && fp32_range(fb)) {
    const float t = __fmul_rn((float)alpha, fb);
    if (fa > t * 1.00001f) return true;
    if (fa < t * 0.99999f) return false;
  }
  return mag_ge(a, dmul(alpha, b));
}
__device__ __forceinline__ bool ge_scaled_ratio(double a, double alpha, double b, double c) {
  const float fa = fpconv::d2f(a), fb = fpconv::d2f(b), fc = fpconv::d2f(c);
  if (fp32_range(fa) && fp32_range(fb) && fp32_range(fc)) {
    const float t = __fmul_rn(__fmul_rn((float)alpha, fb), __fdiv_rn(fb, fc));
    if (fa > t * 1.00001f) return true;
    if (fa < t * 0.99999f) return false;
  }
  return mag_ge(a, dmul(dmul(alpha, b), ddiv(b, c)));
}

// Rows kk .. kk + NC - 1 of the backward solve: B(row, c) -= sum_{i < kk} B(i, c) A(i, row)
// for the NR right-hand sides (A packed upper by columns, B n x NR).
template <int NR, int NC>
__device__ __forceinline__ void back_step(const double* A, double* B, int n, int kk, int lane) {
  constexpr int ND = NR * NC;
  // Short rows: the lanes beyond the row's length would hold +0 partials (and the first
  // levels of the tree add only those), so lanes in groups of L, the length rounded up to a
  // power of two, take one dot product each: one multiply-add and log2 L additions.
  int L = 1;
  while (L < kk - 1) L <<= 1;
  if (ND * L <= 32) {
    const int d = lane / L, i = lane & (L - 1);
    const bool on = d < ND && i < kk - 1;
    const int c = d / NC, q = d - c * NC;
    double v = 0.0;
    if (on) v = fma(B[c * n + i], A[(((kk + q) * (kk + q - 1)) >> 1) + i], 0.0);
    for (int o = L >> 1; o > 0; o >>= 1) v = dadd(v, __shfl_xor_sync(kFull, v, o));
    if (on && i == 0) B[c * n + kk - 1 + q] = dsub(B[c * n + kk - 1 + q], v);
    __syncwarp();
    return;
  }
  double part[ND];
#pragma unroll
  for (int d = 0; d < ND; ++d) part[d] = 0.0;
  const double* col0 = A + ((kk * (kk - 1)) >> 1);  // rows 1.. of column kk
  const double* col1 = col0 + kk;                   // and of column kk + 1
  for (int i = lane; i < kk - 1; i += 32) {
    const double a0 = col0[i], a1 = NC > 1 ? col1[i] : 0.0;
#pragma unroll
    for (int c = 0; c < NR; ++c) {
      const double b = B[c * n + i];
      part[c * NC] = fma(b, a0, part[c * NC]);
      if (NC > 1) part[c * NC + NC - 1] = fma(b, a1, part[c * NC + NC - 1]);
    }
  }
  const double sum = fold_sums<ND>(part, lane);
#pragma unroll
  for (int d = 0; d < ND; ++d)
    if (lane == fold_lane(d)) {
      double& x = B[(d / NC) * n + kk - 1 + d % NC];
      x = dsub(x, sum);
    }
  __syncwarp();
}

// Doubles of shared memory one warp of k_weights uses: the upper triangle of A packed by
// columns (nmax (nmax + 1) / 2; Bunch-Kaufman in upper storage reads and writes only
// i <= j), B (dmax nmax), X (dmax kmax), two column-multiplier arrays (2 nmax) and the pivot
// ints (nmax, two to a double); dmax: the largest dimension of the launch's systems.
__host__ __device__ __forceinline__ size_t weights_smem_doubles(int nmax, int kmax, int dmax) {
  return (size_t)nmax * (nmax + 1) / 2 + (size_t)nmax * dmax + (size_t)kmax * dmax +
         (size_t)nmax * 2 + (nmax + 1) / 2;
}

// The size test of the entry points: a system is accepted when its storage with every array
// at three dimensions (and a double per pivot) fits, a bound the layout above stays below.
__host__ __forceinline__ size_t weights_limit_doubles(int nmax, int kmax) {
  return (size_t)nmax * (nmax + 1) / 2 + (size_t)nmax * 6 + (size_t)kmax * 3;
}

// kOrdered: systems are taken in the order of a.order_list (largest first); otherwise
// in node order.
template <bool kOrdered, int W>
__global__ void __launch_bounds__(W == 1 ? 32 * kWarpsPerBlock : 32 * W) k_weights(WArgs a) {
  extern __shared__ double smem[];
  // W == 1: one warp per system, kWarpsPerBlock systems per block.  W > 1: the W warps
  // of a block share one system (large systems: more warps per SM than the per-system
  // shared memory would otherwise allow); the factorisation's element loops and
  // reductions span the block, the triangular solves run in warp 0.
  constexpr int G = 32 * W;  // threads per system
  const int lane = threadIdx.x & 31;
  const int wib = threadIdx.x >> 5;
  const int gt = W == 1 ? lane : (int)threadIdx.x;
  const int nmax = a.nmax;
  __shared__ unsigned long long red_k[W];
  __shared__ int red_i[W];
  __shared__ unsigned long long s_job;
  // per-system shared layout: A[nmax(nmax+1)/2] (upper, packed), B[nmax*dmax],
  // X[kmax*dmax], TC[nmax], TC2[nmax], ipiv[nmax] (ints)
  const size_t per = weights_smem_doubles(nmax, a.kmax, a.dmax);
  double* A = smem + per * (W == 1 ? wib : 0);
  double* B = A + (size_t)nmax * (nmax + 1) / 2;
  double* X = B + (size_t)nmax * a.dmax;
  double* TC = X + (size_t)a.kmax * a.dmax;
  double* TC2 = TC + nmax;
  int* ipiv = reinterpret_cast<int*>(TC2 + nmax);
  for (;;) {
    unsigned long long job = 0;
    if (W == 1) {
      if (lane == 0) job = atomicAdd(a.next, 1ull);
      job = __shfl_sync(kFull, job, 0);
    } else {
      __syncthreads();  // every thread is done with the previous system
      if (gt == 0) s_job = atomicAdd(a.next, 1ull);
      __syncthreads();
      job = s_job;
    }
    if (job >= (unsigned long long)a.nsys) break;
    const int64_t code = kOrdered ? a.order_list[job] : (int64_t)job;
    const int grp = (int)(code >> kGroupShift);
    const int64_t e = code & ((1ll << kGroupShift) - 1);
    const int dim = a.g[grp].dim, npoly = a.g[grp].npoly;
    const int rbf_pow = a.g[grp].rbf_pow, order = a.g[grp].order, periodic = a.g[grp].periodic;
    const int64_t* rowptr = a.g[grp].rowptr;
    const int32_t* cols = a.g[grp].cols;
    const double* xyz = a.g[grp].xyz;
    double* w_out = a.g[grp].w_out;
    double* resid = a.g[grp].resid;
    const int64_t rb = rowptr[e];
    if (!kOrdered) {
      // Unordered work comes from caller-owned device arrays that no host code checked
      // (mft_weights_noalloc; one warp per system).  Before any coordinate is read, a
      // stencil is skipped, its weights set to NaN where its row lies inside cols, and a
      // status word set, when its size is outside 1..kmax (word 2 for > kmax, word 3
      // otherwise), its extent leaves [0, rowptr[n]) or a column is not a node (word 3).
      static_assert(kOrdered || W == 1, "unordered systems run one warp per system");
      const int64_t re = rowptr[e + 1], nnz = rowptr[a.nsys];
      const int64_t k64 = re - rb;
      const bool in_cols = rb >= 0 && re <= nnz && k64 >= 0;
      int why = 0;
      if (!in_cols || k64 < 1) why = 3;
      else if (k64 > a.kmax) why = 2;
      if (why == 0) {
        bool badc = false;
        for (int64_t j = gt; j < k64; j += G) {
          const int32_t cj = cols[rb + j];
          badc |= cj < 0 || (int64_t)cj >= a.nsys;
        }
        if (__any_sync(kFull, badc)) why = 3;
      }
      if (why != 0) {
        if (gt == 0) atomicExch(reinterpret_cast<int*>(a.next + why), 1);
        if (in_cols)
          for (int64_t t = rb * dim + gt; t < re * dim; t += G) w_out[t] = __longlong_as_double(0x7FF8000000000000LL);
        continue;
      }
    }
    const int k = (int)(rowptr[e + 1] - rb);
    const int n = k + npoly;
// upper-packed element (i, j), 1 <= i <= j: column j starts at j (j - 1) / 2
#define AM(i, j) A[(((j) * ((j)-1)) >> 1) + ((i)-1)]
#define BM(i, c) B[(size_t)(c) * n + ((i)-1)]
    const int32_t* st = cols + rb;
    const int64_t ce = st[0];
    // shift_stencil
    for (int j = gt; j < k; j += G)
      for (int d = 0; d < dim; ++d) {
        double t = dsub(xyz[(int64_t)st[j] * dim + d], xyz[ce * dim + d]);
        if (periodic) t = min_image(t, a.g[grp].period[d]);
        X[j * dim + d] = t;
      }
    gsync<W>();
    double s[3] = {1.0, 1.0, 1.0};
    {
      double m[3] = {1.0, 1.0, 1.0};
      for (int d = 0; d < dim; ++d) {
        unsigned long long key = 1;  // 0.0
        for (int j = gt; j < k; j += G) {
          const unsigned long long kx = mag_key(X[j * dim + d]);
          key = kx > key ? kx : key;
        }
        m[d] = key_value(group_max_key<W>(key, red_k));
      }
      // one division for all axes, lane d's
      const double q = ddiv(1.0, (lane & 3) == 0 ? m[0] : (lane & 3) == 1 ? m[1] : m[2]);
      for (int d = 0; d < dim; ++d) s[d] = __shfl_sync(kFull, q, d);
    }
    for (int j = gt; j < k; j += G)
      for (int d = 0; d < dim; ++d) X[j * dim + d] = dmul(X[j * dim + d], s[d]);
    gsync<W>();
    // interpolation block (upper triangle, column-major): the RBF part
    {
      const int T = k * (k + 1) / 2;
      for (int t = gt; t < T; t += G) {
        int r, cidx;
        tri_rc(t, r, cidx);
        double d2 = 0.0;
        for (int d = 0; d < dim; ++d) {
          const double tt = dsub(X[r * dim + d], X[cidx * dim + d]);
          const double t2 = dmul(tt, tt);
          d2 = d == 0 ? t2 : dadd(d2, t2);
        }
        // coincident points (the diagonal): 0, and sqrt off its slow path
        const bool apart = nonzero(d2);
        const double v = pow_int(sqrt(apart ? d2 : 1.0), rbf_pow);
        A[t] = apart ? v : 0.0;
      }
    }
    // the polynomial part, row by row: each monomial one product of two earlier entries of
    // the row; the zero block below it
    for (int j = gt; j < k; j += G)
      for (int m = 0; m < npoly; ++m) {
        const int s0 = a.g[grp].msrc[m][0], s1 = a.g[grp].msrc[m][1];
        double v;
        if (s0 == -1) v = 1.0;
        else if (s0 < 0) v = X[j * dim + (-2 - s0)];
        else
          v = dmul(A[(((k + s0) * (k + s0 + 1)) >> 1) + j], A[(((k + s1) * (k + s1 + 1)) >> 1) + j]);
        A[(((k + m) * (k + m + 1)) >> 1) + j] = v;
      }
    {
      const int T = npoly * (npoly + 1) / 2;
      for (int t = gt; t < T; t += G) {
        int r, cidx;
        tri_rc(t, r, cidx);
        A[(((k + cidx) * (k + cidx + 1)) >> 1) + k + r] = 0.0;
      }
    }
    // right-hand sides, all axes of a row by one thread
    for (int j = gt; j < k; j += G) {
      double pt[3] = {0.0, 0.0, 0.0};
      double d2 = 0.0;
      for (int dd = 0; dd < dim; ++dd) {
        pt[dd] = j == 0 ? 2.220446049250313e-16 : -X[j * dim + dd];
        const double t2 = dmul(pt[dd], pt[dd]);
        d2 = dd == 0 ? t2 : dadd(d2, t2);
      }
      const double r = sqrt(d2);
      for (int d = 0; d < dim; ++d) B[(size_t)d * n + j] = phs_deriv(a.g[grp], pt[d], r);
    }
    for (int m = gt; m < npoly; m += G)
      for (int d = 0; d < dim; ++d) {
        const int* ex = a.g[grp].mono[m];
        bool ok = true;
        for (int dd = 0; dd < dim; ++dd)
          if (ex[dd] != (dd == d ? order : 0)) ok = false;
        B[(size_t)d * n + k + m] = ok ? a.g[grp].fact_order : 0.0;
      }
    gsync<W>();

    // ---------------- Bunch-Kaufman factorisation (upper, dsytf2) with the forward half of
    // the solve (dsytrs: interchange, elimination and pivot division of each right-hand side)
    // run along: step kk of the solve reads only the multipliers step kk of the factorisation
    // has just formed, and each element sees the same operations in the same order.  Every
    // division of a step that shares its divisor is one warp division, a lane per numerator.
    const int nrhs = dim;
    const double alpha = 0.6403882032022076;  // (1 + sqrt(17)) / 8
    int info = 0;
    int kk = n;
    while (kk >= 1) {
      int kstep = 1, kp;
      const double absakk = fabs(AM(kk, kk));
      unsigned long long ckey = 1;  // 0.0 for kk = 1
      int imax = 0;
      if (kk > 1) {
        ckey = 0;
        int iv = 1 << 30;
        for (int i = 1 + gt; i < kk; i += G) {
          const unsigned long long x = mag_key(AM(i, kk));
          if (x > ckey) { ckey = x; iv = i; }
        }
        group_argmax<W>(ckey, iv, 1, red_k, red_i);
        imax = iv;
      }
      const unsigned long long akey = mag_key(absakk);
      // max(|A(kk,kk)|, colmax) == 0 or A(kk,kk) NaN
      if (akey == 0 || (akey == 1 && ckey <= 1)) {
        if (info == 0) info = kk;
        kp = kk;
      } else {
        const double colmax = key_value(ckey);
        if (ge_scaled(absakk, alpha, colmax)) {
          kp = kk;
        } else {
          unsigned long long rkey = 0;
          for (int j = imax + 1 + gt; j <= kk; j += G) {
            const unsigned long long x = mag_key(AM(imax, j));
            rkey = x > rkey ? x : rkey;
          }
          for (int j = 1 + gt; j < imax; j += G) {
            const unsigned long long x = mag_key(AM(j, imax));
            rkey = x > rkey ? x : rkey;
          }
          const double rowmax = key_value(group_max_key<W>(rkey, red_k));
          if (ge_scaled_ratio(absakk, alpha, colmax, rowmax)) kp = kk;
          else if (ge_scaled(fabs(AM(imax, imax)), alpha, rowmax)) kp = imax;
          else { kp = imax; kstep = 2; }
        }
        // every thread has read the pivot candidates (A(imax, imax) above) before the
        // interchange below overwrites them
        gsync<W>();
        const int kkk = kk - kstep + 1;
        if (kp != kkk) {
          for (int i = 1 + gt; i < kp; i += G) {
            const double t = AM(i, kkk); AM(i, kkk) = AM(i, kp); AM(i, kp) = t;
          }
          for (int j = kp + 1 + gt; j < kkk; j += G) {
            const double t = AM(j, kkk); AM(j, kkk) = AM(kp, j); AM(kp, j) = t;
          }
          if (gt == 0) {
            double t = AM(kkk, kkk); AM(kkk, kkk) = AM(kp, kp); AM(kp, kp) = t;
            if (kstep == 2) { t = AM(kk - 1, kk); AM(kk - 1, kk) = AM(kp, kk); AM(kp, kk) = t; }
          }
          if (gt < nrhs) { const double t = BM(kkk, gt); BM(kkk, gt) = BM(kp, gt); BM(kp, gt) = t; }
          gsync<W>();
        }
        if (kstep == 1) {
          const double r1 = ddiv(1.0, AM(kk, kk));
          // scaled column P_j = r1 x_j, then (dsyr with temp_j = -P_j) A(i,j) += x_i temp_j
          // for x_j != 0, one fused multiply-add per element, and B(i,c) -= P_i b_c
          for (int j = gt; j < kk - 1; j += G) TC[j] = dmul(r1, AM(j + 1, kk));
          gsync<W>();
          const int Tu = (kk - 1) * kk / 2;
          const double* xk = &AM(1, kk);
          // two elements per thread and iteration, their loads ahead of the stores
          for (int t0 = 0; t0 < Tu; t0 += 2 * G) {
            const int ta = t0 + gt, tb = ta + G;
            const bool ona = ta < Tu, onb = tb < Tu;
            int ia, ja, ib, jb;
            tri_rc(ona ? ta : 0, ia, ja);
            tri_rc(onb ? tb : 0, ib, jb);
            const double pa = TC[ja], pb = TC[jb], xa = xk[ia], xb = xk[ib];
            const double va = A[ona ? ta : 0], vb = A[onb ? tb : 0];
            if (ona && nonzero(pa)) A[ta] = fma(xa, -pa, va);
            if (t0 + G < Tu && onb && nonzero(pb)) A[tb] = fma(xb, -pb, vb);
          }
          for (int t = gt; t < (kk - 1) * nrhs; t += G) {
            const int c = (t >= kk - 1) + (t >= 2 * (kk - 1)), i = t - c * (kk - 1);
            const double bk = BM(kk, c);
            if (nonzero(bk)) BM(i + 1, c) = fma(TC[i], -bk, BM(i + 1, c));
          }
          gsync<W>();
          for (int j = gt; j < kk - 1; j += G) AM(j + 1, kk) = TC[j];
          if (gt < nrhs) BM(kk, gt) = dmul(r1, BM(kk, gt));
        } else {
          // divisors: d22, d11 (lanes 0, 1) and the right-hand sides' entries kk-1 (lanes
          // 2..4) and kk (lanes 8..10) over A(kk-1,kk)
          const double d12o = AM(kk - 1, kk);
          const int cb = lane >= 2 && lane < 2 + nrhs ? lane - 2 : lane >= 8 && lane < 8 + nrhs ? lane - 8 : -1;
          double num = 1.0;
          if (lane == 0) num = AM(kk - 1, kk - 1);
          else if (lane == 1) num = AM(kk, kk);
          else if (cb >= 0) num = BM(lane < 8 ? kk - 1 : kk, cb);
          const double q1 = div0(num, d12o);
          const double d22 = __shfl_sync(kFull, q1, 0), d11 = __shfl_sync(kFull, q1, 1);
          const double den = dsub(dmul(d11, d22), 1.0);
          const double other = __shfl_sync(kFull, q1, lane < 8 ? lane + 6 : lane - 6);
          num = cb >= 0 ? dsub(dmul(lane < 8 ? d11 : d22, q1), other) : 1.0;
          const double q2 = div0(num, den);  // lane 0: tt
          if (kk > 2) {
            const double d12 = ddiv(__shfl_sync(kFull, q2, 0), d12o);
            // wkm1, wk of every column j <= kk-2 from the original entries, then
            // A(i,j) -= A(i,kk) wk + A(i,kk-1) wkm1 as two fused multiply-adds, then
            // columns kk-1, kk take wkm1, wk (dsytf2 order: each update reads only
            // rows i <= j, which the column overwrite has not reached)
            for (int j = gt; j < kk - 2; j += G) {
              const double a1 = AM(j + 1, kk - 1), a2 = AM(j + 1, kk);
              TC[j] = dmul(d12, dsub(dmul(d11, a1), a2));
              TC2[j] = dmul(d12, dsub(dmul(d22, a2), a1));
            }
            gsync<W>();
            const int Tu = (kk - 2) * (kk - 1) / 2;
            const double *xk = &AM(1, kk), *xm = &AM(1, kk - 1);
            for (int t = gt; t < Tu; t += G) {
              int i0, j0;
              tri_rc(t, i0, j0);
              A[t] = fma(-xm[i0], TC[j0], fma(-xk[i0], TC2[j0], A[t]));
            }
            for (int t = gt; t < (kk - 2) * nrhs; t += G) {
              const int c = (t >= kk - 2) + (t >= 2 * (kk - 2)), i = t - c * (kk - 2);
              const double bk = BM(kk, c), bm = BM(kk - 1, c);
              double v = BM(i + 1, c);
              if (nonzero(bk)) v = fma(TC2[i], -bk, v);
              if (nonzero(bm)) v = fma(TC[i], -bm, v);
              BM(i + 1, c) = v;
            }
          }
          gsync<W>();
          for (int j = gt; j < kk - 2; j += G) {
            AM(j + 1, kk) = TC2[j];
            AM(j + 1, kk - 1) = TC[j];
          }
          if (gt == lane && cb >= 0) BM(lane < 8 ? kk - 1 : kk, cb) = q2;
        }
      }
      if (gt == 0) {
        if (kstep == 1) ipiv[kk - 1] = kp;
        else { ipiv[kk - 1] = -kp; ipiv[kk - 2] = -kp; }
      }
      gsync<W>();
      kk -= kstep;
    }

    if (info != 0) {
      if (gt == 0) atomicMin(a.bad, (int)e);
      for (int t = gt; t < k * dim; t += G) w_out[(rb + t / dim) * dim + t % dim] = NAN;
      if (resid && gt == 0) resid[e] = NAN;
      gsync<W>();
      continue;
    }

    if (W == 1 || wib == 0) {
    // ---------------- backward half of the solve (dsytrs): U' from the top
    kk = 1;
    while (kk <= n) {
      const bool one = ipiv[kk - 1] > 0;
      // dot products in a fixed 32-way strided order, then a pairwise tree
      if (one) {
        if (nrhs == 2) back_step<2, 1>(A, B, n, kk, lane);
        else if (nrhs == 3) back_step<3, 1>(A, B, n, kk, lane);
        else back_step<1, 1>(A, B, n, kk, lane);
      } else {
        if (nrhs == 2) back_step<2, 2>(A, B, n, kk, lane);
        else if (nrhs == 3) back_step<3, 2>(A, B, n, kk, lane);
        else back_step<1, 2>(A, B, n, kk, lane);
      }
      const int kp = one ? ipiv[kk - 1] : -ipiv[kk - 1];
      if (kp != kk && lane < nrhs) {
        const double t = BM(kk, lane); BM(kk, lane) = BM(kp, lane); BM(kp, lane) = t;
      }
      __syncwarp();
      kk += one ? 1 : 2;
    }

    // weights: s_d^order * w[1:k, d]
    double sp[3];
    for (int d = 0; d < 3; ++d) sp[d] = pow_int(s[d], order);
    for (int t = lane; t < k * dim; t += 32) {
      const int j = t / dim, d = t % dim;
      w_out[(rb + j) * dim + d] = dmul(d == 0 ? sp[0] : d == 1 ? sp[1] : sp[2], BM(j + 1, d));
    }
    if (resid) {
      // ||M w - b||_inf / ||b||_inf per column, M and b re-evaluated from X^
      double worst = 0.0;
      for (int d = 0; d < dim; ++d) {
        double rn = 0.0, bn = 0.0;
        for (int r = lane; r < n; r += 32) {
          double acc = 0.0;
          for (int cidx = 0; cidx < n; ++cidx) {
            const int lo = min(r, cidx), hi = max(r, cidx);
            double v;
            if (hi < k) {
              double d2 = 0.0;
              for (int dd = 0; dd < dim; ++dd) {
                const double tt = dsub(X[lo * dim + dd], X[hi * dim + dd]);
                d2 = dadd(d2, dmul(tt, tt));
              }
              v = pow_int(sqrt(d2), rbf_pow);
            } else if (lo < k) {
              const int* ex = a.g[grp].mono[hi - k];
              v = 1.0;
              for (int dd = 0; dd < dim; ++dd) v = dmul(v, pow_int(X[lo * dim + dd], ex[dd]));
            } else {
              v = 0.0;
            }
            acc += v * BM(cidx + 1, d);
          }
          double bv;
          if (r < k) {
            double pt[3];
            for (int dd = 0; dd < dim; ++dd) pt[dd] = r == 0 ? 2.220446049250313e-16 : -X[r * dim + dd];
            double d2 = 0.0;
            for (int dd = 0; dd < dim; ++dd) d2 = dadd(d2, dmul(pt[dd], pt[dd]));
            bv = phs_deriv(a.g[grp], pt[d], sqrt(d2));
          } else {
            const int* ex = a.g[grp].mono[r - k];
            bool ok = true;
            for (int dd = 0; dd < dim; ++dd)
              if (ex[dd] != (dd == d ? order : 0)) ok = false;
            bv = ok ? a.g[grp].fact_order : 0.0;
          }
          rn = fmax(rn, fabs(acc - bv));
          bn = fmax(bn, fabs(bv));
        }
        rn = warp_max(rn);
        bn = warp_max(bn);
        worst = fmax(worst, bn > 0 ? rn / bn : rn);
      }
      if (lane == 0) resid[e] = worst;
    }
    __syncwarp();
    }
#undef AM
#undef BM
  }
}

int make_monomials(int dim, int deg, int (*ex)[3], int cap) {
  int m = 0;
  for (int q = 0; q <= deg; ++q) {
    if (dim == 1) {
      if (m < cap) { ex[m][0] = q; ex[m][1] = 0; ex[m][2] = 0; }
      m++;
      continue;
    }
    for (int a = q; a >= 0; --a) {
      if (dim == 2) {
        if (m < cap) { ex[m][0] = a; ex[m][1] = q - a; ex[m][2] = 0; }
        m++;
        continue;
      }
      for (int b = q - a; b >= 0; --b) {
        if (m < cap) { ex[m][0] = a; ex[m][1] = b; ex[m][2] = q - a - b; }
        m++;
      }
    }
  }
  return m;
}

// The node-independent constants of a group (after mono, rbf_pow and order are set): the
// monomials' products and phs_deriv's terms, in the CPU restatement's operation order.
void make_constants(WGroup& g) {
  auto find = [&](int x, int y, int z) {
    for (int m = 0; m < g.npoly; ++m)
      if (g.mono[m][0] == x && g.mono[m][1] == y && g.mono[m][2] == z) return m;
    return -1;
  };
  for (int m = 0; m < g.npoly; ++m) {
    int e[3] = {g.mono[m][0], g.mono[m][1], g.mono[m][2]};
    const int deg = e[0] + e[1] + e[2];
    int last = e[2] ? 2 : e[1] ? 1 : 0;
    if (deg <= 1) {
      g.msrc[m][0] = (int16_t)(deg == 0 ? -1 : -2 - last);
      g.msrc[m][1] = 0;
      continue;
    }
    int p[3] = {0, 0, 0};  // the second factor
    p[last] = e[last] == deg ? 1 : e[last];
    g.msrc[m][0] = (int16_t)find(e[0] - p[0], e[1] - p[1], e[2] - p[2]);
    g.msrc[m][1] = (int16_t)find(p[0], p[1], p[2]);
  }
  auto fact = [](int k) {
    double r = 1.0;
    for (int i = 2; i <= k; ++i) r = r * (double)i;
    return r;
  };
  const int k = g.order;
  g.fact_order = fact(k);
  g.nterm = 0;
  for (int j = 0; 2 * j <= k; ++j) {
    const int m = k - j;
    double cm = 1.0;
    for (int i = 0; i < m; ++i) cm = cm * (0.5 * (double)g.rbf_pow - (double)i);
    if (cm == 0.0) continue;
    const int q = g.nterm++;
    g.term_cc[q] = fact(k) / (fact(j) * fact(k - 2 * j));
    g.term_cm[q] = cm;
    g.term_ex[q] = k - 2 * j;
    g.term_er[q] = g.rbf_pow - 2 * m;
  }
}

}  // namespace

// Host description of one group of a weight batch (host arrays).
struct HostGroup {
  int dim, rbf_pow, polydeg, order;
  const double* period;  // dim lengths or null
  int64_t n;
  const double* d_xyz;   // device coordinates (n x dim)
  const int64_t* rowptr; // host, n + 1
  const int32_t* cols;   // host, rowptr[n]
  const int32_t* d_cols; // the same on the device, or null
  double* w_out;         // host, rowptr[n] x dim
  bool keep_on_error;    // leave w_out alone when a system is singular
};

// All groups' systems, largest first, in persistent launches over size buckets of the
// system order n = k + monomials (one launch per non-empty bucket, each with the shared
// memory and occupancy its largest system allows).
constexpr int kBucketEdges[] = {48, 64, 80, 104};

static void weights_run(mft_ctx* c, const std::vector<HostGroup>& gs, double* max_resid) {
  cudaStream_t s = c->stream;
  MFT_REQUIRE(!gs.empty() && gs.size() <= (size_t)kMaxGroups, MFT_ERR_ARG,
              "between 1 and 2 weight groups");
  WArgs a{};
  int kmax = 0, nmax = 0;
  int64_t nsys = 0;
  std::vector<int64_t> order;
  std::vector<int> ks, ns;
  int64_t total = 0;
  for (const HostGroup& h : gs) total += h.n;
  order.reserve(total);
  ks.reserve(total);
  ns.reserve(total);
  for (size_t g = 0; g < gs.size(); ++g) {
    const HostGroup& h = gs[g];
    WGroup& G = a.g[g];
    G.dim = h.dim;
    G.npoly = make_monomials(h.dim, h.polydeg, G.mono, kMaxMono);
    MFT_REQUIRE(G.npoly <= kMaxMono, MFT_ERR_ARG, "polynomial degree too high");
    G.rbf_pow = h.rbf_pow;
    G.order = h.order;
    make_constants(G);
    G.periodic = h.period ? 1 : 0;
    for (int d = 0; d < 3; ++d) G.period[d] = (h.period && d < h.dim) ? h.period[d] : 0.0;
    int km = 0;
    for (int64_t i = 0; i < h.n; ++i) {
      const int k = (int)(h.rowptr[i + 1] - h.rowptr[i]);
      MFT_REQUIRE(k >= 1, MFT_ERR_ARG, "empty stencil");
      km = std::max(km, k);
      order.push_back(((int64_t)g << kGroupShift) | i);
      ks.push_back(k);
      ns.push_back(k + G.npoly);
    }
    kmax = std::max(kmax, km);
    nmax = std::max(nmax, km + G.npoly);
    nsys += h.n;
  }
  // systems by size, largest first, ties in input order: a counting sort on n
  std::vector<int64_t> perm(order.size());
  {
    std::vector<int64_t> start((size_t)nmax + 2, 0);
    for (int v : ns) start[(size_t)(nmax - v) + 1]++;
    for (size_t q = 1; q < start.size(); ++q) start[q] += start[q - 1];
    for (size_t q = 0; q < ns.size(); ++q) perm[start[(size_t)(nmax - ns[q])]++] = (int64_t)q;
  }
  std::vector<int64_t> order_sorted(order.size());
  for (size_t q = 0; q < perm.size(); ++q) order_sorted[q] = order[perm[q]];
  (void)kmax;
  MFT_REQUIRE(weights_limit_doubles(nmax, nmax) * sizeof(double) * kWarpsPerBlock <=
                  227 * 1024 - 256,
              MFT_ERR_ARG, "stencil too large for the weight kernel");
  // buckets: [begin, end) ranges of the sorted list with their largest n and k
  struct Bucket { int64_t begin, end; int nmax, kmax, dmax; };
  std::vector<Bucket> buckets;
  auto bucket_of = [](int n) {
    int b = 0;
    for (int edge : kBucketEdges) { if (n <= edge) return b; ++b; }
    return b;
  };
  for (size_t q = 0; q < perm.size(); ++q) {
    const int n = ns[perm[q]], k = ks[perm[q]];
    if (buckets.empty() || bucket_of(n) != bucket_of(buckets.back().nmax))
      buckets.push_back({(int64_t)q, (int64_t)q, n, k, 1});
    Bucket& b = buckets.back();
    b.end = (int64_t)q + 1;
    b.kmax = std::max(b.kmax, k);
    b.dmax = std::max(b.dmax, gs[order[perm[q]] >> kGroupShift].dim);
  }
  DBuf<int64_t> d_order, d_rp[kMaxGroups];
  DBuf<int32_t> d_ci[kMaxGroups];
  DBuf<double> d_w[kMaxGroups], d_res[kMaxGroups];
  DBuf<int> d_bad;
  DBuf<unsigned long long> d_next;
  d_order.upload(order_sorted, s);
  for (size_t g = 0; g < gs.size(); ++g) {
    const HostGroup& h = gs[g];
    const int64_t nnz = h.rowptr[h.n];
    d_rp[g].upload(h.rowptr, h.n + 1, s);
    if (!h.d_cols) d_ci[g].upload(h.cols, nnz, s);
    d_w[g].alloc((size_t)nnz * h.dim);
    if (max_resid) d_res[g].alloc(h.n);
    a.g[g].rowptr = d_rp[g].p;
    a.g[g].cols = h.d_cols ? h.d_cols : d_ci[g].p;
    a.g[g].xyz = h.d_xyz;
    a.g[g].w_out = d_w[g].p;
    a.g[g].resid = max_resid ? d_res[g].p : nullptr;
  }
  d_bad.alloc(1);
  const int big = 0x7fffffff;
  MFT_CUDA(cudaMemcpyAsync(d_bad.p, &big, sizeof(int), cudaMemcpyHostToDevice, s));
  d_next.alloc(buckets.size());
  d_next.zero(s);
  a.bad = d_bad.p;
  int dev = 0, sms = 0;
  MFT_CUDA(cudaGetDevice(&dev));
  MFT_CUDA(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
  for (size_t b = 0; b < buckets.size(); ++b) {
    const Bucket& bk = buckets[b];
    WArgs ab = a;
    ab.nmax = bk.nmax;
    ab.kmax = bk.kmax;
    ab.dmax = bk.dmax;
    ab.nsys = bk.end - bk.begin;
    ab.order_list = d_order.p + bk.begin;
    ab.next = d_next.p + b;
    const int warps = system_warps(bk.nmax);
    const int spb = warps > 1 ? 1 : kWarpsPerBlock;  // systems per block
    const int threads = 32 * (warps > 1 ? warps : kWarpsPerBlock);
    const size_t shmem = weights_smem_doubles(bk.nmax, bk.kmax, bk.dmax) * sizeof(double) * spb;
    // the opt-in dynamic shared memory this bucket needs (the static part is small)
    void (*const kern)(WArgs) = warps == 3 ? k_weights<true, 3>
                                : warps == 2 ? k_weights<true, 2> : k_weights<true, 1>;
    int per_sm = 0;
    MFT_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)shmem));
    MFT_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, threads, shmem));
    per_sm = std::max(per_sm, 1);
    const int64_t want = (ab.nsys + spb - 1) / spb;
    const unsigned grid =
        (unsigned)std::max<int64_t>(1, std::min<int64_t>((int64_t)sms * per_sm, want));
    kern<<<grid, threads, shmem, s>>>(ab);
    MFT_LAUNCH_CHECK();
  }
  int bad = big;
  MFT_CUDA(cudaMemcpyAsync(&bad, d_bad.p, sizeof(int), cudaMemcpyDeviceToHost, s));
  MFT_CUDA(cudaStreamSynchronize(s));
  std::vector<std::vector<double>> res(gs.size());
  for (size_t g = 0; g < gs.size(); ++g) {
    const HostGroup& h = gs[g];
    if (bad == big || !h.keep_on_error)
      copy_out(c, h.w_out, d_w[g].p, (size_t)h.rowptr[h.n] * h.dim * sizeof(double));
    if (max_resid) {
      res[g].resize(h.n);
      MFT_CUDA(cudaMemcpyAsync(res[g].data(), d_res[g].p, h.n * sizeof(double),
                               cudaMemcpyDeviceToHost, s));
    }
  }
  MFT_CUDA(cudaStreamSynchronize(s));
  MFT_REQUIRE(bad == big, MFT_ERR_SINGULAR,
              "saddle-point system of node " + std::to_string(bad) + " has an exactly zero pivot");
  if (max_resid) {
    double m = 0.0;
    for (auto& r : res)
      for (double x : r) m = std::max(m, x);
    *max_resid = m;
  }
}

void weights_device(mft_ctx* c, int rbf_pow, int polydeg, int deriv_order, double* w,
                    double* max_resid) {
  HostGroup h{};
  h.dim = c->dim;
  h.rbf_pow = rbf_pow;
  h.polydeg = polydeg;
  h.order = deriv_order;
  h.period = c->periodic ? c->period : nullptr;
  h.n = c->n;
  h.d_xyz = c->d_xyz.p;
  h.rowptr = c->st_rp.data();
  h.cols = c->st_ci.data();
  h.d_cols = c->d_st_ci.n == c->st_ci.size() ? c->d_st_ci.p : nullptr;
  h.w_out = w;
  h.keep_on_error = true;
  weights_run(c, {h}, max_resid);
}

void weights_batch(mft_ctx* c, int ngroups, const mft_weight_group* groups, double* max_resid) {
  MFT_REQUIRE(ngroups >= 1 && ngroups <= kMaxGroups && groups, MFT_ERR_ARG,
              "between 1 and 2 weight groups");
  std::vector<HostGroup> hs(ngroups);
  std::vector<DBuf<double>> xyz(ngroups);
  for (int g = 0; g < ngroups; ++g) {
    const mft_weight_group& q = groups[g];
    MFT_REQUIRE(q.dim >= 1 && q.dim <= 3 && q.n >= 1 && q.xyz && q.rowptr && q.cols && q.w,
                MFT_ERR_ARG, "bad weight group");
    MFT_REQUIRE(q.rbf_pow >= 1 && q.polydeg >= 0 && q.polydeg <= 6 && q.deriv_order >= 1 &&
                    q.deriv_order <= 8, MFT_ERR_ARG, "bad basis or derivative order");
    MFT_REQUIRE(q.rowptr[0] == 0, MFT_ERR_ARG, "rowptr[0] must be 0");
    for (int64_t i = 0; i < q.n; ++i) {
      MFT_REQUIRE(q.rowptr[i + 1] > q.rowptr[i], MFT_ERR_ARG, "empty stencil");
      for (int64_t p = q.rowptr[i]; p < q.rowptr[i + 1]; ++p)
        MFT_REQUIRE(q.cols[p] >= 0 && q.cols[p] < q.n, MFT_ERR_ARG, "stencil index out of range");
    }
    xyz[g].upload(q.xyz, (size_t)q.n * q.dim, c->stream);
    HostGroup& h = hs[g];
    h.keep_on_error = false;
    h.d_cols = nullptr;
    h.dim = q.dim;
    h.rbf_pow = q.rbf_pow;
    h.polydeg = q.polydeg;
    h.order = q.deriv_order;
    h.period = nullptr;
    h.n = q.n;
    h.d_xyz = xyz[g].p;
    h.rowptr = q.rowptr;
    h.cols = q.cols;
    h.w_out = q.w;
  }
  weights_run(c, hs, max_resid);
}

}  // namespace mft

// ---------------------------------------------------------------- allocation-free variant
//
// mft_weights_noalloc is for callers that cannot allocate device memory while they
// compute weights: a solver running inside a stream-ordered memory pool it does not own,
// a host that has handed all device memory to its own allocator, or code that must not
// call cudaMalloc/cudaFree because those calls synchronise the device.  The caller passes
// every input and output as device memory; the only global scratch the solve needs (the
// work counter and two status words) lives in the file-scope array below.

namespace {

// [0] work counter, [1] first node with a zero pivot (low 32 bits, 0x7F7F7F7F = none),
// [2] oversize-stencil flag, [3] invalid-stencil flag (empty or decreasing rowptr, a row
// outside cols, a column that is not a node).  32 bytes on every GPU that loads the
// library, held until the process exits.
constexpr int kNoAllocWords = 4;
static __device__ __align__(256) unsigned long long g_weights_scratch[kNoAllocWords];

constexpr int kNoAllocMaxDevices = 64;
std::mutex g_scratch_mu;
unsigned long long* g_scratch_addr[kNoAllocMaxDevices] = {};

void put_err(char* err, int len, const std::string& msg) {
  if (err && len > 0) {
    const size_t m = std::min<size_t>((size_t)len - 1, msg.size());
    memcpy(err, msg.data(), m);
    err[m] = '\0';
  }
}

}  // namespace

extern "C" mft_status mft_weights_noalloc(int dim, int64_t n, const double* xyz,
                                          const double* period, const int64_t* rowptr,
                                          const int32_t* cols, int kmax, int rbf_pow,
                                          int polydeg, int deriv_order, double* w,
                                          void* stream, char* err, int err_len) {
  using namespace mft;
  put_err(err, err_len, "");
  if (dim < 1 || dim > 3 || n < 1 || n > (int64_t)INT32_MAX || !xyz || !rowptr || !cols || !w ||
      kmax < 1 || rbf_pow < 1 || rbf_pow > 15 || polydeg < 0 || polydeg > 6 || deriv_order < 1 ||
      deriv_order > 8) {
    put_err(err, err_len, "mft_weights_noalloc: invalid argument");
    return MFT_ERR_ARG;
  }
  WArgs a{};
  WGroup& G = a.g[0];
  G.dim = dim;
  G.npoly = make_monomials(dim, polydeg, G.mono, kMaxMono);
  G.rbf_pow = rbf_pow;
  G.order = deriv_order;
  G.periodic = period ? 1 : 0;
  for (int d = 0; d < 3; ++d) G.period[d] = (period && d < dim) ? period[d] : 0.0;
  a.kmax = kmax;
  a.nmax = kmax + G.npoly;
  a.dmax = 3;
  const size_t shmem = weights_smem_doubles(a.nmax, kmax, a.dmax) * sizeof(double) * kWarpsPerBlock;
  const size_t need = weights_limit_doubles(a.nmax, kmax) * sizeof(double) * kWarpsPerBlock;
  const size_t kMaxShmem = 227 * 1024;
  if (G.npoly > kMaxMono || need > kMaxShmem) {
    put_err(err, err_len,
            "mft_weights_noalloc: stencil size " + std::to_string(kmax) + " plus " +
                std::to_string(G.npoly) + " monomials needs " + std::to_string(need) +
                " bytes of shared memory; the maximum is " + std::to_string(kMaxShmem) +
                " (kmax + monomials <= 161)");
    return MFT_ERR_ARG;
  }
  make_constants(G);
  int dev = 0;
  if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= kNoAllocMaxDevices) {
    put_err(err, err_len, "mft_weights_noalloc: no current CUDA device");
    return MFT_ERR_CUDA;
  }
  unsigned long long* scratch = nullptr;
  {
    // First call on this device (with it current): resolve the device address of the
    // scratch array.  Later calls reuse it.  Make the first call before any capture.  The
    // address is kept for the life of the process: a cudaDeviceReset after the first call
    // on a device is not supported (the kept address would be stale).
    std::lock_guard<std::mutex> lock(g_scratch_mu);
    if (!g_scratch_addr[dev]) {
      void* ptr = nullptr;
      const cudaError_t e = cudaGetSymbolAddress(&ptr, g_weights_scratch);
      if (e != cudaSuccess || !ptr) {
        put_err(err, err_len, std::string("cudaGetSymbolAddress: ") + cudaGetErrorString(e));
        return MFT_ERR_CUDA;
      }
      g_scratch_addr[dev] = reinterpret_cast<unsigned long long*>(ptr);
    }
    scratch = g_scratch_addr[dev];
  }
  cudaStream_t s = reinterpret_cast<cudaStream_t>(stream);
  // the counter and the status words must start from their initial values
  if (cudaMemsetAsync(scratch, 0, sizeof(unsigned long long), s) != cudaSuccess ||
      cudaMemsetAsync(scratch + 1, 0x7F, sizeof(int), s) != cudaSuccess ||
      cudaMemsetAsync(scratch + 2, 0, 2 * sizeof(unsigned long long), s) != cudaSuccess) {
    put_err(err, err_len, "mft_weights_noalloc: cudaMemsetAsync failed");
    return MFT_ERR_CUDA;
  }
  a.nsys = n;
  a.order_list = nullptr;
  G.rowptr = rowptr;
  G.cols = cols;
  G.xyz = xyz;
  G.w_out = w;
  G.resid = nullptr;
  a.bad = reinterpret_cast<int*>(scratch + 1);
  a.next = scratch;
  int sms = 0, per_sm = 0;
  if (cudaFuncSetAttribute(k_weights<false, 1>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                           (int)shmem) != cudaSuccess ||
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_weights<false, 1>,
                                                    32 * kWarpsPerBlock, shmem) != cudaSuccess) {
    put_err(err, err_len, "mft_weights_noalloc: kernel configuration failed");
    return MFT_ERR_CUDA;
  }
  per_sm = std::max(per_sm, 1);
  const int64_t want = (n + kWarpsPerBlock - 1) / kWarpsPerBlock;
  const unsigned grid =
      (unsigned)std::max<int64_t>(1, std::min<int64_t>((int64_t)sms * per_sm, want));
  k_weights<false, 1><<<grid, 32 * kWarpsPerBlock, shmem, s>>>(a);
  cudaError_t e = cudaGetLastError();
  int status[3] = {0, 0, 0};
  if (e == cudaSuccess) e = cudaMemcpyAsync(&status[0], scratch + 1, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&status[1], scratch + 2, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaMemcpyAsync(&status[2], scratch + 3, sizeof(int), cudaMemcpyDeviceToHost, s);
  if (e == cudaSuccess) e = cudaStreamSynchronize(s);
  if (e != cudaSuccess) {
    put_err(err, err_len, std::string("mft_weights_noalloc: ") + cudaGetErrorString(e));
    return MFT_ERR_CUDA;
  }
  if (status[2] != 0) {
    put_err(err, err_len,
            "mft_weights_noalloc: a stencil is empty, leaves cols (rowptr not increasing "
            "up to rowptr[n]) or lists a column outside 0..n-1; its weights are NaN");
    return MFT_ERR_ARG;
  }
  if (status[1] != 0) {
    put_err(err, err_len, "mft_weights_noalloc: a stencil is longer than kmax = " +
                              std::to_string(kmax) + "; its weights were not computed (NaN)");
    return MFT_ERR_ARG;
  }
  if (status[0] != 0x7F7F7F7F) {
    put_err(err, err_len, "mft_weights_noalloc: node " + std::to_string(status[0]) +
                              " has an exactly zero pivot");
    return MFT_ERR_SINGULAR;
  }
  return MFT_OK;
}
