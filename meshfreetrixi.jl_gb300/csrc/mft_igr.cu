// Information geometric regularisation source (SourceIGR, src/sources/IGR.jl:17-239) for
// the 2D Euler equations, FP64:
//   b = alpha (tr(Du)^2 + tr(Du^2)), with tr(Du) formed as the reference writes it,
//       Dx rho + Dy v1 (update_igr_rhs!, :143-145), tr(Du^2) = (Dx v1)^2 +
//       2 (Dy v1)(Dx v2) + (Dy v2)^2 (:151-153);
//   sigma from (rho^-1 - alpha (Dx rho^-1 Dx + Dy rho^-1 Dy)) sigma = b by unpreconditioned
//       conjugate gradients from sigma = 0, at most maxiter iterations, relative
//       tolerance sqrt(eps) (the in-place cg! the reference intends at :189);
//   du[rho v1] -= Dx sigma, du[rho v2] -= Dy sigma (:214-237).
// The CG runs as a fixed sequence of kernels (four per iteration, or three where every row group
// is staged) whose scalars live in device memory; once converged, the remaining kernels return
// at entry, so one rhs! evaluation is a fixed launch sequence that a CUDA graph can hold.
// Reductions are block partials added in a fixed order (deterministic).
#include <algorithm>
#include <cfloat>

#include "mft_device.cuh"
#include "mft_halo.cuh"

namespace mft {
namespace {

using namespace dev;

template <int W>
__device__ __forceinline__ void block_sum_igr(double (&v)[W]) {
  __shared__ double sh[W][kBlock / 32];
  const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
#pragma unroll
  for (int k = 0; k < W; ++k) {
    double x = v[k];
    for (int o = 16; o > 0; o >>= 1) x += __shfl_down_sync(0xffffffffu, x, o);
    if (lane == 0) sh[k][wid] = x;
  }
  __syncthreads();
  if (threadIdx.x == 0) {
#pragma unroll
    for (int k = 0; k < W; ++k) {
      double x = sh[k][0];
      for (int w = 1; w < kBlock / 32; ++w) x += sh[k][w];
      v[k] = x;
    }
  }
  __syncthreads();
}

// Block partial of one sum; returns true in thread 0 of the last block to finish, with
// the total in *total (fixed order over the partials).
__device__ bool last_block_total(double x, double* partial, unsigned* counter, double* total) {
  double v[1] = {x};
  block_sum_igr<1>(v);
  __shared__ int last;
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = v[0];
    __threadfence();
    last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double a[1] = {0.0};
  for (unsigned b = threadIdx.x; b < gridDim.x; b += kBlock) a[0] += __ldcg(partial + b);
  block_sum_igr<1>(a);
  if (threadIdx.x == 0) {
    *total = a[0];
    *counter = 0u;
  }
  return threadIdx.x == 0;
}

// The CG scalars from the first residual's squared norm, and after an update.
__device__ __forceinline__ void igr_start(const IgrArgs& a, double total) {
  IgrScalars* s = a.sc;
  s->res = sqrt(total);
  s->prev = 1.0;
  s->tol = dmul(s->res, sqrt(DBL_EPSILON));
  s->beta = ddiv(dmul(s->res, s->res), 1.0);
  s->iter = 0;
  s->done = (s->res <= s->tol) || a.maxiter <= 0;
}
__device__ __forceinline__ void igr_next(const IgrArgs& a, double total) {
  IgrScalars* s = a.sc;
  s->prev = s->res;
  s->res = sqrt(total);
  s->iter += 1;
  s->beta = ddiv(dmul(s->res, s->res), dmul(s->prev, s->prev));
  s->done = (s->iter >= a.maxiter) || (s->res <= s->tol);
}

// prim = (rho, v1, v2), rinv = 1 / rho
__global__ void k_igr_prim(int64_t n, const double* __restrict__ u, double* prim, double* rinv) {
  const int64_t i = blockIdx.x * (int64_t)kBlock + threadIdx.x;
  if (i >= n) return;
  const double rho = u[i * 4], m1 = u[i * 4 + 1], m2 = u[i * 4 + 2];
  prim[i * 3] = rho;
  prim[i * 3 + 1] = ddiv(m1, rho);
  prim[i * 3 + 2] = ddiv(m2, rho);
  rinv[i] = ddiv(1.0, rho);
}

// b, x = 0, r = b, u_old = 0 and the initial residual norm.
__global__ void __launch_bounds__(kBlock) k_igr_rhs(IgrArgs a) {
  const int64_t r = blockIdx.x * (int64_t)kBlock + threadIdx.x;  // layout row
  double rr = 0.0;
  if (r < a.n) {
    const int64_t i = ell_node(a.ell, r);
    const int64_t base = a.ell.slice_off[r >> 5] + (r & 31);
    const int len = a.ell.row_len[r];
    double dxr = 0, dxv1 = 0, dxv2 = 0, dyv1 = 0, dyv2 = 0;
    for (int j = 0; j < len; ++j) {
      const int64_t p = base + ((int64_t)j << 5);
      const int64_t c = __ldg(a.ell.col + p);
      const double wx = __ldg(a.wx + p), wy = __ldg(a.wy + p);
      const double rc = a.prim[c * 3], v1 = a.prim[c * 3 + 1], v2 = a.prim[c * 3 + 2];
      dxr = fma(wx, rc, dxr);
      dxv1 = fma(wx, v1, dxv1);
      dxv2 = fma(wx, v2, dxv2);
      dyv1 = fma(wy, v1, dyv1);
      dyv2 = fma(wy, v2, dyv2);
    }
    const double tr = dadd(dxr, dyv1);
    const double tsq = dadd(dadd(dmul(dxv1, dxv1), dmul(dmul(2.0, dyv1), dxv2)), dmul(dyv2, dyv2));
    const double b = dmul(a.alpha, dadd(dmul(tr, tr), tsq));
    a.x[i] = 0.0;
    a.r[i] = b;
    a.u0[i] = 0.0;
    rr = dmul(b, b);
  }
  double total;
  if (last_block_total(rr, a.partial, a.counter, &total)) igr_start(a, total);
}

// u_new = r + beta u_old (elementwise; the gathers below then read u_new directly)
__global__ void k_igr_newdir(IgrArgs a, const double* uo, double* un) {
  if (a.sc->done) return;
  const int64_t i = blockIdx.x * (int64_t)kBlock + threadIdx.x;
  if (i >= a.n) return;
  un[i] = dadd(a.r[i], dmul(a.sc->beta, uo[i]));
}

// t1 = rinv (Dx u_new), t2 = rinv (Dy u_new)
__global__ void __launch_bounds__(kBlock) k_igr_dir(IgrArgs a, const double* un) {
  if (a.sc->done) return;
  const int64_t r = blockIdx.x * (int64_t)kBlock + threadIdx.x;  // layout row
  if (r >= a.n) return;
  const int64_t i = ell_node(a.ell, r);
  const int64_t base = a.ell.slice_off[r >> 5] + (r & 31);
  const int len = a.ell.row_len[r];
  double sx = 0.0, sy = 0.0;
#pragma unroll 4
  for (int j = 0; j < len; ++j) {
    const int64_t p = base + ((int64_t)j << 5);
    const int64_t c = __ldg(a.ell.col + p);
    const double uc = un[c];
    sx = fma(__ldg(a.wx + p), uc, sx);
    sy = fma(__ldg(a.wy + p), uc, sy);
  }
  a.t[i * 2] = dmul(a.rinv[i], sx);
  a.t[i * 2 + 1] = dmul(a.rinv[i], sy);
}

// c = rinv u_new - alpha (Dx t1 + Dy t2); alpha_cg = res^2 / (u_new . c)
__global__ void __launch_bounds__(kBlock) k_igr_op(IgrArgs a, const double* un) {
  if (a.sc->done) return;
  const int64_t r = blockIdx.x * (int64_t)kBlock + threadIdx.x;  // layout row
  double uc = 0.0;
  if (r < a.n) {
    const int64_t i = ell_node(a.ell, r);
    const int64_t base = a.ell.slice_off[r >> 5] + (r & 31);
    const int len = a.ell.row_len[r];
    double sx = 0.0, sy = 0.0;
    const double2* __restrict__ t2 = reinterpret_cast<const double2*>(a.t);
#pragma unroll 4
    for (int j = 0; j < len; ++j) {
      const int64_t p = base + ((int64_t)j << 5);
      const int64_t c = __ldg(a.ell.col + p);
      const double2 tc = t2[c];  // (t1, t2) of the neighbour in one 16-byte load
      sx = fma(__ldg(a.wx + p), tc.x, sx);
      sy = fma(__ldg(a.wy + p), tc.y, sy);
    }
    const double ci = dsub(dmul(a.rinv[i], un[i]), dmul(a.alpha, dadd(sx, sy)));
    a.c[i] = ci;
    uc = dmul(un[i], ci);
  }
  double total;
  if (last_block_total(uc, a.partial, a.counter, &total)) {
    IgrScalars* s = a.sc;
    s->alpha_cg = ddiv(dmul(s->res, s->res), total);
  }
}

// x += alpha_cg u_new; r -= alpha_cg c; new residual, beta, convergence
__global__ void __launch_bounds__(kBlock) k_igr_update(IgrArgs a, const double* un) {
  if (a.sc->done) return;
  const int64_t i = blockIdx.x * (int64_t)kBlock + threadIdx.x;
  double rr = 0.0;
  if (i < a.n) {
    const double al = a.sc->alpha_cg;
    a.x[i] = dadd(a.x[i], dmul(al, un[i]));
    const double r = dsub(a.r[i], dmul(al, a.c[i]));
    a.r[i] = r;
    rr = dmul(r, r);
  }
  double total;
  if (last_block_total(rr, a.partial, a.counter, &total)) igr_next(a, total);
}

// add = (-(Dx sigma), -(Dy sigma)) for the momentum rows of du
__global__ void __launch_bounds__(kBlock) k_igr_flux(IgrArgs a) {
  const int64_t r = blockIdx.x * (int64_t)kBlock + threadIdx.x;  // layout row
  if (r >= a.n) return;
  const int64_t i = ell_node(a.ell, r);
  const int64_t base = a.ell.slice_off[r >> 5] + (r & 31);
  const int len = a.ell.row_len[r];
  double sx = 0.0, sy = 0.0;
#pragma unroll 4
  for (int j = 0; j < len; ++j) {
    const int64_t p = base + ((int64_t)j << 5);
    const int64_t c = __ldg(a.ell.col + p);
    sx = fma(__ldg(a.wx + p), a.x[c], sx);
    sy = fma(__ldg(a.wy + p), a.x[c], sy);
  }
  a.add[i * 2] = -sx;
  a.add[i * 2 + 1] = -sy;
}

// ---------------------------------------------------------------- staged form
//
// The same iteration in three kernels over the staged layout (mft_halo.cuh), for clouds whose
// row groups are all staged; the arithmetic is the kernels' above, operation by operation, but
// for the order in which the blocks' parts of the two dot products are added.  (In double-word
// sums, as the engine's own gathers, the solve was faster still, 1.43 ms for the case below, but
// its part of du was 50 to 100 times further from a quad-precision solve, up to 1.4e-10 of its
// largest value against 2e-12, and at alpha = 20 h^2 du as a whole up to eight times.)
// What bounds it: the FP64 pipe, 37 us for the 70 multiply-adds per node of one gather at 262,144
// nodes, and the 630 B of weights and positions per node.  The new direction is formed while
// staging (no pass of its own), the gathers read neighbours from shared memory, and the
// operator's gather walks the row groups in the opposite order of the direction's, so that the
// weights one reads last are still in L2 for the other (165 MB of weights at 262,144 nodes
// against 129 MB of L2).  Each kernel is the programmatic dependent of the one before: what that
// one wrote (vectors and CG scalars) is read after pdl_wait and past L1.  One rhs! with a solve
// of 16 iterations (of at most 20) at 262,144 nodes: 2.25 ms with the kernels above, 1.90 with
// these; of 20: 2.67 / 2.25, and at 16,384 nodes 0.87 / 0.46, at 65,536 1.05 / 1.00.

// Sum of x over the block, in thread 0 (fixed order).
__device__ __forceinline__ double block_total(double x) {
  __shared__ double sh[kHaloRows / 32];
  for (int o = 16; o > 0; o >>= 1) x = dadd(x, __shfl_xor_sync(0xffffffffu, x, o));
  if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = x;
  __syncthreads();
  x = threadIdx.x < blockDim.x / 32 ? sh[threadIdx.x] : 0.0;
  if (threadIdx.x < 32)
    for (int o = kHaloRows / 64; o > 0; o >>= 1) x = dadd(x, __shfl_xor_sync(0xffffffffu, x, o));
  __syncthreads();
  return x;
}

// As last_block_total for any block size of whole warps up to kHaloRows.
__device__ bool last_block_sum(double x, double* partial, unsigned* counter, double* total) {
  __shared__ int last;
  x = block_total(x);
  if (threadIdx.x == 0) {
    partial[blockIdx.x] = x;
    __threadfence();
    last = (atomicAdd(counter, 1u) == gridDim.x - 1);
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  double a = 0.0;
  for (unsigned b = threadIdx.x; b < gridDim.x; b += blockDim.x) a = dadd(a, __ldcg(partial + b));
  a = block_total(a);
  if (threadIdx.x == 0) {
    *total = a;
    *counter = 0u;
  }
  return threadIdx.x == 0;
}

// Entries per register group of the gathers, and blocks per SM their registers are capped for.
// One rhs! of 20 iterations at 16,384 / 65,536 / 262,144 nodes, us: 3 entries at four blocks 571 /
// 1304 / 2300, 4 at three 586 / 1168 / 2344, 5 at three 466 / 998 / 2250, 6 at three 481 / 1035 /
// 2409, 6 at two 614 / 995 / 2544, 3 at five 575 / 1423 / 2224.
constexpr int kIgrGroup = 5, kIgrBlocks = 3;

// The gather of row group `group` (the block's): per entry of this thread's row
// sum(w_x, w_y, value of the neighbour), the values staged in shared memory as value(c).  What
// does not depend on the kernel before -- the row, the list, and the first 2 G entries' weights
// -- is requested before wait(), which returns whether there is anything to do: the weights'
// latency and the launch then overlap that kernel's tail and the staging.  Every thread of the
// block must call it.
struct IgrStream {
  int lc;
  double wx, wy;
};
template <typename T, typename Wait, typename Value, typename Sum>
__device__ __forceinline__ bool igr_gather(const IgrArgs& a, unsigned group, T* sm, Wait wait,
                                           Value value, Sum sum) {
  const int h0 = __ldg(a.ell.halo_off + group), nh = __ldg(a.ell.halo_off + group + 1) - h0;
  const int64_t r = group * (int64_t)blockDim.x + threadIdx.x;  // layout row
  const bool live = r < a.n;
  const int64_t base = live ? a.ell.slice_off[r >> 5] + (r & 31) : 0;
  const int len = live ? a.ell.row_len[r] : 0;
  IgrStream e[2][kIgrGroup];
  auto load = [&](IgrStream& x, int j) {
    const int64_t p = base + (int64_t)j * 32;
    x.lc = __ldg(a.ell.lcol + p);
    x.wx = __ldg(a.wx + p);
    x.wy = __ldg(a.wy + p);
  };
  const int q0 = threadIdx.x, q1 = q0 + blockDim.x;
  const int c0 = q0 < nh ? __ldg(a.ell.halo_col + h0 + q0) : -1;
  const int c1 = q1 < nh ? __ldg(a.ell.halo_col + h0 + q1) : -1;
  pipelined_open<kIgrGroup>(len, e, load);
  if (!wait()) return false;
  const T v0 = c0 >= 0 ? value(c0) : T{};
  const T v1 = c1 >= 0 ? value(c1) : T{};
  if (c0 >= 0) sm[q0] = v0;
  if (c1 >= 0) sm[q1] = v1;
  for (int q = q1 + blockDim.x; q < nh; q += blockDim.x)
    sm[q] = value((int64_t)__ldg(a.ell.halo_col + h0 + q));
  __syncthreads();
  pipelined_run<kIgrGroup>(len, e, load,
                           [&](const IgrStream& x) { sum(x.wx, x.wy, sm[x.lc]); });
  return true;
}

// t = rinv (Dx u_new, Dy u_new), u_new = r + beta u_old formed while staging and written for the
// node's own row; or, FLUX, add = -(Dx sigma, Dy sigma).
template <bool FLUX>
__global__ void __launch_bounds__(kHaloRows, kIgrBlocks) k_igr_dir_staged(IgrArgs a, const double* uo, double* un) {
  extern __shared__ double2 sm2[];
  pdl_trigger();
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;  // layout row
  const int64_t i = r < a.n ? ell_node(a.ell, r) : 0;
  const double ri = !FLUX && r < a.n ? a.rinv[i] : 0.0;
  double beta = 0.0;
  auto value = [&](int64_t c) { return FLUX ? __ldcg(a.x + c) : dadd(__ldcg(a.r + c), dmul(beta, __ldcg(uo + c))); };
  double sx = 0.0, sy = 0.0;
  const bool ran = igr_gather(
      a, blockIdx.x, reinterpret_cast<double*>(sm2),
      [&] {
        pdl_wait();
        beta = FLUX ? 0.0 : __ldcg(&a.sc->beta);
        return FLUX || !__ldcg(&a.sc->done);
      },
      value,
      [&](double wx, double wy, double v) {
        sx = fma(wx, v, sx);
        sy = fma(wy, v, sy);
      });
  if (!ran || r >= a.n) return;
  if (FLUX) {
    reinterpret_cast<double2*>(a.add)[i] = make_double2(-sx, -sy);
    return;
  }
  un[i] = value(i);
  reinterpret_cast<double2*>(a.t)[i] = make_double2(dmul(ri, sx), dmul(ri, sy));
}

// c = rinv u_new - alpha (Dx t1 + Dy t2) and the block's part of u_new . c.  Block b takes the
// group gridDim.x - 1 - b.  The update's blocks add the parts up, each for itself: a last block
// that did it here would hold every one of the 1024 blocks at a fence and an atomic.
__global__ void __launch_bounds__(kHaloRows, kIgrBlocks) k_igr_op_staged(IgrArgs a, const double* un) {
  extern __shared__ double2 sm2[];
  pdl_trigger();
  const unsigned group = gridDim.x - 1 - blockIdx.x;
  const double2* t2 = reinterpret_cast<const double2*>(a.t);
  const int64_t r = group * (int64_t)blockDim.x + threadIdx.x;  // layout row
  const int64_t i = r < a.n ? ell_node(a.ell, r) : 0;
  const double ri = r < a.n ? a.rinv[i] : 0.0;
  double sx = 0.0, sy = 0.0;
  const bool ran = igr_gather(
      a, group, sm2,
      [&] {
        pdl_wait();
        return !__ldcg(&a.sc->done);
      },
      [&](int64_t c) { return __ldcg(t2 + c); },
      [&](double wx, double wy, double2 t) {
        sx = fma(wx, t.x, sx);
        sy = fma(wy, t.y, sy);
      });
  if (!ran) return;
  double uc = 0.0;
  if (r < a.n) {
    const double ui = __ldcg(un + i);
    const double ci = dsub(dmul(ri, ui), dmul(a.alpha, dadd(sx, sy)));
    a.c[i] = ci;
    uc = dmul(ui, ci);
  }
  uc = block_total(uc);
  if (threadIdx.x == 0) a.partial[group] = uc;
}

// alpha_cg = res^2 / (u_new . c) from the nparts parts; x += alpha_cg u_new; r -= alpha_cg c;
// new residual, beta, convergence
__global__ void __launch_bounds__(kHaloRows) k_igr_update_staged(IgrArgs a, const double* un,
                                                                 unsigned nparts, double* partial) {
  pdl_trigger();
  pdl_wait();
  if (__ldcg(&a.sc->done)) return;
  __shared__ double al_s;
  double uc = 0.0;
  for (unsigned b = threadIdx.x; b < nparts; b += blockDim.x) uc = dadd(uc, __ldcg(a.partial + b));
  uc = block_total(uc);
  if (threadIdx.x == 0) {
    const double res = __ldcg(&a.sc->res);
    al_s = ddiv(dmul(res, res), uc);
  }
  __syncthreads();
  const double al = al_s;
  double rr = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n;
       i += (int64_t)gridDim.x * blockDim.x) {
    a.x[i] = dadd(__ldcg(a.x + i), dmul(al, __ldcg(un + i)));
    const double r = dsub(__ldcg(a.r + i), dmul(al, __ldcg(a.c + i)));
    a.r[i] = r;
    rr = dadd(rr, dmul(r, r));
  }
  double total;
  if (last_block_sum(rr, partial, a.counter, &total)) igr_next(a, total);
}

void launch_igr_staged(const IgrArgs& a, cudaStream_t s) {
  const int rows = a.ell.halo_rows;
  const unsigned g = (unsigned)((a.n + rows - 1) / rows);
  const size_t one = (size_t)a.ell.halo_stride * sizeof(double);
  const unsigned gu = std::min<unsigned>((unsigned)((a.n + kHaloRows - 1) / kHaloRows), a.update_blocks);
  for (int it = 0; it < a.maxiter; ++it) {
    const double* uo = (it & 1) ? a.u1 : a.u0;
    double* un = (it & 1) ? a.u0 : a.u1;
    launch_k(k_igr_dir_staged<false>, g, rows, one, s, true, a, uo, un);
    launch_k(k_igr_op_staged, g, rows, 2 * one, s, true, a, (const double*)un);
    launch_k(k_igr_update_staged, gu, kHaloRows, 0, s, true, a, (const double*)un, g, a.partial + g);
  }
  launch_k(k_igr_dir_staged<true>, g, rows, one, s, true, a, (const double*)nullptr, (double*)nullptr);
}

}  // namespace

void launch_igr(const IgrArgs& a, const double* u, cudaStream_t s) {
  if (a.n <= 0) return;
  const unsigned g = (unsigned)((a.n + kBlock - 1) / kBlock);
  k_igr_prim<<<g, kBlock, 0, s>>>(a.n, u, a.prim, a.rinv);
  MFT_LAUNCH_CHECK();
  k_igr_rhs<<<g, kBlock, 0, s>>>(a);
  MFT_LAUNCH_CHECK();
  if (a.staged) return launch_igr_staged(a, s);
  for (int it = 0; it < a.maxiter; ++it) {
    const double* uo = (it & 1) ? a.u1 : a.u0;
    double* un = (it & 1) ? a.u0 : a.u1;
    k_igr_newdir<<<g, kBlock, 0, s>>>(a, uo, un);
    MFT_LAUNCH_CHECK();
    k_igr_dir<<<g, kBlock, 0, s>>>(a, un);
    MFT_LAUNCH_CHECK();
    k_igr_op<<<g, kBlock, 0, s>>>(a, un);
    MFT_LAUNCH_CHECK();
    k_igr_update<<<g, kBlock, 0, s>>>(a, un);
    MFT_LAUNCH_CHECK();
  }
  k_igr_flux<<<g, kBlock, 0, s>>>(a);
  MFT_LAUNCH_CHECK();
}

}  // namespace mft
