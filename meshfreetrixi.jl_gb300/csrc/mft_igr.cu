// Information geometric regularisation source (SourceIGR, src/sources/IGR.jl:17-239) for
// the 2D Euler equations, FP64:
//   b = alpha (tr(Du)^2 + tr(Du^2)), with tr(Du) formed as the reference writes it,
//       Dx rho + Dy v1 (update_igr_rhs!, :143-145), tr(Du^2) = (Dx v1)^2 +
//       2 (Dy v1)(Dx v2) + (Dy v2)^2 (:151-153);
//   sigma from (rho^-1 - alpha (Dx rho^-1 Dx + Dy rho^-1 Dy)) sigma = b by unpreconditioned
//       conjugate gradients from sigma = 0, at most maxiter iterations, relative
//       tolerance sqrt(eps) (the in-place cg! the reference intends at :189);
//   du[rho v1] -= Dx sigma, du[rho v2] -= Dy sigma (:214-237).
// The CG runs as a fixed sequence of kernels (four per iteration) whose scalars live in
// device memory; once converged, the remaining kernels return at entry, so one rhs!
// evaluation is a fixed launch sequence that a CUDA graph can hold.  Reductions are
// block partials finished by the last block in a fixed order (deterministic).
#include <algorithm>
#include <cfloat>

#include "mft_device.cuh"
#include "mft_dw.cuh"
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

// ---------------------------------------------------------------- double-word form
//
// The same iteration with the gathers' sums in double-word arithmetic over the staged layout
// (mft_dw.cuh, mft_halo.cuh), where the engine's FP64 form uses it; the CG scalars, vectors and
// their updates stay FP64.  The FP64 gathers issued 70 multiply-adds per node on a pipe that
// takes 35 us for 262,144 nodes of them and fetched every neighbour value from L2; here one
// packed product serves an entry and the gathers are bound by the 630 B of weights and
// positions per node.  What the iteration spends: the new direction is formed while staging
// (no pass of its own), and the operator's gather walks the row groups in the opposite order of
// the direction's, so that the weights one reads last are still in L2 for the other (165 MB of
// weights at 262,144 nodes against 129 MB of L2).  Each kernel is the programmatic dependent of
// the one before (what that one wrote is read past L1, after pdl_wait).  One solve of
// 14 iterations (of at most 20) at 262,144 nodes: 1947 -> 1219 us (the order of the groups
// alone: 1604 -> 1511 when it was measured); where all 20 run, 2.44 -> 1.63 ms per rhs!.

// Per node: rinv and the records of the right-hand side's gather, chunks (v1, v2), (rho, rho).
__global__ void k_igr_prim_dw(int64_t n, const double* __restrict__ u, float4* rec, double* rinv) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double2 a = reinterpret_cast<const double2*>(u)[i * 2];
  const double m2 = u[i * 4 + 2];
  const float2 rho = dw::split(a.x), r = dw::recip(rho);
  rec[i * 2] = dw::chunk(dw::mul(dw::split(a.y), r), dw::mul(dw::split(m2), r));
  rec[i * 2 + 1] = dw::chunk(rho, rho);
  rinv[i] = ddiv(1.0, a.x);
}

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
// Measured (262,144 nodes, one solve): groups of 2 / 3 / 4 / 5 uncapped 1371 / 1322 / 1398 / 1450
// us; 3 capped at four blocks 1219, 2 at five 1507 (spills), 5 at three 1369.
constexpr int kIgrGroup = 3, kIgrBlocks = 4;

// One entry of a row's stream.
struct IgrStream {
  int lc;
  float4 wxy;
};

// The gather of row group `group` (the block's): per entry of this thread's row
// sum(weights, record of the neighbour), the record staged in shared memory as chunk(c) or, in a
// group without a list, chunk(c) itself.  What does not depend on the kernel before -- the row,
// the list, and the first 2 G entries' weights -- is requested before wait(), which returns
// whether there is anything to do: the weights' latency and the launch then overlap that
// kernel's tail and the staging.  (STAGED: two loops, because one that chose the source per entry loaded
// through generic addresses.)  Every thread of the block must call it.
template <int G, bool STAGED, typename Wait, typename Chunk, typename Sum>
__device__ __forceinline__ bool igr_gather_as(const IgrArgs& a, int64_t r, int h0, int nh, float4* sm,
                                              Wait wait, Chunk chunk, Sum sum) {
  const bool live = r < a.n;
  const int64_t base = live ? a.ell.slice_off[r >> 5] + (r & 31) : 0;
  const int len = live ? a.ell.row_len[r] : 0;
  IgrStream e[2][G];
  auto load = [&](IgrStream& x, int j) {
    const int64_t p = base + (int64_t)j * 32;
    x.lc = STAGED ? (int)__ldg(a.ell.lcol + p) : __ldg(a.ell.col + p);
    x.wxy = __ldg(a.wxydw + p);
  };
  auto use = [&](const IgrStream& x) { sum(x.wxy, STAGED ? sm[x.lc] : chunk((int64_t)x.lc)); };
  const int q0 = threadIdx.x, q1 = q0 + blockDim.x;
  const int c0 = STAGED && q0 < nh ? __ldg(a.ell.halo_col + h0 + q0) : -1;
  const int c1 = STAGED && q1 < nh ? __ldg(a.ell.halo_col + h0 + q1) : -1;
  pipelined_open<G>(len, e, load);
  if (!wait()) return false;
  if (STAGED) {
    const float4 v0 = c0 >= 0 ? chunk(c0) : make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 v1 = c1 >= 0 ? chunk(c1) : make_float4(0.f, 0.f, 0.f, 0.f);
    if (c0 >= 0) sm[q0] = v0;
    if (c1 >= 0) sm[q1] = v1;
    for (int q = q1 + blockDim.x; q < nh; q += blockDim.x)
      sm[q] = chunk((int64_t)__ldg(a.ell.halo_col + h0 + q));
    __syncthreads();
  }
  pipelined_run<G>(len, e, load, use);
  return true;
}
template <int G, typename Wait, typename Chunk, typename Sum>
__device__ __forceinline__ bool igr_gather(const IgrArgs& a, unsigned group, float4* sm, Wait wait,
                                           Chunk chunk, Sum sum) {
  const int h0 = __ldg(a.ell.halo_off + group), nh = __ldg(a.ell.halo_off + group + 1) - h0;
  const int64_t r = group * (int64_t)blockDim.x + threadIdx.x;  // layout row
  if (nh > 0) return igr_gather_as<G, true>(a, r, h0, nh, sm, wait, chunk, sum);
  return igr_gather_as<G, false>(a, r, h0, nh, sm, wait, chunk, sum);
}

__global__ void __launch_bounds__(kHaloRows) k_igr_rhs_dw(IgrArgs a) {
  extern __shared__ float4 sm[];
  const float4* rec = reinterpret_cast<const float4*>(a.prim);
  const bool staged = stage_halo<2>(a.ell, sm, [&](int k, int64_t c) { return rec + c * 2 + k; });
  const int hs = a.ell.halo_stride;
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;  // layout row
  double rr = 0.0;
  if (r < a.n) {
    const int64_t i = ell_node(a.ell, r);
    const int64_t base = a.ell.slice_off[r >> 5] + (r & 31);
    dw::Acc2 sx = dw::zero2(), sy = dw::zero2();  // (Dx v1, Dx v2), (Dy v1, Dy v2)
    dw::Acc sr = dw::zero();
    auto sum = [&](float4 wxy, float4 v, float4 d) {
      const float2 wx = dw::chunk_a(wxy);
      dw::fma_acc2(sx, dw::both(wx), dw::pair2(v));
      dw::fma_acc2(sy, dw::both(dw::chunk_b(wxy)), dw::pair2(v));
      dw::fma_acc(sr, wx, dw::chunk_a(d));
    };
    if (staged) {
      pipelined_row<3, IgrStream>(
          a.ell.row_len[r],
          [&](IgrStream& e, int j) {
            e.lc = __ldg(a.ell.lcol + base + j * 32);
            e.wxy = __ldg(a.wxydw + base + j * 32);
          },
          [&](const IgrStream& e) {
            sum(e.wxy, sm[halo_at<2>(0, e.lc, hs)], sm[halo_at<2>(1, e.lc, hs)]);
          });
    } else {
      for (int j = 0; j < a.ell.row_len[r]; ++j) {
        const int64_t c = __ldg(a.ell.col + base + j * 32);
        sum(__ldg(a.wxydw + base + j * 32), __ldg(rec + c * 2), __ldg(rec + c * 2 + 1));
      }
    }
    const double dxv1 = dw::to_double(dw::first(sx)), dxv2 = dw::to_double(dw::second(sx));
    const double dyv1 = dw::to_double(dw::first(sy)), dyv2 = dw::to_double(dw::second(sy));
    const double tr = dadd(dw::to_double(sr), dyv1);
    const double tsq = dadd(dadd(dmul(dxv1, dxv1), dmul(dmul(2.0, dyv1), dxv2)), dmul(dyv2, dyv2));
    const double b = dmul(a.alpha, dadd(dmul(tr, tr), tsq));
    a.x[i] = 0.0;
    a.r[i] = b;
    a.u0[i] = 0.0;
    rr = dmul(b, b);
  }
  double total;
  if (last_block_sum(rr, a.partial, a.counter, &total)) igr_start(a, total);
}

// t = rinv (Dx u_new, Dy u_new) as chunks (t1, t2), u_new = r + beta u_old formed while staging
// and written for the node's own row; or, FLUX, add = -(Dx sigma, Dy sigma).
template <bool FLUX>
__global__ void __launch_bounds__(kHaloRows, kIgrBlocks) k_igr_dir_dw(IgrArgs a, const double* uo, double* un) {
  extern __shared__ float4 sm[];
  pdl_trigger();
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;  // layout row
  const int64_t i = r < a.n ? ell_node(a.ell, r) : 0;
  const double ri = !FLUX && r < a.n ? a.rinv[i] : 0.0;
  double beta = 0.0;
  auto value = [&](int64_t c) { return FLUX ? __ldcg(a.x + c) : dadd(__ldcg(a.r + c), dmul(beta, __ldcg(uo + c))); };
  dw::Acc2 s = dw::zero2();
  const bool ran = igr_gather<kIgrGroup>(
      a, blockIdx.x, sm,
      [&] {
        pdl_wait();
        beta = FLUX ? 0.0 : a.sc->beta;
        return FLUX || !a.sc->done;
      },
      [&](int64_t c) {
        const float2 v = dw::split(value(c));
        return dw::chunk(v, v);
      },
      [&](float4 wxy, float4 v) { dw::fma_acc2(s, dw::pair2(wxy), dw::pair2(v)); });
  if (!ran || r >= a.n) return;
  const double sx = dw::to_double(dw::first(s)), sy = dw::to_double(dw::second(s));
  if (FLUX) {
    reinterpret_cast<double2*>(a.add)[i] = make_double2(-sx, -sy);
    return;
  }
  un[i] = value(i);
  reinterpret_cast<float4*>(a.t)[i] = dw::chunk(dw::split(dmul(ri, sx)), dw::split(dmul(ri, sy)));
}

// c = rinv u_new - alpha (Dx t1 + Dy t2) and the block's part of u_new . c.  Block b takes the
// group gridDim.x - 1 - b.  The update's blocks add the parts up, each for itself: a last block
// that did it here would hold every one of the 1024 blocks at a fence and an atomic.
__global__ void __launch_bounds__(kHaloRows, kIgrBlocks) k_igr_op_dw(IgrArgs a, const double* un) {
  extern __shared__ float4 sm[];
  pdl_trigger();
  const unsigned group = gridDim.x - 1 - blockIdx.x;
  const float4* t4 = reinterpret_cast<const float4*>(a.t);
  const int64_t r = group * (int64_t)blockDim.x + threadIdx.x;  // layout row
  const int64_t i = r < a.n ? ell_node(a.ell, r) : 0;
  const double ri = r < a.n ? a.rinv[i] : 0.0;
  dw::Acc2 s = dw::zero2();
  const bool ran = igr_gather<kIgrGroup>(
      a, group, sm,
      [&] {
        pdl_wait();
        return !a.sc->done;
      },
      [&](int64_t c) { return __ldcg(t4 + c); },
      [&](float4 wxy, float4 v) { dw::fma_acc2(s, dw::pair2(wxy), dw::pair2(v)); });
  if (!ran) return;
  double uc = 0.0;
  if (r < a.n) {
    const double ui = __ldcg(un + i);
    const double ci = dsub(dmul(ri, ui), dmul(a.alpha, dw::sum_double(dw::first(s), dw::second(s))));
    a.c[i] = ci;
    uc = dmul(ui, ci);
  }
  uc = block_total(uc);
  if (threadIdx.x == 0) a.partial[group] = uc;
}

// alpha_cg = res^2 / (u_new . c) from the nparts parts; x += alpha_cg u_new; r -= alpha_cg c;
// new residual, beta, convergence
__global__ void __launch_bounds__(kHaloRows) k_igr_update_dw(IgrArgs a, const double* un,
                                                             unsigned nparts, double* partial) {
  pdl_trigger();
  pdl_wait();
  if (a.sc->done) return;
  __shared__ double al_s;
  double uc = 0.0;
  for (unsigned b = threadIdx.x; b < nparts; b += blockDim.x) uc = dadd(uc, __ldcg(a.partial + b));
  uc = block_total(uc);
  if (threadIdx.x == 0) al_s = ddiv(dmul(a.sc->res, a.sc->res), uc);
  __syncthreads();
  const double al = al_s;
  double rr = 0.0;
  for (int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; i < a.n;
       i += (int64_t)gridDim.x * blockDim.x) {
    a.x[i] = dadd(a.x[i], dmul(al, __ldcg(un + i)));
    const double r = dsub(a.r[i], dmul(al, __ldcg(a.c + i)));
    a.r[i] = r;
    rr = dadd(rr, dmul(r, r));
  }
  double total;
  if (last_block_sum(rr, partial, a.counter, &total)) igr_next(a, total);
}

void launch_igr_dw(const IgrArgs& a, const double* u, cudaStream_t s) {
  const int rows = a.ell.halo_rows;
  const unsigned g = (unsigned)((a.n + rows - 1) / rows);
  const size_t one = (size_t)a.ell.halo_stride * sizeof(float4);
  // the update's grid: two blocks of 256 threads per SM leave its last-block sum short
  const unsigned gu = std::min<unsigned>((unsigned)((a.n + kHaloRows - 1) / kHaloRows), 304u);
  k_igr_prim_dw<<<(unsigned)((a.n + 255) / 256), 256, 0, s>>>(a.n, u, reinterpret_cast<float4*>(a.prim), a.rinv);
  MFT_LAUNCH_CHECK();
  k_igr_rhs_dw<<<g, rows, 2 * one, s>>>(a);
  MFT_LAUNCH_CHECK();
  for (int it = 0; it < a.maxiter; ++it) {
    const double* uo = (it & 1) ? a.u1 : a.u0;
    double* un = (it & 1) ? a.u0 : a.u1;
    launch_k(k_igr_dir_dw<false>, g, rows, one, s, true, a, uo, un);
    launch_k(k_igr_op_dw, g, rows, one, s, true, a, (const double*)un);
    launch_k(k_igr_update_dw, gu, kHaloRows, 0, s, true, a, (const double*)un, g, a.partial + g);
  }
  launch_k(k_igr_dir_dw<true>, g, rows, one, s, true, a, (const double*)nullptr, (double*)nullptr);
}

}  // namespace

void launch_igr(const IgrArgs& a, const double* u, cudaStream_t s) {
  if (a.n <= 0) return;
  if (a.wxydw && a.ell.halo_off && a.ell.halo_rows > 0) return launch_igr_dw(a, u, s);
  const unsigned g = (unsigned)((a.n + kBlock - 1) / kBlock);
  k_igr_prim<<<g, kBlock, 0, s>>>(a.n, u, a.prim, a.rinv);
  MFT_LAUNCH_CHECK();
  k_igr_rhs<<<g, kBlock, 0, s>>>(a);
  MFT_LAUNCH_CHECK();
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
