// FP64 form of the 2D Euler rhs! gathers in double-word FP32 arithmetic (mft_dw.cuh).
//
// Same passes, layouts and epilogues as the FP64 kernels (mft_apply.cu); what changes is
// how the sums over a stencil are formed.  Operator weights, the per-node fluxes and the
// neighbour states are read as double-word pairs (h, l) -- 8 bytes per value, the
// footprint of an FP64 value -- and the products and sums run on the FP32 pipe with
// error-free transformations; per-node values (the stage epilogue, the viscosity) stay
// in FP64.  Accumulation order per row is the layout's entry order (ascending columns, or
// in the rows of staged groups the bank-spreading order of build_ell), shared by every
// variant.
#include <cuda_runtime.h>
#include <math.h>

#include <mutex>
#include <set>
#include <utility>

#include "mft_device.cuh"
#include "mft_dw.cuh"
#include "mft_eps.cuh"
#include "mft_halo.cuh"
#include "mft_internal.cuh"
#include "mft_tma.cuh"

namespace mft {

namespace {

using namespace dev;

inline unsigned grid_for(int64_t n, int block) { return (unsigned)((n + block - 1) / block); }

// The streamed arrays of a warp's slice (column indices and up to three weight arrays,
// read once per launch) requested into L2 a chunk of kPfSlots slots at a time by one
// lane, ahead of the slots the warp gathers (the weights otherwise arrive from DRAM on
// each slot's critical path).  The range stays inside the slice.
constexpr int kPfSlots = 8;
struct SliceArrays {
  const void* arr[4];
  int esize[4];
  int narr;
};
static __device__ __forceinline__ void prefetch_chunk(const SliceArrays& sa, int64_t s_lo,
                                                      int64_t s_hi, int chunk) {
  const int64_t e0 = s_lo + (int64_t)chunk * kPfSlots * 32;
  if (e0 >= s_hi) return;
  const int64_t ne = min((int64_t)kPfSlots * 32, s_hi - e0);
#pragma unroll
  for (int k = 0; k < 4; ++k)
    if (k < sa.narr)
      tma::bulk_prefetch_l2(static_cast<const char*>(sa.arr[k]) + e0 * sa.esize[k],
                            (uint32_t)(ne * sa.esize[k]));
}

// Per node: the state as double-word pairs and the Euler flux pair evaluated from them in
// double-word arithmetic (the textbook flux, one reciprocal for both velocities; each
// operation is accurate to about 2 u^2 of its operands, u = 2^-24), as the records the
// forward gather reads, in chunks of two values (dw::chunk): U = (rho, m1), (m2, E) and
// F = (fx1, f12), (f12, fy2), (fx3, fy3), (m1, m2), with f12 = m1 m2 / rho the x flux of m2
// and the y flux of m1; the mass fluxes are m1 and m2.  gm1 = gamma - 1 as a pair.  The state is
// split on the integer pipe.  Shared by the flux kernel and the staged gathers that form the
// records while staging, so both give the same bits.
static __device__ __forceinline__ void euler_records(double2 a, double2 b, float2 gm1,
                                                     float4* F, float4* U) {
  const float2 rho = dw::split(a.x), m1 = dw::split(a.y), m2 = dw::split(b.x);
  const float2 en = dw::split(b.y);
  const float2 r = dw::recip(rho);
  const float2 v1 = dw::mul(m1, r), v2 = dw::mul(m2, r);
  const float2 a1 = dw::mul(m1, v1), a2 = dw::mul(m2, v2);
  const float2 p = dw::mul(gm1, dw::add(en, dw::neg(dw::scale2(dw::add(a1, a2), 0.5f))));
  const float2 ep = dw::add(en, p);
  const float2 fx1 = dw::add(a1, p), f12 = dw::mul(m1, v2), fx3 = dw::mul(ep, v1);
  const float2 fy2 = dw::add(a2, p), fy3 = dw::mul(ep, v2);
  F[0] = dw::chunk(fx1, f12);
  F[1] = dw::chunk(f12, fy2);
  F[2] = dw::chunk(fx3, fy3);
  F[3] = dw::chunk(m1, m2);
  U[0] = dw::chunk(rho, m1);
  U[1] = dw::chunk(m2, en);
}

__global__ void k_prep_euler_dw(int64_t n, float2 gm1, const double* __restrict__ u,
                                float4* __restrict__ F, float4* __restrict__ U) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double2* ui = reinterpret_cast<const double2*>(u) + i * 2;
  float4 f[4], uu[2];
  euler_records(ui[0], ui[1], gm1, f, uu);
  float4* Fi = F + i * 4;
#pragma unroll
  for (int k = 0; k < 4; ++k) Fi[k] = f[k];
  U[i * 2] = uu[0];
  U[i * 2 + 1] = uu[1];
}

// Chunks of a staged forward record: with the state needed (t, q or the Flyer term) the
// three flux chunks and the two state chunks, whose m1 and m2 serve the mass flux too; else
// the four flux chunks.
template <bool NEEDU>
constexpr int kFwdChunks = NEEDU ? 5 : 4;

// Staging with the records formed on the fly: each thread reads the FP64 states of list
// entries q and q + blockDim.x (both loads in flight together), forms their records
// (euler_records) and writes their chunks into shared memory where stage_halo's copies would
// (halo_at).  Returns false for a group without a list.
template <bool NEEDU>
static __device__ __forceinline__ bool stage_halo_records(const EllView& ell, float4* sm,
                                                          const double* __restrict__ u,
                                                          float2 gm1) {
  const int h0 = __ldg(ell.halo_off + blockIdx.x);
  const int nh = __ldg(ell.halo_off + blockIdx.x + 1) - h0;
  if (nh <= 0) return false;  // block-uniform
  const int hs = ell.halo_stride;
  const double2* __restrict__ u2 = reinterpret_cast<const double2*>(u);
  auto put = [&](int q, double2 a, double2 b) {
    float4 F[4], U[2];
    euler_records(a, b, gm1, F, U);
#pragma unroll
    for (int k = 0; k < 3; ++k) sm[halo_at<kFwdChunks<NEEDU>>(k, q, hs)] = F[k];
    if (NEEDU) {
      sm[halo_at<5>(3, q, hs)] = U[0];
      sm[halo_at<5>(4, q, hs)] = U[1];
    } else {
      sm[halo_at<4>(3, q, hs)] = F[3];
    }
  };
  for (int q0 = threadIdx.x; q0 < nh; q0 += 2 * blockDim.x) {
    const int q1 = q0 + blockDim.x;
    const int64_t c0 = __ldg(ell.halo_col + h0 + q0);
    const int64_t c1 = q1 < nh ? (int64_t)__ldg(ell.halo_col + h0 + q1) : c0;
    const double2 a0 = __ldg(u2 + c0 * 2), b0 = __ldg(u2 + c0 * 2 + 1);
    const double2 a1 = __ldg(u2 + c1 * 2), b1 = __ldg(u2 + c1 * 2 + 1);
    put(q0, a0, b0);
    if (q1 < nh) put(q1, a1, b1);
  }
  __syncthreads();
  return true;
}

// One stencil entry of the forward gather: the weight pairs (wxy: the chunk of w_x and w_y)
// and the neighbour's flux and state chunks, requested together.  f[3] = (m1, m2) only
// without the state chunks.
struct FwdEntry {
  float4 wxy;
  float2 wl;
  float4 f[4], u[2];
};

// The entry of a directly gathered row: 32-byte loads, so that a record's sector is looked up once
// (with 16-byte ones 262,144 scattered nodes, none staged, took 166 us per rhs! without sources
// and 318 with residual viscosity; with these 130 and 266).
template <bool NEEDU, bool NEEDL>
static __device__ __forceinline__ FwdEntry fwd_load(const FwdArgs& a, const float4* F,
                                                    const float4* U, int64_t p, int64_t c) {
  FwdEntry e;
  e.wxy = __ldg(a.wxydw + p);
  const F8 f = ldg_f8(reinterpret_cast<const float*>(F + c * 4));
  e.f[0] = f.lo;
  e.f[1] = f.hi;
  if (NEEDU) {
    e.f[2] = __ldg(F + c * 4 + 2);
    const F8 u = ldg_f8(reinterpret_cast<const float*>(U + c * 2));
    e.u[0] = u.lo;
    e.u[1] = u.hi;
  } else {
    const F8 g = ldg_f8(reinterpret_cast<const float*>(F + c * 4 + 2));
    e.f[2] = g.lo;
    e.f[3] = g.hi;
  }
  if (NEEDL) e.wl = __ldg(a.wldw + p);
  return e;
}

// The streamed arrays of a row in the staged loop: the row's element of slot j is element
// 32 j of each.
struct RowStream {
  const uint16_t* lc;
  const float4* wxy;
  const float2* wl;
};

constexpr int kPipelined = 10;  // PIPE: pipelined_row

// The streamed part of entry j of the row.
struct Streamed {
  int lc;
  float4 wxy;
  float2 wl;
};
template <bool XY, bool L, bool HINT = false>
static __device__ __forceinline__ void stream_load(Streamed& e, const RowStream& w, int j,
                                                   uint64_t pol = 0) {
  const int o = j * 32;
  e.lc = HINT ? ldg_hint(w.lc + o, pol) : __ldg(w.lc + o);
  if (XY) e.wxy = HINT ? ldg_hint(w.wxy + o, pol) : __ldg(w.wxy + o);
  if (L) e.wl = HINT ? ldg_hint(w.wl + o, pol) : __ldg(w.wl + o);
}

// The entry with the neighbour's records read from the staged halo.
template <bool NEEDU, bool NEEDL>
static __device__ __forceinline__ FwdEntry fwd_load_halo(const Streamed& x, const float4* sm,
                                                         int hs) {
  FwdEntry e;
  e.wxy = x.wxy;
  if (NEEDL) e.wl = x.wl;
  constexpr int N = kFwdChunks<NEEDU>;
#pragma unroll
  for (int k = 0; k < (NEEDU ? 3 : 4); ++k) e.f[k] = sm[halo_at<N>(k, x.lc, hs)];
  if (NEEDU) {
    e.u[0] = sm[halo_at<N>(3, x.lc, hs)];
    e.u[1] = sm[halo_at<N>(4, x.lc, hs)];
  }
  return e;
}

// The forward gather's running sums, two values each: f12 = (momentum rows), f3 = (x part,
// y part) of the energy row, f0 the same of the mass row (where t does not give it), and
// t = (Dx u, Dy u), q over the four variables.
struct FwdSums {
  dw::Acc2 f0, f12, f3, tx[2], ty[2], q[2];
};

template <bool WT, bool NEEDL>
static __device__ __forceinline__ void fwd_accum(const FwdEntry& e, FwdSums& s) {
  constexpr bool NEEDU = WT || NEEDL;
  const dw::DW2 wxy = dw::pair2(e.wxy);
  const dw::DW2 wx = dw::both(dw::chunk_a(e.wxy)), wy = dw::both(dw::chunk_b(e.wxy));
  dw::fma_acc2(s.f12, wx, dw::pair2(e.f[0]));
  dw::fma_acc2(s.f12, wy, dw::pair2(e.f[1]));
  dw::fma_acc2(s.f3, wxy, dw::pair2(e.f[2]));
  // with t formed, the rho row is tx_1 + ty_2
  if (!WT)
    dw::fma_acc2(s.f0, wxy,
                 NEEDU ? dw::pair2(dw::chunk_b(e.u[0]), dw::chunk_a(e.u[1])) : dw::pair2(e.f[3]));
  if (WT) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      dw::fma_acc2(s.tx[k], wx, dw::pair2(e.u[k]));
      dw::fma_acc2(s.ty[k], wy, dw::pair2(e.u[k]));
    }
  }
  if (NEEDL) {
    const dw::DW2 wl = dw::both(e.wl);
#pragma unroll
    for (int k = 0; k < 2; ++k) dw::fma_acc2(s.q[k], wl, dw::pair2(e.u[k]));
  }
}

// Forward gather (Euler), one node per thread over the sliced ELL: the flux divergence
// -sum_j (Dx F_x + Dy F_y), t = (Dx u, Dy u) (WT), q = lap u (WQ) or the Flyer term
// H u (FLY), as in k_fwd_euler_f64.  Per stencil entry: the weights' 16-byte chunk (and 8 bytes
// more for q or H u), and of the neighbour three flux chunks and the state's two, or four flux
// chunks where the state is not needed (read directly: 256-bit loads).
// PIPE = 0: one entry per loop iteration; PIPE = 2: two (the compiler overlaps their
// loads); PIPE = 1: software pipeline -- the column index is loaded two entries ahead and
// the weights and records one entry ahead, so that the gathers of entry j + 1 are in flight while entry j is
// accumulated (the gathers are latency-bound: most samples stall on their results).
// MINB: minimum resident blocks per SM requested from the compiler (register cap).
// The variants form the same sums in the same order; the autotuner picks one.
// HALO: blocks of one row group (ell.halo_rows rows) first stage the group's neighbour
// records in shared memory and read them from there (groups without a list gather
// directly); PIPE then sets the loop's unrolling, or kPipelined.  HINT: the staged loop reads the
// streamed positions and weights with an L2 evict-first policy and the epilogue writes t,
// q and the partial du with evict-last, which the transpose gather reads next.  FUSE: the
// staged records are formed from the FP64 state while staging (stage_halo_records), so
// the flux kernel's pairs are not read; launched only when every group is staged (a group
// without a list sets MFT_ERR_STATE in *a.err and its rows are not written).
template <bool WT, bool WQ, int FLY, int PIPE, int MINB, bool PREF, bool HALO, bool HINT = false,
          bool FUSE = false>
__global__ void __launch_bounds__(HALO ? kHaloRows : kBlock, MINB) k_fwd_euler_dw(FwdArgs a) {
  const int64_t r = blockIdx.x * (int64_t)(HALO ? (int)blockDim.x : kBlock) + threadIdx.x;
  constexpr bool NEEDL = WQ || FLY != 0, NEEDU = WT || NEEDL;
  const float4* __restrict__ F = reinterpret_cast<const float4*>(a.Fdw);
  const float4* __restrict__ U = reinterpret_cast<const float4*>(a.udw);
  extern __shared__ float4 hsm[];
  bool staged = false;
  if (HALO && FUSE) {
    staged = stage_halo_records<NEEDU>(a.ell, hsm, a.ustate, a.gm1dw);
    if (!staged) {
      if (threadIdx.x == 0) atomicExch(a.err, MFT_ERR_STATE);
      return;
    }
  } else if (HALO) {
    staged = stage_halo<kFwdChunks<NEEDU>>(a.ell, hsm, [&](int k, int64_t c) {
      return !NEEDU || k < 3 ? F + c * 4 + k : U + c * 2 + (k - 3);
    });
  }
  if (r >= a.n) return;
  const int64_t i = ell_node(a.ell, r);
  const int64_t base = a.ell.slice_off[r >> 5] + (r & 31);
  const int len = a.ell.row_len[r];
  const int32_t* __restrict__ col = a.ell.col;
  FwdSums sum;
  sum.f0 = sum.f12 = sum.f3 = dw::zero2();
#pragma unroll
  for (int k = 0; k < 2; ++k) sum.tx[k] = sum.ty[k] = sum.q[k] = dw::zero2();
  const uint16_t* __restrict__ lcol = a.ell.lcol;
  const int hs = a.ell.halo_stride;
  if (HALO && staged) {
    SliceArrays sa{};
    int64_t s_lo = 0, s_hi = 0;
    const bool pf_lane = PREF && (threadIdx.x & 31) == 0;
    if (pf_lane) {
      sa.arr[0] = lcol; sa.esize[0] = 2;
      sa.arr[1] = a.wxydw; sa.esize[1] = 16;
      sa.arr[2] = a.wldw; sa.esize[2] = 8;
      sa.narr = NEEDL ? 3 : 2;
      s_lo = a.ell.slice_off[r >> 5];
      s_hi = a.ell.slice_off[(r >> 5) + 1];
      prefetch_chunk(sa, s_lo, s_hi, 0);
      prefetch_chunk(sa, s_lo, s_hi, 1);
    }
    constexpr int UNR = PIPE < 1 || PIPE == kPipelined ? 1 : PIPE;
    const uint64_t pol = HINT ? l2_evict_first() : 0;
    RowStream w{lcol + base, a.wxydw + base, a.wldw + base};
    auto load = [&](Streamed& x, int j) { stream_load<true, NEEDL, HINT>(x, w, j, pol); };
    auto use = [&](const Streamed& x) {
      fwd_accum<WT, NEEDL>(fwd_load_halo<NEEDU, NEEDL>(x, hsm, hs), sum);
    };
    if constexpr (PIPE == kPipelined) {
      pipelined_row<3, Streamed>(len, load, use);
    } else {
      int j = 0;
      for (; j + UNR <= len; j += UNR) {
        if (pf_lane && (j % kPfSlots) < UNR) prefetch_chunk(sa, s_lo, s_hi, j / kPfSlots + 2);
        Streamed x[UNR];
#pragma unroll
        for (int k = 0; k < UNR; ++k) load(x[k], k);
#pragma unroll
        for (int k = 0; k < UNR; ++k) use(x[k]);
        w.lc += UNR * 32;
        w.wxy += UNR * 32;
        w.wl += UNR * 32;
      }
      for (; j < len; ++j) {
        Streamed x;
        load(x, 0);
        use(x);
        w.lc += 32;
        w.wxy += 32;
        w.wl += 32;
      }
    }
  } else if (PIPE == 0) {
#pragma unroll 1
    for (int j = 0; j < len; ++j) {
      const int64_t p = base + ((int64_t)j << 5);
      const int64_t c = __ldg(col + p);
      fwd_accum<WT, NEEDL>(fwd_load<NEEDU, NEEDL>(a, F, U, p, c), sum);
    }
  } else if (PIPE == 2 || (HALO && PIPE > 2)) {
    SliceArrays sa{};
    int64_t s_lo = 0, s_hi = 0;
    const bool pf_lane = PREF && (threadIdx.x & 31) == 0;
    if (pf_lane) {
      sa.arr[0] = col; sa.esize[0] = 4;
      sa.arr[1] = a.wxydw; sa.esize[1] = 16;
      sa.arr[2] = a.wldw; sa.esize[2] = 8;
      sa.narr = NEEDL ? 3 : 2;
      s_lo = a.ell.slice_off[r >> 5];
      s_hi = a.ell.slice_off[(r >> 5) + 1];
      prefetch_chunk(sa, s_lo, s_hi, 0);
      prefetch_chunk(sa, s_lo, s_hi, 1);
    }
#pragma unroll 2
    for (int j = 0; j < len; ++j) {
      if (pf_lane && (j % kPfSlots) == 0) prefetch_chunk(sa, s_lo, s_hi, j / kPfSlots + 2);
      const int64_t p = base + ((int64_t)j << 5);
      const int64_t c = __ldg(col + p);
      fwd_accum<WT, NEEDL>(fwd_load<NEEDU, NEEDL>(a, F, U, p, c), sum);
    }
  } else if (len > 0) {
    int64_t c_next = len > 1 ? (int64_t)__ldg(col + base + 32) : 0;
    FwdEntry cur = fwd_load<NEEDU, NEEDL>(a, F, U, base, __ldg(col + base));
    for (int j = 0; j < len; ++j) {
      const int64_t p1 = base + ((int64_t)(j + 1) << 5);
      const int64_t c2 = j + 2 < len ? (int64_t)__ldg(col + p1 + 32) : 0;
      FwdEntry nxt;
      if (j + 1 < len) nxt = fwd_load<NEEDU, NEEDL>(a, F, U, p1, c_next);
      fwd_accum<WT, NEEDL>(cur, sum);
      cur = nxt;
      c_next = c2;
    }
  }
  double du[4];
  if (WT) du[0] = -dw::sum_double(dw::second(sum.tx[0]), dw::first(sum.ty[1]));
  else du[0] = -dw::sum_double(dw::first(sum.f0), dw::second(sum.f0));
  du[1] = -dw::to_double(dw::first(sum.f12));
  du[2] = -dw::to_double(dw::second(sum.f12));
  du[3] = -dw::sum_double(dw::first(sum.f3), dw::second(sum.f3));
  double qv[4] = {0, 0, 0, 0};
  if (FLY) {
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      qv[2 * k] = dw::to_double(dw::first(sum.q[k]));
      qv[2 * k + 1] = dw::to_double(dw::second(sum.q[k]));
    }
  }
  if (FLY == 1) {
#pragma unroll
    for (int v = 0; v < 4; ++v) du[v] = fma(-a.hv_gamma, qv[v], du[v]);
  }
  if (WT) {
    float4* t4 = reinterpret_cast<float4*>(a.tdw) + i * 4;
    dw::DW2 t[4] = {dw::to_pair2(sum.tx[0]), dw::to_pair2(sum.tx[1]), dw::to_pair2(sum.ty[0]),
                    dw::to_pair2(sum.ty[1])};
    if (a.fuse_eps) {
      // the viscosity of this node (FP64, as k_eps forms it from the partial du held
      // here) and s = eps * t written in place of t; this FP64 work overlaps the FP32
      // gathers of other warps.  The norms come from the reductions this grid may have
      // been launched beside (launch_k with a.pdl): wait for them here, not earlier.
      pdl_wait();
      const double eps = visc::eps_value<4>(a.ea, i, du);
      if (a.ea.eps) a.ea.eps[i] = eps;
      const dw::DW2 e2 = dw::both(dw::split(eps));
#pragma unroll
      for (int k = 0; k < 4; ++k) t[k] = dw::mul(e2, t[k]);
    }
    const uint64_t keep = HINT ? l2_evict_last() : 0;
#pragma unroll
    for (int k = 0; k < 4; ++k) {
      if (HINT) st_hint(t4 + k, dw::chunk(t[k]), keep);
      else t4[k] = dw::chunk(t[k]);
    }
  }
  if (WQ) {
    float4* q4 = reinterpret_cast<float4*>(a.qdw) + i * 2;
    const uint64_t keep = HINT ? l2_evict_last() : 0;
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      const float4 o = dw::chunk(dw::to_pair2(sum.q[k]));
      if (HINT) st_hint(q4 + k, o, keep);
      else q4[k] = o;
    }
  }
  if (FLY == 2) {
    double2* h2 = reinterpret_cast<double2*>(a.hvf) + i * 2;
    h2[0] = make_double2(-a.hv_gamma * qv[0], -a.hv_gamma * qv[1]);
    h2[1] = make_double2(-a.hv_gamma * qv[2], -a.hv_gamma * qv[3]);
  }
  if (a.final_epilogue) {
    finish_node<4>(a.ep, i, du);
  } else {
    double2* d2 = reinterpret_cast<double2*>(a.du_p) + i * 2;
    if (HINT) {
      const uint64_t keep = l2_evict_last();
      st_hint(d2, make_double2(du[0], du[1]), keep);
      st_hint(d2 + 1, make_double2(du[2], du[3]), keep);
    } else {
      d2[0] = make_double2(du[0], du[1]);
      d2[1] = make_double2(du[2], du[3]);
    }
  }
}

// One entry of the transpose gather: weights and the neighbour's s = eps t (x part, y part;
// two chunks each) and q chunks.
struct RevEntry {
  float4 wxy;
  float2 wl;
  float4 s[4], q[2];
};

template <bool RV, bool LAP>
static __device__ __forceinline__ RevEntry rev_load(const RevArgs& a, const float4* S,
                                                    const float4* Q, int64_t p, int64_t c) {
  RevEntry e;
  if (RV) {
    e.wxy = __ldg(a.wxydw + p);
    const F8 x = ldg_f8(reinterpret_cast<const float*>(S + c * 4));
    const F8 y = ldg_f8(reinterpret_cast<const float*>(S + c * 4 + 2));
    e.s[0] = x.lo;
    e.s[1] = x.hi;
    e.s[2] = y.lo;
    e.s[3] = y.hi;
  }
  if (LAP) {
    e.wl = __ldg(a.wldw + p);
    const F8 q = ldg_f8(reinterpret_cast<const float*>(Q + c * 2));
    e.q[0] = q.lo;
    e.q[1] = q.hi;
  }
  return e;
}

template <bool RV, bool LAP>
static __device__ __forceinline__ RevEntry rev_load_halo(const Streamed& x, const float4* sm,
                                                         int hs) {
  RevEntry e;
  constexpr int N = (RV ? 4 : 0) + (LAP ? 2 : 0), kq = RV ? 4 : 0;  // first chunk of the q record
  if (RV) {
    e.wxy = x.wxy;
#pragma unroll
    for (int k = 0; k < 4; ++k) e.s[k] = sm[halo_at<N>(k, x.lc, hs)];
  }
  if (LAP) {
    e.wl = x.wl;
#pragma unroll
    for (int k = 0; k < 2; ++k) e.q[k] = sm[halo_at<N>(kq + k, x.lc, hs)];
  }
  return e;
}

// r: sums of Dx' s_x + Dy' s_y, l: of lap' q, two variables each
template <bool RV, bool LAP>
static __device__ __forceinline__ void rev_accum(const RevEntry& e, dw::Acc2* r, dw::Acc2* l) {
  if (RV) {
    const dw::DW2 wx = dw::both(dw::chunk_a(e.wxy)), wy = dw::both(dw::chunk_b(e.wxy));
#pragma unroll
    for (int k = 0; k < 2; ++k) {
      dw::fma_acc2(r[k], wx, dw::pair2(e.s[k]));
      dw::fma_acc2(r[k], wy, dw::pair2(e.s[2 + k]));
    }
  }
  if (LAP) {
    const dw::DW2 wl = dw::both(e.wl);
#pragma unroll
    for (int k = 0; k < 2; ++k) dw::fma_acc2(l[k], wl, dw::pair2(e.q[k]));
  }
}

// Transpose gather (Euler) over the reverse adjacency, as k_rev_f64:
// du_i = du_p_i - sum_j (Dx[j,i] s_x[j] + Dy[j,i] s_y[j]) - gamma sum_j lap[j,i] q[j],
// with s = eps * t and q as double-word pairs.  PIPE and MINB as for k_fwd_euler_dw.
template <bool RV, bool LAP, int PIPE, int MINB, bool PREF, bool HALO, bool HINT = false>
__global__ void __launch_bounds__(HALO ? kHaloRows : kBlock, MINB) k_rev_euler_dw(RevArgs a) {
  constexpr int NCH = (RV ? 4 : 0) + (LAP ? 2 : 0);
  const int64_t r = blockIdx.x * (int64_t)(HALO ? (int)blockDim.x : kBlock) + threadIdx.x;
  const float4* __restrict__ S = reinterpret_cast<const float4*>(a.sdw);
  const float4* __restrict__ Q = reinterpret_cast<const float4*>(a.qdw);
  extern __shared__ float4 hsm[];
  bool staged = false;
  if (HALO && NCH > 0) {
    staged = stage_halo<NCH>(a.ell, hsm, [&](int k, int64_t c) {
      return (RV && k < 4) ? S + c * 4 + k : Q + c * 2 + (k - (RV ? 4 : 0));
    });
  }
  if (r >= a.n) return;
  const int64_t i = ell_node(a.ell, r);
  const int64_t base = a.ell.slice_off[r >> 5] + (r & 31);
  const int len = a.ell.row_len[r];
  const int32_t* __restrict__ col = a.ell.col;
  dw::Acc2 sr[2], sl[2];
#pragma unroll
  for (int k = 0; k < 2; ++k) sr[k] = sl[k] = dw::zero2();
  const uint16_t* __restrict__ lcol = a.ell.lcol;
  const int hs = a.ell.halo_stride;
  if (HALO && staged) {
    SliceArrays sa{};
    int64_t s_lo = 0, s_hi = 0;
    const bool pf_lane = PREF && (threadIdx.x & 31) == 0;
    if (pf_lane) {
      int k = 0;
      sa.arr[k] = lcol; sa.esize[k++] = 2;
      if (RV) { sa.arr[k] = a.wxydw; sa.esize[k++] = 16; }
      if (LAP) { sa.arr[k] = a.wldw; sa.esize[k++] = 8; }
      sa.narr = k;
      s_lo = a.ell.slice_off[r >> 5];
      s_hi = a.ell.slice_off[(r >> 5) + 1];
      prefetch_chunk(sa, s_lo, s_hi, 0);
      prefetch_chunk(sa, s_lo, s_hi, 1);
    }
    constexpr int UNR = PIPE < 1 || PIPE == kPipelined ? 1 : PIPE;
    const uint64_t pol = HINT ? l2_evict_first() : 0;
    RowStream w{lcol + base, a.wxydw + base, a.wldw + base};
    auto load = [&](Streamed& x, int j) { stream_load<RV, LAP, HINT>(x, w, j, pol); };
    auto use = [&](const Streamed& x) {
      rev_accum<RV, LAP>(rev_load_halo<RV, LAP>(x, hsm, hs), sr, sl);
    };
    if constexpr (PIPE == kPipelined) {
      pipelined_row<3, Streamed>(len, load, use);
    } else {
      int j = 0;
      for (; j + UNR <= len; j += UNR) {
        if (pf_lane && (j % kPfSlots) < UNR) prefetch_chunk(sa, s_lo, s_hi, j / kPfSlots + 2);
        Streamed x[UNR];
#pragma unroll
        for (int k = 0; k < UNR; ++k) load(x[k], k);
#pragma unroll
        for (int k = 0; k < UNR; ++k) use(x[k]);
        w.lc += UNR * 32;
        w.wxy += UNR * 32;
        w.wl += UNR * 32;
      }
      for (; j < len; ++j) {
        Streamed x;
        load(x, 0);
        use(x);
        w.lc += 32;
        w.wxy += 32;
        w.wl += 32;
      }
    }
  } else if (PIPE == 0) {
#pragma unroll 1
    for (int j = 0; j < len; ++j) {
      const int64_t p = base + ((int64_t)j << 5);
      const int64_t c = __ldg(col + p);
      rev_accum<RV, LAP>(rev_load<RV, LAP>(a, S, Q, p, c), sr, sl);
    }
  } else if (PIPE == 2 || (HALO && PIPE > 2)) {
    SliceArrays sa{};
    int64_t s_lo = 0, s_hi = 0;
    const bool pf_lane = PREF && (threadIdx.x & 31) == 0;
    if (pf_lane) {
      int k = 0;
      sa.arr[k] = col; sa.esize[k++] = 4;
      if (RV) { sa.arr[k] = a.wxydw; sa.esize[k++] = 16; }
      if (LAP) { sa.arr[k] = a.wldw; sa.esize[k++] = 8; }
      sa.narr = k;
      s_lo = a.ell.slice_off[r >> 5];
      s_hi = a.ell.slice_off[(r >> 5) + 1];
      prefetch_chunk(sa, s_lo, s_hi, 0);
      prefetch_chunk(sa, s_lo, s_hi, 1);
    }
#pragma unroll 2
    for (int j = 0; j < len; ++j) {
      if (pf_lane && (j % kPfSlots) == 0) prefetch_chunk(sa, s_lo, s_hi, j / kPfSlots + 2);
      const int64_t p = base + ((int64_t)j << 5);
      const int64_t c = __ldg(col + p);
      rev_accum<RV, LAP>(rev_load<RV, LAP>(a, S, Q, p, c), sr, sl);
    }
  } else if (len > 0) {
    int64_t c_next = len > 1 ? (int64_t)__ldg(col + base + 32) : 0;
    RevEntry cur = rev_load<RV, LAP>(a, S, Q, base, __ldg(col + base));
    for (int j = 0; j < len; ++j) {
      const int64_t p1 = base + ((int64_t)(j + 1) << 5);
      const int64_t c2 = j + 2 < len ? (int64_t)__ldg(col + p1 + 32) : 0;
      RevEntry nxt;
      if (j + 1 < len) nxt = rev_load<RV, LAP>(a, S, Q, p1, c_next);
      rev_accum<RV, LAP>(cur, sr, sl);
      cur = nxt;
      c_next = c2;
    }
  }
  double du[4];
  const double2* dp2 = reinterpret_cast<const double2*>(a.du_p) + i * 2;
  const double2 d0 = dp2[0], d1 = dp2[1];
  const double dp[4] = {d0.x, d0.y, d1.x, d1.y};
#pragma unroll
  for (int v = 0; v < 4; ++v) {
    double d = dp[v];
    if (RV) d = dsub(d, dw::to_double(v & 1 ? dw::second(sr[v >> 1]) : dw::first(sr[v >> 1])));
    if (LAP)
      d = fma(-a.hv_gamma, dw::to_double(v & 1 ? dw::second(sl[v >> 1]) : dw::first(sl[v >> 1])), d);
    if (a.hvf) d = dadd(d, a.hvf[i * 4 + v]);
    du[v] = d;
  }
  if (a.final_epilogue) {
    finish_node<4>(a.ep, i, du);
  } else {
    double2* o2 = reinterpret_cast<double2*>(a.du_p_out) + i * 2;
    o2[0] = make_double2(du[0], du[1]);
    o2[1] = make_double2(du[2], du[3]);
  }
}

}  // namespace

float2 gm1_pair(double gamma) {
  const double gm1 = gamma - 1.0;
  const float h = (float)gm1;
  return make_float2(h, (float)(gm1 - (double)h));
}

bool dw_fwd_fuses(int variant) {
  return variant == 7 || variant == 9 || variant == 11 || variant == 12;
}

void launch_prep_euler_dw(int64_t n, double gamma, const double* u, float2* F, float2* U,
                          cudaStream_t s) {
  if (n <= 0) return;
  k_prep_euler_dw<<<grid_for(n, 256), 256, 0, s>>>(n, gm1_pair(gamma), u,
                                                   reinterpret_cast<float4*>(F),
                                                   reinterpret_cast<float4*>(U));
  MFT_LAUNCH_CHECK();
}

namespace {

// Kernel variants: 0 = one entry per loop iteration (fewest registers, most resident
// warps), 1 = two entries per iteration with the register count capped at six blocks per
// SM, 2 = two entries per iteration uncapped, 3 = software pipeline, 4 = variant 1 with
// the slice's streamed arrays prefetched into L2 ahead of use, 5 = variant 2 with it,
// 6 / 7 = neighbour records staged per row group in shared memory (one / two entries per
// iteration, registers capped at three blocks of kHaloRows per SM), 8 = variant 7 capped
// at four blocks, 9 = staged with the streamed loads in software pipeline (pipelined_row,
// groups of three entries, registers capped at two blocks), 11 = staged with three entries
// per iteration, 10 = variant 7 with the streamed position and weight arrays prefetched into
// L2 (as variant 4), 12 = variant 7 with L2 eviction-priority hints (streamed arrays
// evict-first; the forward gather's t, q and partial du evict-last for the transpose gather).
// Without halos (not built) the staged variants run as variant 2.
// A staged launch: one block per row group, NCH chunks of the layout's longest list
// in dynamic shared memory (above 48 KB that needs a per-kernel opt-in, made once per
// kernel and device).
template <typename Args>
void launch_staged(void (*k)(Args), const Args& a, int nch, int64_t n, cudaStream_t s,
                   bool pdl = false) {
  const size_t smem = (size_t)nch * a.ell.halo_stride * sizeof(float4);
  if (smem > 48 * 1024) {
    static std::mutex mu;
    static std::set<std::pair<const void*, int>> done;
    int dev = 0;
    MFT_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (done.insert({reinterpret_cast<const void*>(k), dev}).second)
      MFT_CUDA(cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(6 * kHaloMax * sizeof(float4))));
  }
  const int rows = a.ell.halo_rows;
  launch_k(k, grid_for(n, rows), rows, smem, s, pdl, a);
}

template <bool WT, bool WQ, int FLY>
void fwd_variant(const FwdArgs& a, int variant, int64_t n, cudaStream_t s) {
  const unsigned g = grid_for(n, kBlock);
  constexpr int nch = kFwdChunks<WT || WQ || FLY != 0>;
  const bool pdl = a.pdl != 0;
  if (variant >= 6 && !a.ell.halo_off) variant = 2;
  if (a.fuse_flux && a.ell.halo_off && dw_fwd_fuses(variant)) {
    MFT_REQUIRE(a.ustate && a.err, MFT_ERR_STATE, "fused staging needs the state and error word");
    switch (variant) {
      case 7: launch_staged(k_fwd_euler_dw<WT, WQ, FLY, 2, 3, false, true, false, true>, a, nch, n, s, pdl); break;
      case 9: launch_staged(k_fwd_euler_dw<WT, WQ, FLY, kPipelined, 2, false, true, false, true>, a, nch, n, s, pdl); break;
      case 11: launch_staged(k_fwd_euler_dw<WT, WQ, FLY, 3, 3, false, true, false, true>, a, nch, n, s, pdl); break;
      default: launch_staged(k_fwd_euler_dw<WT, WQ, FLY, 2, 3, false, true, true, true>, a, nch, n, s, pdl); break;
    }
    return;
  }
  switch (variant) {
    case 1: launch_k(k_fwd_euler_dw<WT, WQ, FLY, 2, 6, false, false>, g, kBlock, 0, s, pdl, a); break;
    case 2: launch_k(k_fwd_euler_dw<WT, WQ, FLY, 2, 1, false, false>, g, kBlock, 0, s, pdl, a); break;
    case 3: launch_k(k_fwd_euler_dw<WT, WQ, FLY, 1, 1, false, false>, g, kBlock, 0, s, pdl, a); break;
    case 4: launch_k(k_fwd_euler_dw<WT, WQ, FLY, 2, 6, true, false>, g, kBlock, 0, s, pdl, a); break;
    case 5: launch_k(k_fwd_euler_dw<WT, WQ, FLY, 2, 1, true, false>, g, kBlock, 0, s, pdl, a); break;
    case 6: launch_staged(k_fwd_euler_dw<WT, WQ, FLY, 0, 3, false, true>, a, nch, n, s, pdl); break;
    case 7: launch_staged(k_fwd_euler_dw<WT, WQ, FLY, 2, 3, false, true>, a, nch, n, s, pdl); break;
    case 8: launch_staged(k_fwd_euler_dw<WT, WQ, FLY, 2, 4, false, true>, a, nch, n, s, pdl); break;
    case 9: launch_staged(k_fwd_euler_dw<WT, WQ, FLY, kPipelined, 2, false, true>, a, nch, n, s, pdl); break;
    case 10: launch_staged(k_fwd_euler_dw<WT, WQ, FLY, 2, 3, true, true>, a, nch, n, s, pdl); break;
    case 11: launch_staged(k_fwd_euler_dw<WT, WQ, FLY, 3, 3, false, true>, a, nch, n, s, pdl); break;
    case 12: launch_staged(k_fwd_euler_dw<WT, WQ, FLY, 2, 3, false, true, true>, a, nch, n, s, pdl); break;
    default: launch_k(k_fwd_euler_dw<WT, WQ, FLY, 0, 1, false, false>, g, kBlock, 0, s, pdl, a); break;
  }
}

template <bool RV, bool LAP>
void rev_variant(const RevArgs& a, int variant, int64_t n, cudaStream_t s) {
  const unsigned g = grid_for(n, kBlock);
  constexpr int nch = (RV ? 4 : 0) + (LAP ? 2 : 0);
  if (variant >= 6 && !a.ell.halo_off) variant = 2;
  switch (variant) {
    case 1: k_rev_euler_dw<RV, LAP, 2, 6, false, false><<<g, kBlock, 0, s>>>(a); break;
    case 2: k_rev_euler_dw<RV, LAP, 2, 1, false, false><<<g, kBlock, 0, s>>>(a); break;
    case 3: k_rev_euler_dw<RV, LAP, 1, 1, false, false><<<g, kBlock, 0, s>>>(a); break;
    case 4: k_rev_euler_dw<RV, LAP, 2, 6, true, false><<<g, kBlock, 0, s>>>(a); break;
    case 5: k_rev_euler_dw<RV, LAP, 2, 1, true, false><<<g, kBlock, 0, s>>>(a); break;
    case 6: launch_staged(k_rev_euler_dw<RV, LAP, 0, 3, false, true>, a, nch, n, s); break;
    case 7: launch_staged(k_rev_euler_dw<RV, LAP, 2, 3, false, true>, a, nch, n, s); break;
    case 8: launch_staged(k_rev_euler_dw<RV, LAP, 2, 4, false, true>, a, nch, n, s); break;
    case 9: launch_staged(k_rev_euler_dw<RV, LAP, kPipelined, 2, false, true>, a, nch, n, s); break;
    case 10: launch_staged(k_rev_euler_dw<RV, LAP, 2, 3, true, true>, a, nch, n, s); break;
    case 11: launch_staged(k_rev_euler_dw<RV, LAP, 3, 3, false, true>, a, nch, n, s); break;
    case 12: launch_staged(k_rev_euler_dw<RV, LAP, 2, 3, false, true, true>, a, nch, n, s); break;
    default: k_rev_euler_dw<RV, LAP, 0, 1, false, false><<<g, kBlock, 0, s>>>(a); break;
  }
}

}  // namespace

void launch_fwd_dw(const FwdArgs& a, int variant, cudaStream_t s) {
  if (a.n <= 0) return;
  MFT_REQUIRE(a.V == 4, MFT_ERR_UNSUPPORTED, "double-word gathers: 2D Euler only");
  MFT_REQUIRE(!(a.flyer && a.want_q), MFT_ERR_UNSUPPORTED,
              "Flyer and Tominec hyperviscosity together are not supported");
  const int64_t n = a.n;
  const bool wt = a.want_t != 0, wq = a.want_q != 0;
  if (a.flyer == 0) {
    if (wt && wq) fwd_variant<true, true, 0>(a, variant, n, s);
    else if (wt) fwd_variant<true, false, 0>(a, variant, n, s);
    else if (wq) fwd_variant<false, true, 0>(a, variant, n, s);
    else fwd_variant<false, false, 0>(a, variant, n, s);
  } else if (a.flyer == 1) {
    if (wt) fwd_variant<true, false, 1>(a, variant, n, s);
    else fwd_variant<false, false, 1>(a, variant, n, s);
  } else {
    if (wt) fwd_variant<true, false, 2>(a, variant, n, s);
    else fwd_variant<false, false, 2>(a, variant, n, s);
  }
  MFT_LAUNCH_CHECK();
}

void launch_rev_dw(const RevArgs& a, int variant, cudaStream_t s) {
  if (a.n <= 0) return;
  MFT_REQUIRE(a.V == 4, MFT_ERR_UNSUPPORTED, "double-word gathers: 2D Euler only");
  const int64_t n = a.n;
  if (a.rv && a.lap) rev_variant<true, true>(a, variant, n, s);
  else if (a.rv) rev_variant<true, false>(a, variant, n, s);
  else if (a.lap) rev_variant<false, true>(a, variant, n, s);
  else rev_variant<false, false>(a, variant, n, s);
  MFT_LAUNCH_CHECK();
}

}  // namespace mft
