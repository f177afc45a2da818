// rhs! on 3D point clouds: the plain flux divergence of calc_fluxes!
// (src/solvers/pointcloudsolver/rbfsolver.jl:247-265) over the three gradient operators of
// compute_flux_operator (compute_operators.jl:500-546), FP64, fused with the strong-BC pass
// 2 and the SSP-RK stage combination (finish_node).  CompressibleEulerEquations3D (5
// variables, fluxes formed once per node and gathered) and scalar advection (the flux a_d u
// formed at the neighbour).  The sliced-ELL layout and its row order are those of the 2D
// kernels.
#include <cuda_runtime.h>

#include <mutex>
#include <set>

#include "mft_device.cuh"
#include "mft_dw.cuh"
#include "mft_halo.cuh"
#include "mft_internal.cuh"

namespace mft {

namespace {

using namespace dev;

constexpr int kRec3 = 6;  // chunks of a node's double-word flux record

inline unsigned grid_for(int64_t n, int block) { return (unsigned)((n + block - 1) / block); }

// F[i] = (F_x, F_y, F_z), each the 5 components (rho v_d, rho v v_d + p e_d, (E + p) v_d):
// the textbook flux with one reciprocal of rho for the three velocities.
__global__ void k_flux_euler3d(int64_t n, double g, const double* __restrict__ u,
                               double* __restrict__ F) {
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* ui = u + i * 5;
  const double rho = ui[0], m1 = ui[1], m2 = ui[2], m3 = ui[3], en = ui[4];
  const double rinv = ddiv(1.0, rho);
  const double v1 = dmul(m1, rinv), v2 = dmul(m2, rinv), v3 = dmul(m3, rinv);
  const double p = dmul(dsub(g, 1.0),
                        dsub(en, dmul(0.5, dadd(dadd(dmul(m1, v1), dmul(m2, v2)), dmul(m3, v3)))));
  const double ep = dadd(en, p);
  const double m[3] = {m1, m2, m3}, v[3] = {v1, v2, v3};
  double* Fi = F + i * 15;
#pragma unroll
  for (int d = 0; d < 3; ++d) {
    Fi[d * 5 + 0] = m[d];
    Fi[d * 5 + 1] = d == 0 ? dadd(dmul(m[d], v1), p) : dmul(m[d], v1);
    Fi[d * 5 + 2] = d == 1 ? dadd(dmul(m[d], v2), p) : dmul(m[d], v2);
    Fi[d * 5 + 3] = d == 2 ? dadd(dmul(m[d], v3), p) : dmul(m[d], v3);
    Fi[d * 5 + 4] = dmul(ep, v[d]);
  }
}

// du_i = -sum_j (Dx_ij F_x + Dy_ij F_y + Dz_ij F_z)(node j), one node per thread over the
// sliced ELL (lane r of a warp owns row 32 s + r of slice s), then finish_node.
template <int V>
__global__ void __launch_bounds__(kBlock) k_fwd3_f64(FwdArgs a) {
  const int64_t r = blockIdx.x * (int64_t)kBlock + threadIdx.x;  // layout row
  if (r >= a.n) return;
  const int64_t i = ell_node(a.ell, r);
  const int64_t base = a.ell.slice_off[r >> 5] + (r & 31);
  const int len = a.ell.row_len[r];
  const int32_t* __restrict__ col = a.ell.col;
  const double* __restrict__ wx = a.w[0];
  const double* __restrict__ wy = a.w[1];
  const double* __restrict__ wz = a.w[2];
  double f[V];
#pragma unroll
  for (int v = 0; v < V; ++v) f[v] = 0.0;
#pragma unroll 2
  for (int j = 0; j < len; ++j) {
    const int64_t p = base + ((int64_t)j << 5);
    const int64_t c = __ldg(col + p);
    const double x = __ldg(wx + p), y = __ldg(wy + p), z = __ldg(wz + p);
    if constexpr (V == 5) {
      const double* Fc = a.F + c * 15;
#pragma unroll
      for (int v = 0; v < 5; ++v) {
        f[v] = fma(x, __ldg(Fc + v), f[v]);
        f[v] = fma(y, __ldg(Fc + 5 + v), f[v]);
        f[v] = fma(z, __ldg(Fc + 10 + v), f[v]);
      }
    } else {
      const double uc = __ldg(a.u + c);
      f[0] = fma(x, dmul(a.ax, uc), f[0]);
      f[0] = fma(y, dmul(a.ay, uc), f[0]);
      f[0] = fma(z, dmul(a.az, uc), f[0]);
    }
  }
  double du[V];
#pragma unroll
  for (int v = 0; v < V; ++v) du[v] = -f[v];
  finish_node<V>(a.ep, i, du);
}

// Double-word form: the state split into pairs and the flux formed in double-word
// arithmetic (one reciprocal of rho refined by a Newton step).  The momentum flux is
// symmetric, so the 15 flux components hold 12 distinct values, each formed once and stored
// once, in chunks of two (dw::chunk; xy = m1 m2 / rho and so on, xx = m1 m1 / rho + p,
// ex = (E + p) v1):
//   F[i] = (m1, ex), (m2, ey), (m3, ez), (xx, xy), (yy, zz), (xz, yz)
// (96 bytes, three sectors), and F_x = (m1, xx, xy, xz, ex), F_y = (m2, xy, yy, yz, ey),
// F_z = (m3, xz, yz, zz, ez).  The state is split on the integer pipe.
__global__ void k_prep_euler3d_dw(int64_t n, float2 gm1, const double* __restrict__ u,
                                  float4* __restrict__ F) {
  pdl_trigger();  // the gather may be launched: it waits for this kernel before it reads F
  const int64_t i = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  if (i >= n) return;
  const double* ui = u + i * 5;
  const float2 rho = dw::split(ui[0]), en = dw::split(ui[4]);
  const float2 m[3] = {dw::split(ui[1]), dw::split(ui[2]), dw::split(ui[3])};
  const float2 r = dw::recip(rho);
  const float2 v[3] = {dw::mul(m[0], r), dw::mul(m[1], r), dw::mul(m[2], r)};
  const float2 mv = dw::add(dw::add(dw::mul(m[0], v[0]), dw::mul(m[1], v[1])), dw::mul(m[2], v[2]));
  const float2 p = dw::mul(gm1, dw::add(en, dw::neg(dw::scale2(mv, 0.5f))));
  const float2 ep = dw::add(en, p);
  const float2 xx = dw::add(dw::mul(m[0], v[0]), p), yy = dw::add(dw::mul(m[1], v[1]), p);
  const float2 zz = dw::add(dw::mul(m[2], v[2]), p);
  const float2 xy = dw::mul(m[0], v[1]), xz = dw::mul(m[0], v[2]), yz = dw::mul(m[1], v[2]);
  const float2 ex = dw::mul(ep, v[0]), ey = dw::mul(ep, v[1]), ez = dw::mul(ep, v[2]);
  float4* Fi = F + i * kRec3;
  Fi[0] = dw::chunk(m[0], ex);
  Fi[1] = dw::chunk(m[1], ey);
  Fi[2] = dw::chunk(m[2], ez);
  Fi[3] = dw::chunk(xx, xy);
  Fi[4] = dw::chunk(yy, zz);
  Fi[5] = dw::chunk(xz, yz);
}

// Running sums of the 3D gather: (mass, energy), (momentum 1, 2), and momentum 3 in three
// parts (x and y packed, z).
struct Sums3 {
  dw::Acc2 f04, f12, f3;
  dw::Acc f3z;
};

// One stencil entry: the weights (wxy: the chunk of w_x and w_y) against the record's 15 flux
// components, seven packed products and one scalar.
static __device__ __forceinline__ void accum3(Sums3& s, float4 wxy, float2 wz, const float4* q) {
  const dw::DW2 x = dw::both(dw::chunk_a(wxy)), y = dw::both(dw::chunk_b(wxy)), z = dw::both(wz);
  const dw::DW2 xzyz = dw::pair2(q[5]);
  dw::fma_acc2(s.f04, x, dw::pair2(q[0]));
  dw::fma_acc2(s.f12, x, dw::pair2(q[3]));
  dw::fma_acc2(s.f3, dw::pair2(wxy), xzyz);
  dw::fma_acc2(s.f04, y, dw::pair2(q[1]));
  dw::fma_acc2(s.f12, y, dw::pair2(dw::chunk_b(q[3]), dw::chunk_a(q[4])));
  dw::fma_acc(s.f3z, wz, dw::chunk_b(q[4]));
  dw::fma_acc2(s.f04, z, dw::pair2(q[2]));
  dw::fma_acc2(s.f12, z, xzyz);
}

// du_i = -sum_j (Dx_ij F_x + Dy_ij F_y + Dz_ij F_z)(node j) as compensated sums of
// double-word products (mft_dw.cuh), the stage epilogue in FP64.  Per stencil entry: three
// weight pairs and the neighbour's 96-byte flux record.  One block per row group
// (ell.halo_rows rows) first stages the group's neighbour records in shared memory (six
// 16-byte chunks each, mft_halo.cuh) and reads them from there; a group without a list
// gathers directly.  Both read the same records in the same order: the same sums.
// Bound by latency and issue of the packed FP32 products; the row's first weights are requested
// before the staging, whose wait then covers theirs: 262k nodes 100 us -> 92.5 between events.
// Where every group is staged they are also requested before the flux kernel has ended (pdl_wait
// stands before the first read of its records, and of anything else that is not constant):
// rhs! 133.1 -> 129.9 us.  Direct reads take the read-only path through L1, which the records may
// only do once they are complete, so a cloud with an unstaged group gets a plain launch (past L1
// and as a dependent, 64^3 nodes: 378 us against 253 with 60 entries, 1721 of 2048 groups staged).
// With xy, yy and zz in chunks of their own as they are multiplied (112 bytes, no moves) rhs! took
// 133 us against 125, 157 / 141 with 35 entries, 253 / 215 with 60, 208 / 191 with none staged.
__global__ void __launch_bounds__(kHaloRows, 2) k_fwd3_dw(FwdArgs a) {
  const int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
  const float4* F4 = reinterpret_cast<const float4*>(a.Fdw);
  extern __shared__ float4 hsm3[];
  const bool live = r < a.n;
  const int64_t i = live ? ell_node(a.ell, r) : 0;
  const int64_t base = live ? a.ell.slice_off[r >> 5] + (r & 31) : 0;
  const int len = live ? a.ell.row_len[r] : 0;
  struct Streamed {
    int lc;
    float4 wxy;
    float2 wz;
  };
  Streamed ahead[2][4];
  auto load = [&](Streamed& e, int j) {
    e.lc = __ldg(a.ell.lcol + base + j * 32);
    e.wxy = __ldg(a.wxydw + base + j * 32);
    e.wz = __ldg(a.wzdw + base + j * 32);
  };
  if (__ldg(a.ell.halo_off + blockIdx.x + 1) > __ldg(a.ell.halo_off + blockIdx.x))
    pipelined_open<4>(len, ahead, load);
  pdl_wait();
  const bool staged =
      stage_halo<kRec3>(a.ell, hsm3, [&](int k, int64_t c) { return F4 + c * kRec3 + k; });
  if (!live) return;
  const int hs = a.ell.halo_stride;
  Sums3 f;
  f.f04 = f.f12 = f.f3 = dw::zero2();
  f.f3z = dw::zero();
  if (staged) {
    pipelined_run<4>(len, ahead, load, [&](const Streamed& e) {
      float4 q[kRec3];
#pragma unroll
      for (int k = 0; k < kRec3; ++k) q[k] = hsm3[halo_at<kRec3>(k, e.lc, hs)];
      accum3(f, e.wxy, e.wz, q);
    });
  } else {
    const int32_t* __restrict__ col = a.ell.col;
#pragma unroll 2
    for (int j = 0; j < len; ++j) {
      const int64_t p = base + ((int64_t)j << 5);
      const int64_t c = __ldg(col + p);
      const float4 wxy = __ldg(a.wxydw + p);
      const float2 wz = __ldg(a.wzdw + p);
      float4 q[kRec3];
#pragma unroll
      for (int k = 0; k < kRec3; ++k) q[k] = __ldg(F4 + c * kRec3 + k);
      accum3(f, wxy, wz, q);
    }
  }
  double du[5];
  du[0] = -dw::to_double(dw::first(f.f04));
  du[1] = -dw::to_double(dw::first(f.f12));
  du[2] = -dw::to_double(dw::second(f.f12));
  du[3] = -dw::value(dw::add(dw::add(dw::to_pair(dw::first(f.f3)), dw::to_pair(dw::second(f.f3))),
                             dw::to_pair(f.f3z)));
  du[4] = -dw::to_double(dw::second(f.f04));
  finish_node<5>(a.ep, i, du);
}

}  // namespace

void launch_prep_euler3d_dw(int64_t n, double gamma, const double* u, float2* F,
                            cudaStream_t s) {
  if (n <= 0) return;
  const double gm1 = gamma - 1.0;
  const float h = (float)gm1;
  const float2 g2 = make_float2(h, (float)(gm1 - (double)h));
  k_prep_euler3d_dw<<<grid_for(n, 256), 256, 0, s>>>(n, g2, u, reinterpret_cast<float4*>(F));
  MFT_LAUNCH_CHECK();
}

void launch_fwd3_dw(const FwdArgs& a, cudaStream_t s, bool pdl) {
  if (a.n <= 0) return;
  MFT_REQUIRE(a.V == 5 && a.Fdw && a.wxydw && a.wzdw && a.final_epilogue,
              MFT_ERR_STATE, "double-word 3D gather: arguments not set");
  MFT_REQUIRE(a.ell.halo_off && a.ell.halo_rows > 0, MFT_ERR_STATE,
              "double-word 3D gather: row groups not built");
  // one block per row group, six chunks of the longest list in dynamic shared memory
  // (above 48 KB a per-kernel opt-in, made once per device)
  const size_t smem = (size_t)kRec3 * a.ell.halo_stride * sizeof(float4);
  if (smem > 48 * 1024) {
    static std::mutex mu;
    static std::set<int> done;
    int dev = 0;
    MFT_CUDA(cudaGetDevice(&dev));
    std::lock_guard<std::mutex> lock(mu);
    if (done.insert(dev).second)
      MFT_CUDA(cudaFuncSetAttribute(k_fwd3_dw, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                    (int)(kRec3 * kHaloMax * sizeof(float4))));
  }
  const int rows = a.ell.halo_rows;
  launch_k(k_fwd3_dw, grid_for(a.n, rows), rows, smem, s, pdl, a);
  MFT_LAUNCH_CHECK();
}

void launch_flux_euler3d(int64_t n, double gamma, const double* u, double* F, cudaStream_t s) {
  if (n <= 0) return;
  k_flux_euler3d<<<grid_for(n, 256), 256, 0, s>>>(n, gamma, u, F);
  MFT_LAUNCH_CHECK();
}

void launch_fwd3(const FwdArgs& a, cudaStream_t s) {
  if (a.n <= 0) return;
  MFT_REQUIRE(a.w[0] && a.w[1] && a.w[2], MFT_ERR_STATE, "3D gradient operators not set");
  MFT_REQUIRE(a.final_epilogue, MFT_ERR_UNSUPPORTED, "3D gather: final epilogue only");
  const unsigned g = grid_for(a.n, kBlock);
  if (a.V == 5) {
    MFT_REQUIRE(a.F, MFT_ERR_STATE, "3D Euler fluxes not formed");
    k_fwd3_f64<5><<<g, kBlock, 0, s>>>(a);
  } else if (a.V == 1) {
    k_fwd3_f64<1><<<g, kBlock, 0, s>>>(a);
  } else {
    throw Error(MFT_ERR_UNSUPPORTED, "3D gather: 5 (Euler) or 1 (advection) variables");
  }
  MFT_LAUNCH_CHECK();
}

}  // namespace mft
