// Shared-memory staging of a row group's neighbour records (the halos of EllView): used by
// the staged variants of the gathers.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

#include "mft_internal.cuh"

namespace mft {
namespace {

// 16-byte asynchronous copy global -> shared (bypasses registers), and the wait for all
// of this thread's copies.
static __device__ __forceinline__ void cp_async16(float4* smem, const float4* gmem) {
  const unsigned sa = (unsigned)__cvta_generic_to_shared(smem);
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gmem) : "memory");
}
static __device__ __forceinline__ void cp_async_wait_all() {
  asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// L2 eviction-priority hints (createpolicy + .L2::cache_hint): evict_first for the streamed
// operator arrays, read once per launch, and evict_last for the intermediates a gather
// writes for the next one (t, q, the partial du), so that the stream does not push the
// intermediates out of L2 before they are read back.
static __device__ __forceinline__ uint64_t l2_evict_first() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
static __device__ __forceinline__ uint64_t l2_evict_last() {
  uint64_t p;
  asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;\n" : "=l"(p));
  return p;
}
static __device__ __forceinline__ float2 ldg_hint(const float2* ptr, uint64_t pol) {
  float2 v;
  asm("ld.global.nc.L2::cache_hint.v2.f32 {%0, %1}, [%2], %3;\n"
      : "=f"(v.x), "=f"(v.y)
      : "l"(ptr), "l"(pol));
  return v;
}
static __device__ __forceinline__ float4 ldg_hint(const float4* ptr, uint64_t pol) {
  float4 v;
  asm("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;\n"
      : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w)
      : "l"(ptr), "l"(pol));
  return v;
}
static __device__ __forceinline__ int ldg_hint(const uint16_t* ptr, uint64_t pol) {
  unsigned short v;
  asm("ld.global.nc.L2::cache_hint.u16 %0, [%1], %2;\n" : "=h"(v) : "l"(ptr), "l"(pol));
  return (int)v;
}
static __device__ __forceinline__ void st_hint(float4* ptr, float4 v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.v4.f32 [%0], {%1, %2, %3, %4}, %5;\n"
               ::"l"(ptr), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w), "l"(pol)
               : "memory");
}
static __device__ __forceinline__ void st_hint(double2* ptr, double2 v, uint64_t pol) {
  asm volatile("st.global.L2::cache_hint.v2.f64 [%0], {%1, %2}, %3;\n"
               ::"l"(ptr), "d"(v.x), "d"(v.y), "l"(pol)
               : "memory");
}

// Shared-memory place (in 16-byte chunks) of chunk k of list entry q, NCH chunks per record
// and hs the longest list: record-major in runs of an odd number of chunks (an odd count as it
// is; 3 + 3 for six, 3 + 1 for four, 1 + 1 for two), so that one multiplication addresses a run and its other
// chunks are immediate offsets, while lanes reading one chunk of different records still spread
// over the bank groups by q mod 8 (an odd stride permutes them).
template <int NCH>
static __device__ __forceinline__ int halo_at(int k, int q, int hs) {
  constexpr int A = NCH % 2 ? NCH : NCH == 6 || NCH == 4 ? 3 : 1, B = NCH > A ? NCH - A : 1;
  return k < A ? q * A + k : hs * A + q * B + (k - A);
}

// Stages the neighbour records of this block's row group (the group's halo list) into
// shared memory: NCH 16-byte chunks per record, chunk k of list entry q at
// sm[halo_at<NCH>(k, q, ell.halo_stride)].  chunk(k, c) is the address of chunk k of node c's
// record.  Consecutive threads copy consecutive chunks of one record, so each record
// arrives in whole sectors.  Returns false (nothing staged) when the group has no list.
// Every thread of the block must call it (it ends with a block barrier); the block is one
// group (blockDim.x = ell.halo_rows).
template <int NCH, typename Chunk>
__device__ __forceinline__ bool stage_halo(const EllView& ell, float4* sm, Chunk chunk) {
  const int h0 = __ldg(ell.halo_off + blockIdx.x);
  const int nh = __ldg(ell.halo_off + blockIdx.x + 1) - h0;
  if (nh <= 0) return false;  // block-uniform
  for (int q = threadIdx.x; q < nh * NCH; q += blockDim.x) {
    const int rec = q / NCH, k = q - rec * NCH;
    cp_async16(sm + halo_at<NCH>(k, rec, ell.halo_stride),
               chunk(k, (int64_t)__ldg(ell.halo_col + h0 + rec)));
  }
  cp_async_wait_all();
  __syncthreads();
  return true;
}

// A staged row's loop with the streamed loads in software pipeline: Entry (positions, weights;
// load(e, j) requests entry j's) in two register groups of G; a group's loads are issued before
// the other group is used, so that a group's arithmetic covers their latency.  The entries are
// used in order, use(e).  pipelined_open requests the first two groups (where the row has them):
// a kernel does that before it stages its neighbours, whose latency then covers theirs.
template <int G, typename Entry, typename Load>
__device__ __forceinline__ void pipelined_get(Entry* x, int g, Load& load) {
#pragma unroll
  for (int k = 0; k < G; ++k) load(x[k], g * G + k);
}
template <int G, typename Entry, typename Load>
__device__ __forceinline__ void pipelined_open(int len, Entry (&e)[2][G], Load& load) {
  const int ng = len / G;
  if (ng > 0) pipelined_get<G>(e[0], 0, load);
  if (ng > 1) pipelined_get<G>(e[1], 1, load);
}
template <int G, typename Entry, typename Load, typename Use>
__device__ __forceinline__ void pipelined_run(int len, Entry (&e)[2][G], Load& load, Use use) {
  const int ng = len / G;
  for (int g = 0; g < ng; g += 2) {
#pragma unroll
    for (int k = 0; k < G; ++k) use(e[0][k]);
    if (g + 2 < ng) pipelined_get<G>(e[0], g + 2, load);
    if (g + 1 < ng) {
#pragma unroll
      for (int k = 0; k < G; ++k) use(e[1][k]);
      if (g + 3 < ng) pipelined_get<G>(e[1], g + 3, load);
    }
  }
  for (int j = ng * G; j < len; ++j) {
    load(e[0][0], j);
    use(e[0][0]);
  }
}
template <int G, typename Entry, typename Load, typename Use>
__device__ __forceinline__ void pipelined_row(int len, Load load, Use use) {
  Entry e[2][G];
  pipelined_open<G>(len, e, load);
  pipelined_run<G>(len, e, load, use);
}

}  // namespace
}  // namespace mft
