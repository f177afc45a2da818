// Double-word FP32 arithmetic ("double-float": a value is an unevaluated sum h + l of two
// floats with |l| <= ulp(h) / 2, 48 significand bits) for the FP64 form's gathers.
//
// On this part an FP64 fused multiply-add issues at 1/74 of the FP32 rate, and the FP64
// gathers are bound by it.  The sums of products those gathers form are evaluated here
// on the FP32 pipe with error-free transformations instead:
//   * the running sum of the rounded products of the high parts, t = RN(s + p), p = RN(a_h b_h);
//   * the product's rounding error and the larger part of the sum's in one FMA, the smaller part
//     by the rest of Knuth's TwoSum (branch-free; Dekker 1971 for the product's error);
//   * the cross terms a_h b_l + a_l b_h folded in (a_l b_l < 2^-48 |ab| is dropped);
//   * these corrections in a float carry: ten operations a product (fma_acc).
// This is the compensated dot product "Dot2" of Ogita, Rump and Oishi (SIAM J. Sci.
// Comput. 26(6), 2005) on double-word inputs (Joldes, Muller and Popescu, ACM TOMS
// 44(2), 2017), but for the corrections' own rounding: a product's correction is of size
// u |t| (u = 2^-24) and takes four roundings, so 4 u^2 |t| beside the inputs' split error
// (3 u^2 |a b|), and the carry's additions, at most gamma_n^2 sum |a_i b_i| with
// gamma_n = n u / (1 - n u) when every rounding error has the same sign and its largest size:
// with the partial sums |t| <= sum |a_i b_i|, n = 35, together 4.9e-12 of that condition scale;
// errors of mixed sign give about sqrt(n) u^2 of it (~2e-14).  (With the product's error formed
// exactly, twelve operations, the errors of du measure the same within sampling: rms 0..2 % less,
// maxima as often larger as smaller.)  The result is rounded once to FP64.  Every operation is an
// explicitly rounded intrinsic, so no contraction or reassociation by the compiler can break
// the error-free steps.
#pragma once

#include <cuda_runtime.h>

#include "mft_fpbits.h"

namespace mft {
namespace dw {

using fpconv::d2f;
using fpconv::f2d;

// x -> (h, l): h = RN32(x), l = RN32(x - h) (x - h is exact in FP64).
static __device__ __forceinline__ float2 split(double x) { return fpconv::split(x); }

static __device__ __forceinline__ double value(float2 a) {
  return __dadd_rn(f2d(a.x), f2d(a.y));
}

// Running sum of products: s is the float running sum, c the float carry of every
// rounding error (products and sums).
struct Acc {
  float s, c;
};

static __device__ __forceinline__ Acc zero() { return Acc{0.f, 0.f}; }

// acc += a * b (a, b double-word), 10 operations.  With p = RN(a_h b_h), t = RN(s + p) and
// b' = RN(t - s) (Knuth's TwoSum; nb = -b'), the sum's rounding error is (s - (t - b')) +
// (p - b') exactly and the product's a_h b_h - p, so fma(a_h, b_h, nb) = RN(a_h b_h - b') is
// the product's error and the second part of the sum's in one operation.
static __device__ __forceinline__ void fma_acc(Acc& acc, float2 a, float2 b) {
  const float p = __fmul_rn(a.x, b.x);
  const float t = __fadd_rn(acc.s, p);
  const float nb = __fsub_rn(acc.s, t);
  float e = fmaf(a.x, b.x, nb);
  e = fmaf(a.x, b.y, e);
  e = fmaf(a.y, b.x, e);
  e = __fadd_rn(e, __fsub_rn(acc.s, __fadd_rn(t, nb)));
  acc.s = t;
  acc.c = __fadd_rn(acc.c, e);
}

// The accumulated value rounded once to FP64.
static __device__ __forceinline__ double to_double(const Acc& a) {
  return __dadd_rn(f2d(a.s), f2d(a.c));
}

// The accumulated value as a normalised double-word pair (TwoSum of s and c).
static __device__ __forceinline__ float2 to_pair(const Acc& a) {
  const float t = __fadd_rn(a.s, a.c);
  const float bp = __fsub_rn(t, a.s);
  const float err = __fadd_rn(__fsub_rn(a.s, __fsub_rn(t, bp)), __fsub_rn(a.c, bp));
  return make_float2(t, err);
}

// a * b for a double-word a and b, normalised (|e| <= ulp(p), so Fast2Sum is exact).
static __device__ __forceinline__ float2 mul(float2 a, float2 b) {
  const float p = __fmul_rn(a.x, b.x);
  float e = fmaf(a.x, b.x, -p);
  e = fmaf(a.x, b.y, e);
  e = fmaf(a.y, b.x, e);
  const float t = __fadd_rn(p, e);
  return make_float2(t, __fsub_rn(e, __fsub_rn(t, p)));
}

// a + b for double-word a and b: TwoSum of the high parts, the low parts added to its
// error, renormalised (absolute error about 2 u^2 (|a| + |b|)).
static __device__ __forceinline__ float2 add(float2 a, float2 b) {
  const float s = __fadd_rn(a.x, b.x);
  const float bb = __fsub_rn(s, a.x);
  float e = __fadd_rn(__fsub_rn(a.x, __fsub_rn(s, bb)), __fsub_rn(b.x, bb));
  e = __fadd_rn(e, __fadd_rn(a.y, b.y));
  const float t = __fadd_rn(s, e);
  return make_float2(t, __fsub_rn(e, __fsub_rn(t, s)));
}

static __device__ __forceinline__ float2 neg(float2 a) { return make_float2(-a.x, -a.y); }

// a * 2^k for a power of two c = 2^k (exact)
static __device__ __forceinline__ float2 scale2(float2 a, float c) {
  return make_float2(__fmul_rn(a.x, c), __fmul_rn(a.y, c));
}

// 1 / a for a double-word a: the correctly rounded FP32 reciprocal y of a_h and one
// Newton step y + y (1 - a y) with 1 - a y formed exactly up to the low-order product
// (relative error about 2 u^2).
static __device__ __forceinline__ float2 recip(float2 a) {
  const float y = __frcp_rn(a.x);
  const float p = __fmul_rn(a.x, y);
  float ep = fmaf(a.x, y, -p);
  ep = fmaf(a.y, y, ep);
  const float d = __fsub_rn(__fsub_rn(1.0f, p), ep);
  const float c = __fmul_rn(y, d);
  const float t = __fadd_rn(y, c);
  return make_float2(t, __fsub_rn(c, __fsub_rn(t, y)));
}

// The Euler flux-Jacobian-transpose product ub = J_Fx(u)^T gx + J_Fy(u)^T gy (as
// euler_flux_vjp in FP64) in double-word arithmetic: u as pairs, gx / gy as pairs,
// gm1 = gamma - 1 as a pair; each operation is accurate to about 2 u^2 of its operands.
static __device__ __forceinline__ void euler_flux_vjp(float2 gm1, const float2* u,
                                                      const float2* gx, const float2* gy,
                                                      float2* ub) {
  const float2 rho = u[0], m1 = u[1], m2 = u[2], en = u[3];
  const float2 ri = recip(rho);
  const float2 v1 = mul(m1, ri), v2 = mul(m2, ri);
  const float2 p = mul(gm1, add(en, neg(scale2(add(mul(m1, v1), mul(m2, v2)), 0.5f))));
  const float2 ep = add(en, p);
  const float2 pb = add(add(gx[1], mul(gx[3], v1)), add(gy[2], mul(gy[3], v2)));
  const float2 hp = scale2(mul(gm1, pb), 0.5f);
  const float2 v1b = add(add(mul(gx[1], m1), mul(gx[3], ep)), add(mul(gy[1], m2), neg(mul(hp, m1))));
  const float2 v2b = add(add(mul(gx[2], m1), mul(gy[2], m2)), add(mul(gy[3], ep), neg(mul(hp, m2))));
  ub[0] = neg(mul(add(mul(v1b, v1), mul(v2b, v2)), ri));
  ub[1] = add(add(add(gx[0], mul(gx[1], v1)), add(mul(gx[2], v2), neg(mul(hp, v1)))), mul(v1b, ri));
  ub[2] = add(add(add(gy[0], mul(gy[1], v1)), add(mul(gy[2], v2), neg(mul(hp, v2)))), mul(v2b, ri));
  ub[3] = add(add(mul(gx[3], v1), mul(gy[3], v2)), mul(gm1, pb));
}

// ---------------------------------------------------------------- two at a time
// The same operations on two double-word values at once with the packed FP32 instructions
// (add / sub / mul / fma .f32x2: two roundings per instruction, each as the scalar one).
// They run at the scalar instructions' rate per operation (measured 16.5 T packed against
// 28-39 T scalar instructions per second and GPU) but take half the issue slots, which the
// gathers need for their loads.
typedef unsigned long long f32x2;

static __device__ __forceinline__ f32x2 pk(float x, float y) {
  f32x2 r;
  asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(x), "f"(y));
  return r;
}
static __device__ __forceinline__ float2 unpk(f32x2 v) {
  float2 r;
  asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(v));
  return r;
}
static __device__ __forceinline__ f32x2 add2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
static __device__ __forceinline__ f32x2 sub2(f32x2 a, f32x2 b) {
  f32x2 r;
  asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
  return r;
}
static __device__ __forceinline__ f32x2 fma2(f32x2 a, f32x2 b, f32x2 c) {
  f32x2 r;
  asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
  return r;
}

// RN(a b), as the multiply-add a b + (-0) with the -0 read from constant memory: the compiler
// contracts a packed multiplication and the packed addition that reads it into one multiply-add
// (also with .rn on both, with a literal -0 and without -fmad; the scalar instructions keep
// their .rn), which would break the error-free steps.
static __constant__ unsigned long long kNegZero2 = 0x8000000080000000ull;
static __device__ __forceinline__ f32x2 mul2(f32x2 a, f32x2 b) { return fma2(a, b, kNegZero2); }

// Two double-word values a, b: (a_h, b_h) and (a_l, b_l).  In memory the 16-byte chunk
// (a_h, b_h, a_l, b_l), so that a chunk's load leaves them in register pairs.
struct DW2 {
  f32x2 h, l;
};
static __device__ __forceinline__ DW2 pair2(float4 c) { return DW2{pk(c.x, c.y), pk(c.z, c.w)}; }
static __device__ __forceinline__ DW2 pair2(float2 a, float2 b) {
  return DW2{pk(a.x, b.x), pk(a.y, b.y)};
}
static __device__ __forceinline__ DW2 both(float2 a) { return pair2(a, a); }
static __device__ __forceinline__ float4 chunk(float2 a, float2 b) {
  return make_float4(a.x, b.x, a.y, b.y);
}
static __device__ __forceinline__ float4 chunk(DW2 v) {
  const float2 h = unpk(v.h), l = unpk(v.l);
  return make_float4(h.x, h.y, l.x, l.y);
}
static __device__ __forceinline__ float2 chunk_a(float4 c) { return make_float2(c.x, c.z); }
static __device__ __forceinline__ float2 chunk_b(float4 c) { return make_float2(c.y, c.w); }

struct Acc2 {
  f32x2 s, c;
};
static __device__ __forceinline__ Acc2 zero2() { return Acc2{0ull, 0ull}; }
static __device__ __forceinline__ void fma_acc2(Acc2& acc, DW2 a, DW2 b) {
  const f32x2 p = mul2(a.h, b.h);
  const f32x2 t = add2(acc.s, p);
  const f32x2 nb = sub2(acc.s, t);
  f32x2 e = fma2(a.h, b.h, nb);
  e = fma2(a.h, b.l, e);
  e = fma2(a.l, b.h, e);
  e = add2(e, sub2(acc.s, add2(t, nb)));
  acc.s = t;
  acc.c = add2(acc.c, e);
}
static __device__ __forceinline__ Acc first(Acc2 a) { return Acc{unpk(a.s).x, unpk(a.c).x}; }
static __device__ __forceinline__ Acc second(Acc2 a) { return Acc{unpk(a.s).y, unpk(a.c).y}; }

static __device__ __forceinline__ DW2 to_pair2(Acc2 a) {
  const f32x2 t = add2(a.s, a.c);
  const f32x2 bp = sub2(t, a.s);
  return DW2{t, add2(sub2(a.s, sub2(t, bp)), sub2(a.c, bp))};
}
// The sum of two accumulated values rounded to FP64: the pairs added in double-word
// arithmetic (add, about 2 u^2 of their sum), one FP64 addition.
static __device__ __forceinline__ double sum_double(Acc a, Acc b) {
  return value(add(to_pair(a), to_pair(b)));
}

static __device__ __forceinline__ DW2 mul(DW2 a, DW2 b) {
  const f32x2 p = mul2(a.h, b.h);
  f32x2 e = fma2(a.h, b.h, sub2(kNegZero2, p));  // -0 - p = -p
  e = fma2(a.h, b.l, e);
  e = fma2(a.l, b.h, e);
  const f32x2 t = add2(p, e);
  return DW2{t, sub2(e, sub2(t, p))};
}

}  // namespace dw
}  // namespace mft
