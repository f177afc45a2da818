// Exact float <-> double conversions on the integer pipe, for the double-word arithmetic.
//
// On this part the conversions between FP32 and FP64 run on the FP64 pipe, which issues at
// 1/74 of the FP32 rate.  Splitting an FP64 value into a double-word pair takes three of
// them and one subtraction; the staged forward gather that forms its neighbours' flux
// records splits four state values per record at the start of every block, where the
// block's FP64 work is not hidden behind other warps; the FP32-apply form converts its
// partial du to FP64 and every new state to its FP32 shadow in the stage epilogues.  Here
// the conversions are formed from the IEEE-754 bit fields with 32-bit integer operations
// (fpconv::f2d / d2f below, the same bits as the hardware conversions):
//   * float -> double is exact: the exponent is rebiased (127 -> 1023) and the 23-bit
//     significand moved to the top of the 52-bit one;
//   * double -> float rounds to nearest, ties to even: the 52-bit significand is cut to
//     23 bits, and one is added to the truncated bit pattern when the 29 dropped bits
//     exceed half an ulp, or equal it with the kept pattern odd; a carry out of the
//     significand moves into the exponent, and from the largest finite exponent into the
//     infinity pattern, which is the IEEE result in both cases.
// Each function handles the operands whose result is a normal number (and signed zeros)
// and returns false otherwise (subnormal results, infinities, NaN); the caller then uses
// the hardware conversion, so every input gets the IEEE result.  Plain C++ on 32-bit
// words: the same code compiles for the host, where a test checks it against the host's
// own conversions.
#pragma once

#include <stdint.h>

#if defined(__CUDACC__)
#define MFT_FPBITS_FN __host__ __device__ __forceinline__
#else
#define MFT_FPBITS_FN static inline
#endif

namespace mft {
namespace fpbits {

// b: the bits of a float.  On success (*hi, *lo) are the high and low words of the
// double with the same value.
MFT_FPBITS_FN bool f2d_words(uint32_t b, uint32_t* hi, uint32_t* lo) {
  const uint32_t e = (b >> 23) & 0xFFu;
  if (e - 1u < 254u) {  // normal
    *hi = (b & 0x80000000u) | ((e + 896u) << 20) | ((b >> 3) & 0xFFFFFu);
    *lo = b << 29;
    return true;
  }
  if ((b << 1) == 0u) {  // +0 or -0
    *hi = b;
    *lo = 0u;
    return true;
  }
  return false;  // subnormal, infinity, NaN
}

// (hi, lo): the words of a double.  On success *out is the bits of the float nearest to
// it (ties to even).
MFT_FPBITS_FN bool d2f_bits(uint32_t hi, uint32_t lo, uint32_t* out) {
  const uint32_t e = (hi >> 20) & 0x7FFu;
  if (e - 897u < 254u) {  // the float exponent e - 896 is normal (1 .. 254)
    uint32_t r = ((e - 896u) << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29);
    const uint32_t rem = lo & 0x1FFFFFFFu;
    const uint32_t half = 0x10000000u;
    r += (rem > half || (rem == half && (r & 1u))) ? 1u : 0u;
    *out = r | (hi & 0x80000000u);
    return true;
  }
  if (((hi << 1) | lo) == 0u) {  // +0 or -0
    *out = hi;
    return true;
  }
  return false;  // below the normal floats, above them, infinity, NaN
}

// (hi, lo): the words of a double x.  On success *h is the bits of RN32(x) and
// x - RN32(x) = *rem * 2^k exactly, |*rem| <= 2^28, with *scale the bits of the float 2^k; then
// RN32(x - RN32(x)) = (float)*rem * 2^k (the conversion rounds, the product is exact).
// Declines where that product could be subnormal, RN32(x) is not a normal float, or x is zero.
MFT_FPBITS_FN bool split_words(uint32_t hi, uint32_t lo, uint32_t* h, int32_t* rem,
                               uint32_t* scale) {
  const uint32_t e = (hi >> 20) & 0x7FFu;
  if (e - 949u >= 201u) return false;  // 2^-74 <= |x| < 2^127
  uint32_t r = ((e - 896u) << 23) | ((hi & 0xFFFFFu) << 3) | (lo >> 29);
  const uint32_t cut = lo & 0x1FFFFFFFu, half = 0x10000000u;
  const uint32_t up = (cut > half || (cut == half && (r & 1u))) ? 1u : 0u;
  r += up;
  const int32_t d = (int32_t)cut - (up ? 0x20000000 : 0);
  *h = r | (hi & 0x80000000u);
  *rem = (hi & 0x80000000u) ? -d : d;
  *scale = (e - 948u) << 23;  // 2^(e - 1075)
  return true;
}

// ---------------------------------------------------------------- order keys
// The IEEE pattern b of a double as an unsigned integer that orders like the value (NaN beyond
// the infinities on its sign's side), and back; |x| as a pattern.
MFT_FPBITS_FN uint64_t order_bits(uint64_t b) { return b ^ ((b >> 63) ? ~0ull : 1ull << 63); }
MFT_FPBITS_FN uint64_t order_back(uint64_t k) { return k ^ ((k >> 63) ? 1ull << 63 : ~0ull); }
MFT_FPBITS_FN uint64_t abs_bits(uint64_t b) { return b & 0x7FFFFFFFFFFFFFFFull; }

// The lowest and highest order keys of a set start as kLowest, 0 (lo > hi: an empty set).
// Largest pattern of |x - m| over a set whose values lie between its extremes: the rounded
// difference is monotonic in x, so that of an end; 0, the smallest, for an empty set.
// diff(b): the pattern of (value of pattern b) - m.
constexpr uint64_t kLowest = ~0ull;
template <typename Diff>
MFT_FPBITS_FN uint64_t extreme_abs(uint64_t lo, uint64_t hi, Diff diff) {
  if (lo > hi) return 0;
  const uint64_t a = abs_bits(diff(order_back(lo))), b = abs_bits(diff(order_back(hi)));
  return a > b ? a : b;
}

}  // namespace fpbits

#if defined(__CUDACC__)
namespace fpconv {
// (double)f, exact, on the integer pipe where the result is normal or zero.
static __device__ __forceinline__ double f2d(float f) {
  uint32_t hi, lo;
  if (fpbits::f2d_words(__float_as_uint(f), &hi, &lo)) return __hiloint2double((int)hi, (int)lo);
  return (double)f;
}
// RN32(x), on the integer pipe where the result is a normal float or zero.
static __device__ __forceinline__ float d2f(double x) {
  uint32_t r;
  if (fpbits::d2f_bits((uint32_t)__double2hiint(x), (uint32_t)__double2loint(x), &r))
    return __uint_as_float(r);
  return __double2float_rn(x);
}
// x -> (h, l), h = RN32(x), l = RN32(x - h), without the FP64 pipe in the range split_words
// takes.
static __device__ __forceinline__ float2 split(double x) {
  uint32_t h, scale;
  int32_t rem;
  if (fpbits::split_words((uint32_t)__double2hiint(x), (uint32_t)__double2loint(x), &h, &rem,
                          &scale))
    return make_float2(__uint_as_float(h),
                       __fmul_rn(__int2float_rn(rem), __uint_as_float(scale)));
  const float hf = d2f(x);
  return make_float2(hf, d2f(__dsub_rn(x, f2d(hf))));
}
}  // namespace fpconv
#endif
}  // namespace mft

#undef MFT_FPBITS_FN
