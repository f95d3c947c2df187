// Double-float ("float-float") storage of the solution levels in the mixed form.
//
// A value is the unevaluated sum hi + lo of two FP32 numbers with |lo| <= ulp(hi)/2,
// i.e. 48 significant bits.  The time-level accumulation
//   u^{n+1} = 2u^n - u^{n-1} + dt^2/rho (Lu + F)
// is carried out in this format with FP32 error-free transformations (Knuth's
// TwoSum and Dekker's FastTwoSum), so the accumulation keeps FP64-class precision
// while the stencil runs in FP32.  Components of a 3-component level are stored
// component-major: hi[c*npts + p], lo[c*npts + p] (lo = hi + 3*npts).
#pragma once

namespace sw4g {

// s + e == a + b exactly (Knuth TwoSum, 6 FP32 operations, no branch).
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e)
{
   s = __fadd_rn(a, b);
   const float bb = __fsub_rn(s, a);
   e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// s + e == a + b exactly when |a| >= |b| (Dekker FastTwoSum).
__device__ __forceinline__ void fast_two_sum(float a, float b, float& s, float& e)
{
   s = __fadd_rn(a, b);
   e = __fsub_rn(b, __fsub_rn(s, a));
}

// The conversions below work on the bit patterns: GB300 converts between FP32 and FP64 on
// the FP64 pipe (2 per clock and SM), where splitting a level took four operations a value
// and widening three, 0.74 and 0.55 ms for a level of 320^3 whose bytes take 0.24 ms.  Values outside
// the ranges that the integer forms cover (subnormal or overflowing halves, not finite) take
// the conversion instructions.

// (double)x
__device__ __forceinline__ double f64_of(float x)
{
   const unsigned b = __float_as_uint(x), e = (b >> 23) & 0xff;
   if (e - 1 < 254) return __hiloint2double((int)((b & 0x80000000u) | ((e + 896) << 20) | ((b >> 3) & 0xfffff)), (int)(b << 29));
   if ((b << 1) == 0) return __hiloint2double((int)b, 0);
   return (double)x;
}

// FP64 value -> (hi, lo), each rounded to nearest even.
__device__ __forceinline__ void df_split(double v, float& h, float& l)
{
   const unsigned hi = (unsigned)__double2hiint(v), lo = (unsigned)__double2loint(v), s = hi & 0x80000000u;
   const unsigned e = (hi >> 20) & 0x7ff;
   if (e - 950 <= 198) {
      // hi: the upper 23 bits of the significand, rounded; lo: the signed rest r * 2^(e-1075)
      const unsigned t = ((hi & 0xfffff) << 3) | (lo >> 29), rest = lo & 0x1fffffff;
      const unsigned up = rest > 0x10000000u || (rest == 0x10000000u && (t & 1)) ? 1 : 0;
      h = __uint_as_float(s | ((((e - 896) << 23) | t) + up));
      const int r = (int)rest - (int)(up << 29);
      l = (float)(s ? -r : r) * __uint_as_float((e - 948) << 23);
   } else if (((hi << 1) | lo) == 0) {
      h = __uint_as_float(s);
      l = 0.f;
   } else {
      h = __double2float_rn(v);
      l = __double2float_rn(v - (double)h);
   }
}

__device__ __forceinline__ double df_value(float h, float l) { return f64_of(h) + f64_of(l); }

}  // namespace sw4g
