// Block fixed-point arithmetic for the FP64 stage kernels on the integer pipes.
//
// GB300 issues FP64 at 1/64 of its FP32 and integer rate: measured per SM and clock,
// 1.7 FP64 operations against 59 multiply-accumulates of 32 x 32 -> 64 bits, 64 funnel
// shifts and about 110 simple integer operations.  A stencil sum in FP64 aligns, rounds and
// normalises every term; here the values that enter one sum are aligned once, to the largest
// exponent among them, as 57-bit integers (4 bits more than an FP64 significand), the
// differences are exact integer sums, the products are accumulated in 64-bit integers, and
// only the finished sum is normalised.
//
// Every value, coefficient and product carries an exponent of its own, and only what is
// added is aligned: the error of a sum is a few units of 2^-57 of its largest term, against
// 2^-53 for each FP64 operation.  The components of a field, the coefficients of a point and
// the axes of an operator may differ by any power of two.  A result depends on the values of
// the point's own stencil alone, so it does not change with the tiling, the launch shape or a
// decomposition of the grid.
#pragma once

#include <cstdint>

namespace sw4g {

typedef long long i64;

constexpr int kSplit = 26;  // low limb of values and weights
constexpr int kMask = (1 << kSplit) - 1;

// x >> d, arithmetic, for any d >= 0 (PTX clamps the amount)
__device__ __forceinline__ i64 sar(i64 x, int d)
{
   i64 r;
   asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(d));
   return r;
}

// x / 2^d rounded to nearest, halves to even, for d >= 0.  Sums are rounded without a
// bias, which a time loop would accumulate: a constant in every step's acceleration grows
// as the square of the step count, and the amounts are small, so halves are common.
// |x| + 2^61 must fit; an amount above 62 leaves 0 or +-1.
struct Round {
   int d, some;
   i64 half;  // 2^(d-1) - 1, and 0 for d = 0
   __device__ __forceinline__ explicit Round(int amount)
   {
      d = min(amount, 62);
      some = min(amount, 1);
      asm("shr.u64 %0, %1, %2;" : "=l"(half) : "l"(-1LL), "r"(65 - d));
   }
   __device__ __forceinline__ i64 operator()(i64 x) const
   {
      return sar(x + half + (i64)((int)sar(x, d) & some), d);
   }
};

// x / 2^d to an integer beside it, the odd one unless it is exact, for any d >= 0: without a
// bias, for fewer instructions than Round takes and an error of up to 1 against 1/2, where
// the integers have bits to spare.
__device__ __forceinline__ i64 to_odd(i64 x, int d)
{
   const i64 y = sar(x, d);
   i64 z;
   asm("shl.b64 %0, %1, %2;" : "=l"(z) : "l"(y), "r"(d));
   return y | (i64)(z != x);
}

__device__ __forceinline__ i64 madw(int a, int b, i64 c)
{
   i64 r;
   asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
   return r;
}

__device__ __forceinline__ int max4(int a, int b, int c, int d) { return max(max(a, b), max(c, d)); }

// An FP64 value as an integer m with value m * 2^(e - 1079), |m| < 2^57, exact: its 53 bits
// and four below; e is its biased exponent (at least 1, the subnormals').  True if it is not
// finite; it counts as less than the smallest normal number.
__device__ __forceinline__ bool to_fixed(double v, i64& m, int& e)
{
   const int hi = __double2hiint(v), eb = (hi >> 20) & 0x7ff;
   const unsigned mh = (unsigned)(hi & 0xfffff) | (unsigned)(min(eb, 1) << 20);
   const i64 t = (i64)(((unsigned long long)mh << 32) | (unsigned)__double2loint(v)) << 4;
   const i64 s = (i64)(hi >> 31);
   m = (t ^ s) - s;
   e = eb == 2047 ? 1 : max(eb, 1);
   return eb == 2047;
}

// An integer with an exponent of its own
struct Num {
   i64 m;
   int e;
};

constexpr int kNone = -20000;  // below any exponent, in 16 bits: that of zero

// How far |m| < 2^(top + 1) is from reaching bit `top`, from its upper word alone: less than
// the distance where |m| < 2^32
template <int top>
__device__ __forceinline__ int headroom(i64 m)
{
   const int hi = (int)(m >> 32);
   return max(__clz(hi ^ (hi >> 31)) - (63 - top), 0);
}

// m * 2^e with the leading bit of m brought to bit 60 (left at bit 61 if it is there): what is
// formed from a difference keeps its accuracy, however small it is against its terms.  Below
// 2^32 the exponent is lowered by kBelow on top, right for zero, and tiny tells of a difference
// that is not zero, for which `rest` finishes.
constexpr int kBelow = 16384;
__device__ __forceinline__ Num normal(i64 m, int e, bool& tiny)
{
   const int n = headroom<60>(m);
   const bool below = n == 29;  // the upper word is sign alone
   tiny = tiny || (below && m != 0);
   return Num{m << n, e - n - (below ? kBelow : 0)};
}
__device__ __forceinline__ void rest(Num& d)
{
   const int n = max(__clzll(d.m ^ (d.m >> 63)) - 3, 0), e = d.e < -kBelow / 2 ? d.e + kBelow : d.e;
   d = Num{d.m << n, d.m == 0 ? kNone : e - n};
}

// 8 (fp1 - fm1) + (fm2 - fp2)
__device__ __forceinline__ i64 d1i(i64 fm2, i64 fm1, i64 fp1, i64 fp2)
{
   return ((fp1 - fm1) << 3) + (fm2 - fp2);
}

// The difference d1i(x) of values |x| < 2^57 aligned to the exponent e of the largest
__device__ __forceinline__ Num difference(i64 x0, i64 x1, i64 x2, i64 x3, int e0, int e1, int e2, int e3, int e, bool& tiny)
{
   return normal(d1i(sar(x0, e - e0), sar(x1, e - e1), sar(x2, e - e2), sar(x3, e - e3)), e, tiny);
}

// x * C / 2^57 for |x| < 2^62 and a coefficient |C| < 2^57 held as c.x = C >> 26,
// c.y = (C & kMask) << 5; the product of the two low limbs (below 2^-60 of the largest
// result) is dropped, the rest rounded.
__device__ __forceinline__ i64 mulc(i64 x, int2 c)
{
   const int xh = (int)(x >> 31), xl = (int)x & 0x7fffffff;
   const i64 cross = madw(xl, c.x, madw(xh, c.y, 1LL << 30));
   return madw(xh, c.x, cross >> 31);
}

// x * f / 2^e for |x| < 2^62 and any finite factor f, with its full relative precision,
// rounded to nearest; f / 2^e is below 1 in magnitude.  TINY: f may lie below the normal range
// (asked for where the factors are a caller's; the time loop's profiles end at 1e-4, and the test
// costs its stages 8 %).
template <bool TINY>
struct Scale {
   int hi, lo, e;
   bool neg;
   __device__ __forceinline__ explicit Scale(double f)
   {
      const int h = __double2hiint(f), eb = (h >> 20) & 0x7ff;
      i64 c = (i64)(((unsigned long long)((h & 0xfffff) | 0x100000) << 32) | (unsigned)__double2loint(f)) << 4;
      e = eb - 1022;
      if (!TINY) {
         if (eb == 0) c = 0, e = -5000;
      } else if (eb == 0) {  // zero and below the normal range
         c = (__double_as_longlong(f) & 0xfffffffffffffLL) << 4;
         const int n = c == 0 ? 0 : __clzll(c) - 7;
         c <<= n;
         e = c == 0 ? -5000 : -1021 - n;
      }
      hi = (int)(c >> kSplit);
      lo = (int)(c & kMask) << 5;
      neg = h < 0;
   }
   __device__ __forceinline__ i64 operator()(i64 x) const
   {
      const int xh = (int)(x >> 31), xl = (int)x & 0x7fffffff;
      const i64 cross = madw(xl, hi, madw(xh, lo, (madw(xl, lo, 1LL << 30) >> 31) + (1LL << 30)));
      const i64 r = madw(xh, hi, cross >> 31);
      return neg ? -r : r;
   }
};

__device__ __forceinline__ bool is_one(double x) { return __double_as_longlong(x) == 0x3ff0000000000000LL; }

// times a stretching factor
template <bool TINY>
__device__ __forceinline__ Num stretched(const Num& d, double s)
{
   const Scale<TINY> f(s);
   return Num{f(d.m), d.e + f.e};
}

// Products of one point for one outer direction of the mixed terms, value m * 2^(e - 1078):
// la times the sum of the differences s0, s1 with stretching factors f0, f1, and mu times m0
// and m1.  A coefficient is C * 2^(e - 57), its limbs as mulc takes them.
struct Triple {
   Num la, m0, m1;
};

__device__ __forceinline__ Num times(const Num& d, int2 c, int e) { return Num{mulc(d.m, c), d.e + e - 1}; }

template <bool TINY>
__device__ __forceinline__ Triple products(Num s0, Num s1, const Num& m0, const Num& m1, int2 mu, int emu, int2 la, int ela,
                                           double f0, double f1)
{
   if (!is_one(f0)) s0 = stretched<TINY>(s0, f0);
   if (!is_one(f1)) s1 = stretched<TINY>(s1, f1);
   const int es = max(s0.e, s1.e);
   Triple t;
   t.la = Num{mulc(sar(s0.m, es - s0.e + 1) + sar(s1.m, es - s1.e + 1), la), es + ela};
   t.m0 = times(m0, mu, emu);
   t.m1 = times(m1, mu, emu);
   return t;
}

// The outer difference of four products, e the largest of their exponents, value
// m * 2^(e - 1074).  Equal products leave zero, which has no exponent: a component that they do
// not reach keeps its own.
__device__ __forceinline__ Num outer(i64 g0, i64 g1, i64 g2, i64 g3, int e0, int e1, int e2, int e3, int e)
{
   const i64 d = d1i(sar(g0, e - e0 + 4), sar(g1, e - e1 + 4), sar(g2, e - e2 + 4), sar(g3, e - e3 + 4));
   return Num{d, d == 0 ? kNone : e};
}

// p * 2^e as FP64, rounded once, above the range infinite.  Below the normal range it comes
// times 2^kLow, with low set, so that it keeps its digits for the product that follows, whose
// other factor brings 2^-kLow.
constexpr int kLow = 200;
__device__ __forceinline__ double from_block(i64 p, int e, bool& low)
{
   const double r = __ll2double_rn(p);
   int hi = __double2hiint(r), lo = __double2loint(r);
   const int eb = (hi >> 20) & 0x7ff;
   low = eb + e <= 0;
   e += low ? kLow : 0;
   const int n = eb == 0 ? 0 : eb + e;
   hi += (int)((unsigned)e << 20);
   if (n <= 0) hi = lo = 0;
   if (n >= 2047) {
      hi = p < 0 ? 0xfff00000 : 0x7ff00000;
      lo = 0;
   }
   return __hiloint2double(hi, lo);
}

// c * 2^-kLow for a factor c >= 0, by its exponent (0 below 2^(kLow - 1022))
__device__ __forceinline__ double lowered(double c)
{
   const int hi = __double2hiint(c) - (kLow << 20);
   return hi < (1 << 20) ? 0.0 : __hiloint2double(hi, __double2loint(c));
}

}  // namespace sw4g
