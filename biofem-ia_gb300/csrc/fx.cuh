/*
 * Fixed-point arithmetic of the FP64 tangent's contraction K = N^T D N.
 *
 * GB300 issues 2 double-precision multiply-adds per clock and SM but 32 integer
 * ones 32 x 32 + 64 (both measured), so a sum of products whose operands share
 * a known scale is several times cheaper as an exact integer sum.  A value is
 * an integer of up to 62 bits in two signed 32-bit words, v = hi 2^32 + lo.
 *
 *   D   |D| < 2^E per element and Cartesian pair (i, j), E from the largest
 *       entry's exponent: d = D 2^(60-E), |d| <= 2^60
 *   N   regular table: N = k / den exactly up to its own rounding (the
 *       reference's constants are four-decimal numbers, den = 10^4; the exact
 *       ones are multiples of 1/324, den = 31 x 324); others: n = N den 2^48
 *   w = N_a^T D den     (sum k d) / 2^14 = (sum n d) / 2^62: unit 2^(E-46)
 *   K = w N_b den       (sum k w) / 2^15 = (sum n w) / 2^63: unit 2^(E-31), or 2^(E-57.6) of K itself
 *
 * A product with an integer k is two integer multiply-adds and exact, one with
 * a 62-bit n three: the lo.lo product, at most one unit, is left out.  With
 * column sums of |N| up to 2.26 the cross sums stay below 2^62.7 and |w| below
 * 2^60.5, so nothing overflows.
 *
 * What is rounded: D to 2^-61 of the largest entry of its own element's (i, j)
 * group, w and each contribution to half a unit of the ROW's E, 2^-57.8 of it
 * in all.  The sum over the contributions is exact, where a chain of double
 * multiply-adds rounds the running value to 2^-53 at each of them.  One unit a
 * row is coarse for an element far smaller than its neighbours: error over the
 * blocks of soft elements beside one stiff, 24 contributions, regular table,
 * against 2.2e-16 of the double chain: alike 0.8e-16, softer by 2^-4 1.0e-16,
 * 2^-6 2.8e-16, 2^-8 1.1e-15.  So rows stay integer only within kFxSpread and
 * kFxPairSpread (below); beyond, every element's sums keep its own unit and
 * are added as doubles.
 */
#ifndef BIOFEM_FX_CUH
#define BIOFEM_FX_CUH

#include "ff.cuh"

namespace biofem {

struct Fx { int lo, hi; };

constexpr int kFxRaw = 0x7ff;        /* exponent field of an element whose D holds an infinity or NaN (stored as doubles) */

__host__ __device__ __forceinline__ Fx fx_split(long long v)
{
  const int lo = (int)v;
  return {lo, (int)((v - lo) >> 32)};
}

/* the exponent field of |d| (0 for zero and subnormals, kFxRaw for infinities and NaN) */
__host__ __device__ __forceinline__ int fx_exponent(double d) { return (int)((ff_bits64(d) >> 52) & 0x7ff); }

/* d 2^(60-E) rounded to nearest, for an exponent field eb >= d's (E = eb - 1022) */
__host__ __device__ __forceinline__ long long fx_from_double(double d, int eb)
{
  const uint64_t b = ff_bits64(d);
  const int e = (int)((b >> 52) & 0x7ff);
  const long long m = (long long)((b & 0xfffffffffffffull) | 0x10000000000000ull);
  const int k = e - eb + 7;                          /* <= 7 */
  long long v;
  if (k >= 0) v = m << k;
  else if (k > -54) v = (m + (1ll << (-k - 1))) >> -k;
  else v = 0;
  if (e == 0) v = 0;
  return (b >> 63) ? -v : v;
}

/* the double of d 2^(60-E) */
__host__ __device__ __forceinline__ double fx_to_double(Fx d, int eb)
{
  return ldexp((double)(((long long)d.hi << 32) + d.lo), eb - 1022 - 60);
}

/* N den 2^48 to the nearest integer: the product and its rounding error apart,
   which is up to 2^8 of these units */
__host__ __device__ __forceinline__ Fx fx_table(double n, int den)
{
  const double p = n * den, e = fma(n, (double)den, -p), scale = 281474976710656.0;
  return fx_split(llrint(p * scale) + llrint(e * scale));
}

/* a sum of products a b / 2^S, rounded to nearest */
template <int S> struct FxSum {
  long long hh = 0, cr = 1ll << (S - 33);
  __host__ __device__ __forceinline__ void add(Fx a, Fx b)
  {
    hh += (long long)a.hi * b.hi;
    cr += (long long)a.hi * b.lo;
    cr += (long long)a.lo * b.hi;
  }
  __host__ __device__ __forceinline__ long long value() const { return hh * (1 << (64 - S)) + (cr >> (S - 32)); }
};

/* a sum of products k b / 2^S of integers k below 2^15, rounded to nearest */
template <int S> struct FxIntSum {
  long long hi = 0, lo = 1ll << (S - 1);
  __host__ __device__ __forceinline__ void add(int k, Fx b)
  {
    hi += (long long)k * b.hi;
    lo += (long long)k * b.lo;
  }
  __host__ __device__ __forceinline__ long long value() const { return hi * (1ll << (32 - S)) + (lo >> S); }
};

/* one entry of an element's block through a table column n: sum n w, in units of K den^2 */
__host__ __device__ __forceinline__ long long fx_entry(const Fx n[5], const Fx w[5])
{
  FxSum<63> sum;
#pragma unroll
  for (int s = 0; s < 5; s++) sum.add(n[s], w[s]);
  return sum.value();
}

constexpr int kFxDenBits = 27;       /* den^2 < 2^27 */
constexpr int kFxUnit = 31;          /* K den^2 in units of 2^(E - 31) */

/* the regular table as a kernel parameter, and den^2 with its unit of K */
struct FxRegular {
  int n[12][5];
  double den2, unit;                 /* unit = 2^-31 / den^2 */
  double wide, unwide;               /* den^2 / 2^27, its inverse */
};

/* v / 2^s rounded to nearest (s >= 0) */
__host__ __device__ __forceinline__ long long fx_shift(long long v, int s)
{
  if (s > 62) return 0;
  return (v + ((1ll << s) >> 1)) >> s;
}

/* A column's sum of |N| in 1/64, rounded up. */
__host__ __device__ __forceinline__ int fx_column_sum(const double n[5])
{
  double t = 0.0;
  for (int r = 0; r < 5; r++) t += fabs(n[r]);
  return (int)(64.0 * t) + 1;
}

/* Bits a row's accumulators drop so that its sums fit 63 bits.  A
   contribution from row slot a to a block through slot b is at most
   s_a s_b 2^57.6 (s: the columns' sums of |N|); bound is the largest sum of
   fx_column_sum(a) fx_column_sum(b) over the (contribution, slot) pairs of
   one block, plus 64 x 64 for each pressure block (at most 2^57.6 in K's unit,
   the row's E covering it too).  A regular row's diagonal block has 34: no bit. */
__host__ __device__ __forceinline__ int fx_growth(long long bound)
{
  int g = 0;
  while ((172032ll << g) < bound) g++;               /* 42 x 64 x 64; 42 x 2^57.6 < 2^63 */
  return g;
}

/* magnitudes below 2^-894 stay doubles (their units would be subnormal), and
   so do those near overflow, infinities and NaN */
constexpr int kFxMinExp = 128, kFxMaxExp = 1998, kFxMaxWide = 2030;

/* The double of v 2^(E - 31 - 27), rounded to nearest, by integer operations: an
   entry of an element's K in units of 2^27 / den^2, for a row that is summed
   in double (eb from kFxMinExp to kFxMaxWide, |v| < 2^62).  The conversion
   instruction takes the FP64 pipe as long as an addition does. */
__host__ __device__ __forceinline__ double fx_wide(long long v, int eb)
{
  if (v == 0) return 0.0;
  const uint64_t u = (uint64_t)(v < 0 ? -v : v);
#ifdef __CUDA_ARCH__
  const int n = __clzll((long long)u);
#else
  const int n = __builtin_clzll(u);
#endif
  const uint64_t t = u << n, mant = (t >> 11) + ((t >> 10) & 1u);      /* 2^52 .. 2^53 */
  return ff_from_bits64(((uint64_t)(eb + 5 - n) << 52) + mant + ((uint64_t)v & 0x8000000000000000ull));
}

/* Binades that an element's largest entry of all groups, and that of its (i, j)
   group, may lie below the row's of the group.  The first keeps every rounding
   within 2^-52.8 of the element's largest entry.  The second keeps the digits
   of a group that is small in one element only (a coupling of in-plane and
   normal motion vanishes where a sheet is level): within 2^-48.8 of the group
   itself, beside the first's 2^-52.8 of the block it stands in.  Row kernel on
   the 98,304-triangle sheet, nodes displaced at random by a hundredth of a cell:
   0.485 ms without the rule, 0.488 with 7 and more, 0.491 with 6, 0.509 with 5,
   0.66 with 4, 0.96 with all rows in double.  On a small mesh one such row is a
   tail of 8 us, so the line lies where they are rare. */
constexpr int kFxSpread = 4, kFxPairSpread = 8;

/* The exponent fields of an element's (i, j) group in one word: D's (the
   load's where D is zero), how far the load's lies above it, and the largest
   that a row with this element may have (any, for a zero). */
constexpr int kFxExps = 12;          /* words an element: nine, 16-byte aligned */
constexpr int kFxMaxExcess = 1000;   /* a load further above D: the element keeps its doubles */
__host__ __device__ __forceinline__ unsigned fx_pack(int d, int load, int most)
{
  const int lim = d + kFxPairSpread < most + kFxSpread ? d + kFxPairSpread : most + kFxSpread;
  if (!d) return (unsigned)load | (unsigned)kFxRaw << 21;
  return (unsigned)d | (unsigned)(load > d ? load - d : 0) << 11 | (unsigned)(lim < kFxRaw ? lim : kFxRaw) << 21;
}
__host__ __device__ __forceinline__ int fx_d_exp(unsigned x) { return (int)(x & 0x7ffu); }
__host__ __device__ __forceinline__ int fx_row_exp(unsigned x) { return fx_d_exp(x) + (int)(x >> 11 & 0x3ffu); }
__host__ __device__ __forceinline__ int fx_most_exp(unsigned x) { return (int)(x >> 21); }

/* a pressure entry times den^2 in units of K of a row with exponent field eb */
__host__ __device__ __forceinline__ long long fx_load(double v, int eb)
{
  return fx_shift(fx_from_double(v, eb + kFxDenBits), 60 - kFxDenBits - kFxUnit);
}

} /* namespace biofem */
#endif
