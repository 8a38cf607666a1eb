// exp(x), x <= 0, for the kernel-matrix entries, evaluated on the integer
// pipes so that it does not compete with the FP64 work for this part's
// narrow FP64 pipe.
//
//   |y| = |x| log2(e) as a fixed-point number with 64 fractional bits
//         (64 x 128-bit product, exact to 2^-64),
//   2^-|y| = 2^-m 2^(j/256) exp(s ln2),  m = ceil(|y|), m - |y| = j/256 + s,
//   exp(t), 0 <= t < ln2/256: degree-5 Taylor polynomial in 64-bit fixed
//   point (scale 2^63, truncation below 2^-60), then one round-to-nearest
//   into the double (subnormals included).
// Error below 0.51 ulp; measured: never more than 1 ulp from the host libm
// over 16.7M arguments spanning [-745.2, 0].  Two entries: a double argument
// (iexp_neg), and an exact fixed-point argument x = -E 2^e (iexp_fixed),
// which the tensor-core build uses without forming a double.
#pragma once
#include "iexp_table.h"

// exp(-|x|) for |x| = M 2^e2 with M normalised (bit 63 set), 2^-54 <= |x| < 1024
__device__ __forceinline__ double iexp_core(unsigned long long M, int e2) {
  const unsigned __int128 P = (unsigned __int128)M * IEXP_L2E_HI +
                              (unsigned long long)(((unsigned __int128)M * IEXP_L2E_LO) >> 64);
  const unsigned __int128 Y = P >> (-1 - e2);  // |y| 2^64; P = |y| 2^(63 - e2), shift 53..116
  const unsigned int yi = (unsigned int)(Y >> 64);
  const unsigned long long yf = (unsigned long long)Y;
  const unsigned int m = yi + (yf ? 1u : 0u);
  const unsigned long long f = 0ULL - yf;  // (m - |y|) 2^64
  const int j = (int)(f >> 56);
  const unsigned long long t = __umul64hi(f & 0x00FFFFFFFFFFFFFFULL, IEXP_LN2);  // s ln2, 2^64
  unsigned long long q = IEXP_C5;
  q = IEXP_C4 + __umul64hi(q, t);
  q = IEXP_C3 + __umul64hi(q, t);
  q = IEXP_C2 + __umul64hi(q, t);
  q = (1ULL << 63) + __umul64hi(q, t);
  const unsigned long long p = (1ULL << 63) + __umul64hi(q, t);      // exp(t) 2^63
  const unsigned long long Z = __umul64hi(__ldg(&g_iexp_tab[j]), p);  // 2^(j/256) exp(t) 2^62
  const int top = (int)(Z >> 63);                                     // value in [2, 2.01)
  const int sh = 10 + top;                                            // keep 53 bits
  const int be = 1023 + top - (int)m;                                 // biased exponent
  if (be >= 1) {
    const unsigned long long mant = (Z + (1ULL << (sh - 1))) >> sh;  // may carry to 2^53
    return __longlong_as_double((long long)(((unsigned long long)be << 52) + mant - (1ULL << 52)));
  }
  const int tot = sh + 1 - be;  // subnormal result
  if (tot > 64) return 0.0;
  const unsigned long long mant = (tot == 64) ? (Z >> 63) : ((Z + (1ULL << (tot - 1))) >> tot);
  return __longlong_as_double((long long)mant);
}

__device__ __forceinline__ double iexp_neg(double x) {
  const unsigned long long bits = (unsigned long long)__double_as_longlong(x);
  const int ex = (int)((bits >> 52) & 0x7FF);
  if (ex < 969) return 1.0;  // |x| < 2^-54 rounds to 1 (also +-0 and subnormals)
  if (!(x >= -745.1332191019412)) return (x != x) ? x : 0.0;  // underflow, -inf, NaN
  if (x > 0.0) return exp(x);
  const unsigned long long M = ((bits & 0xFFFFFFFFFFFFFULL) | 0x10000000000000ULL) << 11;
  return iexp_core(M, ex - 1086);
}

// exp(-E 2^e) for an exact non-negative integer E
__device__ __forceinline__ double iexp_fixed(unsigned long long E, int e) {
  if (E == 0) return 1.0;
  const int lz = __clzll((long long)E);
  const int top = 63 - lz + e;  // 2^top <= E 2^e < 2^(top + 1)
  if (top >= 10) return 0.0;    // beyond 1024: exp underflows
  if (top < -55) return 1.0;    // below 2^-55: rounds to 1
  return iexp_core(E << lz, e - lz);
}

// exp(-E 2^e) for exact integers E >= 0 sharing one scale 2^e (the
// kernel-matrix build's entries of one distance leaf), with the per-entry
// work cut down:
//  * x = E 2^e as it stands, 2^-64 its fraction's unit: only m, the number of
//    halvings, needs log2(e), from 32 bits of x (13 fractional, rounded
//    up so that m >= x log2(e)), and g = m ln2 - x, 0 < g < ln2 + 2^-12, is one
//    64 x 32-bit product modulo 2^64 (ln2 rounded at 2^-64: m 2^-65 off);
//  * the fraction splits as g = j/1024 + (k + 1/2)/2^20 + t, |t| <= 2^-21, with
//    two 1024-entry tables the caller keeps in shared memory, exp(j/1024)
//    2^62 and expm1((k + 1/2)/2^20) 2^64, and exp(t) = 1 + t + t^2/2 up to
//    t^3/6 < 2^-65;
//  * the small products are single 32 x 32-bit multiplies, and the final one,
//    exp(j/1024) times a correction below 2^-10, three;
//  * one round-to-nearest, subnormals included.
// The integer pipe's wide multiplies bound the build (2.3 cycles each, a
// 64 x 64-bit high product 26): against y = x log2(e) from a 64 x 128-bit product
// and two high products, the form before, 40 problems of N = 4000 (two
// leaves) build in 3.8 instead of 5.5 ms.  Error before the final
// rounding below 2^-60 relative for x < 8 (at most 14 2^-64 on a CPU model
// against 60-digit arithmetic, 15 in the form before), the rounding of m
// ln2 beyond; measured on the GPU through fgpu_diag_exp_fixed.
struct IexpScale {
  int F;  // fractional bits of x
};
__device__ __forceinline__ IexpScale iexp_scale(int e) { return IexpScale{-e}; }

// exp(-E 2^e) = Z 2^-62 2^-m, 2^62 <= Z < 2^63 + 2^52 (m >= 1100: below every double)
struct IexpParts {
  unsigned long long Z;
  int m;
};
// x: 13 fractional bits in x13 (saturated), frac = x 2^64 modulo 2^64
__device__ __forceinline__ IexpParts iexp_parts_core(unsigned x13, unsigned long long frac,
                                                     const unsigned long long* __restrict__ tab1024,
                                                     const unsigned long long* __restrict__ fine1024) {
  const unsigned m = (__umulhi(x13, IEXP_L2E32) + 2u + (1u << 12)) >> 12;
  const unsigned long long g = (unsigned long long)m * IEXP_LN2 - frac;
  const unsigned gh = (unsigned)(g >> 32);
  const unsigned long long dk = *reinterpret_cast<const unsigned long long*>(
      reinterpret_cast<const char*>(fine1024) + ((gh >> 9) & (1023u << 3)));
  const unsigned long long T =
      *reinterpret_cast<const unsigned long long*>(reinterpret_cast<const char*>(tab1024) + ((gh >> 19) & ~7u));
  const long long t = (long long)((g & 0x00000FFFFFFFFFFFULL) - (1ULL << 43));  // 2^64, |t| <= 2^43
  const int th = (int)(t >> 12);
  const long long eps = t + (((long long)th * th) >> 41);                                  // expm1(t) 2^64
  const long long de = ((long long)(int)(unsigned)(dk >> 23) * (int)(eps >> 13)) >> 28;   // their product, 2^64
  const unsigned long long d = dk + (unsigned long long)(eps + de);                        // 0 < d < 2^55
  const unsigned Th = (unsigned)(T >> 32), Tl = (unsigned)T, dh = (unsigned)(d >> 32), dl = (unsigned)d;
  const unsigned long long mid = (unsigned long long)Th * dl + (3ULL << 30) + (unsigned long long)Tl * dh;
  return IexpParts{T + (unsigned long long)Th * dh + (mid >> 32), (int)m};  // exp(g) 2^62
}
// the scales of every ordinary leaf, uniform over a pass
__device__ __forceinline__ bool iexp_common(IexpScale sc) { return sc.F >= 20 && sc.F < 128; }
template <bool COARSE>  // F <= 64
__device__ __forceinline__ IexpParts iexp_common_parts(unsigned long long E, IexpScale sc,
                                                       const unsigned long long* __restrict__ tab1024,
                                                       const unsigned long long* __restrict__ fine1024) {
  // x below 2^19 (exp is 0 far before): the top word alone decides
  const unsigned top = sc.F >= 45 ? ~0u : (1u << (sc.F - 13)) - 1u;
  E = (unsigned long long)min((unsigned)(E >> 32), top) << 32 | (unsigned)E;
  const unsigned long long frac = COARSE ? E << (64 - sc.F) : E >> (sc.F - 64);
  return iexp_parts_core((unsigned)(E >> min(sc.F - 13, 63)), frac, tab1024, fine1024);
}
// the others (a call: inlined it would cost its callers registers)
static __device__ __noinline__ double iexp_other(unsigned long long E, IexpScale sc) { return iexp_fixed(E, -sc.F); }

__device__ __forceinline__ double iexp_fixed_tab(unsigned long long E, IexpScale sc,
                                                 const unsigned long long* __restrict__ tab1024,
                                                 const unsigned long long* __restrict__ fine1024) {
  if (!iexp_common(sc)) return iexp_other(E, sc);
  const IexpParts v = sc.F <= 64 ? iexp_common_parts<true>(E, sc, tab1024, fine1024)
                                 : iexp_common_parts<false>(E, sc, tab1024, fine1024);
  if (v.m >= 1100) return 0.0;
  const int top = (int)(v.Z >> 63);
  const int sh = 10 + top;
  const int be = 1023 + top - v.m;
  if (be >= 1) {
    const unsigned long long mant = (v.Z + (1ULL << (sh - 1))) >> sh;
    return __longlong_as_double((long long)(((unsigned long long)be << 52) + mant - (1ULL << 52)));
  }
  const int tot = sh + 1 - be;
  if (tot > 64) return 0.0;
  const unsigned long long mant = (tot == 64) ? (v.Z >> 63) : ((v.Z + (1ULL << (tot - 1))) >> tot);
  return __longlong_as_double((long long)mant);
}

// round(exp(-E 2^e) 2^(62 - e2)), e2 >= 1: the value straight in the matrix's
// fixed-point unit
__device__ __forceinline__ long long iexp_parts_fixed62(IexpParts v, int e2) {
  unsigned long long h;  // the shift gives 0 from 64 on
  asm("shr.u64 %0, %1, %2;" : "=l"(h) : "l"(v.Z), "r"(v.m + e2 - 1));
  return (long long)((h + 1) >> 1);
}
