// Shared device helpers of the tcgen05 kernels: mbarriers with bounded waits,
// shared-memory matrix descriptors, kind::f16 MMA issue and commit, TMA and
// bulk copies, the FP64 -> 55-bit fixed-point conversion, and the exact
// conversions of level sums.
#pragma once
#include "fgpu_internal.h"

#include <cuda_fp16.h>

namespace fgpu {
namespace {

// one k-chunk of 16 of the digit planes in shared memory (no swizzle,
// K-major core matrices): A = 128 rows, B = 64 rows, 7 planes each
constexpr uint32_t A_STAGE = NSLICE * 4096;  // 7 planes x 2 k-groups x 128 rows x 16 B
constexpr uint32_t B_STAGE = NSLICE * 2048;  // 7 planes x 2 k-groups x 64 rows x 16 B
constexpr uint32_t STAGE = A_STAGE + B_STAGE;  // 43008 B

__device__ __forceinline__ uint32_t su32(const void* p) {
  return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}
__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
  asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(su32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
  asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(su32(bar)), "r"(bytes) : "memory");
}
// wait for the phase of `parity` to complete, giving up after `limit` polls
__device__ __forceinline__ bool mbar_wait_n(uint64_t* bar, uint32_t parity, int limit) {
  for (int it = 0; it < limit; ++it) {
    uint32_t ok;
    asm volatile(
        "{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok)
        : "r"(su32(bar)), "r"(parity)
        : "memory");
    if (ok) return true;
  }
  return false;
}
// the kernels' bounded wait: 2^22 polls
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity) { return mbar_wait_n(bar, parity, 1 << 22); }

// After a bounded wait gave up: wait (bounded) until the copies issued into
// a `nstage`-deep ring have landed, so that no copy writes this CTA's shared
// memory after it exits.  `issued` counts the k-chunks whose copies were
// issued; chunk c went to stage c % nstage and completes that stage's phase
// c / nstage, and the last chunk of each stage is the only one that can
// still be in flight (a stage is reissued only after its previous chunk was
// consumed, i.e. had landed).
__device__ __forceinline__ void drain_ring(uint64_t* full, int nstage, uint32_t issued) {
  for (int st = 0; st < nstage && (uint32_t)st < issued; ++st) {
    const uint32_t last = issued - 1 - ((issued - 1 - (uint32_t)st) % (uint32_t)nstage);
    mbar_wait(&full[st], (last / nstage) & 1);
  }
}

// tcgen05 shared-memory descriptor, no swizzle, K-major core matrices
// (8 rows x 16 bytes): lbo = byte stride between core matrices along K,
// sbo = along M/N; descriptor version 1 (bits 46-47).
__device__ __forceinline__ uint64_t smem_desc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
  return (uint64_t)((saddr >> 4) & 0x3FFF) | ((uint64_t)((lbo >> 4) & 0x3FFF) << 16) |
         ((uint64_t)((sbo >> 4) & 0x3FFF) << 32) | ((uint64_t)1 << 46);
}
// kind::f16 instruction descriptor: f32 accumulator, f16 A/B, both K-major, M=128, N=64.
constexpr uint32_t IDESC_128x64 = (1u << 4) | ((64u >> 3) << 17) | ((128u >> 4) << 24);

__device__ __forceinline__ void mma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(IDESC_128x64), "r"(accumulate));
}
__device__ __forceinline__ void mma_f16_desc(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc,
                                             uint32_t accumulate) {
  asm volatile(
      "{\n .reg .pred p;\n setp.ne.u32 p, %4, 0;\n"
      " tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}\n" ::"r"(d_tmem),
      "l"(a), "l"(b), "r"(idesc), "r"(accumulate));
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
  asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(su32(bar))
               : "memory");
}
// After a bounded wait gave up: one more commit tracks every MMA this thread
// issued; waiting (bounded) on it means none still writes TMEM when the CTA
// deallocates it.  `drain` is an mbarrier of count 1 used for nothing else.
__device__ __forceinline__ void drain_mmas(uint64_t* drain) {
  mma_commit(drain);
  mbar_wait(drain, 0);
}

// round(x * 2^(55 - e)) for |x| <= 2^e, with integer operations only.
// Sets *bad when the scale bound is violated (|x| > 2^(e+3)).
__device__ __forceinline__ long long to_fixed55(double x, int e, bool* bad) {
  const long long bits = __double_as_longlong(x);
  const int E = (int)((bits >> 52) & 0x7FF);
  if (E == 0) return 0;  // zero or subnormal (below 2^-1022: far under the 2^-55 resolution)
  if (E == 0x7FF) {
    *bad = true;
    return 0;
  }
  const long long M = (bits & 0xFFFFFFFFFFFFFLL) | (1LL << 52);
  const int sh = E - 1075 + 55 - e;
  long long F;
  if (sh >= 0) {
    if (sh > 3) {
      *bad = true;
      return 0;
    }
    F = M << sh;
  } else if (sh > -63) {
    F = (M + (1LL << (-sh - 1))) >> (-sh);
  } else {
    F = 0;
  }
  return bits < 0 ? -F : F;
}

__device__ __forceinline__ void tma_load_5d(void* dst, const void* tmap, int c0, int c1, int c2, int c3, int c4,
                                            uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4, %5, "
      "%6}], [%7];" ::"r"(su32(dst)),
      "l"(tmap), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4), "r"(su32(bar))
      : "memory");
}
__device__ __forceinline__ void bulk_g2s(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
  asm volatile(
      "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(su32(dst)),
      "l"(src), "r"(bytes), "r"(su32(bar))
      : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
  asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(su32(bar)) : "memory");
}

// round(x 2^(62 - e)) as an integer, for |x| < 2^e.  What does not fit
// saturates, NaN and infinities too (they also set *nonfinite): an
// off-diagonal entry like that leaves the matrix not positive semidefinite,
// and the factorisation stops at its row's pivot, if not before, where
// dpotrf on the unrounded matrix does.
__device__ __forceinline__ long long to_fixed62(double x, int e, bool* nonfinite) {
  const long long bits = __double_as_longlong(x);
  const int E = (int)((bits >> 52) & 0x7FF);
  const long long M = (bits & 0xFFFFFFFFFFFFFLL) | (1LL << 52);
  const int sh = E - 1075 + 62 - e;
  long long F;
  if (E == 0x7FF) *nonfinite = true;
  if (sh > 9) {
    F = (1LL << 62) - 1;
  } else if (E == 0 || sh <= -63) {
    F = 0;
  } else {
    F = sh >= 0 ? M << sh : (M + (1LL << (-sh - 1))) >> (-sh);
  }
  return bits < 0 ? -F : F;
}

// round(x 2^(54 - e)) for |x| < 2^e (a scale break, NaN and infinities are the
// caller's to have excluded: the same features passed to_fixed55 before)
__device__ __forceinline__ long long to_fixed54(double x, int e) {
  bool bad = false;
  return (to_fixed55(x, e, &bad) + 1) >> 1;
}

// a diagonal entry: kernel value plus nugget, exact up to the matrix's unit.  The
// scale is their sum's: where they cancel (a nugget below zero) neither need
// fit it, and what is converted is their sum and its rounding error.  NaN
// becomes negative, which fails that pivot as NaN does in dpotrf; infinity only
// sets *nonfinite.
__device__ __forceinline__ long long diag_fixed62(double k, double noise, int e, bool* nonfinite) {
  const double d = k + noise;
  if (!(fabs(d) < INFINITY)) {
    *nonfinite = true;
    return d > 0.0 ? (1LL << 62) - 1 : -(1LL << 61);
  }
  if (fmax(fabs(k), fabs(noise)) < ldexp(1.0, e)) return to_fixed62(k, e, nonfinite) + to_fixed62(noise, e, nonfinite);
  const double t = d - k;
  return to_fixed62(d, e, nonfinite) + to_fixed62((k - (d - t)) + (noise - t), e, nonfinite);
}

// T 2^(e - 62) rounded to the nearest double (ties away from zero), T a signed
// 64-bit integer, with integer operations only; the result must be normal or 0
__device__ __forceinline__ double fixed62_to_double(long long T, int e = 0) {
  const long long sgn = T >> 63;
  unsigned long long a = (unsigned long long)((T ^ sgn) - sgn);
  const int lz = __clzll((long long)a);
  a <<= (lz & 63);  // leading one at bit 63
  const unsigned long long mant = (a >> 11) + ((a >> 10) & 1);  // 53 bits; a carry goes on into the exponent
  const unsigned long long be = lz == 64 ? 0ULL : (unsigned long long)(1024 + e - lz) << 52;
  const unsigned long long r = lz == 64 ? 0ULL : be - (1ULL << 52) + mant;
  return __longlong_as_double((long long)(r | ((unsigned long long)sgn & 0x8000000000000000ULL)));
}

// The exact integer W = sum_l S_l 256^(6 - l) of 7 level sums, in wrapping
// 64-bit arithmetic: callers guarantee |W| < 2^63 (partial level sums may
// exceed it; the wrapped total is still exact).
__device__ __forceinline__ long long levels_to_w64(const int S[7]) {
  unsigned long long w = (unsigned long long)(long long)S[6];
  w += (unsigned long long)(long long)S[5] << 8;
  w += (unsigned long long)(long long)S[4] << 16;
  w += (unsigned long long)(long long)S[3] << 24;
  w += (unsigned long long)(long long)S[2] << 32;
  w += (unsigned long long)(long long)S[1] << 40;
  w += (unsigned long long)(long long)S[0] << 48;
  return (long long)w;
}

// Exact integer level sums without the conversion unit.  For an
// integer-valued float x with -2^22 <= x < 2^22, x + 1.5 2^23 is exact and
// its bits are b = 0x4B000000 + (x + 2^22).  Callers establish the range
// first: by a bound on the contraction, or by checking the raw sums of a
// warp's group (|x| < 2^22) and converting with F2I otherwise.
__device__ __forceinline__ uint32_t level_bits(uint32_t v) {
  return __float_as_uint(__uint_as_float(v) + 12582912.0f);
}

// W = sum_l x_l 256^(6 - l) from the valid bits b_l of column jj's 7 level
// sums, in wrapping 64-bit arithmetic.  Adjacent levels pair up exactly in
// 32 bits: b_l 256 + b_(l+1) = (x_l + 2^22) 256 + (x_(l+1) + 2^22) +
// 0x4B000000 (the top byte of b_l leaves modulo 2^32, bit 23 is clear), below
// 2^32; the offsets leave as one constant.
constexpr unsigned long long LEVEL_BITS_BIAS =
    (1ULL << 22) * 0x0001010101010101ULL + 0x4B000000ULL * ((1ULL << 40) + (1ULL << 24) + (1ULL << 8) + 1ULL);
template <int N>
__device__ __forceinline__ long long level_bits_to_w64(const uint32_t (&b)[7][N], int jj) {
  const uint32_t p01 = b[0][jj] * 256u + b[1][jj];
  const uint32_t p23 = b[2][jj] * 256u + b[3][jj];
  const uint32_t p45 = b[4][jj] * 256u + b[5][jj];
  unsigned long long w = (unsigned long long)p45 * 256u + b[6][jj];
  w += (unsigned long long)p23 << 24;
  w += (unsigned long long)p01 << 40;
  return (long long)(w - LEVEL_BITS_BIAS);
}

__device__ __forceinline__ void tmem_ld8(uint32_t (&v)[8], uint32_t addr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7])
               : "r"(addr));
}
// one k-chunk of a tile with the B planes stacked along N: for A plane pp
// the pairs (pp, q), q = 0 .. 6 - pp, accumulate into levels pp .. 6, whose
// TMEM blocks of 64 columns are contiguous, so they are one MMA over B
// planes 0 .. 6 - pp (N = 64 (7 - pp), above N = 256 in two equal halves): 10 MMAs instead of
// 28, and A plane pp is read from shared memory once or twice instead of
// 7 - pp times.  N >= 128 MMAs run at the tensor pipe's full rate; N = 64
// ones are bound by shared-memory operand bandwidth.
__device__ __forceinline__ void issue_chunk_128x64(uint32_t tbase, uint64_t adesc, uint64_t bdesc, bool first) {
#pragma unroll
  for (int pp = 0; pp < NSLICE; ++pp) {
    // N = 64 (7 - pp) in one MMA, or, above the 256 limit, in two equal
    // halves (224 + 224, 192 + 192, 160 + 160): an N = 64 remainder would
    // be bound by the A operand's shared-memory read rather than the tensor
    // pipe.  The stacked B rows and the TMEM columns are both contiguous, so
    // a split at any multiple of 8 rows is one offset in each.
    const int n = 64 * (NSLICE - pp);
    const int nh = n <= 256 ? n : n / 2;
#pragma unroll
    for (int off = 0; off < n; off += nh) {
      const uint32_t idesc = (1u << 4) | ((uint32_t)(nh >> 3) << 17) | ((128u >> 4) << 24);
      mma_f16_desc(tbase + (uint32_t)(pp * 64 + off), adesc + (uint64_t)(pp * 4096 >> 4),
                   bdesc + (uint64_t)((off * 16) >> 4), idesc, (first && pp == 0) ? 0u : 1u);
    }
  }
}

// The 7 fp16 digit planes of 8 entries F = x 2^55, |x| <= 1 (one k-group of a
// row), packed: F has the balanced digits
// d_p in [-128, 127] (p = 1..6, base 256, lowest last) and d_0 = the rest.
// G = F + sum_{k<6} 128 256^k turns them into plain bytes: byte 6 - p of G
// is d_p + 128, and G >> 48 is d_0 (|d_0| <= 128 when |x| <= 1).  A byte
// u under the fp16 exponent bits 0x64 is the half 1024 + u, so one HSUB2 of
// 1152 per pair of entries yields the digits exactly, with no conversion
// instruction; two byte permutes place a pair's bytes under the 0x64 bytes.
__device__ __forceinline__ void digits8_of_fixed55(const long long (&F)[8], uint4 out[NSLICE]) {
  unsigned lo[8], hi[8];
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) {
    const long long G = F[kk] + 0x808080808080LL;
    lo[kk] = (unsigned)G;
    hi[kk] = (unsigned)(G >> 32);
  }
  const __half2 off = __halves2half2(__ushort_as_half(0x6480), __ushort_as_half(0x6480));  // 1152
#pragma unroll
  for (int p = 0; p < NSLICE; ++p) {
    unsigned w[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) {
      unsigned bits;
      if (p == 0) {  // d_0 + 128 may be 256: arithmetic, not a byte
        const unsigned u0 = (unsigned)(((int)hi[2 * m] >> 16) + 128);
        const unsigned u1 = (unsigned)(((int)hi[2 * m + 1] >> 16) + 128);
        bits = (0x6400u + u0) | ((0x6400u + u1) << 16);
      } else {
        const int q = 6 - p;  // byte of G: byte q & 3 of the low or high word
        const unsigned wa = q < 4 ? lo[2 * m] : hi[2 * m], wb = q < 4 ? lo[2 * m + 1] : hi[2 * m + 1];
        const unsigned t = __byte_perm(wa, 0x64646464u, 0x4440u | (unsigned)(q & 3));  // [a_q, 64, 64, 64]
        bits = __byte_perm(wb, t, 0x7054u | ((unsigned)(q & 3) << 8));                  // [a_q, 64, b_q, 64]
      }
      const __half2 h = __hsub2(*reinterpret_cast<const __half2*>(&bits), off);
      w[m] = *reinterpret_cast<const unsigned*>(&h);
    }
    out[p] = make_uint4(w[0], w[1], w[2], w[3]);
  }
}

}  // namespace
}  // namespace fgpu
