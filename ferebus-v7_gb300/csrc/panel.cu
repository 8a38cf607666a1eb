// One panel of the Cholesky factorisation (tensor-core mode): the 128 columns
// [c0, c0 + 128) of every problem in one launch, from the fixed-point Schur
// complement to the factor's digit planes.
//
// Everything is in the problem's scale 2^e (K_ii < 2^2e; every K_ii of these
// kernels is the same): the accumulators hold S_ij 2^(62 - 2e), S = K minus the
// exact products of the earlier panels, and the factor computed here is
// L' = 2^-e L, so that every value lies in [-1, 1].
//
// A CTA owns one 128-row tile of one problem (or a 64- or 32-row part of one)
// and walks the panel's 128 columns in 8 pieces of 16.  For piece t:
//
//   B_ij = S_ij - sum_{k < 16 t} L'_ik L'_jk  in 64-bit integers: the couplings
//          inside the panel come from tcgen05.mma on the digit planes (7 exact
//          level sums, as in the trailing update);
//   x L'_tt^T = B by substitution, one thread per row, in 60-bit fixed point
//          (below);
//   x's 7 fp16 digit planes into shared memory (the A operand of the later
//          pieces' couplings) and to HBM (the trailing update's operands).
//
// The tile that holds the panel's own rows (the diagonal tile) factors the
// 16 x 16 diagonal blocks on the way, and publishes each piece -- the block
// and its reciprocal pivots, its rows' digits, the solved right-hand-side
// entries z -- through release/acquire counters in HBM that the problem's
// other CTAs poll (bounded).  CTAs take their tile from an atomic ticket,
// diagonal tiles first: whoever waits for a diagonal tile holds a later
// ticket than it, so the tile is already running, and a diagonal tile itself
// waits for nobody.  The right-hand sides ride along: each row's thread
// accumulates sum_k L'_ik z_k while x is in registers.
//
// Arithmetic.  This GPU's FP64 unit takes 64 cycles per warp instruction and
// SM quarter, for dependent and independent operations alike, so a piece's 136
// multiply-adds per row cost 10k cycles there whatever their order.  In fixed
// point, X = x 2^60 split as X = Xh 2^30 + Xl (|Xl| <= 2^29),
//   x l = (Xh Lh + (Xh Ll + Xl Lh) 2^-30) 2^-60 + O(2^-62),
// is three 32 x 32 + 64-bit multiply-adds on the integer pipe (~10 cycles).
// The dropped Xl Ll and the final shifts err by a few 2^-61, well below the
// 2^-56 to which x is rounded for the trailing update.  The 64-bit sums cannot
// overflow: rows of L' have norm at most 1, so sum |Xh Ll| <= 2^30 2^29 4.
// That holds while K is positive definite.  Schur complements are kept modulo 4 in
// the matrix's unit, so a row of an indefinite matrix, whose entries' squares
// add up far beyond K_ii, could come round to a positive pivot: every row
// keeps the sum of its squares (rowsq), and one that is beyond K_ii fails the pivot.
// Only the right-hand sides' substitution (32 operations per piece, off the
// critical path) and their running sums (one per row and piece) are FP64.
//
// Bounds.  A lone problem is bound by the diagonal tile's chain of 128
// pivots, a batch by integer issue (one warp per SM quarter: latency).  The 7
// digit chunks the couplings read (28 KB each) stay in shared memory, hence
// one CTA per SM.  Measured, against the FP64 panel in ten launches
// (conversion of the integer sums, 32-column factors, solves and couplings,
// right-hand-side update) that this replaces: a lone problem 250 -> 75 us
// per panel (N = 4000, 32 panels), a swarm of 40 at N = 4000 20.7 -> 9.3 ms
// (6.8 with k_panel_rows below).
#include "fgpu_internal.h"
#include "tc_common.cuh"

#include <cuda_fp16.h>

namespace fgpu {
namespace {

constexpr int PW = 16;                 // piece width
constexpr int NPIECE = NB / PW;        // pieces of a panel
constexpr uint32_t PN_ACHUNK = NSLICE * 4096;       // one piece's digits of 128 rows: [plane][k-group 2][row 128][8 x fp16]
constexpr uint32_t PN_BCHUNK = NSLICE * 2 * PW * 16;  // one piece's digits of the next piece's 16 rows: [k-group 2][plane][row 16][8 x fp16]
constexpr uint32_t PN_LBYTES = sizeof(PanelBlock);
constexpr uint32_t PN_ZBYTES = sizeof(PanelZ);
static_assert(PN_LBYTES % 16 == 0 && PN_ZBYTES % 16 == 0, "copied 16 bytes at a time");
constexpr uint32_t PN_OFF_B = (NPIECE - 1) * PN_ACHUNK;
constexpr uint32_t PN_OFF_L = PN_OFF_B + (NPIECE - 1) * PN_BCHUNK;
constexpr uint32_t PN_OFF_Z = PN_OFF_L + 2 * PN_LBYTES;
constexpr uint32_t PN_OFF_R = PN_OFF_Z + 2 * PN_ZBYTES;
constexpr uint32_t PN_OFF_BAR = PN_OFF_R + MAX_RHS * PW * 8;
constexpr uint32_t PN_SMEM = PN_OFF_BAR + 64;
static_assert(PN_SMEM + 1024 <= 227 * 1024, "shared memory per CTA");
constexpr int PN_MMA_WARP = 4, PN_RHS_WARP = 5;
constexpr int PN_THREADS = 32 * 6;  // 4 row warps, operand loads and MMA issue, right-hand sides
constexpr uint32_t PN_TMEM_COLS = 128;  // 7 levels x 16 columns, rounded up
constexpr int FLAG_L = 0, FLAG_D = 1, FLAG_Z = 2;  // a problem's counters: blocks, digits, z published
constexpr int FLAG_FAIL = 1 << 30;                  // the diagonal tile met a non-positive pivot (or gave up)

__device__ __forceinline__ int ld_acquire(const int* p) {
  int v;
  asm volatile("ld.acquire.gpu.global.s32 %0, [%1];" : "=r"(v) : "l"(p) : "memory");
  return v;
}
// raise a counter to v: FLAG_FAIL stays, whatever the diagonal tile's other warps still publish
__device__ __forceinline__ void publish(int* p, int v) {
  asm volatile("red.release.gpu.global.max.s32 [%0], %1;" ::"l"(p), "r"(v) : "memory");
}
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(su32(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// 1 / sqrt(D 2^-60), 4 <= D < 2^60, as y 2^(sh - 62) with y = (yh, yl) in [2^62,
// 2^63): a single-precision estimate refined once in 64-bit fixed point.  With
// D 2^-60 = m 4^k, 1 <= m < 4 (k < 0, sh = -k - 1), and y0 ~ m^-1/2 (23 bits):
// e = 1 - m y0^2 is formed to 2^-61 (|e| < 2^-20) and m^-1/2 =
// y0 (1 - e)^-1/2 = y0 (1 + e/2 + 3 e^2 / 8 + O(2^-61)).  Relative error below
// 2^-57.  ~50 integer instructions (2 to 3 cycles
// of issue each on this GPU, ~220 of latency together); the library's FP64
// rsqrt takes ~380 cycles, and 128 of them follow one another in a panel.
__device__ __forceinline__ void rsqrt_fixed(long long D, unsigned& yh, unsigned& yl, int& sh) {
  const unsigned hi = (unsigned)((unsigned long long)D >> 32), lo = (unsigned)D;
  // leading one to bit 63 of (ah, al); D 2^-60 = 1.f 2^E
  const unsigned h1 = hi ? hi : lo, l1 = hi ? lo : 0u;
  const int z = __clz(h1), E = (hi ? 3 : -29) - z, r = E & 1;
  const unsigned ah = __funnelshift_l(l1, h1, z), al = l1 << (z & 31);
  sh = -(E >> 1) - 1;
  const float mf = __uint_as_float((ah >> 8) + ((unsigned)(126 + r) << 23));  // the leading one carries into the exponent
  float y0;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(mf));
  const unsigned Y = __float_as_uint(y0 + 1.0f) - 0x3F800000u;  // y0 2^23, y0 in [0.5, 1]
  // e 2^61 = 2^61 - m y0^2 2^61, m 2^62 in (mh, ml), y0^2 2^63 in (qh, ql); the
  // product of the low words (below 2^-61) is left out
  const unsigned mh = r ? ah : ah >> 1, ml = r ? al : __funnelshift_r(al, ah, 1);
  const unsigned long long q = ((unsigned long long)Y * Y) << 17;
  const unsigned qh = (unsigned)(q >> 32), ql = (unsigned)q;
  const unsigned long long t1 = (unsigned long long)mh * ql, t2 = (unsigned long long)ml * qh;
  const long long e = (long long)((1ULL << 61) - (t2 >> 32) - ((unsigned long long)mh * qh + (t1 >> 32)));
  const int eh = (int)(e >> 10);
  const unsigned e2 = (unsigned)((unsigned long long)((long long)eh * eh) >> 32);  // e^2 2^70
  const unsigned c2 = (e2 * 3u) >> 14;                                             // 3 e^2 / 8 2^59
  // y0 (1 + e/2 + c2) 2^63, less one unit: never 2^63
  const unsigned long long v = (((unsigned long long)(Y * 256u - 1u) << 32) | 0xFFFFFFFFu) +
                               (unsigned long long)(((long long)Y * (e >> 3) + (long long)((unsigned long long)Y * c2)) >> 19);
  yh = (unsigned)(v >> 32);
  yl = (unsigned)v;
}

// X = x 2^60 of x = T 2^-60 / L'_jj, split in Xh 2^30 + Xl.  |x| <= 1 while
// the matrix is positive semidefinite, i.e. |T| < 2^(60 - sh); a larger |T|
// clamps, to |x| = 1 up to 2^-28, which fails the row's pivot.
__device__ __forceinline__ void scale_entry(long long T, unsigned yh, unsigned yl, int sh, int& Xh, int& Xl) {
  const int lim = 1 << (29 - sh);  // |T| up to twice its bound
  const unsigned tl = (unsigned)T;
  const int th = min(max((int)(T >> 32), -lim), lim - 1);
  // T 2^(sh + 2) y 2^-64: high product, and the two cross products' high parts
  const int uh = (int)__funnelshift_l(tl, (unsigned)th, sh + 2);
  const unsigned ul = tl << (sh + 2);
  const long long X = (long long)uh * (int)yh + (long long)(((unsigned long long)ul * yh) >> 32) +
                      (((long long)uh * (int)(yl >> 1)) >> 31);
  const long long Xr = X + (1LL << 29);
  const int hi = min(max((int)(Xr >> 32), -(1 << 28)), (1 << 28) - 1);
  Xh = (int)__funnelshift_l((unsigned)Xr, (unsigned)hi, 2);
  Xl = (int)((unsigned)X - ((unsigned)Xh << 30));
}

// a Schur complement entry from units of 2^-62 to 2^-60, rounded
__device__ __forceinline__ long long to_unit60(unsigned long long w) { return ((long long)w + 2) >> 2; }

// S + M 2^-30 += x l in units of 2^-60
__device__ __forceinline__ void mac_entry(long long& S, long long& M, int xh, int xl, int lh, int ll) {
  S += (long long)xh * lh;
  M += (long long)xh * ll;
  M += (long long)xl * lh;
}
// shift a register array down by n: a[i] = a[i + n]
template <int n, typename T, int N>
__device__ __forceinline__ void shift_down(T (&a)[N]) {
#pragma unroll
  for (int i = 0; i + n < N; ++i) a[i] = a[i + n];
}

// S + M 2^-30 += sum over c0 <= c < n of x_c l_kc, two block entries a load
template <int c0>
__device__ __forceinline__ void mac_row(long long& S, long long& M, const int (&Xh)[PW], const int (&Xl)[PW],
                                        const PanelBlock& Lt, int k, int n) {
  const int4* l = reinterpret_cast<const int4*>(&Lt.x[k][0]);
#pragma unroll
  for (int c = c0; c < PW; c += 2) {
    if (c < n) {
      const int4 v = l[c / 2];
      mac_entry(S, M, Xh[c], Xl[c], v.x, v.y);
      if (c + 1 < n) mac_entry(S, M, Xh[c + 1], Xl[c + 1], v.z, v.w);
    }
  }
}

// A row's sum of squares, sum_{k <= i} x_ik^2 = K_ii < 1 where the leading minors are
// positive, in units of 2^-SQ_BITS, cut off every 8 entries (16 2^-22 a panel).  The
// pivot K_ii - sum_{k < i} is formed modulo 4: one that came round shows in the
// sum, and one that did not is negative where the matrix is not positive
// definite.  That holds whatever the row's entries were: until one of them clamps
// they are exact, right-hand sides beyond the range +-2 (but below 1 +
// SQ_LIMIT^1/2 = 2.2) come round to ones that clamp, and a clamped entry adds 1.
// 8 multiply-adds and 3 instructions per 8 entries, off the pivots' chain but for
// the diagonal block's rows.
constexpr int SQ_BITS = 22;
constexpr int SQ_LIMIT = (1 << SQ_BITS) + (1 << (SQ_BITS - 2));  // 1.25
constexpr int SQ_MAX = 1 << 30;                                  // where the stored sum saturates
template <int c0>
__device__ __forceinline__ int squares8(const int (&Xh)[PW]) {
  unsigned long long q = 0;  // 2^-60; at most 8
#pragma unroll
  for (int c = c0; c < c0 + 8; ++c) q += (unsigned long long)((long long)Xh[c] * Xh[c]);
  return (int)(q >> (60 - SQ_BITS));
}

// the digit planes of 8 entries X = x 2^60 of a row
__device__ __forceinline__ void digits8_packed(const int* Xh, const int* Xl, uint4 out[NSLICE]) {
  long long F[8];
#pragma unroll
  for (int kk = 0; kk < 8; ++kk) F[kk] = ((long long)Xh[kk] * (1LL << 30) + Xl[kk] + 16) >> 5;
  digits8_of_fixed55(F, out);
}

// the whole warp waits for an mbarrier phase (bounded), or until the CTA
// stops: 0 the phase completed, 1 stopped, 2 gave up (the same in every lane)
__device__ __forceinline__ int wait_or_stop(uint64_t* bar, uint32_t parity, const int* stop) {
  int r = 2;
  for (int it = 0; it < (1 << 22); ++it) {
    if (mbar_wait_n(bar, parity, 1)) {
      r = 0;
      break;
    }
    if (*(volatile const int*)stop) {
      r = 1;
      break;
    }
  }
  if (__all_sync(0xffffffffu, r == 0)) return 0;
  return __any_sync(0xffffffffu, r == 2) ? 2 : 1;
}

__device__ __forceinline__ uint32_t tmem_ld1(uint32_t addr) {
  uint32_t v;
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x1.b32 {%0}, [%1];" : "=r"(v) : "r"(addr));
  return v;
}

// T -= the couplings' exact sums of this warp's 32 rows and 16 columns, from
// their 7 level sums at `addr` in TMEM: by the magic add where they lie in
// (-2^22, 2^22) (the sum's exponent bits tell), else by F2I
__device__ __forceinline__ void drain_couplings(long long (&T)[PW], uint32_t addr) {
#pragma unroll
  for (int g = 0; g < 2; ++g) {
    uint32_t v[NSLICE][8], off = 0;
#pragma unroll
    for (int l = 0; l < NSLICE; ++l) tmem_ld8(v[l], addr + (uint32_t)(l * PW + g * 8));
    asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
    for (int l = 0; l < NSLICE; ++l)
#pragma unroll
      for (int jj = 0; jj < 8; ++jj) {
        v[l][jj] = level_bits(v[l][jj]);
        off |= v[l][jj] ^ 0x4B000000u;
      }
    if (__any_sync(0xffffffffu, off >> 23)) {
#pragma unroll 1
      for (int c = 0; c < 8; ++c) {
        int I[NSLICE];
#pragma unroll
        for (int l = 0; l < NSLICE; ++l) I[l] = (int)tmem_ld1(addr + (uint32_t)(l * PW + g * 8 + c));
        asm volatile("tcgen05.wait::ld.sync.aligned;");
#pragma unroll
        for (int l = 0; l < NSLICE; ++l) I[l] = __float2int_rn(__int_as_float(I[l]));
        const unsigned long long W = (unsigned long long)levels_to_w64(I);
#pragma unroll
        for (int k = 0; k < 8; ++k)
          if (k == c) T[g * 8 + k] = (long long)((unsigned long long)T[g * 8 + k] - W);
      }
    } else {
#pragma unroll
      for (int jj = 0; jj < 8; ++jj)
        T[g * 8 + jj] = (long long)((unsigned long long)T[g * 8 + jj] - (unsigned long long)level_bits_to_w64(v, jj));
    }
  }
}

// one lane polls a problem's counter until it reaches `want` (bounded)
__device__ __forceinline__ int poll_flag(const int* f, int want) {
  for (int it = 0; it < (1 << 22); ++it) {
    const int v = ld_acquire(f);
    if (v >= want) return v;
    __nanosleep(it < 64 ? 20 : 200);
  }
  return -1;
}

}  // namespace

__global__ void __launch_bounds__(PN_THREADS, 1)
    k_panel(const Prob* __restrict__ probs, int s, const int* __restrict__ order, int ndiag, int sub_shift,
            int* __restrict__ counter, int* __restrict__ flags) {
  extern __shared__ __align__(1024) unsigned char smp[];
  unsigned char* As = smp;
  unsigned char* Bs = smp + PN_OFF_B;
  PanelBlock* Ls = reinterpret_cast<PanelBlock*>(smp + PN_OFF_L);  // [2]: this piece's diagonal block
  PanelZ* Zs = reinterpret_cast<PanelZ*>(smp + PN_OFF_Z);          // [2]: this piece's z
  double* Rs = reinterpret_cast<double*>(smp + PN_OFF_R);  // diagonal tile: right-hand-side entries of the piece's rows
  uint64_t* b_mma = reinterpret_cast<uint64_t*>(smp + PN_OFF_BAR);  // a piece's couplings are in TMEM
  uint64_t* b_blk = b_mma + 1;                                      // its block is in Ls
  uint64_t* b_z = b_mma + 2;                                        // its z is in Zs
  uint64_t* b_drained = b_mma + 3;                                  // the row warps hold its couplings in registers
  uint64_t* b_digits = b_mma + 4;                                   // the row warps' digits are in As (and in HBM)
  uint64_t* b_half = b_mma + 5;                                     // the first half of its block's columns is in Ls
  uint64_t* b_rhs = b_mma + 6;                                      // diagonal tile: the piece's right-hand-side entries are in Rs
  uint64_t* b_quiet = b_mma + 7;                                    // quiescing before an early exit
  __shared__ int s_tile, s_sub, s_skip, s_stop, s_abort;
  __shared__ uint32_t s_tmem;
  __shared__ long long s_D[2][PW];  // the pieces' pivots, in units of 2^-60
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  if (tid == 0) {
    const int u = atomicAdd(counter, 1);
    // the order lists every problem's own row tile first, then the others
    const int v = u - ndiag;
    const int id = u < ndiag ? order[u] : order[ndiag + (v >> sub_shift)];
    s_tile = id;
    s_skip = *(volatile int*)&probs[id >> 16].status[1];  // one read: the exit below is block-uniform
    s_sub = u < ndiag ? 0 : (v & ((1 << sub_shift) - 1));
    s_stop = 0;
    s_abort = 0;
  }
  __syncthreads();
  if (s_skip) return;
  const int p = s_tile >> 16, ti = s_tile & 0xFFFF;
  const bool diag = ti == s;
  const int nrw = diag ? 4 : 4 >> sub_shift;  // row warps
  const int row0 = ti * NB + s_sub * 32 * nrw;
  const Prob& P = probs[p];
  const int c0 = s * NB;
  int* fl = flags + PANEL_FLAGS * p;
  const int fbase = s * NPIECE;  // the counters grow through the whole sweep
  const int np = min(NPIECE, (P.N - c0 + PW - 1) / PW);  // pieces that hold more than identity padding
  if (tid == 0) {
    mbar_init(b_mma, 1);
    mbar_init(b_blk, 1);
    mbar_init(b_z, 1);
    mbar_init(b_drained, nrw);
    mbar_init(b_digits, nrw);
    mbar_init(b_half, 1);
    mbar_init(b_rhs, 1);
    mbar_init(b_quiet, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == PN_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(su32(&s_tmem)),
                 "n"(PN_TMEM_COLS));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = s_tmem;
  bool quiet = false;  // MMA warp: its MMAs were waited for after a stop

  if (warp < nrw) {
    // ---------------- row warps: one thread per row ----------------
    const int i = row0 + tid;
    const int rl = i & (NB - 1);  // row inside its 128-row tile
    const size_t ld = (size_t)P.ld;
    double* krow = P.K + (size_t)c0 * ld + i;  // read by alpha and the adjoint (keep_l)
    const int kexp = *P.kscale;
    // the accumulators of this row, column 0 of the panel (tiles 2 s and 2 s + 1)
    const long long* acc0 = P.acc + acc_tile(ti, 2 * s, P.nt128) * ACC_TILE_ELEMS + acc_elem(rl, 0);
    const long long* acc1 = P.acc + acc_tile(ti, 2 * s + 1, P.nt128) * ACC_TILE_ELEMS + acc_elem(rl, 0);
    unsigned char* gdig = P.slices + (size_t)(diag ? P.nt128 : ti) * NSLICE * SLICE_BYTES + (size_t)rl * 16;
    long long wv[PW];
    auto load_piece = [&](int t) {
      const long long* a = (t < 4 ? acc0 : acc1) + (size_t)(t & 3) * 2048;  // 16 columns: 2 groups of 8
#pragma unroll
      for (int c = 0; c < PW; ++c) wv[c] = a[(c >> 3) * 1024 + (c & 7) * 32];
    };
    load_piece(0);
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);  // this warp's TMEM lanes
    double r0 = 0.0, r1 = 0.0;  // sum_k L_ik z_k; the diagonal tile: the entries themselves
    const bool two = P.nrhs > 1;
    const double rhs0 = P.rhs[i], rhs1 = two ? P.rhs[P.Nc + i] : 0.0;
    int sq = P.rowsq[i];  // the row's squares so far
    bool live = true;
    auto wait = [&](uint64_t* bar, int parity) -> bool {
      const int r = wait_or_stop(bar, (uint32_t)parity, &s_stop);
      if (r == 2) s_abort = s_stop = 1;
      live = r == 0;
      return live;
    };
    int Xh[PW], Xl[PW];  // this row's entries of the current piece
    int Ph[PW], Pl[PW];  // and of the previous one
    // the row's own pivot, once its block is factored (kept here: the shared copies are overwritten two pieces on)
    long long D_own = 0;
    unsigned yh_own = 0, yl_own = 0;
    int sh_own = 0;
#pragma unroll 1
    for (int t = 0;; ++t) {
      const bool tail = t == np;  // only the last piece's leftovers
      const bool done = diag && warp < (t >> 1);  // the diagonal tile: every row of this warp is factored
      const bool was_done = diag && warp < ((t - 1) >> 1);
      const bool pivot = diag && warp == (t >> 1);
      long long T[PW];  // the row's right-hand sides B, in units of 2^-60
      if (t > 0 && !tail) {
        if (!wait(b_mma, (t - 1) & 1)) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
      }
      if (tail) {
      } else if (!done) {
        if (t > 0) {
#pragma unroll
          for (int c = 0; c < PW; ++c) T[c] = wv[c];
          drain_couplings(T, trow);
          asm volatile("tcgen05.fence::before_thread_sync;");
          __syncwarp();
          if (lane == 0) mbar_arrive(b_drained);
        } else {
#pragma unroll
          for (int c = 0; c < PW; ++c) T[c] = wv[c];
        }
#pragma unroll
        for (int c = 0; c < PW; ++c) T[c] = to_unit60((unsigned long long)T[c]);
        if (t + 1 < np) load_piece(t + 1);
      } else if (lane == 0) {
        mbar_arrive(b_drained);
      }
      PanelBlock& Lt = Ls[t & 1];
      if (pivot && !tail) {
        // The 16 x 16 diagonal block on the whole warp (rows below the block in
        // the same warp are solved on the way), four columns a round: within
        // the four each entry is taken off the next columns at once (the
        // pivot rows' entries by shuffles), then the four together off the
        // columns beyond (from shared memory), which move down by four.  A
        // rolled loop: unrolled whole, it is 50 KB of code that the
        // instruction fetch shares with the other warps' (a piece's pivots 14k
        // cycles; rolled, 9.6k to 11.3k of the piece's ~16k: 1.6k go to the
        // couplings' sums, 2.9k to the digits, the rest to the couplings themselves).
        // A non-positive pivot is remembered and what
        // follows it is discarded.
        const int base = (t & 1) * PW;
        const int c_own = lane - base;  // this row's index in the block; < 0: above, >= 16: below
        long long M[PW];                // with T: B = T + M 2^-30
#pragma unroll
        for (int k = 0; k < PW; ++k) M[k] = 0;
        int fail = PW;
#pragma unroll 1
        for (int b = 0; b < 4; ++b) {
          int xh[4], xl[4], nxh[4], nxl[4];
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            const int j = 4 * b + q;
            const long long Tj = T[q] + (M[q] >> 30);
            const long long D = __shfl_sync(0xffffffffu, Tj, base + j);
            if (D < 4 && fail == PW) fail = j;  // 2^-58 of 2^2e: far below what K's own rounding leaves of a pivot
            unsigned yh, yl;
            int sh;
            rsqrt_fixed(D, yh, yl, sh);
            sh = min(max(sh, 0), 28);  // discarded columns only
            scale_entry(Tj, yh, yl, sh, xh[q], xl[q]);
            if (c_own < j) xh[q] = xl[q] = 0;  // above the diagonal
            nxh[q] = -xh[q];
            nxl[q] = -xl[q];
            if (c_own == j) {
              yh_own = yh;
              yl_own = yl;
              sh_own = sh;
              D_own = D;
              Lt.y[j] = make_uint2(yh, yl);
              Lt.sh[j] = sh;
              s_D[t & 1][j] = D;
            }
#pragma unroll
            for (int k = q + 1; k < 4; ++k) {
              const int lh = __shfl_sync(0xffffffffu, xh[q], base + 4 * b + k);
              const int ll = __shfl_sync(0xffffffffu, xl[q], base + 4 * b + k);
              mac_entry(T[k], M[k], nxh[q], nxl[q], lh, ll);
            }
          }
          if (c_own >= 0 && c_own < PW) {
            int4* lx = reinterpret_cast<int4*>(&Lt.x[c_own][4 * b]);
            lx[0] = make_int4(xh[0], xl[0], xh[1], xl[1]);
            lx[1] = make_int4(xh[2], xl[2], xh[3], xl[3]);
          }
          shift_down<4>(Xh);
          shift_down<4>(Xl);
#pragma unroll
          for (int q = 0; q < 4; ++q) {
            Xh[PW - 4 + q] = xh[q];
            Xl[PW - 4 + q] = xl[q];
          }
          __syncwarp();
          if (b == 1 && lane == 0) mbar_arrive(b_half);
          const int4* lb = reinterpret_cast<const int4*>(&Lt.x[4 * b + 4][4 * b]);
#pragma unroll
          for (int g = 0; g < 3; ++g) {
            if (b < 3 - g) {  // the columns left: uniform
#pragma unroll
              for (int i = 4 * g; i < 4 * g + 4; ++i) {
                const int4 l0 = lb[i * (PW / 2)], l1 = lb[i * (PW / 2) + 1];
                T[i] = T[i + 4];
                M[i] = M[i + 4];
                mac_entry(T[i], M[i], nxh[0], nxl[0], l0.x, l0.y);
                mac_entry(T[i], M[i], nxh[1], nxl[1], l0.z, l0.w);
                mac_entry(T[i], M[i], nxh[2], nxl[2], l1.x, l1.y);
                mac_entry(T[i], M[i], nxh[3], nxl[3], l1.z, l1.w);
              }
            }
          }
        }
        // the block's rows, their own entries included: K_ii, or 4 and more beyond it if the pivot came round
        sq += squares8<0>(Xh) + squares8<8>(Xh);
        const unsigned over = (__ballot_sync(0xffffffffu, sq > SQ_LIMIT) >> base) & 0xFFFF;
        if (over) fail = min(fail, __ffs(over) - 1);
        if (fail < PW) {
          if (lane == 0) {
            P.status[0] = c0 + t * PW + fail + 1;  // LAPACK info: 1-based column
            P.status[1] = 1;
            s_stop = 1;
            __threadfence();
            for (int f = 0; f < 3; ++f) publish(&fl[f], FLAG_FAIL);
          }
          live = false;
          break;
        }
        // the right-hand-side warp has taken the previous block: no barrier's
        // phase can pass a warp that still waits for the one before
        if (t > 0 && !wait(b_z, (t - 1) & 1)) break;
        __syncwarp();
        if (lane == 0) mbar_arrive(b_blk);
      }
      // Two rounds around one copy of the leftovers' code: the pivot warp writes
      // its digits first, the others do the leftovers while they wait for the
      // pivots.
      bool out = false;
#pragma unroll 1
      for (int round = 0; round < 2; ++round) {
        if ((round == 1) == (pivot && !tail) && t > 0 && !was_done) {
          // the previous piece's leftovers, which nothing on the pivots' chain
          // waits for: the factor's entries for alpha and the adjoint, and the
          // right-hand sides' sum_k L'_ik z_k, z in 60-bit fixed point of the
          // piece's own scale
          const int tp = t - 1;
          if (P.keep_l) {
            // as they are, X = x 2^60: k_factor_doubles converts them where they are wanted
            const int c_own = diag ? rl - tp * PW : PW;
            if (c_own >= 0 && c_own < PW)  // the row's own L_jj = d d^-1/2
              P.ldiag[i] = fixed62_to_double(D_own, 2) * fixed62_to_double((long long)yh_own << 32 | yl_own, sh_own + kexp);
            long long* kp = reinterpret_cast<long long*>(krow) + (size_t)(tp * PW) * ld;
#pragma unroll
            for (int c = 0; c < PW; ++c) kp[(size_t)c * ld] = (long long)Ph[c] * (1LL << 30) + Pl[c];
          }
          if (!wait(b_z, tp & 1)) {
            out = true;
            break;
          }
          const PanelZ& Z = Zs[tp & 1];
          long long s = 0, m = 0;
#pragma unroll
          for (int c = 0; c < PW; ++c) {
            mac_entry(s, m, Ph[c], Pl[c], Z.x[0][c].x, Z.x[0][c].y);
          }
          r0 = fma(Z.scale[0], fixed62_to_double((s << 2) + (m >> 28)), r0);
          if (two) {
            s = m = 0;
#pragma unroll
            for (int c = 0; c < PW; ++c) {
              mac_entry(s, m, Ph[c], Pl[c], Z.x[1][c].x, Z.x[1][c].y);
            }
            r1 = fma(Z.scale[1], fixed62_to_double((s << 2) + (m >> 28)), r1);
          }
        }
        if (tail) break;
        if (round == 0) {
          if (!done && !pivot) {
            // x L'_tt^T = B: the first 8 columns, their part of the last 8, the last 8
            if (!wait(b_half, t & 1)) {
              out = true;
              break;
            }
            constexpr int HW = PW / 2;
#pragma unroll
            for (int k = 0; k < HW; ++k) {
              long long S = 0, M = 0;
              mac_row<0>(S, M, Xh, Xl, Lt, k, k);
              scale_entry(T[k] - S - (M >> 30), Lt.y[k].x, Lt.y[k].y, Lt.sh[k], Xh[k], Xl[k]);
            }
            long long M2[HW];
#pragma unroll
            for (int q = 0; q < HW; ++q) {
              long long S = 0;
              M2[q] = 0;
              mac_row<0>(S, M2[q], Xh, Xl, Lt, HW + q, HW);
              T[HW + q] -= S;
            }
            if (!wait(b_blk, t & 1)) {
              out = true;
              break;
            }
#pragma unroll
            for (int k = HW; k < PW; ++k) {
              long long S = 0;
              mac_row<HW>(S, M2[k - HW], Xh, Xl, Lt, k, k);
              scale_entry(T[k] - S - (M2[k - HW] >> 30), Lt.y[k].x, Lt.y[k].y, Lt.sh[k], Xh[k], Xl[k]);
            }
          }
          if (!done) {
            unsigned char* ad = As + t * PN_ACHUNK + tid * 16;
            unsigned char* gd = gdig + (size_t)(2 * t) * 2048;
            unsigned char* bd = Bs + t * PN_BCHUNK + (rl & 15) * 16;
            const bool own_b = diag && (rl >> 4) == t + 1;  // the diagonal tile's own B operand of the next piece
#pragma unroll
            for (int g = 0; g < 2; ++g) {
              uint4 d[NSLICE];
              digits8_packed(&Xh[g * 8], &Xl[g * 8], d);
#pragma unroll
              for (int q = 0; q < NSLICE; ++q) {
                if (t + 1 < NPIECE) *reinterpret_cast<uint4*>(ad + g * 2048 + q * 4096) = d[q];
                *reinterpret_cast<uint4*>(gd + (size_t)q * SLICE_BYTES + g * 2048) = d[q];
                if (own_b) *reinterpret_cast<uint4*>(bd + g * (NSLICE * PW * 16) + q * (PW * 16)) = d[q];
              }
            }
            asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // digits visible to the tensor cores
          }
          __syncwarp();
          if (lane == 0) mbar_arrive(b_digits);
          if (!done && !pivot) sq += squares8<0>(Xh) + squares8<8>(Xh);
        }
      }
      if (out || tail) break;
      if (pivot) {
        const int c_own = lane - (t & 1) * PW;
        if (c_own >= 0 && c_own < PW) {
          Rs[c_own] = rhs0 - r0;
          Rs[PW + c_own] = rhs1 - r1;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(b_rhs);
      }
#pragma unroll
      for (int c = 0; c < PW; ++c) {
        Ph[c] = Xh[c];
        Pl[c] = Xl[c];
      }
    }
    if (diag && live && P.keep_l) {
      // columns of the identity padding, which the pieces leave out
      for (int c = np * PW; c < NB; ++c) krow[(size_t)c * ld] = 0.0;
      if (rl >= np * PW) P.ldiag[i] = ldexp(0.5, kexp);
    }
    if (!diag && live) {
      P.rowsq[i] = min(sq, SQ_MAX);
      P.rhs[i] = rhs0 - r0;
      if (two) P.rhs[P.Nc + i] = rhs1 - r1;
    }
  } else if (warp == PN_MMA_WARP) {
    // ---------------- operand loads and MMA issue ----------------
    const uint64_t adesc = smem_desc(su32(As), 2048, 128);
    const uint64_t bdesc = smem_desc(su32(Bs), NSLICE * PW * 16, 128);
    // chunk c against the next piece's 16 rows: A plane q against B planes
    // 0 .. 6 - q stacked along N, levels q .. 6 in one instruction
    auto issue_chunk = [&](int c) {
#pragma unroll
      for (int q = 0; q < NSLICE; ++q)
        mma_f16_desc(tmem + (uint32_t)q * PW, adesc + (uint64_t)((c * PN_ACHUNK + q * 4096) >> 4),
                     bdesc + (uint64_t)((c * PN_BCHUNK) >> 4),
                     (1u << 4) | ((uint32_t)(PW * (NSLICE - q) >> 3) << 17) | ((128u >> 4) << 24),
                     (c == 0 && q == 0) ? 0u : 1u);
    };
    // the digits of rows 16 (t + 1) .. + 15 of the diagonal tile, chunk c
    auto load_chunk = [&](int t, int c) {
      const unsigned char* src = P.slices + (size_t)P.nt128 * NSLICE * SLICE_BYTES + (size_t)(t + 1) * PW * 16;
      for (int q = lane; q < (int)PN_BCHUNK / 16; q += 32) {
        const int row = q & 15, pl = (q >> 4) % NSLICE, g = (q >> 4) / NSLICE;
        cp_async16(Bs + c * PN_BCHUNK + q * 16, src + (size_t)pl * SLICE_BYTES + (size_t)(2 * c + g) * 2048 + row * 16);
      }
    };
    // a problem's counter, as the whole warp sees it: 0 reached, 1 failed, 2 gave up
    auto wait_flag = [&](int f, int t) -> int {
      int r = 0;
      if (lane == 0) {
        const int v = poll_flag(&fl[f], fbase + t + 1);
        r = v < 0 ? 2 : (v >= FLAG_FAIL ? 1 : 0);
      }
      __syncwarp();  // the other lanes' reads come after lane 0's acquire too
      return __shfl_sync(0xffffffffu, r, 0);
    };
    int st = 0;  // 1: the problem failed, 2: a wait gave up
#pragma unroll 1
    for (int t = 0; t < np && !st; ++t) {
      if (!diag) {
        if ((st = wait_flag(FLAG_L, t))) break;
        const unsigned char* pub = reinterpret_cast<const unsigned char*>(P.lpub + t);
        unsigned char* dst = reinterpret_cast<unsigned char*>(Ls + (t & 1));
        for (int q = lane; q < (int)PN_LBYTES / 16; q += 32) cp_async16(dst + q * 16, pub + q * 16);
        cp_async_wait();
        __syncwarp();
        if (lane == 0) {
          mbar_arrive(b_half);
          mbar_arrive(b_blk);
        }
      }
      if (t + 1 < np) {
        if (t > 0) {
          // earlier chunks against the next piece, while the rows are solved
          if ((st = wait_or_stop(b_mma, (t - 1) & 1, &s_stop))) break;  // the couplings of piece t have read Bs
          for (int c = 0; c < t; ++c) load_chunk(t, c);
          cp_async_wait();
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
          if ((st = wait_or_stop(b_drained, (t - 1) & 1, &s_stop))) break;
          asm volatile("tcgen05.fence::after_thread_sync;");
          if (lane == 0)
            for (int c = 0; c < t; ++c) issue_chunk(c);
          __syncwarp();
        }
        if (!diag) {
          if ((st = wait_flag(FLAG_D, t))) break;
          load_chunk(t, t);
          cp_async_wait();
          asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
          __syncwarp();
        }
        if ((st = wait_or_stop(b_digits, t & 1, &s_stop))) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        if (lane == 0) {
          issue_chunk(t);
          mma_commit(b_mma);
          // the row warps' digits, written to HBM before they arrived (release:
          // cumulative over what this warp has observed)
          if (diag) publish(&fl[FLAG_D], fbase + t + 1);
        }
        __syncwarp();
      } else if (!diag) {
        if ((st = wait_or_stop(b_digits, t & 1, &s_stop))) break;  // the rows have taken the previous z
      }
      if (!diag) {
        if ((st = wait_flag(FLAG_Z, t))) break;
        if (lane < (int)PN_ZBYTES / 16)
          cp_async16(reinterpret_cast<unsigned char*>(Zs + (t & 1)) + lane * 16,
                     reinterpret_cast<const unsigned char*>(P.zpub + t) + lane * 16);
        cp_async_wait();
        __syncwarp();
        if (lane == 0) mbar_arrive(b_z);
      }
    }
    if (st) {
      // the problem failed or a wait gave up: every warp falls out of its
      // waits, and no MMA still writes TMEM when it is freed
      if (st == 2) s_abort = 1;
      s_stop = 1;
    }
    __syncwarp();
    quiet = st != 0;
    if (quiet && lane == 0) drain_mmas(b_quiet);
  } else if (warp == PN_RHS_WARP && diag) {
    // ---------------- right-hand sides and log-determinant of the panel ----------------
    // lane j + 16 q: entry j of right-hand side q
    const int j = lane & 15;
    const bool have = lane < 16 || P.nrhs > 1;
    double prod = 1.0;  // product of the pivots' significands; their exponents add up in esum
    int esum = 0;
    const int ke = *P.kscale;
    bool ok = true;
#pragma unroll 1
    for (int t = 0; t < np; ++t) {
      int w = wait_or_stop(b_blk, t & 1, &s_stop);
      if (w == 2) s_abort = s_stop = 1;
      ok = w == 0;
      if (!ok) break;
      const PanelBlock& Lt = Ls[t & 1];
      const long long lb = __double_as_longlong(fixed62_to_double(s_D[t & 1][j], 2));
      {
        // publish the block (release: cumulative over what this warp has
        // observed, the pivot warp's stores before b_blk included)
        const uint4* src = reinterpret_cast<const uint4*>(&Lt);
        uint4* dst = reinterpret_cast<uint4*>(P.lpub + t);
        for (int q = lane; q < (int)PN_LBYTES / 16; q += 32) dst[q] = src[q];
        __syncwarp();
        if (lane == 0) publish(&fl[FLAG_L], fbase + t + 1);
      }
      // row j of the block, and 1 / L'_jj = y 2^(sh - 62), as doubles
      double lrow[PW];
#pragma unroll
      for (int c = 0; c < PW; ++c) {
        const int2 l = Lt.x[j][c];
        lrow[c] = fixed62_to_double(((long long)l.x * (1LL << 30) + l.y) * 4);
      }
      const double rdj = fixed62_to_double((long long)Lt.y[j].x << 32 | Lt.y[j].y, Lt.sh[j]);
      w = wait_or_stop(b_rhs, t & 1, &s_stop);
      if (w == 2) s_abort = s_stop = 1;
      ok = w == 0;
      if (!ok) break;
      double r = have ? Rs[lane] : 0.0, z = 0.0;
#pragma unroll
      for (int c = 0; c < PW; ++c) {
        const double b = __shfl_sync(0xffffffffu, r * rdj, (lane & 16) + c);
        if (j == c) z = b;
        r = fma(-b, lrow[c], r);
      }
      // z in fixed point of the piece's scale, 4 max |z| or more: then |sum x z| <= 1 in that
      // scale (16 entries, |x| of norm 1) and no 64-bit sum overflows; NaN and infinity go on through the scale
      int q = (int)((unsigned)__double2hiint(z) >> 20) & 0x7FF;
      for (int o = 8; o > 0; o >>= 1) q = max(q, __shfl_xor_sync(0xffffffffu, q, o));
      PanelZ& Z = Zs[t & 1];
      {
        bool nf = false;
        const long long X = (to_fixed62(z, q - 1020, &nf) + 2) >> 2;
        const int xh = (int)((X + (1LL << 29)) >> 30);
        const int2 v = make_int2(xh, (int)((unsigned)X - ((unsigned)xh << 30)));
        // 2^(q - 1020); beyond the double range the sums are infinite anyway
        const double sc = q == 0x7FF ? nan("") : __longlong_as_double((long long)min(q + 3, 2046) << 52);
        Z.x[lane >> 4][j] = v;
        P.zpub[t].x[lane >> 4][j] = v;
        if (j == 0) {
          Z.scale[lane >> 4] = sc;
          P.zpub[t].scale[lane >> 4] = sc;
        }
      }
      if (have) P.rhs[(size_t)(lane >> 4) * P.Nc + c0 + t * PW + j] = z;
      // every row warp has taken the previous z before this one is signalled
      w = wait_or_stop(b_digits, t & 1, &s_stop);
      if (w == 2) s_abort = s_stop = 1;
      ok = w == 0;
      if (!ok) break;
      __syncwarp();
      if (lane == 0) {
        mbar_arrive(b_z);
        publish(&fl[FLAG_Z], fbase + t + 1);
      }
      if (c0 + t * PW + j < P.N) {  // not the identity padding
        esum += (int)(lb >> 52) - 1023 + 2 * ke;
        prod *= __longlong_as_double((lb & 0xFFFFFFFFFFFFFLL) | 0x3FF0000000000000LL);
      }
    }
    if (ok) {
      for (int o = 8; o > 0; o >>= 1) {
        prod *= __shfl_xor_sync(0xffffffffu, prod, o);
        esum += __shfl_xor_sync(0xffffffffu, esum, o);
      }
      if (lane == 0) P.logdet_part[s] = 0.5 * (log(prod) + (double)esum * 0.69314718055994530942);  // sum of log L_jj
    }
  }
  __syncthreads();
  if (s_abort && warp == PN_MMA_WARP && lane == 0 && !quiet) drain_mmas(b_quiet);
  if (tid == 0 && s_abort) {
    // a bounded wait gave up: report, and release the problem's other CTAs
    atomicExch(&P.status[2], 1);
    __threadfence();
    for (int f = 0; f < 3; ++f) publish(&fl[f], FLAG_FAIL);
  }
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == PN_MMA_WARP) __syncwarp();
  if (warp == PN_MMA_WARP)
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(PN_TMEM_COLS));
}

// ---------------------------------------------------------------------------
// the rows of a panel whose diagonal tiles are done (batches): the same pieces,
// arranged for throughput.  A row tile's integer work (~2.1k instructions per
// piece and warp at 2.5 cycles of issue) keeps one warp per SM quarter only half
// busy -- it waits for its couplings, loads and barriers -- so two CTAs share
// an SM.  That leaves 113 KB each: the digits of the current piece stay in
// shared memory, those of the earlier pieces come back from the L2 by TMA (21
// chunks of 28 KB per tile) through a 2-stage ring, and are multiplied into the
// other one of two TMEM accumulators while the rows are solved.  One thread
// issues the copies and the MMAs.  Every word is the one k_panel computes: the
// sums are exact integers.  All panels of 40 problems of N = 4000: 9.3 -> 6.8
// ms, of 16 of N = 10000: 21.8 -> 16.6 ms, of 50 of N = 2000: 3.3 -> 2.6 ms.
// ---------------------------------------------------------------------------
namespace {
constexpr int PR_THREADS = 160;
constexpr uint32_t PR_STAGE = PN_ACHUNK + PN_BCHUNK;
constexpr uint32_t PR_OFF_RING = PN_ACHUNK;
constexpr uint32_t PR_OFF_B = PR_OFF_RING + 2 * PR_STAGE;  // [2]: B operand of the current piece's own chunk
constexpr uint32_t PR_OFF_L = PR_OFF_B + 2 * PN_BCHUNK;
constexpr uint32_t PR_OFF_Z = PR_OFF_L + 2 * PN_LBYTES;
constexpr uint32_t PR_OFF_BAR = PR_OFF_Z + NPIECE * PN_ZBYTES;
constexpr uint32_t PR_SMEM = PR_OFF_BAR + 96;
static_assert(2 * (PR_SMEM + 2048) <= 228 * 1024, "two CTAs per SM");
static_assert(PN_LBYTES % 16 == 0 && PR_OFF_L % 16 == 0 && PR_STAGE % 128 == 0 && PR_OFF_B % 128 == 0, "bulk and TMA alignment");
}  // namespace

__global__ void __launch_bounds__(PR_THREADS, 2)
    k_panel_rows(const Prob* __restrict__ probs, int s, const int* __restrict__ order) {
  extern __shared__ __align__(1024) unsigned char smr[];
  unsigned char* As = smr;                 // the current piece's digits
  unsigned char* ring = smr + PR_OFF_RING;  // [2]: an earlier piece's digits and its B operand
  unsigned char* Bs = smr + PR_OFF_B;
  PanelBlock* Ls = reinterpret_cast<PanelBlock*>(smr + PR_OFF_L);  // [2]
  PanelZ* Zs = reinterpret_cast<PanelZ*>(smr + PR_OFF_Z);          // [NPIECE]
  uint64_t* b_mma = reinterpret_cast<uint64_t*>(smr + PR_OFF_BAR);  // a piece's couplings are in TMEM
  uint64_t* b_digits = b_mma + 1;                                   // its digits are in As and in HBM, its couplings drained
  uint64_t* b_quiet = b_mma + 2;                                    // quiescing before an early exit
  uint64_t* b_blk = b_mma + 3;                                      // [2]: Ls
  uint64_t* b_own = b_mma + 5;                                      // [2]: Bs
  uint64_t* full = b_mma + 7;                                       // [2]: ring
  uint64_t* empty = b_mma + 9;                                      // [2]
  __shared__ int s_skip, s_stop, s_abort;
  __shared__ uint32_t s_tmem;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const int id = order[blockIdx.x], p = id >> 16, ti = id & 0xFFFF;
  const Prob& P = probs[p];
  if (tid == 0) {
    s_skip = *(volatile int*)&P.status[1];  // one read: the exit below is block-uniform
    s_stop = 0;
    s_abort = 0;
    mbar_init(b_mma, 1);
    mbar_init(b_digits, 4);
    mbar_init(b_quiet, 1);
    for (int k = 0; k < 2; ++k) {
      mbar_init(&b_blk[k], 1);
      mbar_init(&b_own[k], 1);
      mbar_init(&full[k], 1);
      mbar_init(&empty[k], 1);
    }
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  for (int q = tid; q < NPIECE * (int)PN_ZBYTES / 16; q += PR_THREADS)
    reinterpret_cast<uint4*>(Zs)[q] = reinterpret_cast<const uint4*>(P.zpub)[q];
  __syncthreads();
  if (s_skip) return;
  if (warp == 4) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 256;" ::"r"(su32(&s_tmem)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tmem = s_tmem;
  uint32_t issued = 0;  // the issuing thread: ring loads

  if (warp < 4) {
    // ---------------- row warps: one thread per row ----------------
    const int rl = tid, i = ti * NB + rl;
    const long long* acc0 = P.acc + acc_tile(ti, 2 * s, P.nt128) * ACC_TILE_ELEMS + acc_elem(rl, 0);
    const long long* acc1 = P.acc + acc_tile(ti, 2 * s + 1, P.nt128) * ACC_TILE_ELEMS + acc_elem(rl, 0);
    unsigned char* gdig = P.slices + (size_t)ti * NSLICE * SLICE_BYTES + (size_t)rl * 16;
    const uint32_t trow = tmem + ((uint32_t)(warp * 32) << 16);
    const bool two = P.nrhs > 1;
    double r0 = 0.0, r1 = 0.0;  // sum_k L'_ik z_k
    int sq = 0;                 // the row's squares
    bool live = true;
    auto wait = [&](uint64_t* bar, int parity) -> bool {
      const int r = wait_or_stop(bar, (uint32_t)parity, &s_stop);
      if (r == 2) s_abort = s_stop = 1;
      live = r == 0;
      return live;
    };
    long long T[PW];
    auto load_piece = [&](int t) {
      const long long* a = (t < 4 ? acc0 : acc1) + (size_t)(t & 3) * 2048;  // 16 columns: 2 groups of 8
#pragma unroll
      for (int c = 0; c < PW; ++c) T[c] = a[(c >> 3) * 1024 + (c & 7) * 32];
    };
    load_piece(0);
#pragma unroll 1
    for (int t = 0; t < NPIECE; ++t) {
      if (t > 0) {
        if (!wait(b_mma, (t - 1) & 1)) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        drain_couplings(T, trow + (uint32_t)((t & 1) * PN_TMEM_COLS));
        asm volatile("tcgen05.fence::before_thread_sync;");
      }
#pragma unroll
      for (int c = 0; c < PW; ++c) T[c] = to_unit60((unsigned long long)T[c]);
      if (!wait(&b_blk[t & 1], (t >> 1) & 1)) break;
      const PanelBlock& Lt = Ls[t & 1];
      int Xh[PW], Xl[PW];
#pragma unroll
      for (int k = 0; k < PW; ++k) {
        long long S = 0, M = 0;
        mac_row<0>(S, M, Xh, Xl, Lt, k, k);
        scale_entry(T[k] - S - (M >> 30), Lt.y[k].x, Lt.y[k].y, Lt.sh[k], Xh[k], Xl[k]);
      }
      if (t + 1 < NPIECE) load_piece(t + 1);
      unsigned char* ad = As + rl * 16;
      unsigned char* gd = gdig + (size_t)(2 * t) * 2048;
#pragma unroll
      for (int g = 0; g < 2; ++g) {
        uint4 d[NSLICE];
        digits8_packed(&Xh[g * 8], &Xl[g * 8], d);
#pragma unroll
        for (int q = 0; q < NSLICE; ++q) {
          if (t + 1 < NPIECE) *reinterpret_cast<uint4*>(ad + g * 2048 + q * 4096) = d[q];
          *reinterpret_cast<uint4*>(gd + (size_t)q * SLICE_BYTES + g * 2048) = d[q];
        }
      }
      asm volatile("fence.proxy.async;" ::: "memory");  // digits visible to the MMAs and to the TMA reloads
      __syncwarp();
      if (lane == 0) mbar_arrive(b_digits);
      sq += squares8<0>(Xh) + squares8<8>(Xh);
      // the right-hand sides: sum_k L'_ik z_k, z in 60-bit fixed point of the piece's scale
      const PanelZ& Z = Zs[t];
      long long S = 0, M = 0;
#pragma unroll
      for (int c = 0; c < PW; ++c) mac_entry(S, M, Xh[c], Xl[c], Z.x[0][c].x, Z.x[0][c].y);
      r0 = fma(Z.scale[0], fixed62_to_double((S << 2) + (M >> 28)), r0);
      if (two) {
        S = M = 0;
#pragma unroll
        for (int c = 0; c < PW; ++c) mac_entry(S, M, Xh[c], Xl[c], Z.x[1][c].x, Z.x[1][c].y);
        r1 = fma(Z.scale[1], fixed62_to_double((S << 2) + (M >> 28)), r1);
      }
    }
    if (live) {
      P.rowsq[i] = min(P.rowsq[i] + sq, SQ_MAX);
      P.rhs[i] -= r0;
      if (two) P.rhs[P.Nc + i] -= r1;
    }
  } else if (lane == 0) {
    // ---------------- copies and MMA issue ----------------
    const void* ma = P.tmap_a;
    const void* mb = P.tmap_b16;
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(ma) : "memory");
    asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(mb) : "memory");
    bool ok = true;
    auto wait = [&](uint64_t* bar, uint32_t parity) -> bool {
      if (ok) {
        ok = false;
        for (int it = 0; it < (1 << 22) && !ok && !*(volatile int*)&s_stop; ++it) ok = mbar_wait_n(bar, parity, 1);
        if (!ok && !*(volatile int*)&s_stop) s_abort = 1;
      }
      return ok;
    };
    auto load_block = [&](int t) {
      mbar_expect_tx(&b_blk[t & 1], PN_LBYTES);
      bulk_g2s(Ls + (t & 1), P.lpub + t, PN_LBYTES, &b_blk[t & 1]);
    };
    // B operand: rows 16 t .. + 15 of the diagonal tile, chunk c
    auto load_b = [&](unsigned char* dst, int t, int c, uint64_t* bar) {
      tma_load_5d(dst, mb, (t & 1) * 128, t >> 1, 0, 2 * c, P.nt128, bar);
    };
    auto issue = [&](uint32_t acc, unsigned char* a, unsigned char* b, bool first) {
      const uint64_t ad = smem_desc(su32(a), 2048, 128), bd = smem_desc(su32(b), NSLICE * PW * 16, 128);
#pragma unroll
      for (int q = 0; q < NSLICE; ++q)
        mma_f16_desc(acc + (uint32_t)q * PW, ad + (uint64_t)((q * 4096) >> 4), bd,
                     (1u << 4) | ((uint32_t)(PW * (NSLICE - q) >> 3) << 17) | ((128u >> 4) << 24),
                     first && q == 0 ? 0u : 1u);
    };
    load_block(0);
    load_block(1);
    uint32_t g = 0;  // ring loads consumed
#pragma unroll 1
    for (int t = 1; t < NPIECE && ok; ++t) {  // the couplings of piece t
      const uint32_t acc = tmem + (uint32_t)((t & 1) * PN_TMEM_COLS);
      unsigned char* bo = Bs + (t & 1) * PN_BCHUNK;
      const int older = t - 1;  // chunks 0 .. t - 2 through the ring, chunk t - 1 from As
      // the digits of piece t - 2 were waited for: its couplings are drained,
      // its accumulator and its B slot free
      mbar_expect_tx(&b_own[t & 1], PN_BCHUNK);
      load_b(bo, t, t - 1, &b_own[t & 1]);
      auto load_older = [&](int c) {
        const uint32_t st = issued & 1;
        if (issued >= 2 && !wait(&empty[st], ((issued >> 1) & 1) ^ 1)) return;
        unsigned char* dst = ring + st * PR_STAGE;
        mbar_expect_tx(&full[st], PR_STAGE);
        tma_load_5d(dst, ma, 0, 0, 2 * c, 0, ti, &full[st]);
        load_b(dst + PN_ACHUNK, t, c, &full[st]);
        ++issued;
      };
      if (older > 0) load_older(0);
      if (older > 1) load_older(1);
#pragma unroll 1
      for (int c = 0; c < older && ok; ++c, ++g) {
        const uint32_t st = g & 1;
        if (!wait(&full[st], (g >> 1) & 1)) break;
        asm volatile("tcgen05.fence::after_thread_sync;");
        issue(acc, ring + st * PR_STAGE, ring + st * PR_STAGE + PN_ACHUNK, c == 0);
        mma_commit(&empty[st]);
        if (c + 2 < older) load_older(c + 2);
      }
      if (!wait(&b_own[t & 1], (uint32_t)((t - (t & 1 ? 1 : 2)) >> 1) & 1)) break;
      if (!wait(b_digits, (uint32_t)(t - 1) & 1)) break;
      asm volatile("tcgen05.fence::after_thread_sync;");
      asm volatile("fence.proxy.async;" ::: "memory");
      issue(acc, As, bo, older == 0);
      mma_commit(b_mma);
      if (t + 1 < NPIECE) load_block(t + 1);  // the rows are done with block t - 1
    }
    if (!ok) s_stop = 1;
  }
  __syncthreads();
  if (s_stop) {
    // a bounded wait gave up: the copies and MMAs this CTA issued finish
    // (bounded waits) before it frees its TMEM and exits
    if (warp == 4 && lane == 0) {
      drain_ring(full, 2, issued);
      drain_mmas(b_quiet);
      for (int k = 0; k < 2; ++k) {
        // either phase of these two-deep buffers may be the one in flight
        mbar_wait_n(&b_blk[k], 0, 1 << 16);
        mbar_wait_n(&b_blk[k], 1, 1 << 16);
        mbar_wait_n(&b_own[k], 0, 1 << 16);
        mbar_wait_n(&b_own[k], 1, 1 << 16);
      }
    }
    if (tid == 0 && s_abort) atomicExch(&P.status[2], 1);
    __syncthreads();
  }
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == 4) {
    __syncwarp();
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 256;" ::"r"(tmem));
  }
}

// ---------------------------------------------------------------------------
// the factor the panels left in K (lower triangle, X = L' 2^60, its diagonal in
// ldiag) as doubles, in place: only alpha and the adjoint read it, and on the
// panels' chain the conversions cost 1.2k cycles a piece.  One CTA per 128 x 128
// tile
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_factor_doubles(const Prob* __restrict__ pp) {
  const Prob& P = *pp;
  const int ti = blockIdx.x, tj = blockIdx.y;
  if (ti < tj || P.status[1]) return;
  const size_t ld = (size_t)P.ld;
  const int kexp = *P.kscale, i = ti * NB + (threadIdx.x & 127);
#pragma unroll
  for (int c = 0; c < 8; ++c) {
    const int j = tj * NB + blockIdx.z * 16 + (threadIdx.x >> 7) * 8 + c;
    double* k = P.K + (size_t)j * ld + i;
    const double x = fixed62_to_double(__double_as_longlong(*k) * 4, kexp);
    *k = i > j ? x : (i == j ? P.ldiag[i] : 0.0);
  }
}

cudaError_t launch_factor_doubles(const Prob* prob, int nt128, cudaStream_t s) {
  k_factor_doubles<<<dim3(nt128, nt128, NB / 16), 256, 0, s>>>(prob);
  return cudaGetLastError();
}

// Rows per CTA: 128, or 64 or 32 while that still gives every tile an SM of
// its own: a row tile's chain is shorter on four SMs than on one, and once the
// tiles outnumber the SMs, splitting them only repeats the per-CTA work.
cudaError_t launch_panel(const Prob* probs, int step, const int* order, int ndiag, int total_tiles, int* counter,
                         int* flags, int num_sms, cudaStream_t s) {
  cudaError_t e = ensure_smem_attr((const void*)k_panel, SMEM_PANEL, PN_SMEM);
  if (e != cudaSuccess) return e;
  if (ndiag <= 0) return cudaSuccess;
  const int rest = total_tiles - ndiag;
  int sh = 0;
  while (sh < 2 && ndiag + (rest << (sh + 1)) <= num_sms) ++sh;
  k_panel<<<ndiag + (rest << sh), PN_THREADS, PN_SMEM, s>>>(probs, step, order, ndiag, sh, counter, flags);
  return cudaGetLastError();
}

cudaError_t launch_panel_rows(const Prob* probs, int step, const int* order, int ntiles, cudaStream_t s) {
  cudaError_t e = ensure_smem_attr((const void*)k_panel_rows, SMEM_PANEL_ROWS, PR_SMEM);
  if (e != cudaSuccess || ntiles <= 0) return e;
  k_panel_rows<<<ntiles, PR_THREADS, PR_SMEM, s>>>(probs, step, order);
  return cudaGetLastError();
}

}  // namespace fgpu
