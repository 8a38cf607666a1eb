// Kernel-matrix build on the tensor cores (tensor-core mode, kernels whose
// leaves are rbf, periodic, linear or constant with at most two rbf/periodic
// leaves).
//
// Both rbf and periodic leaves are exp(-|f_i - f_j|^2 / 2) of a per-leaf
// feature vector: f = sqrt(l) (x - mean) for rbf (stationary_kernel.f90:
// 101-122), f = (cos x, sin x) / exp(theta) per dimension for periodic
// (periodic_kernel.f90:181-206, since 2 sin^2(d/2) = 1 - cos d).  The
// squared distance is formed exactly in integers:
//
//  * Each leaf gets a power-of-two scale 2^s >= max |f| (from the per-plane
//    maxima of |x|, so it needs no reduction); f 2^-s is rounded to 55
//    fractional bits and split into 7 signed base-256 digits, one fp16 plane
//    per digit, written into the (otherwise idle) digit-plane buffer of the
//    factorisation at k offset koff.
//  * tcgen05.mma kind::f16 over the leaf's k range gives 8 exact level sums
//    S_L, L = p + q <= 7, of <f_i, f_j> (the same exactness argument as the
//    trailing update: at most 7 pairs x 128 terms x 129^2 < 2^24).  With
//    f 2^-s = sum_p d_p 2^(-7 - 8p), sum_L S_L 2^(56 - 8L) = <f_i, f_j>
//    2^(70 - 2s) up to the dropped levels L > 7 (below 2^-54 of 2^2s, under
//    the digits' own rounding), which the epilogue rounds to
//    W_ij = <f_i, f_j> 2^(u - 2 - 2s) (u = 60 - ceil(log2 nf): 4 max W < 2^61).
//    The 8 levels of a 128 x 64 tile fill the 512 TMEM columns.
//  * E = W_ii + W_jj - 2 W_ij (W_ii from the same digits, computed
//    exactly when the digits are written) is |f_i - f_j|^2 2^(u - 2 - 2s):
//    zero on the diagonal, and exp(-E 2^(2s + 1 - u)) is evaluated by the
//    fixed-point exponential straight from the integer (the leaf-scale form
//    iexp_fixed_tab: a fixed binary point, two 1024-entry tables in shared
//    memory, a degree-2 polynomial).
//
// The leaf values combine through the kernel expression, which is
// multilinear in the (at most two) distance leaves: k = a + b v0 + c v1 +
// d v0 v1, with a..d from the constant / linear leaves (one thread per
// problem, before the build).  The persistent kernel has the update's
// structure: TMA producer warp, MMA warp, 16 epilogue warps (the epilogue's
// integer work is what bounds the kernel, so it gets the warps); one pass per
// distance leaf per 128 x 64 tile, the first leaf's values kept in shared
// memory for the second pass.  FP64 instructions run at 2 lanes per cycle
// per SM on this part (FP32: 128), so one leaf, a sum of two and a product of
// two combine in fixed point (k_prep decides which, once per problem), and the
// nugget goes onto the one diagonal entry afterwards.
#include "../../include/fgpu.h"
#include "fgpu_internal.h"
#include "iexp.cuh"
#include "tc_common.cuh"

#include <cmath>

namespace fgpu {

namespace {

constexpr int NLEV = 8;  // digit-pair levels p + q = 0..7
enum Form { FORM_FP64 = 0, FORM_SUM = 1, FORM_PROD = 2 };  // how the leaves' values combine (Prob::fscale[2])

// W = round(sum_L S_L 2^(u - 16 - 8L)) from the 8 exact level sums (48 <= u <= 63)
__device__ __forceinline__ long long assemble_w(const int S[NLEV], int u) {
  const long long H = (long long)S[0] * (1LL << 32) + (long long)S[1] * (1LL << 24) + (long long)S[2] * 65536 +
                      (long long)S[3] * 256 + S[4];
  const long long Lo = (long long)S[5] * 65536 + (long long)S[6] * 256 + S[7];
  return (long long)((unsigned long long)H << (u - 48)) + ((Lo + (1LL << (71 - u))) >> (72 - u));
}

// The same W from the magic-add bits b_L = 0x4B400000 + S_L of level sums
// with |S_L| < 2^22 (level_bits): adjacent levels pair up in 32 bits
// (b_L 256 + b_(L+1) = (S_L + 2^22) 256 + (S_(L+1) + 2^22) + 0x4B000000 <
// 2^32, the top byte of b_L leaving modulo 2^32) and the offsets leave as two
// constants, one for the top five levels and one for the last three.
constexpr long long BUILD_BIAS_H = (1LL << 22) * 0x0101010101LL + 0x4B000000LL * ((1LL << 24) + (1LL << 8) + 1);
constexpr long long BUILD_BIAS_LO = (1LL << 22) * 0x010101LL + 0x4B000000LL * ((1LL << 8) + 1);
// (the first of them once per row and pass: this is W + (BUILD_BIAS_H << (u - 48)), modulo 2^64)
__device__ __forceinline__ long long assemble_w_bits(const uint32_t b[NLEV], int u) {
  const uint32_t p01 = b[0] * 256u + b[1];
  const uint32_t p23 = b[2] * 256u + b[3];
  const uint32_t p56 = b[5] * 256u + b[6];
  // sum_{L<=4} S_L 256^(4-L) + BUILD_BIAS_H
  const unsigned long long H = ((unsigned long long)p01 << 24) + ((unsigned long long)p23 << 8) + b[4];
  const long long Lo = (long long)(((unsigned long long)p56 << 8) + b[7]);
  return (long long)((H << (u - 48)) + (unsigned long long)((Lo + ((1LL << (71 - u)) - BUILD_BIAS_LO)) >> (72 - u)));
}

__device__ __forceinline__ void tmem_ldw(uint32_t (&v)[8], uint32_t addr) { tmem_ld8(v, addr); }
__device__ __forceinline__ void tmem_ldw(uint32_t (&v)[4], uint32_t addr) {
  asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0,%1,%2,%3}, [%4];"
               : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3])
               : "r"(addr));
}

}  // namespace

// ---------------------------------------------------------------------------
// preparation of an evaluation, one CTA per 128 points: the features' weights,
// the problem's scale, the right-hand sides, the scaled features and, for the
// tensor-core build, their digit planes and exact self products.
// grid (nt128, nprob) x (128, PREP_Y) threads: the digits of a point's groups of 8
// features, and the right-hand sides, side by side (one thread per point: 20
// us for a lone problem of 500 points and 12 features, now 14; 31 with 24
// features, now 17)
//
// An exponential is ~50 FP64 instructions of 64 cycles each on this GPU, so each
// weight is formed once per CTA, a thread per parameter, and not by every
// point (prep and digits as two kernels with an exponential per point and
// feature, and a serial one per leaf: 13 + 26 us for a lone problem of 500
// points, 29 + 57 us at N = 4000).
// ---------------------------------------------------------------------------
constexpr int PREP_Y = 4;
__global__ void __launch_bounds__(NB * PREP_Y) k_prep(const Prob* __restrict__ probs) {
  const Prob& P = probs[blockIdx.y];
  const int rb = blockIdx.x;
  if (P.mode != 1 || rb >= P.nt128) return;
  const Spec& sp = *P.spec;
  const int tid = threadIdx.x, y = threadIdx.y, i = rb * NB + tid;
  const size_t nc = (size_t)P.Nc;
  __shared__ double w[MAX_PARAMS];  // rbf, rbf-cyclic sqrt(exp(theta)), periodic 1 / exp(theta), linear 1 / c, constant theta
  int form = FORM_FP64;  // thread 0
  __shared__ int s_e[2], s_k;
  __shared__ bool s_huge[MAX_LEAF];
  __shared__ long long s_mul[MAX_PLANES];
  __shared__ int s_lev[2][PREP_Y][NLEV][NB];
  for (int q = y * NB + tid; q < sp.nkparams; q += NB * PREP_Y) {
    int type = L_CONSTANT;
    for (int l = 0; l < sp.nleaf; ++l) {
      const int cnt = sp.leaf[l].type == L_CONSTANT ? 1 : sp.leaf[l].n;
      if (q >= sp.leaf[l].param0 && q < sp.leaf[l].param0 + cnt) type = sp.leaf[l].type;
    }
    const double t = P.theta[q];
    // linear_kernel.f90:70-76, order 0: sum_k 1 / exp(-theta_k); constant.f90:62-68
    w[q] = type == L_CONSTANT ? t : 1.0;
    if (type != L_CONSTANT) {
      const bool half = type == L_RBF || type == L_RBF_CYCLIC;
      const double x = exp(half ? 0.5 * t : (type == L_LINEAR ? -t : t));
      w[q] = half ? x : 1.0 / x;
    }
  }
  __syncthreads();
  if (y > 0) {
  } else if (tid >= 64) {
    // scale of distance leaf d, 2^s > max |f| over every point (from the per-plane maxima)
    const int d = (tid - 64) >> 5, lane = tid & 31;
    if (sp.tc_build && d < sp.ndot) {
      const Leaf& L = sp.leaf[sp.dot_leaf[d]];
      const int per = L.type == L_PERIODIC ? 2 : 1;
      double m = 0.0;
      for (int k = lane; k < per * L.n; k += 32) m = fmax(m, w[L.param0 + k / per] * P.plane_max[L.plane0 + k]);
      for (int o = 16; o > 0; o >>= 1) m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
      if (lane == 0) {
        s_e[d] = m == 0.0 ? 0 : (int)((__double_as_longlong(m) >> 52) & 0x7FF) - 1022;
        if (rb == 0) P.fscale[d] = s_e[d];
      }
    }
    // the dot-product build's constants.  rbf-cyclic: |weighted difference| <= m <
    // 2^q; in units of 2^-t, t = 56 while that leaves the factors below 2^62
    // (q <= 5, i.e. weights e^theta up to 100 for a wrapped feature)
    for (int l = d; !sp.tc_build && l < sp.nleaf; l += 2) {
      const Leaf& L = sp.leaf[l];
      double m = 0.0, c = 0.0;
      bool huge = false;  // or NaN, which fmax passes over
      for (int k = lane; k < L.n; k += 32) {
        const double u = w[L.param0 + k];
        huge |= !(u < 0x1p900);
        if (L.type == L_RBF_CYCLIC)
          m = fmax(m, u * (0.5 * P.plane_max[L.plane0 + k]));
        else
          c += L.type == L_PERIODIC ? u * u : u;
      }
      for (int o = 16; o > 0; o >>= 1) {
        m = fmax(m, __shfl_xor_sync(0xffffffffu, m, o));
        c += __shfl_xor_sync(0xffffffffu, c, o);
      }
      const int q = m == 0.0 ? 0 : (int)((__double_as_longlong(m) >> 52) & 0x7FF) - 1022;
      const int t = 56 - max(0, q - 5);
      huge = __any_sync(0xffffffffu, huge || !(m < 0x1p900));
      if (lane == 0) {
        s_huge[l] = huge;
        if (rb == 0) {
          P.dotc->leaf_c[l] = L.type == L_CONSTANT ? w[L.param0] : c;
          P.dotc->unit[l] = t;
          P.dotc->clamp[l] = q > 4;
        }
      }
      if (L.type == L_RBF_CYCLIC)
        for (int k = lane; k < L.n; k += 32) {
          // sqrt(l) to l's own rounding, its product with g to the factor's unit
          const double u = w[L.param0 + k], g = P.plane_max[L.plane0 + k], ug = u * g;
          const double l = exp(P.theta[L.param0 + k]);
          const double e = u > 0.0 && l < INFINITY ? fma(fma(-u, u, l) / (2.0 * u), g, fma(u, g, -ug)) : 0.0;
          const long long f = llrint(ldexp(ug, t)) + llrint(ldexp(e, t));
          s_mul[L.plane0 + k] = f;
          if (rb == 0) P.dotc->mul[L.plane0 + k] = make_int2((int)(f >> 32), (int)((unsigned)f >> 1));
        }
    }
  } else if (tid == 0) {
    // the kernel expression in the (at most two) distance leaves of the
    // tensor-core build, c0 + c1 v0 + c2 v1 + c3 v0 v1; with other leaves only
    // its value at zero distance, in c0
    double stk[MAX_POST][4];
    int top = 0;
    for (int tk = 0; tk < sp.npost; ++tk) {
      const int tok = sp.post[tk];
      if (tok >= 0) {
        const Leaf& L = sp.leaf[tok];
        double c[4] = {0.0, 0.0, 0.0, 0.0};
        if (L.type == L_LINEAR) {
          for (int k = 0; k < L.n; ++k) c[0] += w[L.param0 + k];
        } else if (L.type == L_CONSTANT) {
          c[0] = w[L.param0];
        } else if (sp.tc_build) {
          c[tok == sp.dot_leaf[0] ? 1 : 2] = 1.0;
        } else {
          c[0] = 1.0;
        }
        for (int q = 0; q < 4; ++q) stk[top][q] = c[q];
        ++top;
      } else {
        const double* y = stk[--top];
        double* x = stk[top - 1];
        if (tok == P_SUM) {
          for (int q = 0; q < 4; ++q) x[q] += y[q];
        } else if (sp.tc_build) {  // each leaf occurs once: no squared terms
          const double c0 = x[0] * y[0];
          const double c1 = x[0] * y[1] + x[1] * y[0];
          const double c2 = x[0] * y[2] + x[2] * y[0];
          const double c3 = x[0] * y[3] + x[3] * y[0] + x[1] * y[2] + x[2] * y[1];
          x[0] = c0;
          x[1] = c1;
          x[2] = c2;
          x[3] = c3;
        } else {
          x[0] *= y[0];
        }
      }
    }
    const double* c = stk[0];
    if (rb == 0 && sp.tc_build)
      for (int q = 0; q < 4; ++q) P.fcoef[q] = c[q];
    form = c[0] != 0.0                                                             ? FORM_FP64
           : c[3] == 0.0 && c[1] == 1.0 && (sp.ndot == 1 || c[2] == 1.0)           ? FORM_SUM
           : sp.ndot == 2 && c[1] == 0.0 && c[2] == 0.0 && c[3] == 1.0             ? FORM_PROD
                                                                                   : FORM_FP64;
    // the scale 2^e > sqrt(K_ii): the kernels are stationary, so K_ii is one
    // value, the expression with every distance leaf at 1, plus the nugget
    const double d = (sp.tc_build ? (stk[0][3] + stk[0][2]) + (stk[0][1] + stk[0][0]) : stk[0][0]) +
                     (P.optimise_noise ? P.theta[sp.nkparams] : P.noise);
    int e = 0;
    if (d > 0.0 && d < INFINITY) frexp(sqrt(d) * (1.0 + 0x1p-20), &e);  // sqrt(K_ii) (1 + 2^-20) < 2^e
    s_k = e;
    if (rb == 0) P.kscale[0] = e;
  }
  __syncthreads();
  if (rb == 0 && tid == 0 && y == 0 && sp.tc_build) {
    // fixed point throughout (K_ii >= 1, so e >= 1 unless the nugget is
    // negative), with scales in the exponential's common form
    bool fixed = s_k >= 1;
    for (int l = 0; l < sp.ndot; ++l) fixed &= iexp_common(iexp_scale(2 * s_e[l] + 1 - sp.dot_u[l]));
    P.fscale[2] = fixed ? form : FORM_FP64;
  }
  if (y == PREP_Y - 1) {
    // right-hand sides: y - mu (marginal), or y and 1 (concentrated), in the factor's scale; zero on the padding
    const double u = ldexp(1.0, -s_k);
    P.rhs[i] = i < P.N ? u * (P.likelihood == 1 ? P.y[i] : P.y[i] - P.mu[i]) : 0.0;
    if (P.nrhs > 1) P.rhs[nc + i] = i < P.N ? u : 0.0;
    P.rowsq[i] = 0;
  }
  if (!sp.tc_build) {
    // the dot-product build's scaled planes and rbf norms (the workspace is not
    // cleared between evaluations: norms of other leaves are zeroed here)
    __shared__ double s_norm[PREP_Y][NB];
    for (int l = 0; l < MAX_LEAF; ++l) {
      double a = 0.0;
      if (l < sp.nleaf) {
        const Leaf& L = sp.leaf[l];
        const int per = L.type == L_PERIODIC ? 2 : 1;
        const int cnt = L.type == L_LINEAR || L.type == L_CONSTANT ? 0 : per * L.n;
        for (int k = y; k < cnt; k += PREP_Y) {
          const size_t o = (size_t)(L.plane0 + k) * nc + i;
          if (L.type == L_RBF_CYCLIC) {
            // integers: fractions of a turn as they are, the others in the leaf's unit; a
            // point (or a leaf) that is not finite is marked in its norm
            const long long u = __double_as_longlong(P.planes[o]), f = s_mul[L.plane0 + k];
            const long long F = __mul64hi(u, f) + (long long)(((unsigned long long)u * (unsigned long long)f) >> 63);
            P.splanes[o] = __longlong_as_double(sp.cyclic[L.plane0 + k] ? u : F);
            if (u == (long long)TURN_NOT_FINITE || s_huge[l]) a = 1.0;
            continue;
          }
          const double u = w[L.param0 + k / per] * P.planes[o];
          P.splanes[o] = u;
          if (L.type == L_RBF) a = fma(u, u, a);
        }
      }
      if (l < sp.nleaf) {
        s_norm[y][tid] = a;
        __syncthreads();
        a = (s_norm[0][tid] + s_norm[1][tid]) + (s_norm[2][tid] + s_norm[3][tid]);
        __syncthreads();
      }
      if (y == 0) P.norms[(size_t)l * nc + i] = a;
    }
    return;
  }
  bool bad = false;
  for (int t = 0; t < sp.ndot; ++t) {
    const Leaf& L = sp.leaf[sp.dot_leaf[t]];
    const int per = L.type == L_PERIODIC ? 2 : 1, nf = per * L.n;
    const int e = s_e[t];
    int S[NLEV] = {0, 0, 0, 0, 0, 0, 0, 0};
    unsigned char* base = P.slices + (size_t)rb * NSLICE * SLICE_BYTES + (size_t)tid * 16;
    for (int kg = t == 0 ? y : PREP_Y - 1 - y; kg < sp.dot_kch[t] * 2; kg += PREP_Y) {
      long long F[8];
#pragma unroll
      for (int kk = 0; kk < 8; ++kk) {
        const int k = kg * 8 + kk;
        F[kk] = 0;
        if (k < nf) {
          const size_t o = (size_t)(L.plane0 + k) * nc + i;
          const double x = w[L.param0 + k / per] * P.planes[o];
          if (P.keep_l) P.splanes[o] = x;  // the adjoint's features
          F[kk] = to_fixed55(x, e, &bad);
        }
        // W_ii's level sums, from the same digits as the products'
        const long long G = F[kk] + 0x808080808080LL;
        int d[NSLICE];
        d[0] = (int)(G >> 48);
#pragma unroll
        for (int p = 1; p < NSLICE; ++p) d[p] = (int)((G >> (8 * (6 - p))) & 0xFF) - 128;
#pragma unroll
        for (int p = 0; p < NSLICE; ++p)
#pragma unroll
          for (int q = p; q < NSLICE; ++q)
            if (p + q < NLEV) S[p + q] += (p == q ? 1 : 2) * d[p] * d[q];
      }
      uint4 out[NSLICE];
      digits8_of_fixed55(F, out);
      const int kgl = sp.dot_koff[t] / 8 + kg;
#pragma unroll
      for (int p = 0; p < NSLICE; ++p)
        *reinterpret_cast<uint4*>(base + (size_t)p * SLICE_BYTES + (size_t)kgl * 2048) = out[p];
    }
#pragma unroll
    for (int l = 0; l < NLEV; ++l) s_lev[t][y][l][tid] = S[l];
  }
  __syncthreads();
  if (y < sp.ndot) {
    int S[NLEV];
#pragma unroll
    for (int l = 0; l < NLEV; ++l) {
      S[l] = 0;
#pragma unroll
      for (int q = 0; q < PREP_Y; ++q) S[l] += s_lev[y][q][l][tid];
    }
    P.fnorm[(size_t)y * nc + i] = assemble_w(S, sp.dot_u[y]);
  }
  if (bad) atomicOr(&P.status[3], 1);
}

// ---------------------------------------------------------------------------
// persistent tensor-core build of the lower triangle (128 x 64 tiles)
// ---------------------------------------------------------------------------
constexpr int BLD_EPI_WARPS = 16;                      // 4 lane quarters x 4 groups of 16 columns
constexpr int BLD_THREADS = (BLD_EPI_WARPS + 2) * 32;  // + TMA warp + MMA warp
constexpr int NSTAGE = 3;
constexpr uint32_t BLD_TAB = NSTAGE * STAGE + 256;    // the exponential's two tables (2 x 1024 x 8 B)
constexpr uint32_t BLD_STASH = BLD_TAB + 2 * 1024 * 8;  // the first leaf's 16 values per epilogue thread
constexpr uint32_t BLD_SMEM = BLD_STASH + BLD_EPI_WARPS * 32 * 16 * 8;
static_assert(BLD_SMEM <= 227 * 1024, "shared memory per CTA");

// PROD: with the fixed-point product of two leaves.  Its own instance, because
// the loops it adds cost the others up to 18% (40 problems of N = 4000, a sum of
// two: 3.8 -> 4.5 ms, the compiler's schedule).  Against the FP64
// combination, the product's build: 7.5 -> 4.1 ms.
// NC: columns per epilogue thread.  A tile takes 16; where a problem has so few
// tiles that its parts still fit one wave, a CTA takes 4 NC of a tile's 64
// columns (and all of its products): the epilogue's chain is what a small
// build costs.  A lone N = 59 34 -> 18 us, N = 500 25 -> 16.5.
template <bool PROD, int NC>
__global__ void __launch_bounds__(BLD_THREADS, 1)
    k_build_tc(const Prob* __restrict__ probs, int nprob, const unsigned long long* __restrict__ tiles, int total) {
  extern __shared__ __align__(1024) unsigned char smb[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smb + NSTAGE * STAGE);
  uint64_t* empty = full + NSTAGE;
  uint64_t* tfull = full + 2 * NSTAGE;
  uint64_t* tempty = tfull + 1;
  uint64_t* drain = tfull + 2;  // quiescing after a give-up
  uint32_t* slot = reinterpret_cast<uint32_t*>(tfull + 3);
  __shared__ int s_abort;
  constexpr int SUB = 16 / NC;      // CTAs per tile
  constexpr int GW = NC < 8 ? NC : 8;  // columns drained together
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t issued = 0;  // producer lane: k-chunks whose operand copies were issued
  if (tid == 0) {
    s_abort = 0;
    mbar_init(drain, 1);
    for (int k = 0; k < NSTAGE; ++k) {
      mbar_init(&full[k], 1);
      mbar_init(&empty[k], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, BLD_EPI_WARPS * 32);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == BLD_EPI_WARPS + 1) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(su32(slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tbase = *slot;
  unsigned long long* tab = reinterpret_cast<unsigned long long*>(smb + BLD_TAB);
  unsigned long long* fine = tab + 1024;
  double* stash = reinterpret_cast<double*>(smb + BLD_STASH);
  for (int k = tid; k < 1024; k += BLD_THREADS) {
    tab[k] = g_iexp_tab1024[k];
    fine[k] = g_iexp_fine1024[k];
  }
  __syncthreads();
  // tile t: (problem << 40 | 128-row tile << 20 | 64-column tile), host-built
  auto tile_of = [&](int t, int& p, int& ti, int& tj) {
    const unsigned long long e = tiles[t / SUB];
    p = (int)(e >> 40);
    ti = (int)((e >> 20) & 0xFFFFF);
    tj = (int)(e & 0xFFFFF);
  };

  if (warp == BLD_EPI_WARPS) {
    // ---------------- TMA producer: digit planes of each leaf's k chunks ----------------
    if (lane == 0) {
      uint32_t g = 0;
      for (int t = blockIdx.x; t < total * SUB && !s_abort; t += gridDim.x) {
        int p, ti, tj;
        tile_of(t, p, ti, tj);
        const Prob& P = probs[p];
        const Spec& sp = *P.spec;
        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(P.tmap_a) : "memory");
        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(P.tmap_b) : "memory");
        for (int d = 0; d < sp.ndot; ++d) {
          const int c0 = sp.dot_koff[d] / 16;
          for (int c = 0; c < sp.dot_kch[d]; ++c, ++g) {
            const int st = g % NSTAGE;
            if (!mbar_wait(&empty[st], ((g / NSTAGE) & 1) ^ 1)) {
              s_abort = 1;
              break;
            }
            unsigned char* As = smb + st * STAGE;
            mbar_expect_tx(&full[st], STAGE);
            tma_load_5d(As, P.tmap_a, 0, 0, 2 * (c0 + c), 0, ti, &full[st]);
            tma_load_5d(As + A_STAGE, P.tmap_b, 0, (tj & 1) * 2, 2 * (c0 + c), 0, tj >> 1, &full[st]);
            issued = g + 1;
          }
          if (s_abort) break;
        }
      }
    }
  } else if (warp == BLD_EPI_WARPS + 1) {
    // ---------------- MMA issuer: one pass of 35 pairs per chunk per leaf ----------------
    if (lane == 0) {
      uint32_t g = 0, it = 0;
      const uint64_t adesc0 = smem_desc(su32(smb), 2048, 128);
      const uint64_t bdesc0 = smem_desc(su32(smb) + A_STAGE, 1024, 128);
      for (int t = blockIdx.x; t < total * SUB && !s_abort; t += gridDim.x) {
        int p, ti, tj;
        tile_of(t, p, ti, tj);
        const Spec& sp = *probs[p].spec;
        for (int d = 0; d < sp.ndot; ++d, ++it) {
          if (!mbar_wait(tempty, (it & 1) ^ 1)) {
            s_abort = 1;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          for (int c = 0; c < sp.dot_kch[d]; ++c, ++g) {
            const int st = g % NSTAGE;
            if (!mbar_wait(&full[st], (g / NSTAGE) & 1)) {
              s_abort = 1;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint64_t soff = (uint64_t)((st * STAGE) >> 4);
#pragma unroll
            for (int pp = 0; pp < NSLICE; ++pp) {
#pragma unroll
              for (int q = 0; q < NSLICE && q + pp < NLEV; ++q) {
                // the first pair of level L = pp + q is (max(0, L - 6), .): it starts the sum
                const bool first = c == 0 && pp == (pp + q > NSLICE - 1 ? pp + q - (NSLICE - 1) : 0);
                mma_f16(tbase + (uint32_t)(pp + q) * 64, adesc0 + soff + (uint64_t)(pp * 4096 >> 4),
                        bdesc0 + soff + (uint64_t)(q * 2048 >> 4), first ? 0u : 1u);
              }
            }
            mma_commit(&empty[st]);
          }
          if (s_abort) break;
          mma_commit(tfull);
        }
      }
    }
  } else {
    // ---------------- epilogue (warps 0-15) ----------------
    const int r = (warp & 3) * 32 + lane;  // TMEM lane = tile row
    const int h = warp >> 2;               // group of NC columns
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    uint32_t it = 0;
    for (int t = blockIdx.x; t < total * SUB; t += gridDim.x) {
      int p, ti, tj;
      tile_of(t, p, ti, tj);
      const Prob& P = probs[p];
      const Spec& sp = *P.spec;
      const size_t nc = (size_t)P.Nc;
      const int i = ti * NB + r;
      const int cb0 = (t % SUB * 4 + h) * NC;  // this thread's columns of the tile
      const int j0 = tj * TB + cb0;
      const int form = P.fscale[2];
      bool stop = false;
      for (int d = 0; d < sp.ndot; ++d, ++it) {
        if (!mbar_wait(tfull, it & 1)) {
          s_abort = 1;
          stop = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        long long W[NC];
        const int u = sp.dot_u[d];
        // level sums of a leaf with at most 36 features stay below 2^22 (7
        // digit pairs x 36 terms x 2^14): converted by the exact magic add
        // (one FP32 add each, no conversion instruction), otherwise by F2I
        const Leaf& LF = sp.leaf[sp.dot_leaf[d]];
        const bool small = (LF.type == L_PERIODIC ? 2 * LF.n : LF.n) <= 36;
#pragma unroll
        for (int gq = 0; gq < NC / GW; ++gq) {
          uint32_t v[NLEV][GW];
#pragma unroll
          for (int l = 0; l < NLEV; ++l) {
            tmem_ldw(v[l], tbase + lane_base + (uint32_t)(l * 64 + cb0 + gq * GW));
          }
          asm volatile("tcgen05.wait::ld.sync.aligned;");
          if (small) {
#pragma unroll
            for (int jj = 0; jj < GW; ++jj) {
              uint32_t b[NLEV];
#pragma unroll
              for (int l = 0; l < NLEV; ++l) b[l] = level_bits(v[l][jj]);
              W[gq * GW + jj] = assemble_w_bits(b, u);
            }
          } else {
#pragma unroll
            for (int jj = 0; jj < GW; ++jj) {
              int S[NLEV];
#pragma unroll
              for (int l = 0; l < NLEV; ++l) S[l] = __float2int_rn(__uint_as_float(v[l][jj]));
              W[gq * GW + jj] = assemble_w(S, u);
            }
          }
        }
        // TMEM drained: the next pass's MMAs may start
        asm volatile("tcgen05.fence::before_thread_sync;");
        mbar_arrive(tempty);
        // the squared distances, in the leaf's unit
        const long long wi = (long long)((unsigned long long)P.fnorm[(size_t)d * nc + i] +
                                         (small ? (unsigned long long)BUILD_BIAS_H << (u - 47) : 0ULL));
        // W_jj of this thread's NC columns (the same for the whole warp), two at a time
        const longlong2* wj2 = reinterpret_cast<const longlong2*>(P.fnorm + (size_t)d * nc + j0);
#pragma unroll
        for (int q = 0; q < NC; ++q) {
          const longlong2 w2 = __ldg(wj2 + q / 2);
          W[q] = (long long)((unsigned long long)wi + (unsigned long long)((q & 1) ? w2.y : w2.x) - 2 * (unsigned long long)W[q]);
          if (W[q] < 0) W[q] = 0;
        }
        const IexpScale esc = iexp_scale(2 * P.fscale[d] + 1 - u);
        const int N = P.N;
        const int e2 = 2 * *P.kscale;
        bool nonfinite = false;
        // entries (i, j0 + q), in the accumulator layout; the lower triangle of
        // the N x N block, zeros beyond
        long long* A = P.acc + acc_tile(ti, tj, P.nt128) * ACC_TILE_ELEMS;
        const int jmax = i < N ? i : -1;
        auto put = [&](int q, long long F) {
          A[acc_elem(r, cb0 + q)] = j0 + q <= jmax ? F : 0LL;
        };
        // One leaf, a plain sum of two or a plain product of two: fixed point
        // throughout.  Any other expression, and scales outside the
        // exponential's common form, combine in FP64, 64 cycles an operation
        // and warp.
        const bool sum = form == FORM_SUM, prod = PROD && form == FORM_PROD;
        constexpr int tstash = BLD_EPI_WARPS * 32;
        auto fixed = [&](auto parts) {
          long long* st = reinterpret_cast<long long*>(stash) + tid;  // the first leaf's values, for the second pass
          if (d < sp.ndot - 1) {
            const int unit = PROD && prod ? 0 : e2;  // a product's first factor: v0 2^62
#pragma unroll
            for (int q = 0; q < NC; ++q) st[q * tstash] = iexp_parts_fixed62(parts((unsigned long long)W[q]), unit);
          } else if (d == 0) {
#pragma unroll
            for (int q = 0; q < NC; ++q) put(q, iexp_parts_fixed62(parts((unsigned long long)W[q]), e2));
          } else if (PROD && prod) {
#pragma unroll
            for (int q = 0; q < NC; ++q) {
              IexpParts v = parts((unsigned long long)W[q]);
              v.Z = __umul64hi((unsigned long long)st[q * tstash], v.Z);  // v0 v1 2^(60 + m)
              put(q, iexp_parts_fixed62(v, e2 - 2));
            }
          } else {
#pragma unroll
            for (int q = 0; q < NC; ++q) put(q, st[q * tstash] + iexp_parts_fixed62(parts((unsigned long long)W[q]), e2));
          }
        };
        if ((sum || prod) && iexp_common(esc) && esc.F <= 64) {
          fixed([&](unsigned long long E) { return iexp_common_parts<true>(E, esc, tab, fine); });
        } else if ((sum || prod) && iexp_common(esc)) {
          fixed([&](unsigned long long E) { return iexp_common_parts<false>(E, esc, tab, fine); });
        } else {
          const double ca = P.fcoef[0], cb = P.fcoef[1], cc = P.fcoef[2], cd = P.fcoef[3];
          auto leaf = [&](int q) { return iexp_fixed_tab((unsigned long long)W[q], esc, tab, fine); };
          double* st = stash + tid;
          if (d < sp.ndot - 1) {
#pragma unroll
            for (int q = 0; q < NC; ++q) st[q * tstash] = leaf(q);
          } else if (d == 0) {
#pragma unroll
            for (int q = 0; q < NC; ++q) put(q, to_fixed62(fma(cb, leaf(q), ca), e2, &nonfinite));
          } else {
#pragma unroll
            for (int q = 0; q < NC; ++q) {
              // second distance leaf: k = (d v0 + c) v1 + (b v0 + a)
              const double v0 = st[q * tstash];
              put(q, to_fixed62(fma(fma(cd, v0, cc), leaf(q), fma(cb, v0, ca)), e2, &nonfinite));
            }
          }
        }
        // the diagonal entry: every leaf 1, with the nugget; identity padding (1/4 in the matrix's unit) beyond N
        if (d == sp.ndot - 1 && i >= j0 && i < j0 + NC) {
          const double noise = P.optimise_noise ? P.theta[sp.nkparams] : P.noise;
          const double ca = P.fcoef[0], cb = P.fcoef[1], cc = P.fcoef[2], cd = P.fcoef[3];
          const double kd = sp.ndot == 1 ? cb + ca : (cd + cc) + (cb + ca);
          A[acc_elem(r, i - j0 + cb0)] = i < N ? diag_fixed62(kd, noise, e2, &nonfinite) : 1LL << 60;
        }
        if (nonfinite) atomicOr(&P.status[3], 1);
      }
      if (stop) break;
    }
  }
  __syncthreads();
  if (s_abort) {
    // a bounded wait gave up: the copies and MMAs this CTA issued finish
    // (bounded waits) before it frees its TMEM and exits
    if (warp == BLD_EPI_WARPS && lane == 0) drain_ring(full, NSTAGE, issued);
    if (warp == BLD_EPI_WARPS + 1 && lane == 0) drain_mmas(drain);
    __syncthreads();
    if (tid == 0)
      for (int q = 0; q < nprob; ++q) atomicExch(&probs[q].status[2], 1);
  }
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == BLD_EPI_WARPS + 1) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tbase));
}

// ---------------------------------------------------------------------------
// launch helpers
// ---------------------------------------------------------------------------
cudaError_t launch_prep(const Prob* probs, int nprob, int max_nt128, cudaStream_t s) {
  k_prep<<<dim3(max_nt128, nprob), dim3(NB, PREP_Y), 0, s>>>(probs);
  return cudaGetLastError();
}

cudaError_t launch_build_tc(const Prob* probs, int nprob, const unsigned long long* tiles, int total_tiles,
                            bool products, int num_sms, cudaStream_t s) {
  // the parts of the tiles fill one wave at most
  const int sub = 4 * total_tiles <= num_sms ? 4 : (2 * total_tiles <= num_sms ? 2 : 1);
  using Kernel = void (*)(const Prob*, int, const unsigned long long*, int);
  const Kernel kernels[2][3] = {{k_build_tc<false, 16>, k_build_tc<false, 8>, k_build_tc<false, 4>},
                                {k_build_tc<true, 16>, k_build_tc<true, 8>, k_build_tc<true, 4>}};
  const Kernel kernel = kernels[products][sub / 2];
  cudaError_t e = ensure_smem_attr((const void*)kernel, SMEM_BUILD_TC + products * 3 + sub / 2, BLD_SMEM);
  if (e != cudaSuccess) return e;
  if (total_tiles <= 0) return cudaSuccess;
  const int grid = total_tiles * sub < num_sms ? total_tiles * sub : num_sms;
  kernel<<<grid, BLD_THREADS, BLD_SMEM, s>>>(probs, nprob, tiles, total_tiles);
  return cudaGetLastError();
}

}  // namespace fgpu
