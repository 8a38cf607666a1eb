// Adjoint of the log-likelihood (FP64):
//   d logL / d theta_q = 1/2 sum_ij W_ij dK_ij/dtheta_q,  W = alpha alpha^T / s - K^-1,
// s = 1 (marginal) or sigma^2 (concentrated; the profiled mean and variance
// drop out by the envelope theorem), and dK/dnoise = I.
//
// K^-1: the factorisation runs on a taller matrix whose rows below the
// right-hand-side tile start as the identity; the sweep turns them into
// B = L^-T (row i of B = column i of L^-1, zero left of column i), and
// K^-1 = B B^T.  dK/dtheta is never stored: the fused pass recomputes the
// leaf values and their per-feature factors from the feature planes tile by
// tile, exactly as the kernel-matrix build does.
#include "fgpu_internal.h"
#include "iexp.cuh"
#include "tc_common.cuh"

#include <cmath>

namespace fgpu {

namespace {
constexpr int GCHUNK = 32;  // parameters per pass of the fused kernel (+ 1 noise slot)
constexpr int USTRIDE = TB + 8;
__device__ __forceinline__ void dmma(double& c0, double& c1, double a, double b) {
  asm volatile("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0,%1}, {%2}, {%3}, {%0,%1};"
               : "+d"(c0), "+d"(c1)
               : "d"(a), "d"(b));
}
}  // namespace

// rows Nc + 64 + q: e_q^T for q < N, zero otherwise
__global__ void __launch_bounds__(256) k_identity_border(const Prob* __restrict__ pp) {
  const Prob& P = *pp;
  const int ct = blockIdx.x, rt = blockIdx.y;
  const size_t ld = (size_t)P.ld;
  const int r0 = P.Nc + TB + rt * TB;
  for (int e = threadIdx.x; e < TB * TB; e += blockDim.x) {
    const int r = e % TB, c = e / TB;
    const int q = rt * TB + r, j = ct * TB + c;
    P.K[(size_t)j * ld + r0 + r] = (q == j && q < P.N) ? 1.0 : 0.0;
  }
}

// K^-1 tile (ti, tj), ti >= tj: sum over k-blocks kb >= ti of B[ti, kb] B[tj, kb]^T
__global__ void __launch_bounds__(128) k_syrk_inv(const Prob* __restrict__ pp) {
  const Prob& P = *pp;
  const int ti = blockIdx.x, tj = blockIdx.y;
  if (ti < tj || ti >= P.nsteps) return;
  extern __shared__ __align__(16) double smg[];
  double* As = smg;                 // [k][m]
  double* Bs = smg + TB * USTRIDE;  // [k][n]
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  const size_t ld = (size_t)P.ld;
  const int R0 = P.Nc + TB;
  const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32, lr = lane >> 2, lk = lane & 3;
  double acc[4][4][2];
  for (int a = 0; a < 4; ++a)
    for (int b = 0; b < 4; ++b) acc[a][b][0] = acc[a][b][1] = 0.0;
  for (int kb = ti; kb < P.nsteps; ++kb) {
    const double* Ag = P.K + (size_t)(kb * TB) * ld + R0 + ti * TB;
    const double* Bg = P.K + (size_t)(kb * TB) * ld + R0 + tj * TB;
    __syncthreads();
    for (int e = tid; e < TB * (TB / 2); e += blockDim.x) {
      const int k = e / (TB / 2), m2 = (e % (TB / 2)) * 2;
      *reinterpret_cast<double2*>(As + k * USTRIDE + m2) = *reinterpret_cast<const double2*>(Ag + (size_t)k * ld + m2);
      *reinterpret_cast<double2*>(Bs + k * USTRIDE + m2) = *reinterpret_cast<const double2*>(Bg + (size_t)k * ld + m2);
    }
    __syncthreads();
    for (int k0 = 0; k0 < TB; k0 += 4) {
      double af[4], bf[4];
      for (int a = 0; a < 4; ++a) af[a] = As[(k0 + lk) * USTRIDE + wm + a * 8 + lr];
      for (int b = 0; b < 4; ++b) bf[b] = Bs[(k0 + lk) * USTRIDE + wn + b * 8 + lr];
      for (int a = 0; a < 4; ++a)
        for (int b = 0; b < 4; ++b) dmma(acc[a][b][0], acc[a][b][1], af[a], bf[b]);
    }
  }
  const size_t nc = (size_t)P.Nc;
  for (int a = 0; a < 4; ++a)
    for (int b = 0; b < 4; ++b) {
      const int m = ti * TB + wm + a * 8 + lr;
      const int n = tj * TB + wn + b * 8 + lk * 2;
      P.kinv[(size_t)n * nc + m] = acc[a][b][0];
      P.kinv[(size_t)(n + 1) * nc + m] = acc[a][b][1];
    }
}

// Fused dK/dtheta pass over the lower tiles; partial sums per CTA for the
// parameters [q0, q0 + GCHUNK) and (slot GCHUNK) the noise.
__global__ void __launch_bounds__(256) k_grad(const Prob* __restrict__ pp, int q0) {
  const Prob& P = *pp;
  const int ti = blockIdx.x, tj = blockIdx.y;
  const int cta = blockIdx.y * gridDim.x + blockIdx.x;
  __shared__ double ls[MAX_PARAMS];
  __shared__ double red[8][GCHUNK + 1];
  __shared__ int lchild[MAX_POST], rchild[MAX_POST];
  const Spec& sp = *P.spec;
  const int tid = threadIdx.x;
  double acc[GCHUNK + 1];
  for (int q = 0; q <= GCHUNK; ++q) acc[q] = 0.0;
  const bool work = ti >= tj && ti < P.nsteps && !P.status[1];
  if (tid == 0) {
    int stk[MAX_POST], top = 0;
    for (int t = 0; t < sp.npost; ++t) {
      lchild[t] = rchild[t] = -1;
      if (sp.post[t] < 0) {
        rchild[t] = stk[--top];
        lchild[t] = stk[--top];
      }
      stk[top++] = t;
    }
  }
  for (int k = tid; k < sp.nkparams; k += blockDim.x) {
    int type = L_CONSTANT;
    for (int l = 0; l < sp.nleaf; ++l) {
      const int cnt = sp.leaf[l].type == L_CONSTANT ? 1 : sp.leaf[l].n;
      if (k >= sp.leaf[l].param0 && k < sp.leaf[l].param0 + cnt) type = sp.leaf[l].type;
    }
    const double t = P.theta[k];
    ls[k] = (type == L_RBF || type == L_RBF_CYCLIC) ? exp(t)
            : (type == L_PERIODIC) ? (1.0 / exp(t)) * (1.0 / exp(t))
            : (type == L_LINEAR) ? exp(-t) : t;
  }
  __syncthreads();
  if (work) {
    const double s2 = P.likelihood == 1 ? P.out[3] : 1.0;
    const size_t nc = (size_t)P.Nc;
    const double* X = P.planes;
    const int r0 = (tid & 31) * 2, c0 = (tid >> 5) * 8;
    for (int cc = 0; cc < 8; ++cc)
      for (int a = 0; a < 2; ++a) {
        const int i = ti * TB + r0 + a, j = tj * TB + c0 + cc;
        if (i < j || i >= P.N || j >= P.N) continue;
        const double w = (P.z[i] * P.z[j] / s2 - P.kinv[(size_t)j * P.ldkinv + i]) * (i == j ? 1.0 : 2.0);
        if (i == j) acc[GCHUNK] += w;
        // forward: leaf values
        double val[MAX_POST], adj[MAX_POST];
        for (int t = 0; t < sp.npost; ++t) {
          const int tok = sp.post[t];
          adj[t] = 0.0;
          if (tok >= 0) {
            const Leaf& L = sp.leaf[tok];
            double e = 0.0, v;
            if (L.type == L_RBF || L.type == L_RBF_CYCLIC) {
              for (int k = 0; k < L.n; ++k) {
                double d = X[(size_t)(L.plane0 + k) * nc + i] - X[(size_t)(L.plane0 + k) * nc + j];
                if (L.type == L_RBF_CYCLIC && sp.cyclic[L.plane0 + k]) {
                  const double aa = fabs(d) + 3.141592653589793;
                  d = copysign(1.0, d) * (fmod(aa, 6.283185307179586) - 3.141592653589793);
                }
                e = fma(ls[L.param0 + k], d * d, e);
              }
              v = iexp_neg(-0.5 * e);
            } else if (L.type == L_PERIODIC) {
              for (int k = 0; k < L.n; ++k) {
                const double si = X[(size_t)(L.plane0 + 2 * k) * nc + i], ci = X[(size_t)(L.plane0 + 2 * k + 1) * nc + i];
                const double sj = X[(size_t)(L.plane0 + 2 * k) * nc + j], cj = X[(size_t)(L.plane0 + 2 * k + 1) * nc + j];
                const double tt = fma(si, cj, -(ci * sj));
                e = fma(ls[L.param0 + k], tt * tt, e);
              }
              v = iexp_neg(-2.0 * e);
            } else if (L.type == L_LINEAR) {
              v = 0.0;
              for (int k = 0; k < L.n; ++k) v += 1.0 / ls[L.param0 + k];
            } else {
              v = ls[L.param0];
            }
            val[t] = v;
          } else {
            val[t] = (tok == P_SUM) ? val[lchild[t]] + val[rchild[t]] : val[lchild[t]] * val[rchild[t]];
          }
        }
        // backward: sensitivity of K to every node
        adj[sp.npost - 1] = 1.0;
        for (int t = sp.npost - 1; t >= 0; --t) {
          const int tok = sp.post[t];
          if (tok < 0) {
            const int l = lchild[t], r = rchild[t];
            if (tok == P_SUM) {
              adj[l] += adj[t];
              adj[r] += adj[t];
            } else {
              adj[l] += adj[t] * val[r];
              adj[r] += adj[t] * val[l];
            }
          }
        }
        // per-parameter factors
        for (int t = 0; t < sp.npost; ++t) {
          const int tok = sp.post[t];
          if (tok < 0) continue;
          const Leaf& L = sp.leaf[tok];
          const double cw = w * adj[t];
          const int cnt = L.type == L_CONSTANT ? 1 : L.n;
          if (L.param0 + cnt <= q0 || L.param0 >= q0 + GCHUNK) continue;
          for (int k = 0; k < cnt; ++k) {
            const int q = L.param0 + k - q0;
            if (q < 0 || q >= GCHUNK) continue;
            double dv;
            if (L.type == L_RBF || L.type == L_RBF_CYCLIC) {
              double d = X[(size_t)(L.plane0 + k) * nc + i] - X[(size_t)(L.plane0 + k) * nc + j];
              if (L.type == L_RBF_CYCLIC && sp.cyclic[L.plane0 + k]) {
                const double aa = fabs(d) + 3.141592653589793;
                d = copysign(1.0, d) * (fmod(aa, 6.283185307179586) - 3.141592653589793);
              }
              dv = val[t] * (-0.5 * ls[L.param0 + k] * d * d);
            } else if (L.type == L_PERIODIC) {
              const double si = X[(size_t)(L.plane0 + 2 * k) * nc + i], ci = X[(size_t)(L.plane0 + 2 * k + 1) * nc + i];
              const double sj = X[(size_t)(L.plane0 + 2 * k) * nc + j], cj = X[(size_t)(L.plane0 + 2 * k + 1) * nc + j];
              const double tt = fma(si, cj, -(ci * sj));
              dv = val[t] * (4.0 * ls[L.param0 + k] * tt * tt);
            } else if (L.type == L_LINEAR) {
              dv = 1.0 / ls[L.param0 + k];  // d exp(theta) / d theta
            } else {
              dv = 1.0;
            }
            acc[q] += cw * dv;
          }
        }
      }
  }
  // block reduction in a fixed order
  const int warp = tid >> 5, lane = tid & 31;
  for (int q = 0; q <= GCHUNK; ++q) {
    double v = acc[q];
    for (int o = 16; o > 0; o >>= 1) v += __shfl_down_sync(0xffffffffu, v, o);
    if (lane == 0) red[warp][q] = v;
  }
  __syncthreads();
  if (tid <= GCHUNK) {
    double v = 0.0;
    for (int w = 0; w < 8; ++w) v += red[w][tid];
    P.gpart[(size_t)cta * (GCHUNK + 1) + tid] = v;
  }
}

__global__ void k_grad_reduce(const Prob* __restrict__ pp, int nblocks, int q0, int nk, int noise_slot,
                              double* __restrict__ g) {
  const Prob& P = *pp;
  const int q = threadIdx.x;
  if (q > GCHUNK) return;
  double v = 0.0;
  for (int b = 0; b < nblocks; ++b) v += P.gpart[(size_t)b * (GCHUNK + 1) + q];
  if (q < GCHUNK && q0 + q < nk) g[q0 + q] = 0.5 * v;
  if (q == GCHUNK && noise_slot >= 0) g[noise_slot] = 0.5 * v;
}

// ---------------------------------------------------------------------------
// the same pass for kernels with one or two rbf / periodic leaves besides
// linear and constant ones (those of the tensor-core build), k = a + b v0 +
// c v1 + d v0 v1.
//
// FP64 costs 64 cycles per warp instruction here, so it is kept to what the
// gradient's own sums need: per entry w_ij = W_ij and its products with the leaf
// values, and per entry and feature the squared difference times that (3
// operations for an rbf feature, 4 for a periodic one).  The leaf values come
// from exact integer distances: the evaluation's scaled features f (v = exp(-|f_i
// - f_j|^2 / 2)) as 54-bit fixed point in the leaf's scale 2^s, a difference
// D = h 2^27 + l squared as h^2 + 2 h l 2^-27 + l^2 2^-54 on the integer
// multiply-add pipe, and the fixed-point exponential.  One CTA per 64 x 64 lower
// tile, 2 rows x 8 columns per thread, the features staged 16 planes at a time.
// N = 4000, d = 24: 1.6 ms, against 4.9 ms for k_grad (all FP64, leaf values and
// differences formed twice) and 0.34 ms for its one-block reduction.
// ---------------------------------------------------------------------------
namespace {
constexpr int GF_CH = 16;  // planes per chunk
constexpr int GF_SMEM = (2 * GF_CH * TB + 256 * GF_CH) * 8;
}  // namespace

// features of the distance leaves in fixed point: F = f 2^(54 - s)
__global__ void __launch_bounds__(256) k_grad_fixed(const Prob* __restrict__ pe, long long* __restrict__ fx) {
  const Prob& P = *pe;
  const Spec& sp = *P.spec;
  const int i = blockIdx.x * blockDim.x + threadIdx.x, p = blockIdx.y;
  if (i >= P.Nc) return;
  for (int d = 0; d < sp.ndot; ++d) {
    const Leaf& L = sp.leaf[sp.dot_leaf[d]];
    const int nf = L.type == L_PERIODIC ? 2 * L.n : L.n;
    if (p >= L.plane0 && p < L.plane0 + nf)
      fx[(size_t)p * P.Nc + i] = to_fixed54(P.splanes[(size_t)p * P.Nc + i], P.fscale[d]);
  }
}

// PER_SM: CTAs per SM.  With more tiles than SMs, two: the tile's integer and
// FP64 halves follow one another behind barriers, and a second CTA fills the
// pipe the first leaves idle, which is worth the 128 registers (N = 4000: 2.08 ->
// 1.57 ms).  With fewer, one CTA with all the registers it wants (N = 1003: 163
// us, and 168 with 128).
template <int PER_SM>
__global__ void __launch_bounds__(256, PER_SM)
    k_grad_fast(const Prob* __restrict__ pp, const Prob* __restrict__ pe, const long long* __restrict__ fx,
                int nslots, int extra) {
  const Prob& P = *pp;   // adjoint: planes, alpha, K^-1
  const Prob& Q = *pe;   // evaluation: scales and expression coefficients
  const Spec& sp = *P.spec;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  // lower tile (ti, tj) of the linear index
  int ti = (int)((sqrtf(8.0f * (float)blockIdx.x + 1.0f) - 1.0f) * 0.5f);
  while ((ti + 1) * (ti + 2) / 2 <= (int)blockIdx.x) ++ti;
  while (ti * (ti + 1) / 2 > (int)blockIdx.x) --ti;
  const int tj = (int)blockIdx.x - ti * (ti + 1) / 2;
  double* gp = P.gpart + (size_t)blockIdx.x * nslots;
  if (P.status[1]) {
    for (int q = tid; q < nslots; q += 256) gp[q] = 0.0;
    return;
  }
  extern __shared__ __align__(16) unsigned char smraw[];
  double* Xi = reinterpret_cast<double*>(smraw);  // [plane of the chunk][64]
  double* Xj = Xi + GF_CH * TB;
  double* red = Xj + GF_CH * TB;  // [plane of the chunk][thread]
  long long* Fi = reinterpret_cast<long long*>(Xi);
  long long* Fj = reinterpret_cast<long long*>(Xj);
  const int r0 = lane * 2, c0 = warp * 8;
  const size_t nc = (size_t)P.Nc, ncq = (size_t)Q.Nc;
  double v[2][16];  // leaf values, then the leaves' weights
#pragma unroll
  for (int d = 0; d < 2; ++d) {
#pragma unroll
    for (int e = 0; e < 16; ++e) v[d][e] = 0.0;
    if (d < sp.ndot) {
      const Leaf& L = sp.leaf[sp.dot_leaf[d]];
      const int nf = L.type == L_PERIODIC ? 2 * L.n : L.n;
      unsigned long long H[16];  // 128 features' 2^56
      long long M[16];
#pragma unroll
      for (int e = 0; e < 16; ++e) H[e] = 0, M[e] = 0;
      for (int k0 = 0; k0 < nf; k0 += GF_CH) {
        const int kn = min(GF_CH, nf - k0);
        __syncthreads();
        for (int q = tid; q < kn * TB; q += 256) {
          const long long* src = fx + (size_t)(L.plane0 + k0 + q / TB) * ncq;
          Fi[q] = src[ti * TB + q % TB];
          Fj[q] = src[tj * TB + q % TB];
        }
        __syncthreads();
        for (int k = 0; k < kn; ++k) {
          const longlong2 fi = *reinterpret_cast<const longlong2*>(Fi + k * TB + r0);
#pragma unroll
          for (int c = 0; c < 8; ++c) {
            const long long fj = Fj[k * TB + c0 + c];
#pragma unroll
            for (int a = 0; a < 2; ++a) {
              const long long D = (a ? fi.y : fi.x) - fj;
              const int h = (int)((D + (1LL << 26)) >> 27);
              const int l = (int)D - (int)((unsigned)h << 27);
              H[c * 2 + a] += (unsigned long long)((long long)h * h);
              M[c * 2 + a] += (long long)h * l + (((long long)l * l) >> 28);
            }
          }
        }
      }
      // |f_i - f_j|^2 = (H + M 2^-26) 2^(2 s - 54), in units of 2^-55 or finer: with
      // those of 2^(2 s - 54) the leaf values of close pairs were 10^-13 off for
      // weights of 50 (s = 6); beyond 2^62 of the unit (128) they are below 2e-28
      const int s2 = 2 * Q.fscale[d], up = max(0, min(26, s2 + 1));
      const IexpScale sc = iexp_scale(s2 - 55 - up);
#pragma unroll
      for (int e = 0; e < 16; ++e) {
        const unsigned long long E =
            H[e] >> (62 - up) && up ? ~0ULL : (H[e] << up) + (unsigned long long)(M[e] >> (26 - up));
        v[d][e] = iexp_fixed_tab(E, sc, g_iexp_tab1024, g_iexp_fine1024);
      }
    }
  }
  // weights: w dk/dv_d v_d, and the sums the linear and constant leaves need
  double s[5] = {0.0, 0.0, 0.0, 0.0, 0.0};  // sum w, w v0, w v1, w v0 v1, trace of w
  {
    const double is2 = P.likelihood == 1 ? 1.0 / P.out[3] : 1.0;
    const double cb = Q.fcoef[1], cc = Q.fcoef[2], cd = Q.fcoef[3];
    const bool plain = cb == 1.0 && cd == 0.0 && (sp.ndot == 1 || cc == 1.0);
    const double zi[2] = {P.z[ti * TB + r0] * is2, P.z[ti * TB + r0 + 1] * is2};
#pragma unroll
    for (int e = 0; e < 16; ++e) {
      const int a = e & 1, i = ti * TB + r0 + a, j = tj * TB + c0 + (e >> 1);
      double w = 0.0;
      if (i >= j && i < P.N) {
        w = fma(zi[a], P.z[j], -P.kinv[(size_t)j * P.ldkinv + i]);
        if (i == j)
          s[4] += w;
        else
          w = 2.0 * w;
      }
      const double v0 = v[0][e], v1 = v[1][e];
      double m0 = w * v0, m1 = sp.ndot > 1 ? w * v1 : 0.0;
      if (extra) {
        s[0] += w;
        s[1] += m0;
        s[2] += m1;
        s[3] = fma(m0, v1, s[3]);
      }
      if (!plain) {
        const double m01 = cd * (m0 * v1);
        m0 = fma(cb, m0, m01);
        m1 = fma(cc, m1, m01);
      }
      v[0][e] = m0;
      v[1][e] = m1;
    }
  }
  // per-feature sums of weight x squared difference
#pragma unroll
  for (int d = 0; d < 2; ++d) {
    if (d < sp.ndot) {
      const Leaf& L = sp.leaf[sp.dot_leaf[d]];
      const int per = L.type == L_PERIODIC ? 2 : 1;
      for (int k0 = 0; k0 < L.n; k0 += GF_CH / per) {
        const int kn = min(GF_CH / per, L.n - k0);
        __syncthreads();
        for (int q = tid; q < kn * per * TB; q += 256) {
          const double* src = P.planes + (size_t)(L.plane0 + k0 * per + q / TB) * nc;
          Xi[q] = src[ti * TB + q % TB];
          Xj[q] = src[tj * TB + q % TB];
        }
        __syncthreads();
        for (int k = 0; k < kn; ++k) {
          double acc = 0.0;
          if (per == 1) {
            const double2 xi = *reinterpret_cast<const double2*>(Xi + k * TB + r0);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const double xj = Xj[k * TB + c0 + c];
#pragma unroll
              for (int a = 0; a < 2; ++a) {
                const double df = (a ? xi.y : xi.x) - xj;
                acc = fma(v[d][c * 2 + a] * df, df, acc);
              }
            }
          } else {
            const double2 si = *reinterpret_cast<const double2*>(Xi + (2 * k) * TB + r0);
            const double2 ci = *reinterpret_cast<const double2*>(Xi + (2 * k + 1) * TB + r0);
#pragma unroll
            for (int c = 0; c < 8; ++c) {
              const double sj = Xj[(2 * k) * TB + c0 + c], cj = Xj[(2 * k + 1) * TB + c0 + c];
#pragma unroll
              for (int a = 0; a < 2; ++a) {
                const double t = fma(a ? si.y : si.x, cj, -((a ? ci.y : ci.x) * sj));
                acc = fma(v[d][c * 2 + a] * t, t, acc);
              }
            }
          }
          red[k * 256 + tid] = acc;
        }
        __syncthreads();
        // 16 threads per feature, in a fixed order
        const int k = tid >> 4;
        double t = 0.0;
        if (k < kn)
          for (int q = tid & 15; q < 256; q += 16) t += red[k * 256 + q];
        for (int o = 8; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o, 16);
        if (k < kn && (tid & 15) == 0) gp[L.param0 + k0 + k] = t;
      }
    }
  }
  __syncthreads();
#pragma unroll
  for (int q = 0; q < 5; ++q) red[q * 256 + tid] = s[q];
  __syncthreads();
  const int k = tid >> 4;
  double t = 0.0;
  if (k < 5)
    for (int q = tid & 15; q < 256; q += 16) t += red[k * 256 + q];
  for (int o = 8; o > 0; o >>= 1) t += __shfl_down_sync(0xffffffffu, t, o, 16);
  if (k < 5 && (tid & 15) == 0) gp[nslots - 5 + k] = t;
}

// sums of the tiles' partials (one CTA per slot, in a fixed order), then d logL /
// d theta: the distance leaves' from their features' sums, the linear and
// constant leaves' through the expression's coefficients
__global__ void __launch_bounds__(256)
    k_grad_fast_reduce(const Prob* __restrict__ pp, int ntiles, int nslots, double* __restrict__ sums) {
  __shared__ double red[256];
  const int q = blockIdx.x, tid = threadIdx.x;
  double t = 0.0;
  for (int b = tid; b < ntiles; b += 256) t += pp->gpart[(size_t)b * nslots + q];
  red[tid] = t;
  __syncthreads();
  for (int o = 128; o > 0; o >>= 1) {
    if (tid < o) red[tid] += red[tid + o];
    __syncthreads();
  }
  if (tid == 0) sums[q] = red[0];
}
__global__ void __launch_bounds__(256)
    k_grad_fast_out(const Prob* __restrict__ pp, const double* __restrict__ sums, int nslots, int noise_slot,
                    double* __restrict__ g) {
  const Prob& P = *pp;
  const Spec& sp = *P.spec;
  const double* s = sums + nslots - 5;
  const int q = threadIdx.x;  // parameter
  if (q == 0 && noise_slot >= 0) g[noise_slot] = 0.5 * s[4];
  if (q >= sp.nkparams) return;
  int leaf = 0;
  for (int l = 0; l < sp.nleaf; ++l) {
    const int cnt = sp.leaf[l].type == L_CONSTANT ? 1 : sp.leaf[l].n;
    if (q >= sp.leaf[l].param0 && q < sp.leaf[l].param0 + cnt) leaf = l;
  }
  const int type = sp.leaf[leaf].type;
  const double t = P.theta[q];
  if (type == L_RBF) {  // dv/dtheta = -v l (x_i - x_j)^2 / 2
    g[q] = 0.5 * (-0.5 * exp(t)) * sums[q];
  } else if (type == L_PERIODIC) {  // 4 v l sin^2(d / 2)
    const double il = 1.0 / exp(t);
    g[q] = 0.5 * (4.0 * (il * il)) * sums[q];
  } else {
    // the expression's coefficients (1, v0, v1, v0 v1) and their derivative by this leaf
    double c[MAX_POST][4], dc[MAX_POST][4];
    int top = 0;
    for (int k = 0; k < sp.npost; ++k) {
      const int tok = sp.post[k];
      if (tok >= 0) {
        const Leaf& L = sp.leaf[tok];
        for (int m = 0; m < 4; ++m) c[top][m] = dc[top][m] = 0.0;
        if (L.type == L_RBF || L.type == L_PERIODIC) {
          c[top][tok == sp.dot_leaf[0] ? 1 : 2] = 1.0;
        } else if (L.type == L_LINEAR) {
          for (int m = 0; m < L.n; ++m) c[top][0] += 1.0 / exp(-P.theta[L.param0 + m]);
          if (tok == leaf) dc[top][0] = 1.0 / exp(-t);
        } else {
          c[top][0] = P.theta[L.param0];
          if (tok == leaf) dc[top][0] = 1.0;
        }
        ++top;
      } else {
        const double* b = c[top - 1];
        const double* db = dc[top - 1];
        --top;
        double* a = c[top - 1];
        double* da = dc[top - 1];
        if (tok == P_SUM) {
          for (int m = 0; m < 4; ++m) {
            a[m] += b[m];
            da[m] += db[m];
          }
        } else {  // each leaf occurs once: no squared terms
          double r[4], dr[4];
          r[0] = a[0] * b[0];
          r[1] = a[0] * b[1] + a[1] * b[0];
          r[2] = a[0] * b[2] + a[2] * b[0];
          r[3] = a[0] * b[3] + a[3] * b[0] + a[1] * b[2] + a[2] * b[1];
          dr[0] = da[0] * b[0] + a[0] * db[0];
          dr[1] = da[0] * b[1] + a[0] * db[1] + da[1] * b[0] + a[1] * db[0];
          dr[2] = da[0] * b[2] + a[0] * db[2] + da[2] * b[0] + a[2] * db[0];
          dr[3] = da[0] * b[3] + a[0] * db[3] + da[3] * b[0] + a[3] * db[0] + da[1] * b[2] + a[1] * db[2] +
                  da[2] * b[1] + a[2] * db[1];
          for (int m = 0; m < 4; ++m) {
            a[m] = r[m];
            da[m] = dr[m];
          }
        }
      }
    }
    g[q] = 0.5 * (dc[0][0] * s[0] + dc[0][1] * s[1] + dc[0][2] * s[2] + dc[0][3] * s[3]);
  }
}

size_t grad_fast_partials(int nsteps, int nk) { return (size_t)nsteps * (nsteps + 1) / 2 * (nk + 5) + (nk + 5); }

cudaError_t enqueue_grad_fast(const Prob* p, const Prob* eval, int nsteps, int nc_eval, int nplanes, int nk, int extra,
                              int optimise_noise, long long* fx, double* sums, double* g_out, int num_sms, cudaStream_t s,
                              long long* nlaunch) {
  const int ntiles = nsteps * (nsteps + 1) / 2, nslots = nk + 5;
  const bool two = ntiles > num_sms;
  const auto kernel = two ? k_grad_fast<2> : k_grad_fast<1>;
  const cudaError_t e = ensure_smem_attr((const void*)kernel, two ? SMEM_GRAD_FAST2 : SMEM_GRAD_FAST, GF_SMEM);
  if (e != cudaSuccess) return e;
  k_grad_fixed<<<dim3((nc_eval + 255) / 256, nplanes), 256, 0, s>>>(eval, fx);
  kernel<<<ntiles, 256, GF_SMEM, s>>>(p, eval, fx, nslots, extra);
  k_grad_fast_reduce<<<nslots, 256, 0, s>>>(p, ntiles, nslots, sums);
  k_grad_fast_out<<<1, 256, 0, s>>>(p, sums, nslots, optimise_noise ? nk : -1, g_out);
  if (nlaunch) *nlaunch += 4;
  return cudaGetLastError();
}

cudaError_t launch_identity_border(const Prob* p, int nc, cudaStream_t s) {
  k_identity_border<<<dim3(nc / TB, nc / TB), 256, 0, s>>>(p);
  return cudaGetLastError();
}

cudaError_t launch_syrk_inv(const Prob* p, int nsteps, cudaStream_t s) {
  const int smem = 2 * TB * USTRIDE * (int)sizeof(double);
  cudaError_t e = ensure_smem_attr((const void*)k_syrk_inv, SMEM_SYRK, smem);
  if (e != cudaSuccess) return e;
  k_syrk_inv<<<dim3(nsteps, nsteps), 128, smem, s>>>(p);
  return cudaGetLastError();
}

// Driver used by the host: all chunks, kernel passes and reductions.
cudaError_t enqueue_grad_passes(const Prob* p, int nsteps, int nk, int optimise_noise, double* g_out,
                                cudaStream_t s, long long* nlaunch) {
  const int nblocks = nsteps * nsteps;
  for (int q0 = 0; q0 < (nk > 0 ? nk : 1); q0 += GCHUNK) {
    k_grad<<<dim3(nsteps, nsteps), 256, 0, s>>>(p, q0);
    k_grad_reduce<<<1, GCHUNK + 1, 0, s>>>(p, nblocks, q0, nk, (q0 == 0 && optimise_noise) ? nk : -1, g_out);
    if (nlaunch) *nlaunch += 2;
  }
  return cudaGetLastError();
}

}  // namespace fgpu
