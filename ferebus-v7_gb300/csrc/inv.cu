// K^-1 from the factor on the tensor cores (the adjoint of tensor-core
// contexts): V = L'^-1 by block recursion, then K'^-1 = V^T V, with L' = 2^-e L the
// factor in the problem's scale.
//
//   * V's 128 x 128 diagonal blocks in FP64 (k_inv_diag32, k_inv_diag128);
//   * for block sizes b = 128, 256, ...: the pair (1, 2) of neighbouring blocks
//     combines as V_21 = -V_22 (L'_21 V_11): two products per level, all
//     pairs in one launch;
//   * K'^-1 = V^T V, lower tiles only.
//
// Every product is a split-integer one (ozaki.cu): the operands' rows (for V_11,
// P and V^T: columns) are scaled by a power of two above their 2-norm over the
// range summed, rounded to 55 bits, written as 7 fp16 digit planes, and
// multiplied exactly on tcgen05 in 7 levels.  By Cauchy-Schwarz every sum stays
// below the product of the two scales, so the exact level sums of all 128-wide
// k blocks of a tile add up in one int64 per element and round once.
//
// Against the FP64 sweep over identity rows and the FP64 product (N^3 / 3
// multiply-adds on a 1.05 TFLOP/s pipe: 51 ms at N = 4000) this is 24 k
// 128 x 64 x 128 tile products at the trailing update's rate (about 1 ms) and
// four launches per doubling of the block size: 1.6 ms at N = 4000 and 0.35 at
// N = 1003 (a gradient took 13.6 ms instead of 62.4, and 2.8 instead of 6.6,
// with this; 6.8 and 1.3 with what else has changed since), with the same
// errors against extended precision (7 kernels and data sets, ratio 0.7 to 1.2).
#include "fgpu_internal.h"
#include "tc_common.cuh"

#include <algorithm>

namespace fgpu {
namespace {

constexpr int IV_NSTAGE = 4;
constexpr int IV_EPI_WARPS = 16;  // 4 TMEM lane quarters x 4 groups of 16 columns
constexpr int IV_TMA_WARP = IV_EPI_WARPS, IV_MMA_WARP = IV_EPI_WARPS + 1;
constexpr int IV_THREADS = 32 * (IV_EPI_WARPS + 2);
constexpr uint32_t IV_SMEM = IV_NSTAGE * STAGE + 128;
constexpr int IV_CH = 8;  // k-chunks of 16 per k block

// exponent e with 2^e above the 2-norm whose square is s (a few float roundings off)
__device__ __forceinline__ int norm_exponent(float s, bool* bad) {
  if (!(s < 1e38f)) {
    *bad = true;
    return 0;
  }
  if (s == 0.0f) return 0;
  const float n = sqrtf(s) * 1.001f;
  return (int)((__float_as_uint(n) >> 23) & 0xFF) - 126;
}

}  // namespace

// ---------------------------------------------------------------------------
// 32 x 32 diagonal inverses: a column per lane, every fourth row per warp, the
// solved rows handed over in shared memory (one warp alone issues 496
// multiply-adds at 64 cycles each: 30 us, all blocks side by side; now 17).
// Written to V's diagonal blocks; grid (nt128 * 4) x (32, 4) threads
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(128) k_inv_diag32(const Prob* __restrict__ pp, double* __restrict__ V) {
  const Prob& P = *pp;
  if (P.status[1]) return;
  const int c0 = blockIdx.x * 32, lane = threadIdx.x, q = threadIdx.y;
  const size_t ld = (size_t)P.ld, nc = (size_t)P.Nc;
  const double w = ldexp(1.0, -*P.kscale);
  __shared__ double L[32][33];  // L[row][col]
  __shared__ double rd[32], xs[32][32];
#pragma unroll
  for (int k = q; k < 32; k += 4) L[lane][k] = k <= lane ? P.K[(size_t)(c0 + k) * ld + c0 + lane] * w : 0.0;
  __syncthreads();
  if (q == 0) rd[lane] = 1.0 / L[lane][lane];
  __syncthreads();
  double v[8];  // rows q, q + 4, ..
#pragma unroll
  for (int m = 0; m < 8; ++m) v[m] = 4 * m + q == lane ? 1.0 : 0.0;
#pragma unroll
  for (int k = 0; k < 32; ++k) {
    if (q == (k & 3)) xs[k][lane] = v[k >> 2] *= rd[k];
    __syncthreads();
    const double x = xs[k][lane];
#pragma unroll
    for (int m = k >> 2; m < 8; ++m)
      if (4 * m + q > k) v[m] = fma(-L[4 * m + q][k], x, v[m]);  // uniform in a warp
  }
#pragma unroll
  for (int m = 0; m < 8; ++m) V[(size_t)(c0 + lane) * nc + c0 + 4 * m + q] = v[m];
}

// ---------------------------------------------------------------------------
// the 128 x 128 diagonal blocks from their 32 x 32 ones: V_I = -V_II (sum_k L_Ik
// V_k), 8 columns per CTA (a lone FP64 pipe would need 90 us per block), and the
// block's sums of squares for the scales.  grid (16, nt128) x 256 threads
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(256) k_inv_diag128(const Prob* __restrict__ pp, double* __restrict__ V) {
  const Prob& P = *pp;
  if (P.status[1]) return;
  const int s0 = blockIdx.y * NB, j0 = blockIdx.x * 8, cb = j0 / 32;  // columns j0 .. + 7 of the block
  const size_t ld = (size_t)P.ld, nc = (size_t)P.Nc;
  const double w = ldexp(1.0, -*P.kscale);
  __shared__ double Lt[32][33];
  __shared__ double Vs[128][9];
  __shared__ double Rt[32][9];
  const int tid = threadIdx.x, r = tid & 31, c = tid >> 5;
  for (int I = 0; I < 4; ++I)  // the column block's own 32 rows; zero above them
    Vs[I * 32 + r][c] = I == cb ? V[(size_t)(s0 + j0 + c) * nc + s0 + I * 32 + r] : 0.0;
  for (int I = cb + 1; I < 4; ++I) {
    double acc = 0.0;
    for (int k = cb; k < I; ++k) {
      __syncthreads();
      for (int q = tid; q < 1024; q += 256)
        Lt[q & 31][q >> 5] = P.K[(size_t)(s0 + k * 32 + (q >> 5)) * ld + s0 + I * 32 + (q & 31)] * w;
      __syncthreads();
#pragma unroll 8
      for (int q = 0; q < 32; ++q) acc = fma(Lt[r][q], Vs[k * 32 + q][c], acc);
    }
    __syncthreads();
    Rt[r][c] = acc;
    for (int q = tid; q < 1024; q += 256)
      Lt[q & 31][q >> 5] = V[(size_t)(s0 + I * 32 + (q >> 5)) * nc + s0 + I * 32 + (q & 31)];
    __syncthreads();
    acc = 0.0;
    for (int q = 0; q <= r; ++q) acc = fma(Lt[r][q], Rt[q][c], acc);
    Vs[I * 32 + r][c] = -acc;
  }
  __syncthreads();
  for (int I = 0; I < 4; ++I)
    if (I != cb) V[(size_t)(s0 + j0 + c) * nc + s0 + I * 32 + r] = Vs[I * 32 + r][c];
}

// sums of squares of the diagonal tiles: per row over groups of 16 columns, per
// column over groups of 32 rows.  grid (nt128, 8) x 128 threads, 16 columns each
// (all 128 in one CTA: a chain of 26 us)
__global__ void __launch_bounds__(128) k_inv_diag_norms(const Prob* __restrict__ pp, const double* __restrict__ V,
                                                        float* __restrict__ rowpart, float* __restrict__ colpart) {
  const Prob& P = *pp;
  if (P.status[1]) return;
  const int t = blockIdx.x, g = blockIdx.y, s0 = t * NB, r = threadIdx.x;
  const size_t nc = (size_t)P.Nc;
  float s = 0.0f;
#pragma unroll
  for (int q = 0; q < 16; ++q) {
    const float x = (float)V[(size_t)(s0 + g * 16 + q) * nc + s0 + r];
    s = fmaf(x, x, s);
    float y = x * x;
    for (int o = 16; o > 0; o >>= 1) y += __shfl_down_sync(0xffffffffu, y, o);
    if ((r & 31) == 0) colpart[(size_t)(t * 4 + (r >> 5)) * nc + s0 + g * 16 + q] = y;
  }
  rowpart[(size_t)(t * 8 + g) * nc + s0 + r] = s;
}

// ---------------------------------------------------------------------------
// digit planes of one 128 x 128 operand tile: four threads per operand row and
// two CTAs per tile, two groups of 8 entries each.  A row's norm is summed by
// its four threads.  A level has fewer tiles than the GPU has SMs at N = 1000,
// and its chain per thread is what it costs: with one thread per row, 51 us a
// level at N = 1003 and 56 at N = 4000, now 13 and 23.
// kind 0: rows of L' (norms below 1); 1: rows of V; 2: columns of V; 3: columns of P
// grid (tasks, 2) x (128, 4) threads
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(512)
    k_inv_split(const Prob* __restrict__ pp, const InvSplit* __restrict__ tasks, const double* __restrict__ V,
                const double* __restrict__ Pm, const float* __restrict__ rowpart, const float* __restrict__ colpart,
                const float* __restrict__ colpart_p, int* __restrict__ exps, unsigned char* __restrict__ dr,
                unsigned char* __restrict__ dc) {
  const Prob& P = *pp;
  if (P.status[1]) return;
  const InvSplit T = tasks[blockIdx.x];
  const int r = threadIdx.x, i = T.row * NB + r;  // operand row: a matrix row (kinds 0, 1) or column (2, 3)
  const size_t nc = (size_t)P.Nc;
  bool bad = false;
  int e = 0;
  if (T.kind > 0) {  // block-uniform
    __shared__ float sum[4][NB];
    const float* part = T.kind == 1 ? rowpart : (T.kind == 2 ? colpart : colpart_p);
    float s = 0.0f;
#pragma unroll 8
    for (int g = T.g0 + threadIdx.y; g < T.g1; g += 4) s += part[(size_t)g * nc + i];
    sum[threadIdx.y][r] = s;
    __syncthreads();
    e = norm_exponent((sum[0][r] + sum[1][r]) + (sum[2][r] + sum[3][r]), &bad);
  }
  if (blockIdx.y == 0 && threadIdx.y == 0) exps[(size_t)T.kind * nc + i] = e;
  const int es = T.kind == 0 ? *P.kscale : e;
  const bool rows = T.kind <= 1;
  const double* src = T.kind == 0 ? P.K : (T.kind == 3 ? Pm : V);
  const size_t ld = T.kind == 0 ? (size_t)P.ld : nc;
  const int k0 = T.k * NB;
  unsigned char* dst = (T.kind <= 1 ? dr : dc) + (size_t)T.slot * NSLICE * SLICE_BYTES + (size_t)r * 16;
  const int kg0 = (blockIdx.y * 4 + threadIdx.y) * 2;
#pragma unroll
  for (int kg = kg0; kg < kg0 + 2; ++kg) {
    long long F[8];
    if (rows) {
#pragma unroll
      for (int q = 0; q < 8; ++q) F[q] = to_fixed55(src[(size_t)(k0 + kg * 8 + q) * ld + i], es, &bad);
    } else {
      const double2* s2 = reinterpret_cast<const double2*>(src + (size_t)i * ld + k0 + kg * 8);
#pragma unroll
      for (int q = 0; q < 4; ++q) {
        const double2 v = s2[q];
        F[2 * q] = to_fixed55(v.x, es, &bad);
        F[2 * q + 1] = to_fixed55(v.y, es, &bad);
      }
    }
    uint4 d[NSLICE];
    digits8_of_fixed55(F, d);
#pragma unroll
    for (int p = 0; p < NSLICE; ++p)
      *reinterpret_cast<uint4*>(dst + (size_t)p * SLICE_BYTES + (size_t)kg * 2048) = d[p];
  }
  if (bad) atomicOr(&P.status[3], 1);
}

// ---------------------------------------------------------------------------
// the tile products: persistent and warp-specialised like the trailing update
// (ozaki.cu), each 128 x 64 tile summed over its nkb k blocks in one int64 per
// element held in registers.  out = +-(A B^T) 2^(eout_mul e), with the sums of
// squares of the tile where asked for
// ---------------------------------------------------------------------------
__global__ void __launch_bounds__(IV_THREADS, 1)
    k_inv_gemm(const Prob* __restrict__ pp, const InvTile* __restrict__ tiles, int total, const void* __restrict__ map_a,
               const void* __restrict__ map_b, const int* __restrict__ ea, const int* __restrict__ eb, int negate,
               int eout_mul, double* __restrict__ out, float* __restrict__ rowpart, float* __restrict__ colpart) {
  const Prob& P = *pp;
  if (P.status[1]) return;
  extern __shared__ __align__(1024) unsigned char smi[];
  uint64_t* full = reinterpret_cast<uint64_t*>(smi + IV_NSTAGE * STAGE);
  uint64_t* empty = full + IV_NSTAGE;
  uint64_t* tfull = full + 2 * IV_NSTAGE;
  uint64_t* tempty = tfull + 1;
  uint64_t* drain = tfull + 2;  // quiescing after a give-up
  uint32_t* slot = reinterpret_cast<uint32_t*>(tfull + 3);
  __shared__ int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t issued = 0;
  if (tid == 0) {
    s_abort = 0;
    for (int k = 0; k < IV_NSTAGE; ++k) {
      mbar_init(&full[k], 1);
      mbar_init(&empty[k], 1);
    }
    mbar_init(tfull, 1);
    mbar_init(tempty, IV_EPI_WARPS * 32);
    mbar_init(drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == IV_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(su32(slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tbase = *slot;

  if (warp == IV_TMA_WARP) {
    if (lane == 0) {
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map_a) : "memory");
      asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(map_b) : "memory");
      uint32_t g = 0;
      for (int t = blockIdx.x; t < total && !s_abort; t += gridDim.x) {
        const InvTile T = tiles[t];
        for (int c = 0; c < IV_CH * T.nkb; ++c, ++g) {
          const int st = g % IV_NSTAGE;
          if (!mbar_wait(&empty[st], ((g / IV_NSTAGE) & 1) ^ 1)) {
            s_abort = 1;
            break;
          }
          unsigned char* As = smi + st * STAGE;
          const int kb = c / IV_CH, cc = c % IV_CH;
          mbar_expect_tx(&full[st], STAGE);
          tma_load_5d(As, map_a, 0, 0, 2 * cc, 0, T.a0 + kb * T.astep, &full[st]);
          tma_load_5d(As + A_STAGE, map_b, 0, (T.col & 1) * 2, 0, 2 * cc, T.b0 + kb * T.bstep, &full[st]);
          issued = g + 1;
        }
      }
    }
  } else if (warp == IV_MMA_WARP) {
    if (lane == 0) {
      uint32_t g = 0, it = 0;
      const uint64_t adesc0 = smem_desc(su32(smi), 2048, 128);
      const uint64_t bdesc0 = smem_desc(su32(smi) + A_STAGE, NSLICE * 1024, 128);
      for (int t = blockIdx.x; t < total && !s_abort; t += gridDim.x) {
        const int nkb = tiles[t].nkb;
        for (int kb = 0; kb < nkb; ++kb, ++it) {
          if (!mbar_wait(tempty, (it & 1) ^ 1)) {
            s_abort = 1;
            break;
          }
          asm volatile("tcgen05.fence::after_thread_sync;");
          bool ok = true;
          for (int c = 0; c < IV_CH; ++c, ++g) {
            const int st = g % IV_NSTAGE;
            if (!mbar_wait(&full[st], (g / IV_NSTAGE) & 1)) {
              ok = false;
              break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;");
            const uint64_t soff = (uint64_t)((st * STAGE) >> 4);
            issue_chunk_128x64(tbase, adesc0 + soff, bdesc0 + soff, c == 0);
            mma_commit(&empty[st]);
          }
          if (!ok) {
            s_abort = 1;
            break;
          }
          mma_commit(tfull);
        }
      }
    }
  } else {
    const int h = warp >> 2;
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    const size_t nc = (size_t)P.Nc;
    uint32_t it = 0;
    bool stop = false;
    for (int t = blockIdx.x; t < total && !stop; t += gridDim.x) {
      const InvTile T = tiles[t];
      unsigned long long acc[16];
#pragma unroll
      for (int q = 0; q < 16; ++q) acc[q] = 0;
      for (int kb = 0; kb < T.nkb; ++kb, ++it) {
        if (!mbar_wait(tfull, it & 1)) {
          s_abort = 1;
          stop = true;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
#pragma unroll
        for (int gq = 0; gq < 2; ++gq) {
          uint32_t v[NSLICE][8];
#pragma unroll
          for (int l = 0; l < NSLICE; ++l) tmem_ld8(v[l], tbase + lane_base + (uint32_t)(l * 64 + h * 16 + gq * 8));
          asm volatile("tcgen05.wait::ld.sync.aligned;");
          // magic-add conversion where the warp's sums lie in (-2^22, 2^22), F2I otherwise
          float mx = 0.0f;
#pragma unroll
          for (int l = 0; l < NSLICE; ++l)
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) mx = fmaxf(mx, fabsf(__uint_as_float(v[l][jj])));
          const bool magic = __all_sync(0xffffffffu, mx < 4194304.0f);
          if (gq == 1) {
            asm volatile("tcgen05.fence::before_thread_sync;");
            mbar_arrive(tempty);
          }
          if (magic) {
#pragma unroll
            for (int l = 0; l < NSLICE; ++l)
#pragma unroll
              for (int jj = 0; jj < 8; ++jj) v[l][jj] = level_bits(v[l][jj]);
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) acc[gq * 8 + jj] += (unsigned long long)level_bits_to_w64(v, jj);
          } else {
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) {
              int S[NSLICE];
#pragma unroll
              for (int l = 0; l < NSLICE; ++l) S[l] = __float2int_rn(__uint_as_float(v[l][jj]));
              acc[gq * 8 + jj] += (unsigned long long)levels_to_w64(S);
            }
          }
        }
      }
      if (stop) break;
      const int i = T.row * NB + (warp & 3) * 32 + lane, j0 = T.col * TB + h * 16;
      const int er = ea[i];
      const double so = ldexp(1.0, eout_mul * *P.kscale);
      float rs = 0.0f;
#pragma unroll
      for (int q = 0; q < 16; ++q) {
        const long long W = negate ? (long long)(0ULL - acc[q]) : (long long)acc[q];
        const double x = so * fixed62_to_double(W, er + __ldg(&eb[j0 + q]));
        out[(size_t)(j0 + q) * nc + i] = x;
        if (colpart) {
          const float f = (float)x;
          rs = fmaf(f, f, rs);
          float y = f * f;
          for (int o = 16; o > 0; o >>= 1) y += __shfl_down_sync(0xffffffffu, y, o);
          if (lane == 0) colpart[(size_t)(T.row * 4 + (warp & 3)) * nc + j0 + q] = y;
        }
      }
      if (rowpart) rowpart[(size_t)(T.col * 4 + h) * nc + i] = rs;
    }
  }
  __syncthreads();
  if (s_abort) {
    if (warp == IV_TMA_WARP && lane == 0) drain_ring(full, IV_NSTAGE, issued);
    if (warp == IV_MMA_WARP && lane == 0) drain_mmas(drain);
    __syncthreads();
    if (tid == 0) atomicExch(&P.status[2], 1);
  }
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == IV_MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tbase));
}

// ---------------------------------------------------------------------------
// host: the levels' task lists, and the launches
// ---------------------------------------------------------------------------
size_t inv_slots(int nt128) { return (size_t)nt128 * (nt128 + 1) / 2; }

void inv_schedule(int nt, std::vector<InvSplit>& splits, std::vector<InvTile>& tiles, std::vector<InvLevel>& levels) {
  splits.clear();
  tiles.clear();
  levels.clear();
  for (int b = 1; b < nt; b *= 2) {
    InvLevel L{};
    int slot_r = 0, slot_c = 0;
    std::vector<InvTile> t1, t2;
    L.split1 = (int)splits.size();
    std::vector<InvSplit> sp;  // P's columns
    for (int c0 = 0; c0 + b < nt; c0 += 2 * b) {
      const int r0 = c0 + b, r1 = std::min(nt, r0 + b);
      const int l21 = slot_r;  // (r, k): l21 + (r - r0) b + (k - c0)
      for (int r = r0; r < r1; ++r)
        for (int k = c0; k < r0; ++k) splits.push_back({slot_r++, 0, r, k, 0, 0});
      std::vector<int> v22(r1 - r0);  // (r, k <= r): v22[r - r0] + (k - r0)
      for (int r = r0; r < r1; ++r) {
        v22[r - r0] = slot_r;
        for (int k = r0; k <= r; ++k) splits.push_back({slot_r++, 1, r, k, r0 * 8, (r + 1) * 8});
      }
      std::vector<int> v11(b);  // (c, k >= c): v11[c - c0] + (k - c)
      for (int c = c0; c < r0; ++c) {
        v11[c - c0] = slot_c;
        for (int k = c; k < r0; ++k) splits.push_back({slot_c++, 2, c, k, c * 4, r0 * 4});
      }
      const int pt = slot_c;  // (c, k in the row block): pt + (c - c0)(r1 - r0) + (k - r0)
      for (int c = c0; c < r0; ++c)
        for (int k = r0; k < r1; ++k) sp.push_back({slot_c++, 3, c, k, r0 * 4, r1 * 4});
      for (int r = r0; r < r1; ++r)
        for (int c = c0; c < r0; ++c)
          for (int half = 0; half < 2; ++half) {
            t1.push_back({l21 + (r - r0) * b + (c - c0), 1, v11[c - c0], 1, r0 - c, r, 2 * c + half, 0});
            t2.push_back({v22[r - r0], 1, pt + (c - c0) * (r1 - r0), 1, r - r0 + 1, r, 2 * c + half, 0});
          }
    }
    L.nsplit1 = (int)splits.size() - L.split1;
    L.split2 = (int)splits.size();
    L.nsplit2 = (int)sp.size();
    splits.insert(splits.end(), sp.begin(), sp.end());
    // longest sums first: the persistent CTAs stride through the list
    auto longer = [](const InvTile& x, const InvTile& y) { return x.nkb > y.nkb; };
    std::stable_sort(t1.begin(), t1.end(), longer);
    std::stable_sort(t2.begin(), t2.end(), longer);
    L.tile1 = (int)tiles.size();
    L.ntile1 = (int)t1.size();
    tiles.insert(tiles.end(), t1.begin(), t1.end());
    L.tile2 = (int)tiles.size();
    L.ntile2 = (int)t2.size();
    tiles.insert(tiles.end(), t2.begin(), t2.end());
    levels.push_back(L);
  }
  // V^T V: columns of V over all their rows
  InvLevel L{};
  L.split1 = (int)splits.size();
  std::vector<int> off(nt);
  int slot = 0;
  for (int c = 0; c < nt; ++c) {
    off[c] = slot;
    for (int k = c; k < nt; ++k) splits.push_back({slot++, 2, c, k, c * 4, nt * 4});
  }
  L.nsplit1 = (int)splits.size() - L.split1;
  L.tile1 = (int)tiles.size();
  for (int i = 0; i < nt; ++i)  // the longest sums first
    for (int j = 0; j < 2 * (i + 1); ++j)
      tiles.push_back({off[i], 1, off[j / 2] + (i - j / 2), 1, nt - i, i, j, 0});
  L.ntile1 = (int)tiles.size() - L.tile1;
  levels.push_back(L);
}

cudaError_t enqueue_inverse(const Prob* p, int nt128, const InvWorkspace& w, const std::vector<InvLevel>& levels,
                            int num_sms, cudaStream_t s, long long* nlaunch) {
  cudaError_t e = ensure_smem_attr((const void*)k_inv_gemm, SMEM_INV_GEMM, IV_SMEM);
  if (e != cudaSuccess) return e;
  const size_t nc = (size_t)nt128 * NB;
  const unsigned char* map_ra = w.tmaps;                   // D_R as the A operand
  const unsigned char* map_ca = w.tmaps + TMAP_BYTES;      // D_C as the A operand
  const unsigned char* map_cb = w.tmaps + TMAP_BYTES + 256;  // D_C as the stacked B operand
  long long n = 0;
  k_inv_diag32<<<nt128 * 4, dim3(32, 4), 0, s>>>(p, w.V);
  k_inv_diag128<<<dim3(16, nt128), 256, 0, s>>>(p, w.V);
  k_inv_diag_norms<<<dim3(nt128, 8), 128, 0, s>>>(p, w.V, w.rowpart, w.colpart);
  n += 3;
  auto split = [&](int first, int count) {
    k_inv_split<<<dim3(count, 2), dim3(NB, 4), 0, s>>>(p, w.splits + first, w.V, w.kinv, w.rowpart, w.colpart, w.colpart_p, w.exps, w.dr,
                                      w.dc);
    ++n;
  };
  auto gemm = [&](int first, int count, const void* ma, int ka, int kb, int negate, int eout, double* out, float* rp,
                  float* cp) {
    k_inv_gemm<<<count < num_sms ? count : num_sms, IV_THREADS, IV_SMEM, s>>>(
        p, w.tiles + first, count, ma, map_cb, w.exps + ka * nc, w.exps + kb * nc, negate, eout, out, rp, cp);
    ++n;
  };
  for (size_t l = 0; l + 1 < levels.size(); ++l) {
    const InvLevel& L = levels[l];
    split(L.split1, L.nsplit1);
    gemm(L.tile1, L.ntile1, map_ra, 0, 2, 0, 0, w.kinv, nullptr, w.colpart_p);
    split(L.split2, L.nsplit2);
    gemm(L.tile2, L.ntile2, map_ra, 1, 3, 1, 0, w.V, w.rowpart, w.colpart);
  }
  const InvLevel& L = levels.back();
  split(L.split1, L.nsplit1);
  gemm(L.tile1, L.ntile1, map_ca, 2, 2, 0, -2, w.kinv, nullptr, nullptr);
  if (nlaunch) *nlaunch += n;
  return cudaGetLastError();
}

}  // namespace fgpu
