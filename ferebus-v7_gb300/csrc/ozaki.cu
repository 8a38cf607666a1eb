// Tensor-core trailing update for the FP64 Cholesky (mode 1).
//
// GB300 executes FP64 at about 1.1 TFLOP/s, so the O(N^3) trailing update is
// moved to the 5th-generation tensor cores as an exact integer computation
// (the error-free splitting of Ozaki, Ogita and Oishi, "Error-free
// transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", Numer. Algorithms 59, 2012, with the
// power-of-two row scaling of its tensor-core use by Mukunoki et al., 2020):
//
//  * The factor has a FIXED power-of-two scale 2^e > sqrt(K_ii) (the kernels
//    here are stationary: every K_ii is the same): since sum_k L_ik^2 =
//    K_ii, every |L_ik| <= 2^e for all panels.
//  * L_ik 2^-e is rounded to 55 fractional bits and written as 7 signed
//    base-256 digits d_0..d_6 (|d| <= 129), one fp16 plane per digit.
//  * For a 128-wide panel, digit planes p (rows i) and q (rows j) are
//    multiplied by tcgen05.mma kind::f16 with f32 accumulation.  Products
//    are exact (|d_p d_q| < 2^15) and every partial sum of one level
//    L = p + q (at most 7 pairs x 128 terms x 129^2 < 2^24) is an exact
//    integer in f32, so the 7 level accumulators in TMEM hold exact integers.
//    Levels p + q > 6 (weights below 2^-62 of 2^2e) are dropped.
//  * The kernel-matrix build stores K itself as 64-bit fixed point,
//    K_ij 2^(62 - 2e) rounded once.  The epilogue turns the 7 exact level sums
//    into one int64 of the same unit and SUBTRACTS it there (every partial
//    sum of L_ik L_jk is below 2^2e by Cauchy-Schwarz, i.e. below 2^62 in the
//    unit, so 64 bits hold K and its Schur complements exactly): the
//    trailing matrix update is exact integer arithmetic, order
//    independent, and uses no FP64 instruction.  When a block column becomes
//    the next panel, the panel kernel (panel.cu) reads it from there.
#include "fgpu_internal.h"
#include "tc_common.cuh"

#include <cuda.h>
#include <cuda_fp16.h>
#include <cudaTypedefs.h>

#include <cmath>
#include <mutex>

namespace fgpu {

// ---------------------------------------------------------------------------
// trailing update of the integer accumulators: persistent, warp-specialised
//
// Output tiles are 128 rows x 64 columns; a tile's 7 level sums occupy 448
// TMEM columns.  Warp 16 (one lane) streams the digit planes of each
// k-chunk of 16 by 5-D TMA into a 4-stage ring; warp 17 (one lane) issues
// the chunk's 28 digit pairs as 10 tcgen05.mma with B's planes stacked
// along N (issue_chunk_128x64); warps 0-15 drain TMEM into registers (16
// columns per thread, two rounds of TMEM loads), release it (so the next
// tile's MMAs start), then stage each 8-column piece of the tile's exact
// sums (2 KB, contiguous in the accumulator layout) in shared memory and
// add it to the accumulators in HBM with one bulk reduction
// (cp.reduce.async.bulk .add.u64: the L2 adds, exactly, modulo 2^64), while
// the tensor cores work on the next tile.  The accumulators never pass
// through the SM, which leaves the shared memory to a fourth operand stage.
// (Per-element 64-bit reductions instead, with a fifth stage in the freed
// staging memory, measured slower: the L2 takes them at about half the
// bulk path's rate.)
//
// Accumulator per element: the Schur complement (int64) in units of
// 2^(2e - 62); tile-major storage of the lower
// triangle's 128 x 64 tiles (acc_tile), column-major inside.  Tiles of a
// step come from a packed list from the host: every problem's next diagonal
// tiles, then problem by problem, column tile major, row tile minor.  (Taken
// by tickets instead of a stride, for the launches that share a step with the
// next diagonal tiles' factorisation: 2-4% slower.)
// ---------------------------------------------------------------------------
constexpr int CH = 8;                                // k-chunks of 16 per 128-panel (one MMA each)
constexpr int NSTAGE = 4;
constexpr uint32_t UPD_PIECE = 8 * 32 * 8;  // one warp's staged accumulator piece: 8 columns x 32 rows (2 KB)
constexpr int UPD_MMA_WARPS = 1;  // the epilogue's conversion below takes all 7 levels of a column group at once
// epilogue warps: 4 TMEM lane quarters x UPD_EPI_WARPS / 4 column groups; the
// tile's 7 levels drain in 64 / (UPD_EPI_WARPS / 4) / 8 rounds of 8 columns
// per thread, and the next tile's MMAs wait for the last round
constexpr int UPD_EPI_WARPS = 16;
constexpr int UPD_COLS = 64 / (UPD_EPI_WARPS / 4);  // columns per epilogue thread
constexpr int UPD_TMA_WARP = UPD_EPI_WARPS, UPD_MMA_WARP = UPD_EPI_WARPS + 1;
constexpr int UPD_THREADS = 32 * (UPD_EPI_WARPS + 1 + UPD_MMA_WARPS);  // epilogue, TMA, MMA issue
static_assert(UPD_COLS % 8 == 0 && UPD_EPI_WARPS % 4 == 0, "epilogue column groups of 8");
constexpr uint32_t UPD_SMEM = NSTAGE * STAGE + UPD_EPI_WARPS * UPD_PIECE + 256;
static_assert(UPD_SMEM <= 227 * 1024, "shared memory per CTA");

static_assert(UPD_MMA_WARPS == 1, "the update epilogue converts all 7 levels of a column group in one pass");

// KSH: a tile's 8 k-chunks are shared by 2^KSH CTAs, each of which subtracts
// its part (the same integers).  Where a step has so few tiles that the parts
// still fit one wave, the loads and MMAs of one tile are what it costs: the
// updates of a lone N = 500 39 -> 28 us, of N = 1501 138 -> 116.
template <int KSH>
__global__ void __launch_bounds__(UPD_THREADS, 1)
    k_ozaki_update(const Prob* __restrict__ probs, int nprob, int s, const unsigned long long* __restrict__ tiles,
                   int total) {
  extern __shared__ __align__(1024) unsigned char smu[];
  unsigned char* pieces = smu + NSTAGE * STAGE;  // [epilogue warp]: its staged accumulator piece
  uint64_t* full = reinterpret_cast<uint64_t*>(smu + NSTAGE * STAGE + UPD_EPI_WARPS * UPD_PIECE);
  uint64_t* empty = full + NSTAGE;
  uint64_t* tfull = full + 2 * NSTAGE;
  uint64_t* tempty = tfull + 1;                     // [UPD_MMA_WARPS]: that warp's levels drained
  uint64_t* drain = tempty + UPD_MMA_WARPS;         // quiescing after a give-up
  uint32_t* slot = reinterpret_cast<uint32_t*>(drain + 1);
  __shared__ int s_abort;
  const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
  uint32_t issued = 0;  // producer lane: k-chunks whose operand copies were issued
  if (tid == 0) {
    s_abort = 0;
    for (int k = 0; k < NSTAGE; ++k) {
      mbar_init(&full[k], 1);
      mbar_init(&empty[k], UPD_MMA_WARPS);  // a commit from each MMA warp
    }
    mbar_init(tfull, UPD_MMA_WARPS);
    for (int k = 0; k < UPD_MMA_WARPS; ++k) mbar_init(&tempty[k], UPD_EPI_WARPS * 32);
    mbar_init(drain, 1);
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
  }
  if (warp == UPD_MMA_WARP) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], 512;" ::"r"(su32(slot)));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
  }
  asm volatile("tcgen05.fence::before_thread_sync;");
  __syncthreads();
  asm volatile("tcgen05.fence::after_thread_sync;");
  const uint32_t tbase = *slot;
  // tile t of the step: one load instead of a search over the problems
  auto tile_of = [&](int t, int& p, int& ti, int& tj) {
    const unsigned long long e = tiles[t >> KSH];
    p = (int)(e >> 40);
    ti = (int)((e >> 20) & 0xFFFFF);
    tj = (int)(e & 0xFFFFF);
  };

  // A problem that failed up to this step's panel is left out.  The next
  // panel's diagonal tile may be factored while this kernel runs, so the
  // column of the failure is looked at: every warp decides alike.
  auto failed = [&](const Prob& P) {
    const int info = P.status[0];
    return info > 0 && info <= (s + 1) * NB;
  };

  if (warp == UPD_TMA_WARP) {
    // ---------------- TMA producer ----------------
    if (lane == 0) {
      uint32_t g = 0;
      for (int t = blockIdx.x; t < total << KSH; t += gridDim.x) {
        int p, ti, tj;
        tile_of(t, p, ti, tj);
        const Prob& P = probs[p];
        if (failed(P)) continue;
        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(P.tmap_a) : "memory");
        asm volatile("fence.proxy.tensormap::generic.acquire.gpu [%0], 128;" ::"l"(P.tmap_bs) : "memory");
        for (int c = 0; c < CH >> KSH; ++c, ++g) {
          const int st = g % NSTAGE, kc = c + (t & ((1 << KSH) - 1)) * (CH >> KSH);
          if (!mbar_wait(&empty[st], ((g / NSTAGE) & 1) ^ 1)) {
            s_abort = 1;
            break;
          }
          unsigned char* As = smu + st * STAGE;
          mbar_expect_tx(&full[st], STAGE);
          tma_load_5d(As, P.tmap_a, 0, 0, 2 * kc, 0, ti, &full[st]);
          tma_load_5d(As + A_STAGE, P.tmap_bs, 0, (tj & 1) * 2, 0, 2 * kc, tj >> 1, &full[st]);
          issued = g + 1;
        }
        if (s_abort) break;
      }
    }
  } else if (warp >= UPD_MMA_WARP) {
    // ---------------- MMA issue ----------------
    const int mw = warp - UPD_MMA_WARP;
    if (lane == 0) {
      uint32_t g = 0, it = 0;
      const uint64_t adesc0 = smem_desc(su32(smu), 2048, 128);
      const uint64_t bdesc0 = smem_desc(su32(smu) + A_STAGE, NSLICE * 1024, 128);  // [k-group][plane][row]
      for (int t = blockIdx.x; t < total << KSH; t += gridDim.x) {
        int p, ti, tj;
        tile_of(t, p, ti, tj);
        if (failed(probs[p])) continue;
        if (!mbar_wait(&tempty[mw], (it & 1) ^ 1)) {  // this warp's levels of the previous tile drained
          s_abort = 1;
          break;
        }
        asm volatile("tcgen05.fence::after_thread_sync;");
        bool ok = true;
        for (int c = 0; c < CH >> KSH; ++c, ++g) {
          const int st = g % NSTAGE;
          if (!mbar_wait(&full[st], (g / NSTAGE) & 1)) {
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
        ++it;
      }
    }
  } else {
    // ---------------- epilogue (warps 0 .. UPD_EPI_WARPS - 1) ----------------
    const int h = warp >> 2;  // column group of UPD_COLS; TMEM lanes (tile rows) 32 (warp & 3) + lane
    const uint32_t lane_base = (uint32_t)((warp & 3) * 32) << 16;
    uint32_t it = 0;
    for (int t = blockIdx.x; t < total << KSH; t += gridDim.x) {
      int p, ti, tj;
      tile_of(t, p, ti, tj);
      const Prob& P = probs[p];
      if (failed(P)) continue;
      if (!mbar_wait(tfull, it & 1)) {
        s_abort = 1;
        break;
      }
      asm volatile("tcgen05.fence::after_thread_sync;");
      // drain the 7 level sums of this thread's columns in groups of 8;
      // W = sum_l S_l 2^(48 - 8 l) is gathered on the way in unsigned,
      // wrapping arithmetic (partial sums may pass 2^63, the total W stays
      // below 2^62)
      unsigned long long wv[UPD_COLS];
#pragma unroll
      for (int gq = 0; gq < UPD_COLS / 8; ++gq) {
        const int col0 = h * UPD_COLS + gq * 8;
        uint32_t v[NSLICE][8];
#pragma unroll
        for (int l = 0; l < NSLICE; ++l)
          asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                       : "=r"(v[l][0]), "=r"(v[l][1]), "=r"(v[l][2]), "=r"(v[l][3]), "=r"(v[l][4]),
                         "=r"(v[l][5]), "=r"(v[l][6]), "=r"(v[l][7])
                       : "r"(tbase + lane_base + (uint32_t)(l * 64 + col0)));
        asm volatile("tcgen05.wait::ld.sync.aligned;");
        // Exact integer level sums without the conversion unit (see
        // level_bits) when every sum of the warp's group lies in (-2^22,
        // 2^22) (up to 2^24 in principle, far rarer in practice); otherwise
        // the warp converts this group with F2I.  The range is checked on the
        // raw sums, so the conversion itself needs no second TMEM read and
        // can follow the release below.
        float mx = 0.0f;
#pragma unroll
        for (int l = 0; l < NSLICE; ++l)
#pragma unroll
          for (int jj = 0; jj < 8; ++jj) mx = fmaxf(mx, fabsf(__uint_as_float(v[l][jj])));
        const bool magic = __all_sync(0xffffffffu, mx < 4194304.0f);
        if (gq == UPD_COLS / 8 - 1) {
          // every level sum of the tile is in registers: the next tile's
          // MMAs may overwrite these TMEM columns while the last group converts
          asm volatile("tcgen05.fence::before_thread_sync;");
          mbar_arrive(&tempty[0]);
        }
        if (magic) {
#pragma unroll
          for (int l = 0; l < NSLICE; ++l)
#pragma unroll
            for (int jj = 0; jj < 8; ++jj) v[l][jj] = level_bits(v[l][jj]);
#pragma unroll
          for (int jj = 0; jj < 8; ++jj) wv[gq * 8 + jj] = 0ULL - (unsigned long long)level_bits_to_w64(v, jj);
        } else {
#pragma unroll
          for (int jj = 0; jj < 8; ++jj) {
            int S[NSLICE];
#pragma unroll
            for (int l = 0; l < NSLICE; ++l) S[l] = __float2int_rn(__uint_as_float(v[l][jj]));
            wv[gq * 8 + jj] = 0ULL - (unsigned long long)levels_to_w64(S);
          }
        }
      }
      // each 8-column group of this warp's 32 rows is one contiguous 2 KB
      // piece of the accumulator tile (acc_elem): staged in shared memory,
      // then subtracted in HBM by one bulk reduction from lane 0
      long long* ga = P.acc + acc_tile(ti, tj, P.nt128) * ACC_TILE_ELEMS;
      unsigned long long* stg = reinterpret_cast<unsigned long long*>(pieces + warp * UPD_PIECE);
#pragma unroll
      for (int pc = 0; pc < UPD_COLS / 8; ++pc) {
        if (lane == 0) asm volatile("cp.async.bulk.wait_group.read 0;" ::: "memory");  // the last reduction has read the buffer
        __syncwarp();
#pragma unroll
        for (int jj = 0; jj < 8; ++jj) stg[jj * 32 + lane] = wv[pc * 8 + jj];
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");  // visible to the bulk copy
        __syncwarp();
        if (lane == 0) {
          long long* dst = ga + acc_elem((warp & 3) * 32, h * UPD_COLS + pc * 8);
          asm volatile("cp.reduce.async.bulk.global.shared::cta.bulk_group.add.u64 [%0], [%1], %2;" ::"l"(dst),
                       "r"(su32(stg)), "r"(UPD_PIECE)
                       : "memory");
          asm volatile("cp.async.bulk.commit_group;" ::: "memory");
        }
      }
      ++it;
    }
  }
  // the accumulator reductions this warp issued complete before the CTA
  // (and its staged pieces) goes away
  if (warp < UPD_EPI_WARPS && lane == 0) asm volatile("cp.async.bulk.wait_group 0;" ::: "memory");
  __syncthreads();
  if (s_abort) {
    // a bounded wait gave up: before the CTA frees its TMEM and exits, the
    // operand copies it issued land and its MMAs complete (each of these
    // waits is bounded too), then every problem of this step is flagged
    if (warp == UPD_TMA_WARP && lane == 0) drain_ring(full, NSTAGE, issued);
    if (warp == UPD_MMA_WARP && lane == 0) drain_mmas(drain);
    __syncthreads();
    if (tid == 0)
      for (int q = 0; q < nprob; ++q) atomicExch(&probs[q].status[2], 1);
  }
  asm volatile("tcgen05.fence::after_thread_sync;");
  if (warp == UPD_MMA_WARP) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, 512;" ::"r"(tbase));
}

// ---------------------------------------------------------------------------
// host: TMA tensor maps over a problem's digit-plane buffer
// buffer layout: [row tile nt128][plane 7][k-group 16][row 128][8 fp16]; a (k-group, plane)
// block is 2 KB contiguous
// ---------------------------------------------------------------------------
int encode_slice_maps(void* host_maps, const void* slices, int tiles) {
  static PFN_cuTensorMapEncodeTiled_v12000 fn = nullptr;
  static std::mutex mu;
  {
    std::lock_guard<std::mutex> lk(mu);
    if (!fn) {
      void* f = nullptr;
      cudaDriverEntryPointQueryResult q;
      if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &f, 12000, cudaEnableDefault, &q) !=
              cudaSuccess ||
          q != cudaDriverEntryPointSuccess || !f)
        return -1;
      fn = reinterpret_cast<PFN_cuTensorMapEncodeTiled_v12000>(f);
    }
  }
  // A (k-group, plane) block of 128 rows x 16 B is 2 KB contiguous: describe it
  // as 4 rows of 256 fp16 (512 B) so each TMA request moves 512 B.
  const cuuint64_t dims[5] = {256, 4, 16, (cuuint64_t)NSLICE, (cuuint64_t)tiles};
  const cuuint64_t strides[4] = {512, 2048, (cuuint64_t)SLICE_BYTES, (cuuint64_t)NSLICE * SLICE_BYTES};
  const cuuint32_t boxA[5] = {256, 4, 2, NSLICE, 1};   // 128 rows
  const cuuint32_t boxB[5] = {256, 2, 2, NSLICE, 1};   // 64 rows
  const cuuint32_t es[5] = {1, 1, 1, 1, 1};
  CUtensorMap* m = static_cast<CUtensorMap*>(host_maps);
  CUresult r = fn(&m[0], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, const_cast<void*>(slices), dims, strides, boxA, es,
                  CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                  CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return (int)r;
  r = fn(&m[1], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, const_cast<void*>(slices), dims, strides, boxB, es,
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return (int)r;
  // a box of 64 rows with the plane and k-group dimensions swapped: it lands
  // as [k-group][plane][row], so the 7 planes of a k-group are one operand of
  // 7 x 64 rows (the stacked-N MMAs of the trailing update)
  const cuuint64_t dimsS[5] = {256, 4, (cuuint64_t)NSLICE, 16, (cuuint64_t)tiles};
  const cuuint64_t stridesS[4] = {512, (cuuint64_t)SLICE_BYTES, 2048, (cuuint64_t)NSLICE * SLICE_BYTES};
  const cuuint32_t boxS[5] = {256, 2, NSLICE, 2, 1};
  r = fn(&m[2], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, const_cast<void*>(slices), dimsS, stridesS, boxS, es,
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  if (r != CUDA_SUCCESS) return (int)r;
  // the same with 16 rows (the panel's couplings)
  const cuuint32_t boxS16[5] = {128, 1, NSLICE, 2, 1};
  r = fn(&m[3], CU_TENSOR_MAP_DATA_TYPE_FLOAT16, 5, const_cast<void*>(slices), dimsS, stridesS, boxS16, es,
         CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_NONE, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
         CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
  return (int)r;
}

// ---------------------------------------------------------------------------
// launch helpers
// ---------------------------------------------------------------------------
cudaError_t launch_ozaki_update(const Prob* probs, int nprob, int step, int max_nt128,
                                const unsigned long long* tiles, int total_tiles, int max_ctas, cudaStream_t s) {
  if (max_nt128 - step - 1 <= 0 || total_tiles <= 0) return cudaSuccess;
  const int ksh = 4 * total_tiles <= max_ctas ? 2 : (2 * total_tiles <= max_ctas ? 1 : 0);
  const auto kernel = ksh == 2 ? k_ozaki_update<2> : (ksh == 1 ? k_ozaki_update<1> : k_ozaki_update<0>);
  const cudaError_t e = ensure_smem_attr((const void*)kernel, SMEM_OZAKI_UPDATE + ksh, UPD_SMEM);
  if (e != cudaSuccess) return e;
  const int units = total_tiles << ksh, grid = units < max_ctas ? units : max_ctas;
  kernel<<<grid, UPD_THREADS, UPD_SMEM, s>>>(probs, nprob, step, tiles, total_tiles);
  return cudaGetLastError();
}

}  // namespace fgpu
