// Internal declarations shared by the engine's translation units.
//
// Data layout in HBM (one problem = one training set evaluated at one theta):
//
//   planes  : nplanes x Nc doubles, plane-major.  One plane per (leaf, active
//             dim): x for rbf / rbf-cyclic / linear, and the pair
//             sin(x/2), cos(x/2) for periodic, so that
//             sin((xi-xj)/2) = s_i c_j - c_i s_j needs no FP64 sin per pair.
//   K       : ld x Nc, column-major (Fortran order, like the reference's
//             covariance_matrix).  Nc = N rounded up to TB; ld = Nc + TB.
//             Rows [0, N) x cols [0, N): k(X, X) + nugget (lower triangle).
//             Rows/cols [N, Nc): identity padding, so every panel is full.
//             Rows [Nc, Nc + nrhs): the right-hand sides r_q^T (border rows);
//             the Cholesky sweep turns them into (L^-1 r_q)^T, which is all
//             the log-likelihood needs.  Rows [Nc + nrhs, ld): zero.
//
// Tensor-core mode keeps the matrix as 64-bit fixed point instead (acc), the
// right-hand sides in an array of their own (rhs), and K only where the
// factor itself is wanted.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <vector>

namespace fgpu {

constexpr int TB = 64;            // panel width and tile edge
constexpr int MAX_LEAF = 8;
constexpr int MAX_POST = 16;
constexpr int MAX_PLANES = 192;
constexpr int MAX_PARAMS = 256;
constexpr int MAX_RHS = 2;

enum LeafType { L_RBF = 1, L_PERIODIC = 2, L_RBF_CYCLIC = 3, L_LINEAR = 4, L_CONSTANT = 5 };
enum PostTok : int8_t { P_SUM = -1, P_PROD = -2 };

struct Leaf {
  int type;     // LeafType
  int n;        // active dims (0 for constant)
  int plane0;   // first plane of this leaf
  int param0;   // first kernel parameter of this leaf
};

struct Spec {
  int nleaf;
  Leaf leaf[MAX_LEAF];
  int npost;
  int8_t post[MAX_POST];          // >= 0: leaf index; P_SUM / P_PROD
  int nplanes;
  int nkparams;
  uint8_t cyclic[MAX_PLANES];     // rbf-cyclic: plane's feature index is 3, 6, 9, ... (1-based)
  // tensor-core build (tensor-core mode; leaves rbf / periodic / linear /
  // constant, at most 2 rbf or periodic "distance" leaves, <= 128 digit columns)
  int tc_build;                   // 0 no, 1 yes, 2 yes and two leaves may be multiplied
  int ndot;                       // distance leaves
  int dot_leaf[2];                // their leaf indices
  int dot_koff[2];                // first digit column (multiple of 16)
  int dot_kch[2];                 // k chunks of 16
  int dot_u[2];                   // W units: <f_i, f_j> 2^(u - 2 - 2s)
};

// A 16 x 16 diagonal block of the factor (panel.cu): its entries L'_jc 2^60 at
// x[j][c] as (high, low) 30-bit halves, and 1 / L'_jj = y 2^(sh - 62).
struct alignas(16) PanelBlock {
  int2 x[16][16];
  uint2 y[16];  // high, low word
  int sh[16];
};
// 16 entries of each solved right-hand side, z = (x as above) 2^-60 scale
struct alignas(16) PanelZ {
  int2 x[MAX_RHS][16];
  double scale[MAX_RHS];
};

// What the dot-product build (engine.cu) needs per evaluation besides the scaled
// planes, from k_prep: per leaf the sum of l (periodic) or of 1 / c (linear), or
// the constant; for rbf-cyclic leaves the unit 2^-t of the weighted differences,
// whether they may pass 2^60 of it, and per plane the factor sqrt(l) g 2^t from
// differences in units of 2^-64 g, as (high word, low word >> 1), where they wrap.
constexpr unsigned long long TURN_NOT_FINITE = 1ULL << 63;  // an rbf-cyclic feature's plane entry that stands for NaN or infinity
struct DotConst {
  double leaf_c[MAX_LEAF];
  int unit[MAX_LEAF], clamp[MAX_LEAF];
  int2 mul[MAX_PLANES];
};

// Per-problem descriptor, resident in device memory.
struct Prob {
  int N, Nc, ld, nsteps, nrhs, likelihood, optimise_noise, nkparams;
  double noise;
  const double* planes;           // nplanes x Nc
  const double* y;                // Nc, zero padded
  const double* mu;               // Nc, zero padded (marginal)
  const Spec* spec;
  const double* theta;            // raw parameters
  double* K;                      // ld x Nc
  double* logdet_part;            // nsteps
  int* status;                    // [0] info (LAPACK convention), [1] failed flag
  double* out;                    // [0] ll, [1] logdet, [2] mean, [3] sigma2
  double* z;                      // Nc: the vector alpha's back-substitution starts from
  double* ll_dst;                 // optional extra destination for ll (batch output)
  int* info_dst;                  // optional extra destination for info
  // tensor-core (split-integer) trailing update; unused in FP64 mode
  int mode;                       // 0: FP64 mma.sync 64-panels, 1: tcgen05 split update, 128-panels
  int nt128;                      // Nc / 128 (mode 1)
  int* kscale;                    // [0]: the scale e, K_ii < 2^2e for every i
  long long* acc;                 // lower-triangle 128 x 64 tiles: K, then its Schur complements, value A 2^(2e - 62)
  unsigned char* slices;          // (nt128 + 1) x 7 x 32 KB: fp16 digit planes of the current panel; the last
                                  // slot holds its diagonal tile's, which no update reads
  const void* tmap_a;             // TMA tensor map over slices, box 8 x 128 rows x 2 kgroups x 7 planes
  const void* tmap_b;             // same, box of 64 rows
  const void* tmap_bs;            // box of 64 rows landing as [k-group][plane][row]: the 7 planes stacked along N
  const void* tmap_b16;           // same, box of 16 rows
  double* rhs;                    // MAX_RHS x Nc: right-hand sides times 2^-e, turned into L^-1 r panel by panel
  int* rowsq;                     // Nc: sums of squares of the factor's rows so far (panel.cu)
  PanelBlock* lpub;               // 8: the current panel's diagonal blocks, as its diagonal tile publishes them
  PanelZ* zpub;                   // 8: and its solved right-hand-side entries
  int keep_l;                     // K exists and receives the factor, as 60-bit fixed point (launch_factor_doubles)
  double* ldiag;                  // Nc: the factor's diagonal (keep_l)
  // dot-product kernel build (mode 1): planes scaled by sqrt(l_k) per evaluation
  double* splanes;                // nplanes x Nc
  double* norms;                  // MAX_LEAF x Nc: sum_k u_ik^2 of rbf leaves
  DotConst* dotc;
  // FP64 kernels: number of 64-row tiles when extra border rows follow the
  // right-hand-side tile (the adjoint's identity rows); 0 = nsteps + 1
  int nrt;
  // adjoint on a tensor-core context: K already holds the final factor L
  // (from the tensor-core evaluation), so the FP64 sweep works only on the
  // identity rows below the right-hand-side tile
  int border_only;
  double* kinv;                   // adjoint: K^-1 (ldkinv x Nc, lower)
  int ldkinv;
  double* gpart;                  // adjoint: per-CTA partial sums
  // tensor-core build
  const double* plane_max;        // nplanes: max_i |planes[p][i]|; rbf-cyclic: g (DotConst)
  long long* fnorm;               // 2 x Nc: W_ii of the distance leaves
  double* fcoef;                  // 4: k = a + b v0 + c v1 + d v0 v1
  int* fscale;                    // 2: s of the distance leaves, max |f| < 2^s; how their values combine
};

// Encode the four 5-D TMA tensor maps of a problem's digit-plane buffer
// (boxes of 128 and 64 rows, and 64 and 16 rows with the planes stacked) into
// host memory (TMAP_BYTES).  Returns 0 or a CUDA driver error code.
constexpr size_t TMAP_BYTES = 4 * 128;
int encode_slice_maps(void* host_maps, const void* slices, int tiles);

// Launch helpers (engine.cu).  All kernels take a device array of problems
// and index it by blockIdx.y; problems whose geometry does not reach the
// current step exit immediately, so ragged batches share one launch.
cudaError_t launch_build(const Prob* probs, int nprob, int max_nsteps, int max_nplanes, cudaStream_t s);
// mode 1: the dot-product form of the build, for kernels the tensor cores do not serve
// (cyclic: some of them have an rbf-cyclic leaf)
cudaError_t launch_build_dot(const Prob* probs, int nprob, int max_nsteps, int max_nplanes, bool cyclic, cudaStream_t s);
size_t build_dot_smem_bytes(int nplanes);
cudaError_t launch_potf2(const Prob* probs, int nprob, int step, cudaStream_t s);
// max_rowtiles: 64-row tiles of the tallest problem (0 = max_nsteps + 1)
cudaError_t launch_trsm(const Prob* probs, int nprob, int step, int max_nsteps, cudaStream_t s,
                        int max_rowtiles = 0);
cudaError_t launch_update(const Prob* probs, int nprob, int step, int max_nsteps, cudaStream_t s,
                          int max_rowtiles = 0);
cudaError_t launch_finalize(const Prob* probs, int nprob, cudaStream_t s);
// the kept factor of a tensor-core problem to doubles, in place, for alpha and the adjoint
cudaError_t launch_factor_doubles(const Prob* prob, int nt128, cudaStream_t s);
// alpha of one problem; sync: two ints of scratch
cudaError_t launch_backsolve(const Prob* prob, int nsteps, int* sync, cudaStream_t s);
size_t build_smem_bytes(int nplanes);

// Split-integer tensor-core path (ozaki.cu): 128-wide panels.
constexpr int NB = 128;
constexpr int NSLICE = 7;                       // fp16 digit planes per FP64 value
constexpr size_t SLICE_BYTES = 128 * 128 * 2;   // one digit plane of a 128-row x 128-k tile
// The fixed-point matrix is kept for lower-triangle tiles only (128 rows x
// 64 columns), one int64 per element: column tile tj holds row tiles tj / 2
// .. nt128 - 1, so a problem stores nt128 (nt128 + 1) tiles instead of
// (2 nt128) nt128.  acc_tile is the tile's index in that packed order.
// Inside a tile the elements are grouped in 32 pieces of 2 KB, one per
// (8-column group, 32-row quarter), each column-major (8 columns x 32 rows):
// the piece one epilogue warp of the trailing update adds in a single bulk
// reduction.  acc_elem is an element's index inside its tile.
__host__ __device__ inline size_t acc_tile(int ti, int tj, int nt128) {
  const long long q = tj >> 1, h = tj & 1;
  return (size_t)(2 * q * nt128 - q * (q - 1) + h * (nt128 - q) + (ti - q));
}
inline size_t acc_tiles(int nt128) { return (size_t)nt128 * (nt128 + 1); }
__host__ __device__ inline int acc_elem(int r, int c) {  // row r < 128, column c < 64 of the tile
  return (((c >> 3) * 4 + (r >> 5)) << 8) + ((c & 7) << 5) + (r & 31);
}
constexpr size_t ACC_TILE_ELEMS = (size_t)NB * TB;

// One panel of the factorisation (panel.cu), of every problem with a panel
// `step`.  order: the step's row tiles as (problem << 16 | tile), first the
// ndiag own row tiles, then the others, total_tiles in all; counter: a
// zeroed int the CTAs take tiles from; flags: PANEL_FLAGS ints per problem,
// zeroed once per evaluation.
constexpr int PANEL_FLAGS = 32;            // one 128-byte line per problem
cudaError_t launch_panel(const Prob* probs, int step, const int* order, int ndiag, int total_tiles, int* counter,
                         int* flags, int num_sms, cudaStream_t s);
cudaError_t launch_panel_rows(const Prob* probs, int step, const int* order, int ntiles, cudaStream_t s);
// Trailing update of `total_tiles` of the step's tiles, packed (problem << 40 | row
// tile << 20 | column tile), by at most max_ctas CTAs.
cudaError_t launch_ozaki_update(const Prob* probs, int nprob, int step, int max_nt128,
                                const unsigned long long* tiles, int total_tiles, int max_ctas, cudaStream_t s);
// Preparation of an evaluation and the tensor-core kernel-matrix build
// (build_tc.cu): weights, scale, right-hand sides, scaled features or feature
// digits; then the persistent build of the lower triangle.
// tiles: the lower triangle's 128 x 64 tiles of every eligible problem,
// packed (problem << 40 | row tile << 20 | column tile).
cudaError_t launch_prep(const Prob* probs, int nprob, int max_nt128, cudaStream_t s);
cudaError_t launch_build_tc(const Prob* probs, int nprob, const unsigned long long* tiles, int total_tiles,
                            bool products, int num_sms, cudaStream_t s);

// K^-1 of a tensor-core context's factor (inv.cu).  A split task turns a
// 128 x 128 operand tile into digit planes: kind 0 rows of L', 1 rows of V, 2
// columns of V, 3 columns of P = L'_21 V_11; row = its operand-row tile, k = its
// k tile, g0 .. g1 the partial sums of squares its rows' scales add up.  A tile
// task is one 128 x 64 output tile: the first slots of its operands' k blocks
// and their strides, the k blocks, row tile (128) and column tile (64).
struct InvSplit {
  int slot, kind, row, k, g0, g1;
};
struct InvTile {
  int a0, astep, b0, bstep, nkb, row, col, pad;
};
struct InvLevel {
  int split1, nsplit1, tile1, ntile1;  // L'_21, V_22, V_11; P
  int split2, nsplit2, tile2, ntile2;  // P; V_21
};
struct InvWorkspace {
  double* V = nullptr;                 // Nc x Nc, lower
  double* kinv = nullptr;              // Nc x Nc, lower: P on the way, then K^-1
  float* rowpart = nullptr;            // sums of squares of V: 16-column groups (Nc / 16) x rows
  float* colpart = nullptr;            // 32-row groups (Nc / 32) x columns
  float* colpart_p = nullptr;          // of P
  int* exps = nullptr;                 // 4 kinds x Nc: scales of the operand rows
  unsigned char* dr = nullptr;         // digit planes: row operands (kinds 0, 1)
  unsigned char* dc = nullptr;         // column operands (kinds 2, 3)
  unsigned char* tmaps = nullptr;      // tensor maps over dr, dc
  InvSplit* splits = nullptr;
  InvTile* tiles = nullptr;
};
size_t inv_slots(int nt128);  // 128 x 128 operand tiles each of dr, dc holds
void inv_schedule(int nt128, std::vector<InvSplit>& splits, std::vector<InvTile>& tiles, std::vector<InvLevel>& levels);
cudaError_t enqueue_inverse(const Prob* p, int nt128, const InvWorkspace& w, const std::vector<InvLevel>& levels,
                            int num_sms, cudaStream_t s, long long* nlaunch);

// Adjoint (grad.cu): identity rows below the right-hand-side tile turn into
// L^-T during the sweep; K^-1 = L^-T (L^-T)^T; fused dK/dtheta pass.
cudaError_t launch_identity_border(const Prob* p, int nc, cudaStream_t s);
cudaError_t launch_syrk_inv(const Prob* p, int nsteps, cudaStream_t s);
cudaError_t enqueue_grad_passes(const Prob* p, int nsteps, int nk, int optimise_noise, double* g_out,
                                cudaStream_t s, long long* nlaunch);
constexpr int GRAD_SLOTS = 33;  // parameters per fused pass + noise slot
// The dK/dtheta pass of kernels the tensor-core build serves: eval is the
// evaluation's descriptor (its scaled features and coefficients), fx nplanes x
// nc_eval int64 of scratch; extra: the kernel has linear or constant leaves.
// grad_fast_partials: doubles of partial and total sums.
size_t grad_fast_partials(int nsteps, int nk);
cudaError_t enqueue_grad_fast(const Prob* p, const Prob* eval, int nsteps, int nc_eval, int nplanes, int nk, int extra,
                              int optimise_noise, long long* fx, double* sums, double* g_out, int num_sms, cudaStream_t s,
                              long long* nlaunch);

// Opt kernel `func` into `bytes` of dynamic shared memory on the CURRENT
// device.  cudaFuncSetAttribute acts per device, so the record of what was
// already set is one bit per (device, slot), updated atomically: a second
// device, or a second thread, sets the attribute for itself.  Devices
// beyond the first 64 set it on every call.
enum SmemSlot {
  SMEM_BUILD, SMEM_UPDATE, SMEM_SYRK, SMEM_PANEL, SMEM_PANEL_ROWS, SMEM_INV_GEMM, SMEM_GRAD_FAST,
  SMEM_BUILD_DOT, SMEM_BUILD_DOT_LAST = SMEM_BUILD_DOT + 1,  // one slot per instance, as below
  SMEM_GRAD_FAST2,
  SMEM_OZAKI_UPDATE, SMEM_OZAKI_UPDATE_LAST = SMEM_OZAKI_UPDATE + 2,  // one slot per instance
  SMEM_BUILD_TC, SMEM_BUILD_TC_LAST = SMEM_BUILD_TC + 5,
  SMEM_NSLOTS
};
cudaError_t ensure_smem_attr(const void* func, int slot, int bytes);

// api.cu hooks for other translation units.
int internal_compile_spec(const int* kspec, int nkspec, int d, Spec& sp, std::vector<int>& plane_dim,
                          std::vector<int>& plane_kind);
int internal_fail(int code, const char* msg);
void internal_clear_error();
void internal_add_launches(long long n);

}  // namespace fgpu
