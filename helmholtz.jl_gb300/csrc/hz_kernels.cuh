// Launch wrappers for the helmgpu kernels (implemented in hz_stencil.cu and
// hz_krylov.cu).  Every wrapper launches on ctx.stream, counts the launch and,
// when profiling is on, brackets it with CUDA events.
#pragma once

#include <string>
#include <vector>

#include "../../include/helmgpu.h"
#include "hz_common.cuh"
#include "hz_fixed.cuh"
#include "hz_host.h"

namespace hz {

// Device ordinals the per-device caches of the library cover.
static constexpr int kMaxDevices = 64;

// Per-handle launch context: stream, launch counter and the optional
// per-kernel event timer.
struct Ctx {
  cudaStream_t stream = nullptr;
  long long launches = 0;
  bool profile = false;
  std::vector<std::string> names;  // kernel name table
  std::vector<long long> counts;   // launches per kernel
  std::vector<long long> timed;    // launches with an event pair (profiling on)
  std::vector<double> total_ms;    // event-timed milliseconds per kernel
  std::vector<double> alg_bytes;   // algorithmic bytes per kernel (all launches)
  std::vector<double> alg_flops;   // algorithmic flops per kernel (tensor-core and native-FP64 outer kernels; 0 elsewhere)
  struct Pending {
    int id;
    cudaEvent_t a, b;
  };
  std::vector<Pending> pending;
  std::vector<cudaEvent_t> pool;
  int name_id(const char* name);
  void before(int id, cudaEvent_t* a);
  void after(int id, cudaEvent_t a, double bytes);
  void resolve();  // after a stream sync: fold pending event pairs into the table
  void add_bytes(const char* name, double bytes) { alg_bytes[name_id(name)] += bytes; }
  void add_flops(const char* name, double flops) { alg_flops[name_id(name)] += flops; }
  // launch-shape choices of the autotuner: CTAs aimed at per launch of the
  // fine-level and the Galerkin stencils (0: the default rule), which set how
  // many right-hand sides a block loops over
  int tune_fine = 0, tune_rap = 0;
  // 3D Galerkin stencils of the complex-FP32 cycle on staged tiles (k_rap_tile)
  // instead of k_rap: opt-in (HELMGPU_RAP_TILED=1) until timed on a GB300
  bool rap_tiled = false;
  void release();
};

// Jacobi / residual modes of the stencil kernels.
enum StencilMode { MODE_APPLY = 0, MODE_RESID = 1, MODE_JACOBI = 2 };

// Fine-level operator: constant-coefficient nodal Laplacian with the
// reference's ghost-reflection boundary rows plus a per-node complex diagonal.
struct FineOp {
  Grid g;
  double o[3];  // 1/h_d^2: interior off-diagonal magnitude per axis
  double b[3];  // BC/h_d^2: boundary-row off-diagonal magnitude per axis
  int adj;      // 1: apply the adjoint (transposed boundary rows, conjugated diagonal)
  int outer = 0;  // 1: the Krylov method's operator H (launch-table names outer_*), 0: a cycle operator
  // FP64 MODE_APPLY: column c's result times 2^basis_exponent(sig[c * sig_stride]) (null: as it is)
  const double* sig = nullptr;
  int sig_stride = 0;
};

// y = op(x) on nodes of a fine level, for the columns cols[0..ncols) of the
// RHS block (column c starts at c*ld), computed in precision T.  b may be
// FP64 while x/y are FP32, and x may be FP32 while y is FP64.
template <typename T, typename TX, typename TB>
void launch_fine(Ctx& ctx, int mode, const FineOp& op, const cplx<T>* diag, const cplx<T>* dinv, const cplx<TX>* x,
                 const cplx<TB>* b, cplx<T>* y, long long ld, const int* cols, int ncols, double w);

// y = op(x), b - op(x) or x + weight dinv (b - op(x)) in FP64 accuracy on the integer pipe (hz_fine_fixed.cu), where
// fine_fixed_fits() and fine_fixed_pays() say so.  Rounds otherwise than launch_fine: not for
// arithmetic whose bits have to be those of another path.
struct FixedRefs {
  int exponent;  // the largest of the operator's coefficients, from launch_fine_setup
  Fixed o[3];    // minus the neighbours' coefficients per axis, from launch_diag_fixed
};
struct FixedDiag {
  const FixedRefs* refs;
  const int4* d;  // the diagonal's limbs, from launch_diag_fixed
};
void launch_diag_fixed(Ctx& ctx, const FineOp& op, const double2* d, FixedRefs* refs, int4* out);
bool fine_fixed_fits(const FineOp& op, int exponent);  // the operator's coefficients
bool fine_fixed_pays(const FineOp& op, int ncols);     // the block
template <typename TX>
void launch_fine_fixed(Ctx& ctx, int mode, const FineOp& op, const double2* diag, const FixedDiag& fd,
                       const cplx<TX>* x, const double2* b, double2* y, long long ld, const int* cols, int ncols,
                       const double2* dinv = nullptr, double weight = 0.0);

// The first Jacobi sweep y = w dinv .* r of a Galerkin level, written by the kernel that makes
// its right-hand side r (y null: none): the same numbers as launch_jacobi0, which on small
// levels is a launch of 1 us for each visit (129^2, one source, V-cycle: 18.2 -> 17.9 ms a
// solve; 257 x 129 x 4, W-cycle: 114 -> 113; 3D: 0.1% to 0.6%).
template <typename T> struct Sweep {
  const cplx<T>* dinv = nullptr;
  cplx<T>* y = nullptr;
  T w = T(0);
};
// Galerkin level: 3^d stored complex coefficients per node, coef[k*cld + p]
// is the entry A(p, p + offset_k), offset_k = (k%3-1, k/3%3-1, k/9-1).
template <typename T, typename TB>
void launch_rap(Ctx& ctx, int mode, const Grid& g, const cplx<T>* coef, long long cld, const cplx<T>* dinv,
                const cplx<T>* x, const cplx<TB>* b, cplx<T>* y, long long ld, const int* cols, int ncols, double w,
                const Sweep<T>& sweep = Sweep<T>());

// y = w * dinv .* b  (first Jacobi sweep from a zero guess); adj conjugates dinv.
template <typename T, typename TB>
void launch_jacobi0(Ctx& ctx, const Grid& g, const cplx<T>* dinv, int adj, const cplx<TB>* b, cplx<T>* y, long long ld,
                    const int* cols, int ncols, double w);

// Full-weighting restriction rc = P^T rf / 2^d (fine grid gf, coarse grid gc).
template <typename T>
void launch_restrict(Ctx& ctx, const Grid& gf, const Grid& gc, const cplx<T>* rf, long long ldf, cplx<T>* rc,
                     long long ldc, const int* cols, int ncols, const Sweep<T>& sweep = Sweep<T>());
// The same of b - y W, y = yt[c*8 + 6].
template <typename T, typename TB>
void launch_restrict_diff(Ctx& ctx, const Grid& gf, const Grid& gc, const cplx<TB>* b, const cplx<T>* W,
                          const cplx<T>* yt, long long ldf, cplx<T>* rc, long long ldc, const int* cols, int ncols,
                          const Sweep<T>& sweep);

// A coarse-grid correction: z0, or Y0 z0 + Y1 z1 with the K-cycle's coefficients kt (slots 6, 7).
template <typename T> struct Correction {
  const cplx<T>* z0 = nullptr;
  const cplx<T>* z1 = nullptr;
  const cplx<T>* kt = nullptr;
};
// xout = base + P e (bi/trilinear nodal prolongation); base: nothing (xin null), xin, or
// y xin with y = yt[c*8 + 6] (yt not null).
template <typename T>
void launch_prolong(Ctx& ctx, const Grid& gf, const Grid& gc, const Correction<T>& e, long long ldc,
                    const cplx<T>* xin, const cplx<T>* yt, cplx<T>* xout, long long ldf, const int* cols, int ncols);

// Coarsest-level direct solve: blocked banded LU (see band_block_operators);
// T / G are the device copies of the forward / backward block operators.
// work holds 3 * ncols * N FP64 complex values.
struct BandSolveOps {
  long long N = 0;
  std::vector<BandBlock> blocks;
  const BandBlock* dblocks = nullptr;  // device copy of blocks: one cooperative launch per solve
  const double2* T = nullptr;
  const double2* G = nullptr;
  int cluster = 0, resident = 0;  // CTAs per cluster and clusters at once, from plan_band_solve (0: no clusters)
};
// The cluster schedule for T columns of op.N rows on the current device.
template <typename T>
void plan_band_solve(BandSolveOps& op);
template <typename T>
void launch_band_solve(Ctx& ctx, const BandSolveOps& op, const cplx<T>* b, cplx<T>* x, long long ld, const int* cols,
                       int ncols, double2* work);

// Allocation-free Y = A X on device memory for hz_apply_noalloc: the column
// list lives in a static device array of kNoAllocMaxCols entries shared by all
// calls on a device.  Returns 0, -1 (bad size) or -2 (CUDA error) with *err set.
static constexpr int kNoAllocMaxCols = HZ_NOALLOC_MAX_COLS;
static constexpr int kNoAllocMaxDevices = 64;
int launch_fine_apply_noalloc(cudaStream_t stream, int dev, const FineOp& op, const double2* diag, const double2* x,
                              double2* y, long long ld, int nrhs, std::string* err);

// ---- emulated-FP64 outer FGMRES (hz_df64.cu) ---------------------------------
// w = H z with z complex FP32, accumulated in df64; w a df64 vector (TO =
// float4) or rounded to FP64 (TO = double2); dHd = diag(H) in df64.
template <typename TO>
void launch_fine_df64(Ctx& ctx, const FineOp& op, const float4* dHd, const float2* z, TO* y, long long ld,
                      const int* cols, int ncols);
// y = s[c] x (FP64 x into df64 y; may run in place on the same memory)
void launch_to_df(Ctx& ctx, long long N, const double2* x, long long xld, float4* y, long long yld, const double* s,
                  const int* cols, int ncols);
void launch_diag_to_df(Ctx& ctx, long long N, const double2* d, float4* out);
// x += sum_{i<kcol[c]} y_i Z_i with the products and their sum in df64, x FP64.
void launch_update_x_df(Ctx& ctx, long long N, const float2* Z, long long zstride, long long ld, const int* kcol,
                        const double2* y, int ystride, double2* x, long long xld, const int* cols, int ncols,
                        long long zcols);
// Coarsest solve with the block operators stored as df64 (op.T / op.G point to
// float4 arrays); work holds 3 * ncols * N df64 values.
template <typename T>
void launch_band_solve_df(Ctx& ctx, const BandSolveOps& op, const cplx<T>* b, cplx<T>* x, long long ld,
                          const int* cols, int ncols, float4* work);

// ---- K-cycle (hz_kcycle.cu) ------------------------------------------------------
// Two-step FGMRES and one-step smoothing on a coarse level; per-column scalars
// ks[c*8 + slot] (FP64 sums) and kt[c*8 + slot] (cplx<T> coefficients) on the device, partial
// sums (kcycle_part_bytes) and block counters (one int per column, zeroed once).
struct KcSums {
  double2* ks = nullptr;
  void* kt = nullptr;
  double* part = nullptr;
  int* count = nullptr;
};
enum KcMode { KC_SMOOTH = 0, KC_FIRST = 1, KC_SECOND = 2 };
size_t kcycle_part_bytes(long long N, int R);
// the sums of a mode: KC_SMOOTH y = <W, b> / ||W||^2; KC_FIRST <b, W>, ||b||^2;
// KC_SECOND <b, W>, <W1, W>
template <typename T, typename TB>
void launch_kc_dots(Ctx& ctx, int mode, long long N, long long ld, const int* cols, int nc, const cplx<TB>* B,
                    const cplx<T>* W1, const cplx<T>* W, const KcSums& s);
// W -= (<b, W> / ||b||^2) b and its norm
template <typename T>
void launch_kc_update(Ctx& ctx, long long N, long long ld, const int* cols, int nc, const cplx<T>* B, cplx<T>* W,
                      const KcSums& s, const Sweep<T>& sweep = Sweep<T>());
// the norm of W2 orthogonalised against b and W1, and the 3x2 least squares -> Y0, Y1
template <typename T>
void launch_kc_last(Ctx& ctx, long long N, long long ld, const int* cols, int nc, const cplx<T>* B, const cplx<T>* W1,
                    const cplx<T>* W2, const KcSums& s);
// X += y Z with y = yt[c*8 + 6]; KC_FIRST / KC_SECOND: also AX = b - R + y W and its sums (KC_SECOND:
// b is the step's W1 and KB its b)
template <typename T, typename TB>
void launch_kc_finish(Ctx& ctx, int mode, long long N, long long ld, const int* cols, int nc, const cplx<T>* yt,
                      cplx<T>* X, const cplx<T>* Z, const cplx<TB>* B, const cplx<T>* R, const cplx<T>* W,
                      const cplx<T>* KB, cplx<T>* AX, const KcSums& s);
// X = Y0 Z0 + Y1 Z1 (add: X +=)
template <typename T>
void launch_kc_combine(Ctx& ctx, bool add, long long N, long long ld, const int* cols, int nc, const cplx<T>* kt,
                       const cplx<T>* Z0, const cplx<T>* Z1, cplx<T>* X);

// ---- setup kernels ---------------------------------------------------------
// Fine-level diagonals on the device from nodal m and gamma (device arrays):
// diag(H), diag(SH) with the shift i*shift*Re(w)^2*m, and 1/diag(SH); refs[2]: the largest
// exponent fields of H's and SH's coefficients.
void launch_fine_setup(Ctx& ctx, const Grid& g, int dim, const double* h, double wr, double wi, double shift, double BC,
                       int neumann_on_top, int sommerfeld, const double* m, const double* gamma, double2* dH,
                       double2* dSH, double2* iSH, FixedRefs* refs);
void launch_probe_init(Ctx& ctx, const Grid& gc, int dim, double2* out, long long ld);
void launch_probe_scatter(Ctx& ctx, const Grid& gc, int dim, const double2* y, long long ld, double2* coef,
                          long long cld);
void launch_coef_transpose(Ctx& ctx, const Grid& g, int dim, const double2* coef, double2* coefT, long long cld);
template <typename T>
void launch_center_inverse(Ctx& ctx, const Grid& g, int dim, const double2* coef, long long cld, cplx<T>* dinv);
template <typename To, typename From>
void launch_cast(Ctx& ctx, const cplx<From>* in, cplx<To>* out, long long n);
// Column-wise cast between RHS blocks (active columns only).
template <typename To, typename From>
void launch_cast_cols(Ctx& ctx, long long N, const cplx<From>* in, long long ldi, cplx<To>* out, long long ldo,
                      const int* cols, int ncols);
template <typename T>
void launch_zero_cols(Ctx& ctx, long long N, cplx<T>* x, long long ld, const int* cols, int ncols);

// ---- Krylov kernels (FP64) -------------------------------------------------
// Conventions: per-column device arrays are indexed by the column number c
// (not by the position in the active list); V_i column c lives at
// V + (i*vstride + c)*ld.  Partial sums go to part[(pos*K1 + slot)*nblk + blk]
// and are folded in a fixed order by launch_reduce (deterministic results).
int krylov_nblk(long long N, int ncols);
// K (0 or 1) dots conj(V) . w and, with want_norm, ||w||^2 in slot K (norms and BiCGSTAB).
void launch_dots(Ctx& ctx, long long N, const double2* V, long long ld, int K, const double2* w, long long wld,
                 const int* cols, int ncols, int nblk, int want_norm, double2* part);
// Classical Gram-Schmidt with the DGKS test on the unnormalised FGMRES basis: stored v_i
// stands for sig_i v_i (sig[c*sstride + i]), w = v_{j+1} on entry.  Pass 0 runs for every
// column, pass 1 only for the columns that the test flagged (||w'||^2 < ||w||^2 / 2).  The
// per-column results and scalar work are in hz_gs.cuh.
struct GsColumn {
  int m = 0;                                      // restart length
  double2 *hA = nullptr, *hB = nullptr;           // dots of pass 0 / 1 (pass 0: ||w||^2 in slot j + 1)
  double2* coef = nullptr;                        // update coefficients sig_i^2 d_i
  int hstride = 0;
  double* sig = nullptr;
  int sstride = 0;
  double2 *Hh = nullptr, *cs = nullptr, *sn = nullptr, *g = nullptr;  // Hessenberg columns, rotations, right-hand side
  int* flag = nullptr;                            // second pass due
  double* host_est = nullptr;                     // pinned: residual estimates
  int* host_flag = nullptr;                       // pinned copy of flag
  int* count = nullptr;                           // block counters, zero
  double* part = nullptr;                         // partial sums, gs_part_bytes
  int* vexp = nullptr;                            // references of the stored basis, gs_exponents (FP64 form)
};
int gs_nblk(long long N, int ncols);
size_t gs_part_bytes(long long N, int R);
size_t gs_exponents(long long N, int vectors);
// the dots of step j (K = j + 1 vectors) and the update w -= sum coef_i V_i of one pass
// (FP64 form: pass 0 leaves V_j as fixed-point words)
void launch_gs_pass(Ctx& ctx, long long N, double2* V, long long vstride, long long ld, int j, int pass,
                    const int* cols, int ncols, const GsColumn& g);
// both passes of the double-float form; fused: the second pass's dots read no basis of their own
void launch_gs_df(Ctx& ctx, long long N, const float4* V, long long vstride, long long ld, int j, const int* cols,
                  int ncols, const GsColumn& g);
bool gs_fused_df(int vectors);
// out[c*ostride + slot] = sum over blocks of part (slot < K1); accum adds to out.
void launch_reduce(Ctx& ctx, const double2* part, const int* cols, int ncols, int K1, int nblk, double2* out,
                   int ostride, int accum);
// Deferred normalisation of the FGMRES basis: sig_0 = 1; y_i *= sig_i.
void launch_sig_init(Ctx& ctx, const int* cols, int ncols, double* sig, int sstride);
void launch_sig_y(Ctx& ctx, const int* cols, int ncols, const int* kcol, const double* sig, int sstride, double2* y,
                  int ystride);
// y[:, c] = s[c] * x[:, c]
void launch_scale_cols(Ctx& ctx, long long N, const double2* x, long long xld, double2* y, long long yld,
                       const double* s, const int* cols, int ncols);
// x[:, c] += sum_{i < kcol[c]} y[c*ystride + i] Z_i[:, c], Z in precision TZ;
// zcols = sum of kcol over the active columns (for the byte count).
template <typename TZ>
void launch_update_x(Ctx& ctx, long long N, const cplx<TZ>* Z, long long zstride, long long ld, const int* kcol,
                     const double2* y, int ystride, double2* x, long long xld, const int* cols, int ncols,
                     long long zcols);
// nrm[c] = sqrt(Re red[c*stride + slot]), inv[c] = 1/nrm[c] (0 for a zero norm).
void launch_norms(Ctx& ctx, const double2* red, int stride, int slot, const int* cols, int ncols, double* nrm,
                  double* inv);
// g[c*(m+1) + 0] = beta[c], the other entries of g zero.
void launch_cycle_init(Ctx& ctx, int m, const int* cols, int ncols, const double* beta, double2* g);
// Hh[c*(m+1)*m + jj*(m+1) + i], cs/sn[c*m + i], g[c*(m+1) + i].
// BiCGSTAB per-column scalars sc[c*8 + k] (0 rho, 1 rho_prev, 2 alpha, 3 omega,
// 4 beta) from reduced dots red[c*rstride + slot]: stage -1 init, 0 beta from
// <rh,r>, 1 alpha from <rh,v>, 2 omega from (conj<t,s>, ||t||^2).
void launch_bicg_scalars(Ctx& ctx, int stage, const int* cols, int ncols, const double2* red, int rstride,
                         double2* sc);
// mode 0: p = r + beta (p - omega v); mode 1: out = r - alpha v.  Blocks of N per column.
void launch_bicg_vec(Ctx& ctx, int mode, long long N, const double2* r, double2* p, const double2* v, double2* out,
                     const double2* sc, const int* cols, int ncols);
// x += alpha ph + omega sh; r = s - omega t.
template <typename TZ>
void launch_bicg_xr(Ctx& ctx, long long N, double2* x, const cplx<TZ>* ph, const cplx<TZ>* sh, const double2* s,
                    const double2* t, double2* r, const double2* sc, const int* cols, int ncols);
// Back substitution R y = g for the first kcol[c] entries: y[c*m + i].
void launch_lsq(Ctx& ctx, int m, const int* cols, int ncols, const int* kcol, const double2* Hh, const double2* g,
                double2* y);

}  // namespace hz
