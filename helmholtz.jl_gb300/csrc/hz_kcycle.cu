// K-cycle coarse-grid correction: two steps of FGMRES on a coarse level's
// operator, right-preconditioned by that level's own cycle, for a block of
// columns at once (the Krylov-accelerated cycle Multigrid.jl offers as
// cycleType 'K', used by test/ShiftedLaplacianTest.jl:137-140).  The same
// kernels run the "Jac-GMRES" smoother (relaxType of that test, :138): one or
// two GMRES steps preconditioned by a damped-Jacobi sweep, added to the iterate.
//
// No vector is normalised: with Z0 = M b, W = A Z0, W1 = W - (d0 / beta^2) b, Z1 = M W1,
// W2 = A Z1 the steps need only the sums below, and the correction is Y0 Z0 + Y1 Z1 (M is
// homogeneous).  Per column c they live on the device in ks[c*8 + slot]:
//   0 beta^2 = ||b||^2, 1 d0 = <b, W>, 2 n1 = ||W1||^2, 3 p0 = <b, W2>, 4 p1 = <W1, W2>,
// and the vectors' coefficients in their precision in kt[c*8 + slot]:
//   0 d0 / beta^2, 1 p0 / beta^2, 2 p1 / n1, 6 Y0, 7 Y1
// (a division or an FP64 -> FP32 conversion in every thread would cost more than the
// vectors: each takes a warp's quarter of an SM 64 clocks).
// One smoothing step needs one number, y = <W, r> / ||W||^2 for W = A Z, Z = w D^-1 r (kt slot 6);
// it also leaves A x = b - r + y W behind, so a K step after it needs no operator
// product and a first step from zero leaves the residual b - y W.
//
// Vectors are level vectors in the cycle's precision T and so is the
// per-element arithmetic (a thread sums a few terms); a warp's totals are exact to
// 48 bits (double-float tree) in FP32 and FP64 otherwise, blocks and columns are
// folded in FP64 in a fixed order (deterministic) by the last block of a column.
//
// Why: these levels are small, so launches and the reduction's FP64 steps were the cost.
// A K step took 14 launches and a smoothing step 11 (normalising copies, separate
// folds, an operator product for each residual); now 4 and 4.  Solves: 3D 193 x 161 x 97 x 16
// 630 -> 494 ms, 3D 129^3 x 8 349 -> 299 ms, 2D 641 x 321 x 33 259 -> 234 ms.
#include "hz_launch.cuh"

namespace hz {

namespace {

constexpr int kNV = 4;  // real sums per kernel

__device__ __forceinline__ void two_sum_f(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// Warp totals of four values; lane l < 32 ends with value 2 (l >= 16) + (l / 8 & 1).
// Each exchange halves the values a lane carries, so four totals take 6 steps.
__device__ __forceinline__ double warp_totals(const double (&v)[kNV], int lane) {
  const bool up = lane & 16, up2 = lane & 8;
  const double a = (up ? v[2] : v[0]) + __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 16);
  const double b = (up ? v[3] : v[1]) + __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 16);
  double s = (up2 ? b : a) + __shfl_xor_sync(0xffffffffu, up2 ? a : b, 8);
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return s;
}
__device__ __forceinline__ double warp_totals(const float (&v)[kNV], int lane) {
  const bool up = lane & 16, up2 = lane & 8;
  float a, ea, b, eb, s, es;
  two_sum_f(up ? v[2] : v[0], __shfl_xor_sync(0xffffffffu, up ? v[0] : v[2], 16), a, ea);
  two_sum_f(up ? v[3] : v[1], __shfl_xor_sync(0xffffffffu, up ? v[1] : v[3], 16), b, eb);
  float lo = (up2 ? eb : ea) + __shfl_xor_sync(0xffffffffu, up2 ? ea : eb, 8);
  two_sum_f(up2 ? b : a, __shfl_xor_sync(0xffffffffu, up2 ? a : b, 8), s, es);
  lo += es;
#pragma unroll
  for (int o = 4; o > 0; o >>= 1) {
    lo += __shfl_xor_sync(0xffffffffu, lo, o);
    two_sum_f(s, __shfl_xor_sync(0xffffffffu, s, o), s, es);
    lo += es;
  }
  return (double)s + (double)lo;
}

// Column totals of four sums over the blocks (gridDim.x, pos): the block's totals go to
// part[(pos * 4 + v) * nblk + blk]; the last block of the column to arrive folds
// them in block order and gets true with tot filled (all threads).  count[c] returns to 0.
template <typename T>
__device__ __forceinline__ bool column_totals(const T (&v)[kNV], double* part, int* count, int pos, int c,
                                              double (&tot)[kNV]) {
  __shared__ double sh[kNV][8];
  __shared__ double out[kNV];
  __shared__ int last;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  const int nblk = gridDim.x;
  const double s = warp_totals(v, lane);
  if ((lane & 7) == 0) sh[2 * (lane >> 4) + ((lane >> 3) & 1)][warp] = s;
  __syncthreads();
  if (warp == 0) {  // lane = 8 value + warp
    double t = sh[lane >> 3][lane & 7];
#pragma unroll
    for (int o = 4; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if ((lane & 7) == 0) {
      __stcg(&part[((long long)pos * kNV + (lane >> 3)) * nblk + blockIdx.x], t);
      __threadfence();
    }
    __syncwarp();
    if (lane == 0) last = atomicInc(reinterpret_cast<unsigned*>(&count[c]), (unsigned)nblk - 1) == (unsigned)nblk - 1;
  }
  __syncthreads();
  if (!last) return false;
  __threadfence();
  if (warp < kNV) {
    double t = 0.0;
    for (int b = lane; b < nblk; b += 32) t += __ldcg(&part[((long long)pos * kNV + warp) * nblk + b]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
    if (lane == 0) out[warp] = t;
  }
  __syncthreads();
#pragma unroll
  for (int k = 0; k < kNV; ++k) tot[k] = out[k];
  return true;
}

template <typename T, typename TB> __device__ __forceinline__ cplx<T> load_b(const cplx<TB>& v) {
  return mk<T>((T)v.x, (T)v.y);
}

// conj(u) w into v[i], v[i + 1]
template <typename T> __device__ __forceinline__ void add_dot(T (&v)[kNV], int i, cplx<T> u, cplx<T> w) {
  v[i] = fma(u.x, w.x, fma(u.y, w.y, v[i]));
  v[i + 1] = fma(u.x, w.y, fma(-u.y, w.x, v[i + 1]));
}
template <typename T> __device__ __forceinline__ void add_norm(T (&v)[kNV], int i, cplx<T> w) {
  v[i] = fma(w.x, w.x, fma(w.y, w.y, v[i]));
}

// coefficient in the vectors' precision; 0 unless finite: a step whose squares leave the range of
// FP32 (vectors beyond 1e19) corrects nothing
template <typename T> __device__ __forceinline__ cplx<T> narrow(double2 a) {
  const T x = (T)a.x, y = (T)a.y;
  return isfinite(x) && isfinite(y) ? mk<T>(x, y) : mk<T>(0, 0);
}
// a / n (0 for n = 0)
template <typename T> __device__ __forceinline__ cplx<T> ratio(double2 a, double n) {
  return n > 0.0 ? narrow<T>(make_double2(a.x / n, a.y / n)) : mk<T>(0, 0);
}

// Two-step least squares from the sums: the 3 x 2 problem min || beta e0 - H y || by two
// complex Givens rotations, H = [[h00, h01], [h10, h11], [0, h21]] of the normalised
// basis, scaled back to the unnormalised Z0, Z1.
template <typename T> __device__ void least_squares(const double2* s, double n2, cplx<T>* kt) {
  const double beta2 = s[0].x, n1 = fmax(s[2].x, 0.0);
  const double beta = sqrt(fmax(beta2, 0.0)), rn1 = sqrt(n1);
  double2 y0 = make_double2(0.0, 0.0), y1 = make_double2(0.0, 0.0);
  if (beta > 0.0) {
    const double2 a = make_double2(s[1].x / beta2, s[1].y / beta2);
    const double c10 = rn1 / beta;
    double2 b = make_double2(0.0, 0.0), d = b;
    double e = 0.0;
    if (rn1 > 0.0) {
      b = make_double2(s[3].x / (beta * rn1), s[3].y / (beta * rn1));
      d = make_double2(s[4].x / n1, s[4].y / n1);
      e = sqrt(fmax(n2, 0.0)) / rn1;
    }
    const double r1 = sqrt(a.x * a.x + a.y * a.y + c10 * c10);
    if (r1 > 0.0) {
      const double2 cs = make_double2(a.x / r1, a.y / r1);  // G1 = [conj(cs) sn; -sn cs], sn = c10 / r1 (real)
      const double sn = c10 / r1;
      // row 0 after G1: (r1, b'), g0 = conj(cs) beta; row 1: (0, d'), g1 = -sn beta
      const double2 bp = make_double2(cs.x * b.x + cs.y * b.y + sn * d.x, cs.x * b.y - cs.y * b.x + sn * d.y);
      const double2 dp = make_double2(-sn * b.x + cs.x * d.x - cs.y * d.y, -sn * b.y + cs.x * d.y + cs.y * d.x);
      const double2 g0 = make_double2(cs.x * beta, -cs.y * beta);
      const double g1 = -sn * beta;
      const double r2 = sqrt(dp.x * dp.x + dp.y * dp.y + e * e);
      if (r2 > 0.0) {
        // G2 on rows 1, 2: g1' = conj(dp / r2) g1, y1 = g1' / r2
        y1 = make_double2(dp.x * g1 / (r2 * r2), -dp.y * g1 / (r2 * r2));
      }
      // y0 = (g0 - b' y1) / r1
      const double2 t = make_double2(g0.x - (bp.x * y1.x - bp.y * y1.y), g0.y - (bp.x * y1.y + bp.y * y1.x));
      y0 = make_double2(t.x / (r1 * beta), t.y / (r1 * beta));
      if (rn1 > 0.0) y1 = make_double2(y1.x / rn1, y1.y / rn1);
    }
  }
  const bool ok = isfinite((T)y0.x) && isfinite((T)y0.y) && isfinite((T)y1.x) && isfinite((T)y1.y);
  kt[6] = ok ? narrow<T>(y0) : mk<T>(0, 0);
  kt[7] = ok ? narrow<T>(y1) : mk<T>(0, 0);
}

}  // namespace

// MODE KC_SMOOTH: kt slot 6 = y = <W, b> / ||W||^2;  KC_FIRST: slots 1, 0 = <b, W>, ||b||^2;
// KC_SECOND: slots 3, 4 = <b, W>, <W1, W>
template <typename T, int MODE>
__device__ __forceinline__ void kc_accumulate(T (&v)[kNV], cplx<T> b, cplx<T> w1, cplx<T> w) {
  add_dot<T>(v, 0, b, w);
  if (MODE == KC_SMOOTH) add_norm<T>(v, 2, w);
  if (MODE == KC_FIRST) add_norm<T>(v, 2, b);
  if (MODE == KC_SECOND) add_dot<T>(v, 2, w1, w);
}
template <typename T, int MODE>
__device__ __forceinline__ void kc_store(const double (&t)[kNV], double2* s, cplx<T>* kt) {
  if (MODE == KC_SMOOTH) {
    kt[6] = ratio<T>(make_double2(t[0], -t[1]), t[2]);
  } else if (MODE == KC_FIRST) {
    s[0] = make_double2(t[2], 0.0);
    s[1] = make_double2(t[0], t[1]);
    kt[0] = ratio<T>(s[1], t[2]);
  } else {
    s[3] = make_double2(t[0], t[1]);
    s[4] = make_double2(t[2], t[3]);
    kt[1] = ratio<T>(s[3], s[0].x);
    kt[2] = ratio<T>(s[4], s[2].x);
  }
}

template <typename T, typename TB, int MODE>
__global__ void __launch_bounds__(256) k_kc_dots(long long N, long long ld, const int* __restrict__ cols,
                                                 const cplx<TB>* __restrict__ B, const cplx<T>* __restrict__ W1,
                                                 const cplx<T>* __restrict__ W, double* part, int* count,
                                                 double2* __restrict__ ks, cplx<T>* __restrict__ kt) {
  const int c = cols[blockIdx.y];
  const long long off = (long long)c * ld;
  T v[kNV] = {0, 0, 0, 0};
#pragma unroll 4
  for (long long p = (long long)blockIdx.x * 256 + threadIdx.x; p < N; p += (long long)gridDim.x * 256)
    kc_accumulate<T, MODE>(v, load_b<T, TB>(B[off + p]), MODE == KC_SECOND ? W1[off + p] : mk<T>(0, 0), W[off + p]);
  double t[kNV];
  if (column_totals(v, part, count, blockIdx.y, c, t) && threadIdx.x == 0) kc_store<T, MODE>(t, ks + c * 8, kt + c * 8);
}

// W -= (d0 / beta^2) b, slot 2 = ||W||^2
template <typename T>
__global__ void __launch_bounds__(256) k_kc_update(long long N, long long ld, const int* __restrict__ cols,
                                                   const cplx<T>* __restrict__ B, cplx<T>* __restrict__ W,
                                                   double* part, int* count, double2* __restrict__ ks,
                                                   cplx<T>* __restrict__ kt, Sweep<T> sw) {
  const int c = cols[blockIdx.y];
  const long long off = (long long)c * ld;
  const cplx<T> h = kt[c * 8];
  T v[kNV] = {0, 0, 0, 0};
#pragma unroll 4
  for (long long p = (long long)blockIdx.x * 256 + threadIdx.x; p < N; p += (long long)gridDim.x * 256) {
    const cplx<T> w = cfms<T>(h, B[off + p], W[off + p]);
    W[off + p] = w;
    if (sw.y) {
      const cplx<T> d = sw.dinv[p];
      sw.y[off + p] = cmul<T>(mk<T>(d.x * sw.w, d.y * sw.w), w);
    }
    add_norm<T>(v, 0, w);
  }
  double t[kNV];
  if (column_totals(v, part, count, blockIdx.y, c, t) && threadIdx.x == 0) ks[c * 8 + 2] = make_double2(t[0], 0.0);
}

// n2 = ||W2 - (p0 / beta^2) b - (p1 / n1) W1||^2 and the least squares: kt slots 6, 7
template <typename T>
__global__ void __launch_bounds__(256) k_kc_last(long long N, long long ld, const int* __restrict__ cols,
                                                 const cplx<T>* __restrict__ B, const cplx<T>* __restrict__ W1,
                                                 const cplx<T>* __restrict__ W2, double* part, int* count,
                                                 double2* __restrict__ ks, cplx<T>* __restrict__ kt) {
  const int c = cols[blockIdx.y];
  const long long off = (long long)c * ld;
  const cplx<T> h0 = kt[c * 8 + 1], h1 = kt[c * 8 + 2];
  T v[kNV] = {0, 0, 0, 0};
#pragma unroll 4
  for (long long p = (long long)blockIdx.x * 256 + threadIdx.x; p < N; p += (long long)gridDim.x * 256)
    add_norm<T>(v, 0, cfms<T>(h1, W1[off + p], cfms<T>(h0, B[off + p], W2[off + p])));
  double t[kNV];
  if (column_totals(v, part, count, blockIdx.y, c, t) && threadIdx.x == 0) least_squares<T>(ks + c * 8, t[0], kt + c * 8);
}

// End of a smoothing step: X += y Z (y: slot 6 of yt).  MODE KC_FIRST / KC_SECOND:
// also AX = b - r + y W = A X for the cycle's right-hand side b and the K step's sums of
// it: the first step's cycle has the step's own b, the second step's has W1 (then KB
// is the step's b).
template <typename T, typename TB, int MODE>
__global__ void __launch_bounds__(256) k_kc_finish(long long N, long long ld, const int* __restrict__ cols,
                                                   const cplx<T>* __restrict__ yt, cplx<T>* __restrict__ X,
                                                   const cplx<T>* __restrict__ Z, const cplx<TB>* __restrict__ B,
                                                   const cplx<T>* __restrict__ R, const cplx<T>* __restrict__ W,
                                                   const cplx<T>* __restrict__ KB, cplx<T>* __restrict__ AX,
                                                   double* part, int* count, double2* __restrict__ ks,
                                                   cplx<T>* __restrict__ kt) {
  const int c = cols[blockIdx.y];
  const long long off = (long long)c * ld;
  const cplx<T> y = yt[c * 8 + 6];
  T v[kNV] = {0, 0, 0, 0};
#pragma unroll 2
  for (long long p = (long long)blockIdx.x * 256 + threadIdx.x; p < N; p += (long long)gridDim.x * 256) {
    X[off + p] = cfma<T>(y, Z[off + p], X[off + p]);
    if (MODE != KC_SMOOTH) {
      const cplx<T> b = load_b<T, TB>(B[off + p]);
      const cplx<T> ax = cfma<T>(y, W[off + p], csub<T>(b, R[off + p]));
      AX[off + p] = ax;
      kc_accumulate<T, MODE>(v, MODE == KC_SECOND ? KB[off + p] : b, b, ax);
    }
  }
  if (MODE == KC_SMOOTH) return;
  double t[kNV];
  if (column_totals(v, part, count, blockIdx.y, c, t) && threadIdx.x == 0) kc_store<T, MODE>(t, ks + c * 8, kt + c * 8);
}

// X = Y0 Z0 + Y1 Z1, or X += (ADD)
template <typename T, bool ADD>
__global__ void __launch_bounds__(256) k_kc_combine(long long N, long long ld, const int* __restrict__ cols,
                                                    const cplx<T>* __restrict__ kt, const cplx<T>* __restrict__ Z0,
                                                    const cplx<T>* __restrict__ Z1, cplx<T>* __restrict__ X) {
  const int c = cols[blockIdx.y];
  const cplx<T> y0 = kt[c * 8 + 6], y1 = kt[c * 8 + 7];
  const long long off = (long long)c * ld;
#pragma unroll 4
  for (long long p = (long long)blockIdx.x * 256 + threadIdx.x; p < N; p += (long long)gridDim.x * 256) {
    const cplx<T> z0 = Z0[off + p];
    X[off + p] = cfma<T>(y1, Z1[off + p], ADD ? cfma<T>(y0, z0, X[off + p]) : cmul<T>(y0, z0));
  }
}

static int kc_nblk(long long N) {
  long long b = (N + 1023) / 1024;
  return (int)std::max<long long>(1, std::min<long long>(64, b));
}

size_t kcycle_part_bytes(long long N, int R) { return (size_t)R * kNV * kc_nblk(N) * sizeof(double); }

template <typename T, typename TB>
void launch_kc_dots(Ctx& ctx, int mode, long long N, long long ld, const int* cols, int nc, const cplx<TB>* B,
                    const cplx<T>* W1, const cplx<T>* W, const KcSums& s) {
  const dim3 grid(kc_nblk(N), nc);
  const double bytes = (double)N * nc * (sizeof(cplx<TB>) + (mode == KC_SECOND ? 2 : 1) * sizeof(cplx<T>));
  if (mode == KC_SMOOTH)
    HZ_LAUNCH(ctx, "smooth_dots", bytes, (k_kc_dots<T, TB, KC_SMOOTH>), grid, 256, 0, N, ld, cols, B, W1, W, s.part,
              s.count, s.ks, (cplx<T>*)s.kt);
  else if (mode == KC_FIRST)
    HZ_LAUNCH(ctx, "kcycle_dots", bytes, (k_kc_dots<T, TB, KC_FIRST>), grid, 256, 0, N, ld, cols, B, W1, W, s.part,
              s.count, s.ks, (cplx<T>*)s.kt);
  else
    HZ_LAUNCH(ctx, "kcycle_dots", bytes, (k_kc_dots<T, TB, KC_SECOND>), grid, 256, 0, N, ld, cols, B, W1, W, s.part,
              s.count, s.ks, (cplx<T>*)s.kt);
}

template <typename T>
void launch_kc_update(Ctx& ctx, long long N, long long ld, const int* cols, int nc, const cplx<T>* B, cplx<T>* W,
                      const KcSums& s, const Sweep<T>& sweep) {
  HZ_LAUNCH(ctx, "kcycle_update", (double)N * nc * (sweep.y ? 4 : 3) * sizeof(cplx<T>), k_kc_update<T>,
            dim3(kc_nblk(N), nc), 256, 0, N, ld, cols, B, W, s.part, s.count, s.ks, (cplx<T>*)s.kt, sweep);
}

template <typename T>
void launch_kc_last(Ctx& ctx, long long N, long long ld, const int* cols, int nc, const cplx<T>* B, const cplx<T>* W1,
                    const cplx<T>* W2, const KcSums& s) {
  HZ_LAUNCH(ctx, "kcycle_last", (double)N * nc * 3 * sizeof(cplx<T>), k_kc_last<T>, dim3(kc_nblk(N), nc), 256, 0, N, ld,
            cols, B, W1, W2, s.part, s.count, s.ks, (cplx<T>*)s.kt);
}

template <typename T, typename TB>
void launch_kc_finish(Ctx& ctx, int mode, long long N, long long ld, const int* cols, int nc, const cplx<T>* yt,
                      cplx<T>* X, const cplx<T>* Z, const cplx<TB>* B, const cplx<T>* R, const cplx<T>* W,
                      const cplx<T>* KB, cplx<T>* AX, const KcSums& s) {
  const dim3 grid(kc_nblk(N), nc);
  const double bytes = (double)N * nc *
                       (3 * sizeof(cplx<T>) + (mode == KC_SMOOTH ? 0 : sizeof(cplx<TB>) + 3 * sizeof(cplx<T>)) +
                        (mode == KC_SECOND ? sizeof(cplx<T>) : 0));
  if (mode == KC_SMOOTH)
    HZ_LAUNCH(ctx, "smooth_update", bytes, (k_kc_finish<T, TB, KC_SMOOTH>), grid, 256, 0, N, ld, cols, yt, X, Z, B, R, W,
              KB, AX, s.part, s.count, s.ks, (cplx<T>*)s.kt);
  else if (mode == KC_FIRST)
    HZ_LAUNCH(ctx, "smooth_update_dots", bytes, (k_kc_finish<T, TB, KC_FIRST>), grid, 256, 0, N, ld, cols, yt, X, Z, B,
              R, W, KB, AX, s.part, s.count, s.ks, (cplx<T>*)s.kt);
  else
    HZ_LAUNCH(ctx, "smooth_update_dots", bytes, (k_kc_finish<T, TB, KC_SECOND>), grid, 256, 0, N, ld, cols, yt, X, Z, B,
              R, W, KB, AX, s.part, s.count, s.ks, (cplx<T>*)s.kt);
}

template <typename T>
void launch_kc_combine(Ctx& ctx, bool add, long long N, long long ld, const int* cols, int nc, const cplx<T>* kt,
                       const cplx<T>* Z0, const cplx<T>* Z1, cplx<T>* X) {
  const dim3 grid(kc_nblk(N), nc);
  const double bytes = (double)N * nc * (add ? 4 : 3) * sizeof(cplx<T>);
  if (add)
    HZ_LAUNCH(ctx, "smooth_update", bytes, (k_kc_combine<T, true>), grid, 256, 0, N, ld, cols, kt, Z0, Z1, X);
  else
    HZ_LAUNCH(ctx, "kcycle_combine", bytes, (k_kc_combine<T, false>), grid, 256, 0, N, ld, cols, kt, Z0, Z1, X);
}

#define HZ_KC_INST_TB(T, TB)                                                                                           \
  template void launch_kc_dots<T, TB>(Ctx&, int, long long, long long, const int*, int, const cplx<TB>*,               \
                                      const cplx<T>*, const cplx<T>*, const KcSums&);                                  \
  template void launch_kc_finish<T, TB>(Ctx&, int, long long, long long, const int*, int, const cplx<T>*, cplx<T>*,    \
                                        const cplx<T>*, const cplx<TB>*, const cplx<T>*, const cplx<T>*,               \
                                        const cplx<T>*, cplx<T>*, const KcSums&);
#define HZ_KC_INST(T)                                                                                                  \
  HZ_KC_INST_TB(T, T)                                                                                                  \
  template void launch_kc_update<T>(Ctx&, long long, long long, const int*, int, const cplx<T>*, cplx<T>*,             \
                                    const KcSums&, const Sweep<T>&);                                                   \
  template void launch_kc_last<T>(Ctx&, long long, long long, const int*, int, const cplx<T>*, const cplx<T>*,         \
                                  const cplx<T>*, const KcSums&);                                                      \
  template void launch_kc_combine<T>(Ctx&, bool, long long, long long, const int*, int, const cplx<T>*,                \
                                     const cplx<T>*, const cplx<T>*, cplx<T>*);
HZ_KC_INST(float)
HZ_KC_INST(double)
HZ_KC_INST_TB(float, double)
HZ_KC_INST_TB(float, df64_tag)
#undef HZ_KC_INST
#undef HZ_KC_INST_TB

}  // namespace hz
