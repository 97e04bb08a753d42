// Multigrid kernels: matrix-free fine-level Helmholtz stencil, Galerkin
// coarse-level stencils, damped Jacobi, full-weighting restriction,
// bi/trilinear prolongation, the banded coarsest solve and the setup kernels.
//
// Replaces the sparse assembly + ParSpMatVec SpMV of the reference
// (src/GetHelmholtz.jl:33-50, 85-95; src/PlainNodalLaplacian.jl:18-46) and
// the Multigrid.jl relaxation / transfer / coarse-solve steps called from
// src/ShiftedLaplacianMultigridSolver.jl:89.
#include <algorithm>
#include <cstdio>
#include <mutex>
#include <stdexcept>
#include <string>
#include <type_traits>

#include <cooperative_groups.h>

#include "hz_launch.cuh"
#include "hz_rap_tile.cuh"

namespace cg = cooperative_groups;

namespace hz {

// ---------------------------------------------------------------------------
// Launch bookkeeping
// ---------------------------------------------------------------------------
int Ctx::name_id(const char* name) {
  for (size_t i = 0; i < names.size(); ++i)
    if (names[i] == name) return (int)i;
  names.emplace_back(name);
  counts.push_back(0);
  timed.push_back(0);
  total_ms.push_back(0.0);
  alg_bytes.push_back(0.0);
  alg_flops.push_back(0.0);
  return (int)names.size() - 1;
}

void Ctx::before(int id, cudaEvent_t* a) {
  (void)id;
  if (!profile) return;
  if (pool.empty()) {
    cudaEvent_t e;
    cudaEventCreate(&e);
    pool.push_back(e);
  }
  *a = pool.back();
  pool.pop_back();
  cudaEventRecord(*a, stream);
}

void Ctx::after(int id, cudaEvent_t a, double bytes) {
  ++launches;
  counts[id] += 1;
  alg_bytes[id] += bytes;
  if (!profile) return;
  cudaEvent_t b;
  if (pool.empty()) {
    cudaEventCreate(&b);
  } else {
    b = pool.back();
    pool.pop_back();
  }
  cudaEventRecord(b, stream);
  pending.push_back({id, a, b});
}

void Ctx::resolve() {
  for (auto& p : pending) {
    float ms = 0.f;
    if (cudaEventElapsedTime(&ms, p.a, p.b) == cudaSuccess) {
      timed[p.id] += 1;
      total_ms[p.id] += ms;
    }
    pool.push_back(p.a);
    pool.push_back(p.b);
  }
  pending.clear();
}

void Ctx::release() {
  resolve();
  for (auto e : pool) cudaEventDestroy(e);
  pool.clear();
}


// ---------------------------------------------------------------------------
// Fine-level stencil
// ---------------------------------------------------------------------------
template <typename T> struct FineOpT {
  int nx, ny, nz;
  long long N;
  T o[3], b[3];
  int adj;
  const double* sig = nullptr;
  int sig_stride = 0;
};

// Off-diagonal magnitudes of the two neighbours of node i on an axis of n
// nodes.  Row i of the 1D operator is (2u_i - u_{i-1} - u_{i+1})/h^2 inside and
// (BC u_0 - BC u_1)/h^2, (BC u_{n-1} - BC u_{n-2})/h^2 on the boundary rows
// (src/PlainNodalLaplacian.jl:18-30).  The adjoint takes entry (j, i).
template <typename T>
__device__ __forceinline__ void axis_coef(int i, int n, T o, T bb, int adj, T& cl, T& cr) {
  if (!adj) {
    cl = (i > 0) ? ((i == n - 1) ? bb : o) : T(0);
    cr = (i < n - 1) ? ((i == 0) ? bb : o) : T(0);
  } else {
    cl = (i > 0) ? ((i - 1 == 0) ? bb : o) : T(0);
    cr = (i < n - 1) ? ((i + 1 == n - 1) ? bb : o) : T(0);
  }
}

template <typename T, typename TX, typename TB, int MODE, bool IS3D>
__global__ void __launch_bounds__(256) k_fine(FineOpT<T> op, const cplx<T>* __restrict__ diag,
                                              const cplx<T>* __restrict__ dinv, const cplx<TX>* __restrict__ x,
                                              const cplx<TB>* __restrict__ b, cplx<T>* __restrict__ y, long long ld,
                                              const int* __restrict__ cols, int ncols, int cpb, T w) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= op.N) return;
  const int nx = op.nx, ny = op.ny;
  const int i = (int)(p % nx);
  const long long t = p / nx;
  const int j = (int)(t % ny);
  const int k = (int)(t / ny);
  T cxl, cxr, cyl, cyr, czl = 0, czr = 0;
  axis_coef<T>(i, nx, op.o[0], op.b[0], op.adj, cxl, cxr);
  axis_coef<T>(j, ny, op.o[1], op.b[1], op.adj, cyl, cyr);
  if (IS3D) axis_coef<T>(k, op.nz, op.o[2], op.b[2], op.adj, czl, czr);
  // clamped neighbour offsets: a missing neighbour has a zero coefficient
  const long long sx = 1, sy = nx, sz = (long long)nx * ny;
  const long long oxl = (i > 0) ? -sx : 0, oxr = (i < nx - 1) ? sx : 0;
  const long long oyl = (j > 0) ? -sy : 0, oyr = (j < ny - 1) ? sy : 0;
  long long ozl = 0, ozr = 0;
  if (IS3D) {
    ozl = (k > 0) ? -sz : 0;
    ozr = (k < op.nz - 1) ? sz : 0;
  }
  cplx<T> d = diag[p];
  if (op.adj) d.y = -d.y;
  cplx<T> di = mk<T>(0, 0);
  if (MODE == MODE_JACOBI) {
    di = dinv[p];
    if (op.adj) di.y = -di.y;
  }
  const int c0 = blockIdx.y * cpb;
  const int c1 = min(ncols, c0 + cpb);
  // columns are independent: unrolled so that several columns' loads are in flight
#pragma unroll 4
  for (int ci = c0; ci < c1; ++ci) {
    const long long off = (long long)cols[ci] * ld;
    const cplx<TX>* xc = x + off + p;
    const cplx<T> xp = ccast<T, TX>(xc[0]);
    const cplx<T> a = ccast<T, TX>(xc[oxl]), bq = ccast<T, TX>(xc[oxr]);
    const cplx<T> c = ccast<T, TX>(xc[oyl]), e = ccast<T, TX>(xc[oyr]);
    T sr = cxl * a.x + cxr * bq.x + cyl * c.x + cyr * e.x;
    T si = cxl * a.y + cxr * bq.y + cyl * c.y + cyr * e.y;
    if (IS3D) {
      const cplx<T> f = ccast<T, TX>(xc[ozl]), g = ccast<T, TX>(xc[ozr]);
      sr += czl * f.x + czr * g.x;
      si += czl * f.y + czr * g.y;
    }
    cplx<T> ax = mk<T>(-sr, -si);
    ax = cfma<T>(d, xp, ax);
    // b is read once and y written once: streaming hints keep the cache for the
    // x planes whose neighbours are read again
    if (MODE == MODE_APPLY) {
      if (std::is_same<T, double>::value && op.sig)
        ax = cscale<T>((T)basis_power(basis_exponent(op.sig[(long long)cols[ci] * op.sig_stride])), ax);
      __stcs(&y[off + p], ax);
    } else {
      const cplx<TB> bb = __ldcs(&b[off + p]);
      const cplx<T> r = mk<T>((T)bb.x - ax.x, (T)bb.y - ax.y);
      if (MODE == MODE_RESID) {
        __stcs(&y[off + p], r);
      } else {
        const cplx<T> dr = cmul<T>(di, r);
        __stcs(&y[off + p], mk<T>(xp.x + w * dr.x, xp.y + w * dr.y));
      }
    }
  }
}

template <typename T, typename TX, typename TB>
void launch_fine(Ctx& ctx, int mode, const FineOp& op, const cplx<T>* diag, const cplx<T>* dinv, const cplx<TX>* x,
                 const cplx<TB>* b, cplx<T>* y, long long ld, const int* cols, int ncols, double w) {
  if (ncols <= 0) return;
  FineOpT<T> o;
  o.nx = op.g.nx;
  o.ny = op.g.ny;
  o.nz = op.g.nz;
  o.N = op.g.N;
  for (int d = 0; d < 3; ++d) {
    o.o[d] = (T)op.o[d];
    o.b[d] = (T)op.b[d];
  }
  o.adj = op.adj;
  o.sig = op.sig;
  o.sig_stride = op.sig_stride;
  const int TPB = 256;
  long long nbx = (op.g.N + TPB - 1) / TPB;
  int ch = ctx.tune_fine > 0 ? chunks_for(nbx, ncols, ctx.tune_fine) : chunks_for(nbx, ncols);
  int cpb = (ncols + ch - 1) / ch;
  dim3 grid((unsigned)nbx, (unsigned)ch);
  const bool is3d = op.g.nz > 1;
  // x (and b) read and y written once per active column, the diagonal (and
  // its inverse) once per node
  double fbytes = (double)op.g.N * ncols * (sizeof(cplx<TX>) + sizeof(cplx<T>)) + (double)op.g.N * sizeof(cplx<T>);
  if (mode != MODE_APPLY) fbytes += (double)op.g.N * ncols * sizeof(cplx<TB>);
  if (mode == MODE_JACOBI) fbytes += (double)op.g.N * sizeof(cplx<T>);
#define HZ_FINE_CASE(M, D, NAME) \
  HZ_LAUNCH(ctx, NAME, fbytes, (k_fine<T, TX, TB, M, D>), grid, TPB, 0, o, diag, dinv, x, b, y, ld, cols, ncols, cpb, (T)w)
  const char* nm_apply = op.outer ? "outer_apply" : "fine_apply";
  const char* nm_resid = op.outer ? "outer_resid" : "fine_resid";
  // FP64 arithmetic of the Krylov method's operator, per node and column: a multiply
  // and an add per component of each real-coefficient neighbour, 8 flops for the
  // complex diagonal, 2 for b - H x
  if (op.outer && std::is_same<T, double>::value && mode != MODE_JACOBI)
    ctx.add_flops(mode == MODE_APPLY ? nm_apply : nm_resid,
                  (8.0 * (is3d ? 3 : 2) + 8.0 + (mode == MODE_RESID ? 2.0 : 0.0)) * (double)op.g.N * ncols);
  if (mode == MODE_APPLY) {
    if (is3d) HZ_FINE_CASE(MODE_APPLY, true, nm_apply);
    else HZ_FINE_CASE(MODE_APPLY, false, nm_apply);
  } else if (mode == MODE_RESID) {
    if (is3d) HZ_FINE_CASE(MODE_RESID, true, nm_resid);
    else HZ_FINE_CASE(MODE_RESID, false, nm_resid);
  } else {
    if (is3d) HZ_FINE_CASE(MODE_JACOBI, true, "fine_jacobi");
    else HZ_FINE_CASE(MODE_JACOBI, false, "fine_jacobi");
  }
#undef HZ_FINE_CASE
}

// ---------------------------------------------------------------------------
// Galerkin (stored-coefficient) stencil
// ---------------------------------------------------------------------------
// w dinv of a node, as k_jacobi0 takes it
template <typename T>
__device__ __forceinline__ cplx<T> scaled_dinv(const Sweep<T>& sw, long long p) {
  const cplx<T> d = sw.dinv[p];
  return mk<T>(d.x * sw.w, d.y * sw.w);
}

template <typename T, typename TB, int MODE, bool IS3D>
__global__ void __launch_bounds__(128) k_rap(Grid g, const cplx<T>* __restrict__ coef, long long cld,
                                             const cplx<T>* __restrict__ dinv, const cplx<T>* __restrict__ x,
                                             const cplx<TB>* __restrict__ b, cplx<T>* __restrict__ y, long long ld,
                                             const int* __restrict__ cols, int ncols, int cpb, T w, Sweep<T> sw) {
  constexpr int NS = IS3D ? 27 : 9;
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= g.N) return;
  const int nx = g.nx, ny = g.ny;
  const int i = (int)(p % nx);
  const long long t = p / nx;
  const int j = (int)(t % ny);
  const int k = (int)(t / ny);
  const long long sy = nx, sz = (long long)nx * ny;
  const long long dxo[3] = {(i > 0) ? -1LL : 0LL, 0LL, (i < nx - 1) ? 1LL : 0LL};
  const long long dyo[3] = {(j > 0) ? -sy : 0LL, 0LL, (j < ny - 1) ? sy : 0LL};
  long long dzo[3] = {0, 0, 0};
  if (IS3D) {
    dzo[0] = (k > 0) ? -sz : 0;
    dzo[2] = (k < g.nz - 1) ? sz : 0;
  }
  cplx<T> c[NS];
#pragma unroll
  for (int s = 0; s < NS; ++s) {
    c[s] = coef[s * cld + p];
  }
  cplx<T> di = mk<T>(0, 0);
  if (MODE == MODE_JACOBI) di = dinv[p];
  if (MODE == MODE_RESID && sw.y) di = scaled_dinv<T>(sw, p);
  const int c0 = blockIdx.y * cpb;
  const int c1 = min(ncols, c0 + cpb);
  // columns are independent: unrolled so that several columns' loads are in flight
#pragma unroll 2
  for (int ci = c0; ci < c1; ++ci) {
    const long long off = (long long)cols[ci] * ld;
    const cplx<T>* xc = x + off + p;
    cplx<T> ax = mk<T>(0, 0);
    cplx<T> xp = mk<T>(0, 0);
#pragma unroll
    for (int s = 0; s < NS; ++s) {
      const long long o = dxo[s % 3] + dyo[(s / 3) % 3] + (IS3D ? dzo[s / 9] : 0LL);
      const cplx<T> v = xc[o];
      if (s == NS / 2) xp = v;
      ax = cfma<T>(c[s], v, ax);
    }
    // b read once, y written once: streaming hints, as in k_fine
    if (MODE == MODE_APPLY) {
      __stcs(&y[off + p], ax);
    } else {
      const cplx<TB> bb = __ldcs(&b[off + p]);
      const cplx<T> r = mk<T>((T)bb.x - ax.x, (T)bb.y - ax.y);
      if (MODE == MODE_RESID) {
        __stcs(&y[off + p], r);
        if (sw.y) __stcs(&sw.y[off + p], cmul<T>(di, r));
      } else {
        const cplx<T> dr = cmul<T>(di, r);
        __stcs(&y[off + p], mk<T>(xp.x + w * dr.x, xp.y + w * dr.y));
      }
    }
  }
}

// The 3D Galerkin stencil of the complex-FP32 cycle on staged tiles (the steps
// and the layout are in hz_rap_tile.cuh); the same outputs, bit for bit, as k_rap.
template <typename TB, int MODE>
__global__ void __launch_bounds__(kRtThreads) k_rap_tile(Grid g, const float2* __restrict__ coef, long long cld,
                                                         const float2* __restrict__ dinv,
                                                         const float2* __restrict__ x, const cplx<TB>* __restrict__ b,
                                                         float2* __restrict__ y, long long ld,
                                                         const int* __restrict__ cols, int ncols, float w) {
  __shared__ float2 sm[kRtSmemElems];
  const RapTileCta t = rap_tile_cta(g, blockIdx.x, blockIdx.y, blockIdx.z, ncols);
  const int tid = threadIdx.x;
  rap_tile_load<float>(t, tid, t.z0 - 1, x, ld, cols, sm);
  rap_tile_load<float>(t, tid, t.z0, x, ld, cols, sm);
  for (int z = t.z0; z < t.z1; ++z) {
    // plane z + 1 takes the slot of plane z - 2, free since the barrier closing the last step
    rap_tile_load<float>(t, tid, z + 1, x, ld, cols, sm);
    __syncthreads();
    rap_tile_node<float, TB, MODE>(t, tid, z, coef, cld, dinv, b, y, ld, cols, sm, w);
    __syncthreads();
  }
}

template <typename TB>
void launch_rap_tile(Ctx& ctx, int mode, const Grid& g, const float2* coef, long long cld, const float2* dinv,
                     const float2* x, const cplx<TB>* b, float2* y, long long ld, const int* cols, int ncols, double w,
                     double bytes) {
  int bx, by, bz;
  rap_tile_grid(g, ncols, bx, by, bz);
  const dim3 grid((unsigned)bx, (unsigned)by, (unsigned)bz);
  if (mode == MODE_APPLY)
    HZ_LAUNCH(ctx, "rap_tile_apply", bytes, (k_rap_tile<TB, MODE_APPLY>), grid, kRtThreads, 0, g, coef, cld, dinv, x,
              b, y, ld, cols, ncols, (float)w);
  else if (mode == MODE_RESID)
    HZ_LAUNCH(ctx, "rap_tile_resid", bytes, (k_rap_tile<TB, MODE_RESID>), grid, kRtThreads, 0, g, coef, cld, dinv, x,
              b, y, ld, cols, ncols, (float)w);
  else
    HZ_LAUNCH(ctx, "rap_tile_jacobi", bytes, (k_rap_tile<TB, MODE_JACOBI>), grid, kRtThreads, 0, g, coef, cld, dinv,
              x, b, y, ld, cols, ncols, (float)w);
}

template <typename T, typename TB>
void launch_rap(Ctx& ctx, int mode, const Grid& g, const cplx<T>* coef, long long cld, const cplx<T>* dinv,
                const cplx<T>* x, const cplx<TB>* b, cplx<T>* y, long long ld, const int* cols, int ncols, double w,
                const Sweep<T>& sweep) {
  if (ncols <= 0) return;
  const int TPB = 128;
  long long nbx = (g.N + TPB - 1) / TPB;
  int ch = ctx.tune_rap > 0 ? chunks_for(nbx, ncols, ctx.tune_rap) : chunks_for(nbx, ncols);
  int cpb = (ncols + ch - 1) / ch;
  dim3 grid((unsigned)nbx, (unsigned)ch);
  const bool is3d = g.nz > 1;
  const int ns = is3d ? 27 : 9;
  double rbytes = (double)g.N * ncols * 2 * sizeof(cplx<T>) + (double)g.N * ns * sizeof(cplx<T>);
  if (mode != MODE_APPLY) rbytes += (double)g.N * ncols * sizeof(cplx<TB>);
  if (mode == MODE_JACOBI) rbytes += (double)g.N * sizeof(cplx<T>);
  if (sweep.y) rbytes += (double)g.N * (ncols + 1) * sizeof(cplx<T>);
  if constexpr (std::is_same<T, float>::value) {
    if (is3d && ctx.rap_tiled) {
      launch_rap_tile<TB>(ctx, mode, g, coef, cld, dinv, x, b, y, ld, cols, ncols, w, rbytes);
      if (sweep.y) launch_jacobi0<T, T>(ctx, g, sweep.dinv, 0, y, sweep.y, ld, cols, ncols, (double)sweep.w);
      return;
    }
  }
#define HZ_RAP_CASE(M, D, NAME)                                                                                         \
  HZ_LAUNCH(ctx, NAME, rbytes, (k_rap<T, TB, M, D>), grid, TPB, 0, g, coef, cld, dinv, x, b, y, ld, cols, ncols, cpb, (T)w, \
            sweep)
  if (mode == MODE_APPLY) {
    if (is3d) HZ_RAP_CASE(MODE_APPLY, true, "rap_apply");
    else HZ_RAP_CASE(MODE_APPLY, false, "rap_apply");
  } else if (mode == MODE_RESID) {
    if (is3d) HZ_RAP_CASE(MODE_RESID, true, "rap_resid");
    else HZ_RAP_CASE(MODE_RESID, false, "rap_resid");
  } else {
    if (is3d) HZ_RAP_CASE(MODE_JACOBI, true, "rap_jacobi");
    else HZ_RAP_CASE(MODE_JACOBI, false, "rap_jacobi");
  }
#undef HZ_RAP_CASE
}

// ---------------------------------------------------------------------------
// First Jacobi sweep from a zero guess: y = w dinv b
// ---------------------------------------------------------------------------
template <typename T, typename TB>
__global__ void __launch_bounds__(256) k_jacobi0(long long N, const cplx<T>* __restrict__ dinv, int adj,
                                                 const cplx<TB>* __restrict__ b, cplx<T>* __restrict__ y, long long ld,
                                                 const int* __restrict__ cols, int ncols, int cpb, T w) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= N) return;
  cplx<T> di = dinv[p];
  if (adj) di.y = -di.y;
  di.x *= w;
  di.y *= w;
  const int c0 = blockIdx.y * cpb;
  const int c1 = min(ncols, c0 + cpb);
  // columns are independent: unrolled so that several columns' loads are in flight
#pragma unroll 4
  for (int ci = c0; ci < c1; ++ci) {
    const long long off = (long long)cols[ci] * ld;
    const cplx<TB> bb = b[off + p];
    y[off + p] = cmul<T>(di, mk<T>((T)bb.x, (T)bb.y));
  }
}

template <typename T, typename TB>
void launch_jacobi0(Ctx& ctx, const Grid& g, const cplx<T>* dinv, int adj, const cplx<TB>* b, cplx<T>* y, long long ld,
                    const int* cols, int ncols, double w) {
  if (ncols <= 0) return;
  const int TPB = 256;
  long long nbx = (g.N + TPB - 1) / TPB;
  int ch = chunks_for(nbx, ncols);
  int cpb = (ncols + ch - 1) / ch;
  dim3 grid((unsigned)nbx, (unsigned)ch);
  const double jbytes = (double)g.N * ncols * (sizeof(cplx<TB>) + sizeof(cplx<T>)) + (double)g.N * sizeof(cplx<T>);
  HZ_LAUNCH(ctx, "jacobi0", jbytes, (k_jacobi0<T, TB>), grid, TPB, 0, g.N, dinv, adj, b, y, ld, cols, ncols, cpb, (T)w);
}

// ---------------------------------------------------------------------------
// Transfers
// ---------------------------------------------------------------------------
// DIFF: the fine vector is rf - y W (a smoothing step from zero leaves that residual)
template <typename T, typename TB, bool IS3D, bool DIFF>
__global__ void __launch_bounds__(256) k_restrict(Grid gf, Grid gc, const cplx<TB>* __restrict__ rf,
                                                  const cplx<T>* __restrict__ W, const cplx<T>* __restrict__ yt,
                                                  long long ldf, cplx<T>* __restrict__ rc, long long ldc,
                                                  const int* __restrict__ cols, int ncols, int cpb, Sweep<T> sw) {
  const long long q = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (q >= gc.N) return;
  const int I = (int)(q % gc.nx);
  const long long t = q / gc.nx;
  const int J = (int)(t % gc.ny);
  const int K = (int)(t / gc.ny);
  const int fi = 2 * I, fj = 2 * J, fk = 2 * K;
  const long long sy = gf.nx, sz = (long long)gf.nx * gf.ny;
  const long long pc = fi + fj * sy + (IS3D ? fk * sz : 0);
  // weights of the three fine nodes per axis; a missing node has weight 0
  const T wx[3] = {(fi > 0) ? T(0.5) : T(0), T(1), (fi < gf.nx - 1) ? T(0.5) : T(0)};
  const T wy[3] = {(fj > 0) ? T(0.5) : T(0), T(1), (fj < gf.ny - 1) ? T(0.5) : T(0)};
  T wz[3] = {T(0), T(1), T(0)};
  if (IS3D) {
    wz[0] = (fk > 0) ? T(0.5) : T(0);
    wz[2] = (fk < gf.nz - 1) ? T(0.5) : T(0);
  }
  const long long ox[3] = {(fi > 0) ? -1LL : 0LL, 0LL, (fi < gf.nx - 1) ? 1LL : 0LL};
  const long long oy[3] = {(fj > 0) ? -sy : 0LL, 0LL, (fj < gf.ny - 1) ? sy : 0LL};
  long long oz[3] = {0, 0, 0};
  if (IS3D) {
    oz[0] = (fk > 0) ? -sz : 0;
    oz[2] = (fk < gf.nz - 1) ? sz : 0;
  }
  const T scale = IS3D ? T(0.125) : T(0.25);
  const cplx<T> di = sw.y ? scaled_dinv<T>(sw, q) : mk<T>(0, 0);
  const int c0 = blockIdx.y * cpb;
  const int c1 = min(ncols, c0 + cpb);
  // columns are independent: unrolled so that several columns' loads are in flight
#pragma unroll 4
  for (int ci = c0; ci < c1; ++ci) {
    const int col = cols[ci];
    const cplx<TB>* r = rf + (long long)col * ldf + pc;
    const cplx<T>* wc = DIFF ? W + (long long)col * ldf + pc : nullptr;
    const cplx<T> y = DIFF ? yt[col * 8 + 6] : mk<T>(0, 0);
    T ar = 0, ai = 0;
#pragma unroll
    for (int c = 0; c < (IS3D ? 3 : 1); ++c) {
#pragma unroll
      for (int bq = 0; bq < 3; ++bq) {
#pragma unroll
        for (int a = 0; a < 3; ++a) {
          const T wgt = wx[a] * wy[bq] * (IS3D ? wz[c] : T(1));
          const long long o = ox[a] + oy[bq] + (IS3D ? oz[c] : 0LL);
          cplx<T> v = mk<T>((T)r[o].x, (T)r[o].y);
          if (DIFF) v = cfms<T>(y, wc[o], v);
          ar += wgt * v.x;
          ai += wgt * v.y;
        }
      }
    }
    const cplx<T> v = mk<T>(scale * ar, scale * ai);
    rc[(long long)col * ldc + q] = v;
    if (sw.y) sw.y[(long long)col * ldc + q] = cmul<T>(di, v);
  }
}

template <typename T, typename TB, bool DIFF>
static void restrict_any(Ctx& ctx, const Grid& gf, const Grid& gc, const cplx<TB>* rf, const cplx<T>* W,
                         const cplx<T>* yt, long long ldf, cplx<T>* rc, long long ldc, const int* cols, int ncols,
                         const Sweep<T>& sweep) {
  if (ncols <= 0) return;
  const int TPB = 256;
  long long nbx = (gc.N + TPB - 1) / TPB;
  int ch = chunks_for(nbx, ncols);
  int cpb = (ncols + ch - 1) / ch;
  dim3 grid((unsigned)nbx, (unsigned)ch);
  const double tbytes =
      (double)ncols * (gf.N * (sizeof(cplx<TB>) + (DIFF ? sizeof(cplx<T>) : 0)) +
                       gc.N * (sweep.y ? 2 : 1) * sizeof(cplx<T>));
  if (gf.nz > 1)
    HZ_LAUNCH(ctx, "restrict", tbytes, (k_restrict<T, TB, true, DIFF>), grid, TPB, 0, gf, gc, rf, W, yt, ldf, rc, ldc,
              cols, ncols, cpb, sweep);
  else
    HZ_LAUNCH(ctx, "restrict", tbytes, (k_restrict<T, TB, false, DIFF>), grid, TPB, 0, gf, gc, rf, W, yt, ldf, rc, ldc,
              cols, ncols, cpb, sweep);
}

template <typename T>
void launch_restrict(Ctx& ctx, const Grid& gf, const Grid& gc, const cplx<T>* rf, long long ldf, cplx<T>* rc,
                     long long ldc, const int* cols, int ncols, const Sweep<T>& sweep) {
  restrict_any<T, T, false>(ctx, gf, gc, rf, (const cplx<T>*)nullptr, nullptr, ldf, rc, ldc, cols, ncols, sweep);
}

template <typename T, typename TB>
void launch_restrict_diff(Ctx& ctx, const Grid& gf, const Grid& gc, const cplx<TB>* b, const cplx<T>* W,
                          const cplx<T>* yt, long long ldf, cplx<T>* rc, long long ldc, const int* cols, int ncols,
                          const Sweep<T>& sweep) {
  restrict_any<T, TB, true>(ctx, gf, gc, b, W, yt, ldf, rc, ldc, cols, ncols, sweep);
}

// COMB: the coarse vector is Y0 e0 + Y1 e1 (a K-cycle correction, formed here instead of
// in a pass of its own).  xin null: base 0; yt: base y xin.
template <typename T, bool COMB>
__global__ void __launch_bounds__(256) k_prolong2(Grid gf, Grid gc, const cplx<T>* __restrict__ ec0,
                                                 const cplx<T>* __restrict__ ec1, const cplx<T>* __restrict__ kt,
                                                 long long ldc, const cplx<T>* xin, const cplx<T>* __restrict__ yt,
                                                 cplx<T>* xout, long long ldf, const int* __restrict__ cols, int ncols,
                                                 int cpb) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= gf.N) return;
  const int i = (int)(p % gf.nx);
  const long long t = p / gf.nx;
  const int j = (int)t;
  // Parent pair per axis: (i>>1, (i+1)>>1).  An even fine index has both
  // entries equal to its single parent, an odd one has its two neighbours, so
  // a uniform weight of 1/2 per axis is exact linear interpolation.
  const long long sy = gc.nx;
  const long long a0 = i >> 1, a1 = (i + 1) >> 1;
  const long long b0 = (long long)(j >> 1) * sy, b1 = (long long)((j + 1) >> 1) * sy;
  const T wgt = T(0.25);
  const int c0 = blockIdx.y * cpb;
  const int c1 = min(ncols, c0 + cpb);
  // columns are independent: unrolled so that several columns' loads are in flight
#pragma unroll 4
  for (int ci = c0; ci < c1; ++ci) {
    const int col = cols[ci];
    const cplx<T>* e0 = ec0 + (long long)col * ldc;
    const cplx<T>* e1 = COMB ? ec1 + (long long)col * ldc : nullptr;
    const cplx<T> y0 = COMB ? kt[col * 8 + 6] : mk<T>(0, 0);
    const cplx<T> y1 = COMB ? kt[col * 8 + 7] : mk<T>(0, 0);
    auto e = [&](long long q) { return COMB ? cfma<T>(y1, e1[q], cmul<T>(y0, e0[q])) : e0[q]; };
    const cplx<T> v0 = e(b0 + a0), v1 = e(b0 + a1), v2 = e(b1 + a0), v3 = e(b1 + a1);
    const T ar = (v0.x + v1.x) + (v2.x + v3.x);
    const T ai = (v0.y + v1.y) + (v2.y + v3.y);
    const long long o = (long long)col * ldf + p;
    // the fine vector is read and written once (streaming); the coarse one stays cached
    cplx<T> base = xin ? __ldcs(&xin[o]) : mk<T>(0, 0);
    if (yt) base = cmul<T>(yt[col * 8 + 6], base);
    __stcs(&xout[o], mk<T>(base.x + wgt * ar, base.y + wgt * ai));
  }
}

// 3D: a thread owns the nodes (i, 2J..2J+1, 2K..2K+1) of its columns.  They share their 8 coarse
// values, where one thread per node loads 8 for each and is bound by L1: 45 -> 40 us per
// launch over the levels of 193 x 161 x 97 x 16 (In 2D the pairs cost more than they save on
// small grids, 6.6 -> 8.0 us at 129^2 x 1, and change nothing on large ones.)
template <typename T, bool COMB>
__global__ void __launch_bounds__(256) k_prolong3(Grid gf, Grid gc, const cplx<T>* __restrict__ ec0,
                                                 const cplx<T>* __restrict__ ec1, const cplx<T>* __restrict__ kt,
                                                 long long ldc, const cplx<T>* xin, const cplx<T>* __restrict__ yt,
                                                 cplx<T>* xout, long long ldf, const int* __restrict__ cols, int ncols,
                                                 int cpb) {
  const int nyh = (gf.ny + 1) >> 1, nzh = (gf.nz + 1) >> 1;
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= (long long)gf.nx * nyh * nzh) return;
  const int i = (int)(p % gf.nx);
  const long long t = p / gf.nx;
  const int J = (int)(t % nyh), K = (int)(t / nyh);
  const bool oddj = 2 * J + 1 < gf.ny, oddk = 2 * K + 1 < gf.nz;  // the odd nodes exist
  const long long sy = gc.nx, sz = (long long)gc.nx * gc.ny;
  const long long q0 = (long long)J * sy + (long long)K * sz + (i >> 1);
  const int da = ((i + 1) >> 1) - (i >> 1);
  const long long dy = oddj ? sy : 0, dz = oddk ? sz : 0;
  const long long o0 = i + (long long)gf.nx * (2 * J + (long long)gf.ny * 2 * K);
  const long long fy = gf.nx, fz = (long long)gf.nx * gf.ny;
  const T wgt = T(0.125);
  const int c0 = blockIdx.y * cpb;
  const int c1 = min(ncols, c0 + cpb);
  // columns are independent: unrolled so that several columns' loads are in flight
#pragma unroll 2
  for (int ci = c0; ci < c1; ++ci) {
    const int col = cols[ci];
    const cplx<T>* e0 = ec0 + (long long)col * ldc;
    const cplx<T>* e1 = COMB ? ec1 + (long long)col * ldc : nullptr;
    const cplx<T> y0 = COMB ? kt[col * 8 + 6] : mk<T>(0, 0);
    const cplx<T> y1 = COMB ? kt[col * 8 + 7] : mk<T>(0, 0);
    auto e = [&](long long q) { return COMB ? cfma<T>(y1, e1[q], cmul<T>(y0, e0[q])) : e0[q]; };
    auto pair = [&](long long q) { return cadd<T>(e(q), e(q + da)); };  // the two parents along x
    const cplx<T> s00 = pair(q0), s01 = pair(q0 + dy), s10 = pair(q0 + dz), s11 = pair(q0 + dz + dy);
    const cplx<T> yb = yt ? yt[col * 8 + 6] : mk<T>(0, 0);
    const cplx<T>* xi = xin ? xin + (long long)col * ldf : nullptr;
    cplx<T>* xo = xout + (long long)col * ldf;
    // the fine vector is read and written once (streaming); the coarse one stays cached
    auto put = [&](long long o, cplx<T> a) {
      cplx<T> base = xi ? __ldcs(&xi[o]) : mk<T>(0, 0);
      if (yt) base = cmul<T>(yb, base);
      __stcs(&xo[o], mk<T>(base.x + wgt * a.x, base.y + wgt * a.y));
    };
    const cplx<T> z0 = cadd<T>(s00, s00), z1 = cadd<T>(s00, s01);
    put(o0, cadd<T>(z0, z0));
    if (oddj) put(o0 + fy, cadd<T>(z1, z1));
    if (oddk) {
      put(o0 + fz, cadd<T>(z0, cadd<T>(s10, s10)));
      if (oddj) put(o0 + fz + fy, cadd<T>(z1, cadd<T>(s10, s11)));
    }
  }
}

template <typename T>
void launch_prolong(Ctx& ctx, const Grid& gf, const Grid& gc, const Correction<T>& e, long long ldc,
                    const cplx<T>* xin, const cplx<T>* yt, cplx<T>* xout, long long ldf, const int* cols, int ncols) {
  if (ncols <= 0) return;
  const int TPB = 256;
  const long long threads = gf.nz > 1 ? (long long)gf.nx * ((gf.ny + 1) / 2) * ((gf.nz + 1) / 2) : gf.N;
  long long nbx = (threads + TPB - 1) / TPB;
  int ch = chunks_for(nbx, ncols);
  int cpb = (ncols + ch - 1) / ch;
  dim3 grid((unsigned)nbx, (unsigned)ch);
  const double pbytes = (double)ncols * ((e.z1 ? 2 : 1) * gc.N + (xin ? 2 : 1) * gf.N) * sizeof(cplx<T>);
#define HZ_PROLONG(K, C)                                                                                             \
  HZ_LAUNCH(ctx, "prolong", pbytes, (K<T, C>), grid, TPB, 0, gf, gc, e.z0, e.z1, e.kt, ldc, xin, yt, xout, ldf, cols, \
            ncols, cpb)
  if (gf.nz > 1) {
    if (e.z1) HZ_PROLONG(k_prolong3, true);
    else HZ_PROLONG(k_prolong3, false);
  } else {
    if (e.z1) HZ_PROLONG(k_prolong2, true);
    else HZ_PROLONG(k_prolong2, false);
  }
#undef HZ_PROLONG
}

// ---------------------------------------------------------------------------
// Coarsest level: blocked banded LU solve, FP64 arithmetic.
//
// The host folds each block of kl elimination steps of the band LU (row
// interchanges included) into a dense window operator T_I, and each block of
// the back substitution into G_I = [U_II^{-1} | -U_II^{-1} U_right]; a solve is
// then N/kl sequential window mat-vecs per direction, each spread over the
// whole GPU: one warp per (output row, column), lanes split the window sum.
// ---------------------------------------------------------------------------
template <typename T, int MODE>
__global__ void __launch_bounds__(256) k_band_block(long long N, long long s, int Win, int split,
                                                    const double2* __restrict__ M, const double2* __restrict__ src0,
                                                    const cplx<T>* __restrict__ b, long long ldb,
                                                    const int* __restrict__ cols, const double2* __restrict__ src1,
                                                    double2* __restrict__ dst, cplx<T>* __restrict__ xout,
                                                    long long ldx, int ncols) {
  const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
  const int i = blockIdx.x;
  const int ci = blockIdx.y * 8 + warp;
  if (ci >= ncols) return;
  const double2* Mr = M + (long long)i * Win;
  const long long base = (long long)ci * N + s;
  double ar = 0.0, ai = 0.0;
  for (int k = lane; k < Win; k += 32) {
    const double2 m = Mr[k];
    double2 v;
    if (k < split) {
      v = src0[base + k];
    } else if (MODE == 0) {
      const cplx<T> bb = b[(long long)cols[ci] * ldb + s + k];
      v = mk<double>((double)bb.x, (double)bb.y);
    } else {
      v = src1[base + k];
    }
    ar = fma(m.x, v.x, ar);
    ar = fma(-m.y, v.y, ar);
    ai = fma(m.x, v.y, ai);
    ai = fma(m.y, v.x, ai);
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    ar += __shfl_xor_sync(0xffffffffu, ar, o);
    ai += __shfl_xor_sync(0xffffffffu, ai, o);
  }
  if (lane == 0) {
    dst[base + i] = mk<double>(ar, ai);
    if (MODE == 1) xout[(long long)cols[ci] * ldx + s + i] = mk<T>((T)ar, (T)ai);
  }
}

// All block steps of the solve in one cooperative launch.  A warp item is one
// row of the current window operator for BCW columns: the row entries are
// loaded once and feed BCW independent accumulators (more loads in flight per
// warp than one column per item).  The grid synchronises between block steps;
// the launch is sized to the co-resident capacity (cudaLaunchCooperativeKernel
// refuses a larger grid rather than deadlocking).
static constexpr int BCW = 1;  // one column per item: more items in flight per step

template <typename T>
__global__ void __launch_bounds__(256) k_band_coop(long long N, int nbk, const BandBlock* __restrict__ blocks,
                                                   const double2* __restrict__ Tops, const double2* __restrict__ Gops,
                                                   const cplx<T>* __restrict__ b, long long ldb,
                                                   const int* __restrict__ cols, int ncols, double2* __restrict__ work,
                                                   cplx<T>* __restrict__ x, long long ldx) {
  cg::grid_group grid = cg::this_grid();
  const int lane = threadIdx.x & 31;
  const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  double2* const Y0 = work;
  double2* const Y1 = work + (long long)ncols * N;
  double2* const X64 = work + 2LL * ncols * N;
  const int ngrp = (ncols + BCW - 1) / BCW;
  long long prev_end = 0;
  for (int I = 0; I < nbk; ++I) {
    const BandBlock B = blocks[I];
    const int split = (I == 0) ? 0 : (int)(prev_end - B.s);
    const double2* src0 = (I & 1) ? Y0 : Y1;  // output of block I-1
    double2* dst = (I & 1) ? Y1 : Y0;
    const long long items = (long long)B.W * ngrp;
    for (long long it = gw; it < items; it += nw) {
      const int i = (int)(it % B.W), c0 = (int)(it / B.W) * BCW;
      const double2* Mr = Tops + B.toff + (long long)i * B.W;
      double ar[BCW], ai[BCW];
#pragma unroll
      for (int c = 0; c < BCW; ++c) ar[c] = ai[c] = 0.0;
      for (int k = lane; k < B.W; k += 32) {
        const double2 m = Mr[k];
#pragma unroll
        for (int c = 0; c < BCW; ++c) {
          const int ci = c0 + c;
          if (ci < ncols) {
            double2 v;
            if (k < split) {
              v = src0[(long long)ci * N + B.s + k];
            } else {
              const cplx<T> bb = b[(long long)cols[ci] * ldb + B.s + k];
              v = mk<double>((double)bb.x, (double)bb.y);
            }
            ar[c] = fma(m.x, v.x, ar[c]);
            ar[c] = fma(-m.y, v.y, ar[c]);
            ai[c] = fma(m.x, v.y, ai[c]);
            ai[c] = fma(m.y, v.x, ai[c]);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < BCW; ++c) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          ar[c] += __shfl_xor_sync(0xffffffffu, ar[c], o);
          ai[c] += __shfl_xor_sync(0xffffffffu, ai[c], o);
        }
        if (lane == 0 && c0 + c < ncols) dst[(long long)(c0 + c) * N + B.s + i] = mk<double>(ar[c], ai[c]);
      }
    }
    prev_end = B.s + B.W;
    grid.sync();
  }
  for (int I = nbk - 1; I >= 0; --I) {
    const BandBlock B = blocks[I];
    const double2* yb = (I & 1) ? Y1 : Y0;
    const long long items = (long long)B.nb * ngrp;
    for (long long it = gw; it < items; it += nw) {
      const int i = (int)(it % B.nb), c0 = (int)(it / B.nb) * BCW;
      const double2* Mr = Gops + B.goff + (long long)i * B.Wb;
      double ar[BCW], ai[BCW];
#pragma unroll
      for (int c = 0; c < BCW; ++c) ar[c] = ai[c] = 0.0;
      for (int k = lane; k < B.Wb; k += 32) {
        const double2 m = Mr[k];
#pragma unroll
        for (int c = 0; c < BCW; ++c) {
          const int ci = c0 + c;
          if (ci < ncols) {
            const long long q = (long long)ci * N + B.s + k;
            const double2 v = (k < B.nb) ? yb[q] : X64[q];
            ar[c] = fma(m.x, v.x, ar[c]);
            ar[c] = fma(-m.y, v.y, ar[c]);
            ai[c] = fma(m.x, v.y, ai[c]);
            ai[c] = fma(m.y, v.x, ai[c]);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < BCW; ++c) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
          ar[c] += __shfl_xor_sync(0xffffffffu, ar[c], o);
          ai[c] += __shfl_xor_sync(0xffffffffu, ai[c], o);
        }
        const int ci = c0 + c;
        if (lane == 0 && ci < ncols) {
          X64[(long long)ci * N + B.s + i] = mk<double>(ar[c], ai[c]);
          x[(long long)cols[ci] * ldx + B.s + i] = mk<T>((T)ar[c], (T)ai[c]);
        }
      }
    }
    grid.sync();
  }
}

// The same block steps, one cluster of CTAs per column: the columns are
// independent, so a step ends with a cluster barrier instead of a grid barrier.
// Every CTA holds the column's vectors in its shared memory; a row's result is
// written into all of them.  The entries of the next step's operator row are
// loaded before the barrier.  A warp-wide FP64 instruction occupies its quarter of
// the SM for 64 clocks, so rows go to the CTAs in turn (one row per quarter up to
// four rows per CTA), the real and imaginary sums share the reduction's
// instructions, and stretches of 32 zero entries are skipped.  Every row sum is
// k_band_coop's, in its order: the results are equal bit for bit.
static constexpr int kBandWarps = 8;

template <int PF, typename V>
__device__ __forceinline__ double2 band_row_sum(const double2* Mr, int W, int lane, const double2 (&m)[PF], bool pre,
                                                V&& value) {
  double ar = 0.0, ai = 0.0;
  auto add = [&](double2 a, int k) {
    if (__any_sync(0xffffffffu, a.x != 0.0 || a.y != 0.0)) {
      const double2 v = k < W ? value(k) : mk<double>(0, 0);
      ar = fma(a.x, v.x, ar);
      ar = fma(-a.y, v.y, ar);
      ai = fma(a.x, v.y, ai);
      ai = fma(a.y, v.x, ai);
    }
  };
#pragma unroll
  for (int q = 0; q < PF; ++q)
    if (32 * q < W) add(pre ? m[q] : (lane + 32 * q < W ? Mr[lane + 32 * q] : mk<double>(0, 0)), lane + 32 * q);
  for (int k = lane + 32 * PF; k - lane < W; k += 32) add(k < W ? Mr[k] : mk<double>(0, 0), k);
  // lanes 0-15 reduce the real sums, lanes 16-31 the imaginary ones, each in the
  // tree of a full exchange
  const bool lower = lane < 16;
  double s = (lower ? ar : ai) + __shfl_xor_sync(0xffffffffu, lower ? ai : ar, 16);
#pragma unroll
  for (int o = 8; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
  return mk<double>(__shfl_sync(0xffffffffu, s, 0), __shfl_sync(0xffffffffu, s, 16));
}

template <int PF>
__device__ __forceinline__ void band_row_prefetch(const double2* Mr, int W, int lane, double2 (&m)[PF]) {
#pragma unroll
  for (int q = 0; q < PF; ++q) m[q] = lane + 32 * q < W ? Mr[lane + 32 * q] : mk<double>(0, 0);
}

template <typename T>
__global__ void __launch_bounds__(32 * kBandWarps) k_band_cluster(int N, int nbk, const BandBlock* __restrict__ blocks,
                                                                  const double2* __restrict__ Tops,
                                                                  const double2* __restrict__ Gops,
                                                                  const cplx<T>* b, long long ldb,
                                                                  const int* __restrict__ cols, cplx<T>* x,
                                                                  long long ldx) {
  extern __shared__ __align__(16) double2 band_sm[];
  double2* const bx = band_sm;  // b, then x from the back
  double2* const Y0 = band_sm + N;
  double2* const Y1 = band_sm + 2 * N;
  cg::cluster_group cluster = cg::this_cluster();
  const int lane = threadIdx.x & 31;
  const int ctas = (int)cluster.num_blocks();
  const int gw = (threadIdx.x >> 5) * ctas + (int)cluster.block_rank(), nw = ctas * kBandWarps;
  constexpr int PF = 4;
  const int col = cols[blockIdx.x / ctas];
  const cplx<T>* bc = b + (long long)col * ldb;
  cplx<T>* xc = x + (long long)col * ldx;
  for (int k = threadIdx.x; k < N; k += 32 * kBandWarps) {
    const cplx<T> v = bc[k];
    bx[k] = mk<double>((double)v.x, (double)v.y);
  }
  double2 m[PF];
  BandBlock B = blocks[0];
  if (gw < B.W) band_row_prefetch<PF>(Tops + B.toff + (long long)gw * B.W, B.W, lane, m);
  cluster.sync();
  long long prev_end = 0;
  for (int I = 0; I < nbk; ++I) {
    const int split = (I == 0) ? 0 : (int)(prev_end - B.s);
    const double2* src0 = ((I & 1) ? Y0 : Y1) + B.s;  // output of block I-1
    const double2* srcb = bx + B.s;
    double2* dst = ((I & 1) ? Y1 : Y0) + B.s;
    for (int i = gw; i < B.W; i += nw) {
      const double2 r = band_row_sum<PF>(Tops + B.toff + (long long)i * B.W, B.W, lane, m, i == gw,
                                         [&](int k) { return k < split ? src0[k] : srcb[k]; });
      if (lane < ctas) cluster.map_shared_rank(dst, lane)[i] = r;
    }
    prev_end = B.s + B.W;
    if (I + 1 < nbk) {
      B = blocks[I + 1];
      if (gw < B.W) band_row_prefetch<PF>(Tops + B.toff + (long long)gw * B.W, B.W, lane, m);
    } else if (gw < B.nb) {
      band_row_prefetch<PF>(Gops + B.goff + (long long)gw * B.Wb, B.Wb, lane, m);
    }
    cluster.sync();
  }
  for (int I = nbk - 1; I >= 0; --I) {
    const double2* yb = ((I & 1) ? Y1 : Y0) + B.s;
    double2* xb = bx + B.s;
    for (int i = gw; i < B.nb; i += nw) {
      const double2 r = band_row_sum<PF>(Gops + B.goff + (long long)i * B.Wb, B.Wb, lane, m, i == gw,
                                         [&](int k) { return k < B.nb ? yb[k] : xb[k]; });
      if (lane < ctas) cluster.map_shared_rank(xb, lane)[i] = r;
      if (lane == 0) xc[B.s + i] = mk<T>((T)r.x, (T)r.y);
    }
    if (I > 0) {
      B = blocks[I - 1];
      if (gw < B.nb) band_row_prefetch<PF>(Gops + B.goff + (long long)gw * B.Wb, B.Wb, lane, m);
    }
    cluster.sync();
  }
}

// Shared memory of a cluster's CTA: the column's three vectors.
static constexpr size_t kBandSmemMax = 220 * 1024;
static size_t band_smem(long long N) { return (size_t)N * 3 * sizeof(double2); }

// Clusters of 16 CTAs (8 where the GPU takes no larger ones) with the column's vectors in
// shared memory that can be resident at once; 0: not available.
template <typename T>
void plan_band_solve(BandSolveOps& op) {
  op.cluster = op.resident = 0;
  const size_t smem = band_smem(op.N);
  if (smem > kBandSmemMax) return;
  static SmemLimit limit;
  try {
    raise_smem_limit(limit, (const void*)k_band_cluster<T>, kBandSmemMax, "band_solve", true);
  } catch (const std::runtime_error&) {
    return;  // no such clusters here: the cooperative kernel
  }
  for (int ctas = 16; ctas >= 8; ctas /= 2) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3((unsigned)ctas);
    cfg.blockDim = dim3(32 * kBandWarps);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.x = (unsigned)ctas;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    int resident = 0;
    if (cudaOccupancyMaxActiveClusters(&resident, k_band_cluster<T>, &cfg) == cudaSuccess && resident > 0) {
      op.cluster = ctas;
      op.resident = resident;
      return;
    }
    cudaGetLastError();
  }
}
template void plan_band_solve<double>(BandSolveOps&);
template void plan_band_solve<float>(BandSolveOps&);

template <typename T>
void launch_band_solve(Ctx& ctx, const BandSolveOps& op, const cplx<T>* b, cplx<T>* x, long long ld, const int* cols,
                       int ncols, double2* work) {
  if (ncols <= 0) return;
  const long long N = op.N;
  const int nbk = (int)op.blocks.size();
  double bytes = 0.0;
  for (const BandBlock& B : op.blocks)
    bytes += ((double)B.W * B.W + (double)B.nb * B.Wb) * sizeof(double2) +
             ncols * (2.0 * B.W + B.Wb + 2.0 * B.nb) * sizeof(double2);
  if (op.dblocks) {
    // one cooperative launch, grid = co-resident capacity
    static int capacity[kMaxDevices] = {};
    int dev = 0;
    cudaGetDevice(&dev);
    if (dev >= 0 && dev < kMaxDevices && capacity[dev] == 0) {
      int per_sm = 0, sms = 0;
      cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_band_coop<T>, 256, 0);
      cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
      capacity[dev] = std::max(1, std::min(per_sm, 4)) * std::max(1, sms);
    }
    // Clocks of both schedules: a cluster per column (as many at once as fit) and a
    // cluster barrier per step, or the columns over the whole GPU and a grid barrier
    // over as many CTAs as the widest step fills; two FP64 FMA lanes per SM and clock.
    const int ctas = op.cluster, resident = op.resident;
    double cl = 0.0, gr = 0.0;
    long long rows = 1;
    for (const BandBlock& B : op.blocks) {
      const double fma = 4.0 * ((double)B.W * B.W + (double)B.nb * B.Wb);
      if (resident) cl += (ncols + resident - 1) / resident * (fma / (2.0 * ctas) + 2 * 2000.0);
      gr += fma * ncols / (2.0 * kSMs) + 2 * 6000.0;
      rows = std::max(rows, (long long)B.W);
    }
    const bool clustered = resident && cl < gr;
    const int full = (dev >= 0 && dev < kMaxDevices) ? capacity[dev] : kSMs;
    const int grid = (int)std::min<long long>(full, (rows * ncols + 7) / 8);
    static thread_local int id = -1;
    if (id < 0 || (size_t)id >= ctx.names.size() || ctx.names[id] != "band_solve") id = ctx.name_id("band_solve");
    cudaEvent_t ev = nullptr;
    ctx.before(id, &ev);
    const BandBlock* blk = op.dblocks;
    if (clustered) {
      cudaLaunchConfig_t cfg{};
      cfg.gridDim = dim3((unsigned)(ctas * ncols));
      cfg.blockDim = dim3(32 * kBandWarps);
      cfg.dynamicSmemBytes = band_smem(N);
      cfg.stream = ctx.stream;
      cudaLaunchAttribute at{};
      at.id = cudaLaunchAttributeClusterDimension;
      at.val.clusterDim.x = (unsigned)ctas;
      at.val.clusterDim.y = at.val.clusterDim.z = 1;
      cfg.attrs = &at;
      cfg.numAttrs = 1;
      const cudaError_t e = cudaLaunchKernelEx(&cfg, k_band_cluster<T>, (int)N, nbk, blk, op.T, op.G, b, ld, cols, x,
                                               ld);
      if (e != cudaSuccess) {
        cudaGetLastError();
        throw std::runtime_error(std::string("band_solve cluster launch failed: ") + cudaGetErrorString(e));
      }
      ctx.after(id, ev, bytes);
      return;
    }
    const double2* Tp = op.T;
    const double2* Gp = op.G;
    long long ldb = ld, ldx = ld;
    void* args[] = {(void*)&N,    (void*)&nbk,  (void*)&blk,   (void*)&Tp,   (void*)&Gp, (void*)&b,
                    (void*)&ldb,  (void*)&cols, (void*)&ncols, (void*)&work, (void*)&x,  (void*)&ldx};
    const cudaError_t e =
        cudaLaunchCooperativeKernel((const void*)k_band_coop<T>, dim3(grid), dim3(256), args, 0, ctx.stream);
    if (e != cudaSuccess) {
      cudaGetLastError();
      throw std::runtime_error(std::string("band_solve cooperative launch failed: ") + cudaGetErrorString(e));
    }
    ctx.after(id, ev, bytes);
    return;
  }
  double2* Y[2] = {work, work + (long long)ncols * N};
  double2* X64 = work + 2LL * ncols * N;
  const unsigned gy = (unsigned)((ncols + 7) / 8);
  long long prev_end = 0;
  for (int I = 0; I < nbk; ++I) {
    const BandBlock& B = op.blocks[(size_t)I];
    const int split = (I == 0) ? 0 : (int)(prev_end - B.s);
    const double fb = (double)B.W * B.W * sizeof(double2) + 2.0 * ncols * B.W * sizeof(double2);
    HZ_LAUNCH(ctx, "band_forward", fb, (k_band_block<T, 0>), dim3((unsigned)B.W, gy), 256, 0, N, B.s, B.W, split,
              op.T + B.toff, Y[(I + 1) % 2], b, ld, cols, (const double2*)nullptr, Y[I % 2], (cplx<T>*)nullptr,
              0LL, ncols);
    prev_end = B.s + B.W;
  }
  for (int I = nbk - 1; I >= 0; --I) {
    const BandBlock& B = op.blocks[(size_t)I];
    const double bb = (double)B.nb * B.Wb * sizeof(double2) + ncols * (B.Wb + 2.0 * B.nb) * sizeof(double2);
    HZ_LAUNCH(ctx, "band_backward", bb, (k_band_block<T, 1>), dim3((unsigned)B.nb, gy), 256, 0, N, B.s, B.Wb,
              B.nb, op.G + B.goff, Y[I % 2], (const cplx<T>*)nullptr, 0LL, cols, X64, X64, x, ld, ncols);
  }
}

// ---------------------------------------------------------------------------
// Allocation-free operator apply (hz_apply_noalloc).  The column-index list
// the stencil kernel reads is kept in a file-scope device array instead of a
// per-call allocation.  Host code must not pass the symbol itself to a kernel
// (in host code it is only a host-side stand-in); its device address is looked
// up with cudaGetSymbolAddress once per device, with that device current.
// ---------------------------------------------------------------------------
static __device__ __align__(256) int g_noalloc_cols[kNoAllocMaxCols];

__global__ void k_iota(int* __restrict__ out, int n) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < n) out[i] = i;
}

static int* noalloc_cols_address(int dev, std::string* err) {
  static std::mutex mu;
  static int* addr[kNoAllocMaxDevices] = {};
  if (dev < 0 || dev >= kNoAllocMaxDevices) {
    *err = "device ordinal out of range for the allocation-free entry point";
    return nullptr;
  }
  std::lock_guard<std::mutex> lock(mu);
  if (!addr[dev]) {
    int* p = nullptr;
    const cudaError_t e = cudaGetSymbolAddress((void**)&p, g_noalloc_cols);
    if (e != cudaSuccess || !p) {
      cudaGetLastError();
      *err = std::string("cudaGetSymbolAddress of the column-list scratch failed: ") + cudaGetErrorString(e);
      return nullptr;
    }
    addr[dev] = p;
  }
  return addr[dev];
}

int launch_fine_apply_noalloc(cudaStream_t stream, int dev, const FineOp& op, const double2* diag, const double2* x,
                              double2* y, long long ld, int nrhs, std::string* err) {
  if (nrhs < 1 || nrhs > kNoAllocMaxCols) {
    *err = "nrhs must be in [1, " + std::to_string(kNoAllocMaxCols) + "] for the allocation-free apply";
    return -1;
  }
  int* cols = noalloc_cols_address(dev, err);
  if (!cols) return -2;
  // every call rewrites the entries it reads: the array keeps the previous call's contents
  k_iota<<<(nrhs + 255) / 256, 256, 0, stream>>>(cols, nrhs);
  FineOpT<double> o;
  o.nx = op.g.nx;
  o.ny = op.g.ny;
  o.nz = op.g.nz;
  o.N = op.g.N;
  for (int d = 0; d < 3; ++d) {
    o.o[d] = op.o[d];
    o.b[d] = op.b[d];
  }
  o.adj = op.adj;
  const int TPB = 256;
  const long long nbx = (op.g.N + TPB - 1) / TPB;
  const int ch = chunks_for(nbx, nrhs);
  const int cpb = (nrhs + ch - 1) / ch;
  const dim3 grid((unsigned)nbx, (unsigned)ch);
  if (op.g.nz > 1)
    k_fine<double, double, double, MODE_APPLY, true><<<grid, TPB, 0, stream>>>(
        o, diag, nullptr, x, (const double2*)nullptr, y, ld, cols, nrhs, cpb, 0.0);
  else
    k_fine<double, double, double, MODE_APPLY, false><<<grid, TPB, 0, stream>>>(
        o, diag, nullptr, x, (const double2*)nullptr, y, ld, cols, nrhs, cpb, 0.0);
  const cudaError_t e = cudaGetLastError();
  if (e != cudaSuccess) {
    *err = std::string("allocation-free apply launch failed: ") + cudaGetErrorString(e);
    return -2;
  }
  return 0;
}

// explicit instantiations
#define HZ_INST_T_TB(T, TB)                                                                                        \
  template void launch_fine<T, T, TB>(Ctx&, int, const FineOp&, const cplx<T>*, const cplx<T>*, const cplx<T>*,     \
                                      const cplx<TB>*, cplx<T>*, long long, const int*, int, double);               \
  template void launch_rap<T, TB>(Ctx&, int, const Grid&, const cplx<T>*, long long, const cplx<T>*,                \
                                  const cplx<T>*, const cplx<TB>*, cplx<T>*, long long, const int*, int, double,    \
                                  const Sweep<T>&);                                                                 \
  template void launch_jacobi0<T, TB>(Ctx&, const Grid&, const cplx<T>*, int, const cplx<TB>*, cplx<T>*, long long, \
                                      const int*, int, double);
HZ_INST_T_TB(double, double)
HZ_INST_T_TB(float, float)
HZ_INST_T_TB(float, double)
HZ_INST_T_TB(float, df64_tag)
template void launch_fine<double, float, double>(Ctx&, int, const FineOp&, const double2*, const double2*,
                                                 const float2*, const double2*, double2*, long long, const int*, int,
                                                 double);
#undef HZ_INST_T_TB
template void launch_restrict<double>(Ctx&, const Grid&, const Grid&, const double2*, long long, double2*, long long,
                                      const int*, int, const Sweep<double>&);
template void launch_restrict<float>(Ctx&, const Grid&, const Grid&, const float2*, long long, float2*, long long,
                                     const int*, int, const Sweep<float>&);
#define HZ_INST_RD(T, TB)                                                                                       \
  template void launch_restrict_diff<T, TB>(Ctx&, const Grid&, const Grid&, const cplx<TB>*, const cplx<T>*,     \
                                            const cplx<T>*, long long, cplx<T>*, long long, const int*, int,     \
                                            const Sweep<T>&);
HZ_INST_RD(double, double)
HZ_INST_RD(float, float)
HZ_INST_RD(float, double)
HZ_INST_RD(float, df64_tag)
#undef HZ_INST_RD
template void launch_prolong<double>(Ctx&, const Grid&, const Grid&, const Correction<double>&, long long,
                                     const double2*, const double2*, double2*, long long, const int*, int);
template void launch_prolong<float>(Ctx&, const Grid&, const Grid&, const Correction<float>&, long long, const float2*,
                                    const float2*, float2*, long long, const int*, int);
template void launch_band_solve<double>(Ctx&, const BandSolveOps&, const double2*, double2*, long long, const int*, int,
                                        double2*);
template void launch_band_solve<float>(Ctx&, const BandSolveOps&, const float2*, float2*, long long, const int*, int,
                                       double2*);

}  // namespace hz
