// Emulated-FP64 ("df64") outer FGMRES kernels: a complex value is stored as
// float4 (re_hi, im_hi, re_lo, im_lo) with x = hi + lo exactly representable to
// about 2^-48 relative, and arithmetic uses error-free FP32 transformations
// (TwoSum: Knuth; TwoProd via fused multiply-add), which run on the FP32 pipe
// (64x the FP64 rate of GB300).  Used for the Krylov basis, H z, Gram-Schmidt
// and the basis scaling of the mixed-precision form; the true residual at
// every restart is still computed in native FP64.
//
// The (re_hi, im_hi) pair is the float2 a complex-FP32 kernel reads, so the
// V-cycle takes a df64 basis vector directly as its right-hand side.
#include <algorithm>

#include <cooperative_groups.h>

#include "hz_gs.cuh"
#include "hz_launch.cuh"

namespace cg = cooperative_groups;

namespace hz {

// ---- error-free transformations (no contraction, no reassociation) ---------
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  const float bb = __fsub_rn(s, a);
  e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}
__device__ __forceinline__ void quick_two_sum(float a, float b, float& s, float& e) {
  s = __fadd_rn(a, b);
  e = __fsub_rn(b, __fsub_rn(s, a));
}
__device__ __forceinline__ void two_prod(float a, float b, float& p, float& e) {
  p = __fmul_rn(a, b);
  e = __fmaf_rn(a, b, -p);
}

// Accumulator: hi + lo, lo collects rounding errors and cross terms and is
// folded back by renorm().
struct DAcc {
  float hi, lo;
  __device__ __forceinline__ void init(float h, float l) {
    hi = h;
    lo = l;
  }
  // += (ah + al) * (bh + bl)
  __device__ __forceinline__ void mac(float ah, float al, float bh, float bl) {
    float p, e, s, t;
    two_prod(ah, bh, p, e);
    two_sum(hi, p, s, t);
    hi = s;
    lo = __fadd_rn(lo, __fadd_rn(t, e));
    lo = __fmaf_rn(ah, bl, lo);
    lo = __fmaf_rn(al, bh, lo);
  }
  // -= (ah + al) * (bh + bl)
  __device__ __forceinline__ void msub(float ah, float al, float bh, float bl) { mac(-ah, -al, bh, bl); }
  // += (ah + al) * b   (b exact float)
  __device__ __forceinline__ void mac1(float ah, float al, float b) {
    float p, e, s, t;
    two_prod(ah, b, p, e);
    two_sum(hi, p, s, t);
    hi = s;
    lo = __fadd_rn(lo, __fadd_rn(t, e));
    lo = __fmaf_rn(al, b, lo);
  }
  // += x (an FP32 value) with the rounding error of the sum kept in lo
  __device__ __forceinline__ void add(float x) {
    float s, t;
    two_sum(hi, x, s, t);
    hi = s;
    lo = __fadd_rn(lo, t);
  }
  __device__ __forceinline__ void renorm() { quick_two_sum(hi, lo, hi, lo); }
  __device__ __forceinline__ double to_double() const { return (double)hi + (double)lo; }
};

__device__ __forceinline__ void split(double x, float& hi, float& lo) {
  hi = __double2float_rn(x);
  lo = __double2float_rn(x - (double)hi);
}

// ---- H z (z complex FP32) into a df64 basis vector ---------------------------
// dHd: diag(H) as float4 (re_hi, im_hi, re_lo, im_lo); c[6] = (hi, lo) of the
// interior / boundary-row magnitudes per axis.
struct DFOp {
  int nx, ny, nz;
  long long N;
  float oh[3], ol[3], bh[3], bl[3];
  int adj;
  const double* sig = nullptr;
  int sig_stride = 0;
};

__device__ __forceinline__ void axis_df(int i, int n, const DFOp& op, int a, float& clh, float& cll, float& crh,
                                        float& crl) {
  // same rule as the FP32/FP64 stencil: boundary rows use BC/h^2, the adjoint takes entry (j, i)
  bool lb, rb;  // left / right coefficient is the boundary one
  if (!op.adj) {
    lb = (i == n - 1);
    rb = (i == 0);
  } else {
    lb = (i - 1 == 0);
    rb = (i + 1 == n - 1);
  }
  if (i > 0) {
    clh = lb ? op.bh[a] : op.oh[a];
    cll = lb ? op.bl[a] : op.ol[a];
  } else {
    clh = cll = 0.f;
  }
  if (i < n - 1) {
    crh = rb ? op.bh[a] : op.oh[a];
    crl = rb ? op.bl[a] : op.ol[a];
  } else {
    crh = crl = 0.f;
  }
}

__device__ __forceinline__ void store_out(float4* y, long long i, const DAcc& re, const DAcc& im) {
  y[i] = make_float4(re.hi, im.hi, re.lo, im.lo);
}
__device__ __forceinline__ void store_out(double2* y, long long i, const DAcc& re, const DAcc& im) {
  y[i] = mk<double>(re.to_double(), im.to_double());
}

// TO = float4: df64 result (basis vector); TO = double2: rounded to FP64
template <bool IS3D, typename TO>
__global__ void __launch_bounds__(256) k_fine_df64(DFOp op, const float4* __restrict__ dHd,
                                                   const float2* __restrict__ z, TO* __restrict__ y, long long ld,
                                                   const int* __restrict__ cols, int ncols, int cpb) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= op.N) return;
  const int nx = op.nx, ny = op.ny;
  const int i = (int)(p % nx);
  const long long t = p / nx;
  const int j = (int)(t % ny);
  const int k = (int)(t / ny);
  float c[12];  // (hi, lo) of left/right per axis
  axis_df(i, nx, op, 0, c[0], c[1], c[2], c[3]);
  axis_df(j, ny, op, 1, c[4], c[5], c[6], c[7]);
  if (IS3D) axis_df(k, op.nz, op, 2, c[8], c[9], c[10], c[11]);
  const long long sy = nx, sz = (long long)nx * ny;
  const long long o[6] = {(i > 0) ? -1LL : 0LL, (i < nx - 1) ? 1LL : 0LL, (j > 0) ? -sy : 0LL,
                          (j < ny - 1) ? sy : 0LL, (IS3D && k > 0) ? -sz : 0LL, (IS3D && k < op.nz - 1) ? sz : 0LL};
  float4 d = dHd[p];
  if (op.adj) {
    d.y = -d.y;
    d.w = -d.w;
  }
  const int c0 = blockIdx.y * cpb;
  const int c1 = min(ncols, c0 + cpb);
  for (int ci = c0; ci < c1; ++ci) {
    const long long off = (long long)cols[ci] * ld;
    const float2* zc = z + off + p;
    const float2 zp = zc[0];
    DAcc re, im;
    re.init(0.f, 0.f);
    im.init(0.f, 0.f);
    // diagonal: (dr + i di)(zr + i zi)
    re.mac1(d.x, d.z, zp.x);
    re.mac1(-d.y, -d.w, zp.y);
    im.mac1(d.x, d.z, zp.y);
    im.mac1(d.y, d.w, zp.x);
#pragma unroll
    for (int q = 0; q < (IS3D ? 6 : 4); ++q) {
      const float2 zn = zc[o[q]];
      re.mac1(-c[2 * q], -c[2 * q + 1], zn.x);
      im.mac1(-c[2 * q], -c[2 * q + 1], zn.y);
    }
    re.renorm();
    im.renorm();
    if (op.sig) {
      const float s = (float)basis_power(basis_exponent(op.sig[(long long)cols[ci] * op.sig_stride]));
      re.init(s * re.hi, s * re.lo);
      im.init(s * im.hi, s * im.lo);
    }
    store_out(y, off + p, re, im);
  }
}

template <typename TO>
void launch_fine_df64(Ctx& ctx, const FineOp& op, const float4* dHd, const float2* z, TO* y, long long ld,
                      const int* cols, int ncols) {
  if (ncols <= 0) return;
  DFOp d;
  d.nx = op.g.nx;
  d.ny = op.g.ny;
  d.nz = op.g.nz;
  d.N = op.g.N;
  for (int a = 0; a < 3; ++a) {
    d.oh[a] = (float)op.o[a];
    d.ol[a] = (float)(op.o[a] - (double)d.oh[a]);
    d.bh[a] = (float)op.b[a];
    d.bl[a] = (float)(op.b[a] - (double)d.bh[a]);
  }
  d.adj = op.adj;
  d.sig = op.sig;
  d.sig_stride = op.sig_stride;
  const int TPB = 256;
  const long long nbx = (op.g.N + TPB - 1) / TPB;
  const int ch = chunks_for(nbx, ncols);
  const int cpb = (ncols + ch - 1) / ch;
  const double bytes = (double)op.g.N * ncols * (8 + 16) + (double)op.g.N * 16;
  if (op.g.nz > 1)
    HZ_LAUNCH(ctx, "outer_apply_df64", bytes, (k_fine_df64<true, TO>), dim3((unsigned)nbx, (unsigned)ch), TPB, 0, d, dHd,
              z, y, ld, cols, ncols, cpb);
  else
    HZ_LAUNCH(ctx, "outer_apply_df64", bytes, (k_fine_df64<false, TO>), dim3((unsigned)nbx, (unsigned)ch), TPB, 0, d, dHd,
              z, y, ld, cols, ncols, cpb);
}
template void launch_fine_df64<float4>(Ctx&, const FineOp&, const float4*, const float2*, float4*, long long,
                                       const int*, int);
template void launch_fine_df64<double2>(Ctx&, const FineOp&, const float4*, const float2*, double2*, long long,
                                        const int*, int);

// ---- Gram-Schmidt: dots and update on df64 vectors ---------------------------
static constexpr int RT = 256;

// dots sum conj(V_{i0+s}) w for s < KT, and ||w||^2
template <int KT>
__global__ void __launch_bounds__(RT, 2) k_dots_df(long long N, const float4* __restrict__ V, long long vstride,
                                                   long long ld, int i0, const float4* __restrict__ w,
                                                   const int* __restrict__ cols, int pass, int want_norm, GsColumn g) {
  __shared__ double tot[2 * KT + 1];
  const int c = cols[blockIdx.y];
  if (pass && !g.flag[c]) return;
  const int nblk = gridDim.x;
  const float4* wc = w + (long long)c * ld;
  const float4* vb = V + ((long long)i0 * vstride + c) * ld;
  const long long vs = vstride * ld;
  DAcc ar[KT], ai[KT], nn;
#pragma unroll
  for (int s = 0; s < KT; ++s) {
    ar[s].init(0.f, 0.f);
    ai[s].init(0.f, 0.f);
  }
  nn.init(0.f, 0.f);
  const long long stride = (long long)nblk * RT;
  for (long long p = (long long)blockIdx.x * RT + threadIdx.x; p < N; p += stride) {
    const float4 wv = wc[p];
#pragma unroll
    for (int s = 0; s < KT; ++s) {
      const float4 v = vb[s * vs + p];
      // conj(v) w = (vr wr + vi wi) + i (vr wi - vi wr)
      ar[s].mac(v.x, v.z, wv.x, wv.z);
      ar[s].mac(v.y, v.w, wv.y, wv.w);
      ai[s].mac(v.x, v.z, wv.y, wv.w);
      ai[s].msub(v.y, v.w, wv.x, wv.z);
    }
    if (want_norm) {
      nn.mac(wv.x, wv.z, wv.x, wv.z);
      nn.mac(wv.y, wv.w, wv.y, wv.w);
    }
  }
  double2 acc[KT];
#pragma unroll
  for (int s = 0; s < KT; ++s) acc[s] = mk<double>(ar[s].to_double(), ai[s].to_double());
  double* part = g.part + (long long)blockIdx.y * (2 * KT + 1) * nblk;
  block_partials<KT>(acc, KT, nn.to_double(), want_norm, part, nblk);
  if (!last_of_column(g.count, c, nblk)) return;
  fold_partials(part, nblk, 2 * KT + want_norm, tot);
  gs_after_dots(g, c, i0, KT, want_norm, pass, tot);
}

// w -= sum_s coef_{i0+s} V_{i0+s}; with the last vectors ||w_new||^2 and the column's step
template <int KT>
__global__ void __launch_bounds__(RT, 2) k_update_df(long long N, const float4* __restrict__ V, long long vstride,
                                                     long long ld, int i0, float4* __restrict__ w,
                                                     const int* __restrict__ cols, int j, int pass, int last,
                                                     GsColumn g) {
  __shared__ double tot[1];
  const int c = cols[blockIdx.y];
  if (pass && !g.flag[c]) return;
  const int nblk = gridDim.x;
  float hrh[KT], hrl[KT], hih[KT], hil[KT];
#pragma unroll
  for (int s = 0; s < KT; ++s) {
    const double2 hv = g.coef[(long long)c * g.hstride + i0 + s];
    split(hv.x, hrh[s], hrl[s]);
    split(hv.y, hih[s], hil[s]);
  }
  const float4* vb = V + ((long long)i0 * vstride + c) * ld;
  const long long vs = vstride * ld;
  float4* wc = w + (long long)c * ld;
  DAcc nn;
  nn.init(0.f, 0.f);
  const long long stride = (long long)nblk * RT;
  for (long long p = (long long)blockIdx.x * RT + threadIdx.x; p < N; p += stride) {
    const float4 wv = wc[p];
    DAcc re, im;
    re.init(wv.x, wv.z);
    im.init(wv.y, wv.w);
#pragma unroll
    for (int s = 0; s < KT; ++s) {
      const float4 v = vb[s * vs + p];
      // (hr + i hi)(vr + i vi) = (hr vr - hi vi) + i (hr vi + hi vr)
      re.msub(hrh[s], hrl[s], v.x, v.z);
      re.mac(hih[s], hil[s], v.y, v.w);
      im.msub(hrh[s], hrl[s], v.y, v.w);
      im.msub(hih[s], hil[s], v.x, v.z);
    }
    re.renorm();
    im.renorm();
    __stcs(&wc[p], make_float4(re.hi, im.hi, re.lo, im.lo));
    if (last) {
      nn.mac(re.hi, re.lo, re.hi, re.lo);
      nn.mac(im.hi, im.lo, im.hi, im.lo);
    }
  }
  if (!last) return;
  double* part = g.part + (long long)blockIdx.y * nblk;
  const double2 none[1] = {mk<double>(0, 0)};
  block_partials<1>(none, 0, nn.to_double(), 1, part, nblk);
  if (!last_of_column(g.count, c, nblk)) return;
  fold_partials(part, nblk, 1, tot);
  gs_after_update(g, c, j, pass, tot[0]);
}

// The first pass's update and the second pass's dots of the new w in one read of the basis:
// HBM is the bound of the separate kernels (6.1 to 6.4 TB/s), so the read saved counts: 193 x
// 161 x 97 x 16, per step averaged over restart 10: 1626 us for both -> 1070; 641 x 321 x 33:
// 267 -> 170.  Near the FP32 pipe's bound at 10 vectors (960 operations per node).  Columns whose
// second pass is not due waste their dots, which cost no traffic; most columns take it.
template <int KT>
__global__ void __launch_bounds__(RT, 2) k_update_dots_df(long long N, const float4* __restrict__ V, long long vstride,
                                                          long long ld, float4* __restrict__ w,
                                                          const int* __restrict__ cols, GsColumn g) {
  __shared__ double tot[2 * KT + 1];
  __shared__ float4 h[KT];  // Re hi, Re lo, Im hi, Im lo
  const int c = cols[blockIdx.y];
  const int nblk = gridDim.x;
  if (threadIdx.x < KT) {
    const double2 hv = g.coef[(long long)c * g.hstride + threadIdx.x];
    float4 q;
    split(hv.x, q.x, q.y);
    split(hv.y, q.z, q.w);
    h[threadIdx.x] = q;
  }
  __syncthreads();
  const float4* vb = V + (long long)c * ld;
  const long long vs = vstride * ld;
  float4* wc = w + (long long)c * ld;
  DAcc ar[KT], ai[KT], nn;
#pragma unroll
  for (int s = 0; s < KT; ++s) {
    ar[s].init(0.f, 0.f);
    ai[s].init(0.f, 0.f);
  }
  nn.init(0.f, 0.f);
  const long long stride = (long long)nblk * RT;
  for (long long p = (long long)blockIdx.x * RT + threadIdx.x; p < N; p += stride) {
    float4 v[KT];
#pragma unroll
    for (int s = 0; s < KT; ++s) v[s] = vb[s * vs + p];
    const float4 wv = wc[p];
    DAcc re, im;
    re.init(wv.x, wv.z);
    im.init(wv.y, wv.w);
#pragma unroll
    for (int s = 0; s < KT; ++s) {
      const float4 q = h[s];
      re.msub(q.x, q.y, v[s].x, v[s].z);
      re.mac(q.z, q.w, v[s].y, v[s].w);
      im.msub(q.x, q.y, v[s].y, v[s].w);
      im.msub(q.z, q.w, v[s].x, v[s].z);
    }
    re.renorm();
    im.renorm();
    __stcs(&wc[p], make_float4(re.hi, im.hi, re.lo, im.lo));
    nn.mac(re.hi, re.lo, re.hi, re.lo);
    nn.mac(im.hi, im.lo, im.hi, im.lo);
#pragma unroll
    for (int s = 0; s < KT; ++s) {
      ar[s].mac(v[s].x, v[s].z, re.hi, re.lo);
      ar[s].mac(v[s].y, v[s].w, im.hi, im.lo);
      ai[s].mac(v[s].x, v[s].z, im.hi, im.lo);
      ai[s].msub(v[s].y, v[s].w, re.hi, re.lo);
    }
  }
  double2 acc[KT];
#pragma unroll
  for (int s = 0; s < KT; ++s) acc[s] = mk<double>(ar[s].to_double(), ai[s].to_double());
  double* part = g.part + (long long)blockIdx.y * (2 * KT + 1) * nblk;
  block_partials<KT>(acc, KT, nn.to_double(), 1, part, nblk);
  if (!last_of_column(g.count, c, nblk)) return;
  fold_partials(part, nblk, 2 * KT + 1, tot);
  gs_after_update(g, c, KT - 1, 0, tot[2 * KT]);
  gs_after_dots(g, c, 0, KT, 0, 1, tot);  // read by the second pass where it is due
}

#define HZ_K_CASES(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)

// The basis in registers beside the sums: up to this many vectors (the restart length's default)
static constexpr int kFuse = 10;
bool gs_fused_df(int vectors) { return vectors <= kFuse; }

// dots: whether the dots are due; update: 1 alone, 2 with the next pass's dots
static void gs_launches_df(Ctx& ctx, long long N, const float4* V, long long vstride, long long ld, int j, int pass,
                           int dots, int update, const int* cols, int ncols, const GsColumn& g) {
  float4* w = const_cast<float4*>(V) + (long long)(j + 1) * vstride * ld;
  const int K = j + 1;
  const dim3 grid(gs_nblk(N, ncols), ncols);
  const double el = pass ? 0.0 : (double)N * ncols;
  for (int i0 = 0; dots && i0 < K; i0 += 16) {
    const int k = std::min(16, K - i0);
    const int wn = (pass == 0 && i0 + 16 >= K) ? 1 : 0;
    switch (k) {
#define HZ_GS_CASE(q)                                                                                             \
  case q:                                                                                                         \
    HZ_LAUNCH(ctx, "krylov_dots", el * (k + 1) * 16.0, k_dots_df<q>, grid, RT, 0, N, V, vstride, ld, i0, w, cols, \
              pass, wn, g);                                                                                       \
    break;
      HZ_K_CASES(HZ_GS_CASE)
#undef HZ_GS_CASE
    }
  }
  if (update == 2) {
    switch (K) {
#define HZ_GS_CASE(q)                                                                                              \
  case q:                                                                                                          \
    HZ_LAUNCH(ctx, "krylov_update", el * (K + 2) * 16.0, k_update_dots_df<q>, grid, RT, 0, N, V, vstride, ld, w, cols, \
              g);                                                                                                  \
    break;
      HZ_GS_CASE(1) HZ_GS_CASE(2) HZ_GS_CASE(3) HZ_GS_CASE(4) HZ_GS_CASE(5)
      HZ_GS_CASE(6) HZ_GS_CASE(7) HZ_GS_CASE(8) HZ_GS_CASE(9) HZ_GS_CASE(10)
#undef HZ_GS_CASE
    }
    return;
  }
  for (int i0 = 0; i0 < K; i0 += 16) {
    const int k = std::min(16, K - i0);
    const int last = i0 + 16 >= K ? 1 : 0;
    switch (k) {
#define HZ_GS_CASE(q)                                                                                               \
  case q:                                                                                                           \
    HZ_LAUNCH(ctx, "krylov_update", el * (k + 2) * 16.0, k_update_df<q>, grid, RT, 0, N, V, vstride, ld, i0, w, cols, \
              j, pass, last, g);                                                                                    \
    break;
      HZ_K_CASES(HZ_GS_CASE)
#undef HZ_GS_CASE
    }
  }
}

void launch_gs_df(Ctx& ctx, long long N, const float4* V, long long vstride, long long ld, int j, const int* cols,
                  int ncols, const GsColumn& g) {
  if (ncols <= 0) return;
  const bool fused = gs_fused_df(j + 1);
  gs_launches_df(ctx, N, V, vstride, ld, j, 0, 1, fused ? 2 : 1, cols, ncols, g);
  gs_launches_df(ctx, N, V, vstride, ld, j, 1, fused ? 0 : 1, 1, cols, ncols, g);
}

// ---- coarsest solve with emulated-FP64 window operators ---------------------
// Same schedule as k_band_coop (one cooperative launch, grid-wide barrier
// between block steps); operators T/G and the work vectors are df64.
__device__ __forceinline__ void cmac_df(DAcc& re, DAcc& im, const float4 m, const float4 v) {
  // (mr + i mi)(vr + i vi)
  re.mac(m.x, m.z, v.x, v.z);
  re.msub(m.y, m.w, v.y, v.w);
  im.mac(m.x, m.z, v.y, v.w);
  im.mac(m.y, m.w, v.x, v.z);
}

__device__ __forceinline__ float4 warp_sum_df(const DAcc& re, const DAcc& im) {
  double a = re.to_double(), b = im.to_double();
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  float rh, rl, ih, il;
  split(a, rh, rl);
  split(b, ih, il);
  return make_float4(rh, ih, rl, il);
}

static constexpr int BCW = 1;  // columns per warp item

template <typename T>
__global__ void __launch_bounds__(256) k_band_coop_df(long long N, int nbk, const BandBlock* __restrict__ blocks,
                                                      const float4* __restrict__ Tops, const float4* __restrict__ Gops,
                                                      const cplx<T>* __restrict__ b, long long ldb,
                                                      const int* __restrict__ cols, int ncols,
                                                      float4* __restrict__ work, cplx<T>* __restrict__ x,
                                                      long long ldx) {
  cg::grid_group grid = cg::this_grid();
  const int lane = threadIdx.x & 31;
  const long long gw = ((long long)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const long long nw = ((long long)gridDim.x * blockDim.x) >> 5;
  float4* const Y0 = work;
  float4* const Y1 = work + (long long)ncols * N;
  float4* const X4 = work + 2LL * ncols * N;
  const int ngrp = (ncols + BCW - 1) / BCW;
  long long prev_end = 0;
  for (int I = 0; I < nbk; ++I) {
    const BandBlock B = blocks[I];
    const int split_k = (I == 0) ? 0 : (int)(prev_end - B.s);
    const float4* src0 = (I & 1) ? Y0 : Y1;
    float4* dst = (I & 1) ? Y1 : Y0;
    const long long items = (long long)B.W * ngrp;
    for (long long it = gw; it < items; it += nw) {
      const int i = (int)(it % B.W), c0 = (int)(it / B.W) * BCW;
      const float4* Mr = Tops + B.toff + (long long)i * B.W;
      DAcc re[BCW], im[BCW];
#pragma unroll
      for (int c = 0; c < BCW; ++c) {
        re[c].init(0.f, 0.f);
        im[c].init(0.f, 0.f);
      }
      for (int k = lane; k < B.W; k += 32) {
        const float4 m = Mr[k];
#pragma unroll
        for (int c = 0; c < BCW; ++c) {
          const int ci = c0 + c;
          if (ci < ncols) {
            float4 v;
            if (k < split_k) {
              v = src0[(long long)ci * N + B.s + k];
            } else {
              const cplx<T> bb = b[(long long)cols[ci] * ldb + B.s + k];
              v = make_float4((float)bb.x, (float)bb.y, 0.f, 0.f);  // FP32 input: exact as a df64 pair
            }
            cmac_df(re[c], im[c], m, v);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < BCW; ++c) {
        const float4 r = warp_sum_df(re[c], im[c]);
        if (lane == 0 && c0 + c < ncols) dst[(long long)(c0 + c) * N + B.s + i] = r;
      }
    }
    prev_end = B.s + B.W;
    grid.sync();
  }
  for (int I = nbk - 1; I >= 0; --I) {
    const BandBlock B = blocks[I];
    const float4* yb = (I & 1) ? Y1 : Y0;
    const long long items = (long long)B.nb * ngrp;
    for (long long it = gw; it < items; it += nw) {
      const int i = (int)(it % B.nb), c0 = (int)(it / B.nb) * BCW;
      const float4* Mr = Gops + B.goff + (long long)i * B.Wb;
      DAcc re[BCW], im[BCW];
#pragma unroll
      for (int c = 0; c < BCW; ++c) {
        re[c].init(0.f, 0.f);
        im[c].init(0.f, 0.f);
      }
      for (int k = lane; k < B.Wb; k += 32) {
        const float4 m = Mr[k];
#pragma unroll
        for (int c = 0; c < BCW; ++c) {
          const int ci = c0 + c;
          if (ci < ncols) {
            const long long q = (long long)ci * N + B.s + k;
            cmac_df(re[c], im[c], m, (k < B.nb) ? yb[q] : X4[q]);
          }
        }
      }
#pragma unroll
      for (int c = 0; c < BCW; ++c) {
        const float4 r = warp_sum_df(re[c], im[c]);
        const int ci = c0 + c;
        if (lane == 0 && ci < ncols) {
          X4[(long long)ci * N + B.s + i] = r;
          x[(long long)cols[ci] * ldx + B.s + i] =
              mk<T>((T)((double)r.x + (double)r.z), (T)((double)r.y + (double)r.w));
        }
      }
    }
    grid.sync();
  }
}

template <typename T>
void launch_band_solve_df(Ctx& ctx, const BandSolveOps& op, const cplx<T>* b, cplx<T>* x, long long ld,
                          const int* cols, int ncols, float4* work) {
  if (ncols <= 0) return;
  const long long N = op.N;
  const int nbk = (int)op.blocks.size();
  double bytes = 0.0;
  for (const BandBlock& B : op.blocks)
    bytes += ((double)B.W * B.W + (double)B.nb * B.Wb) * 16.0 + ncols * (2.0 * B.W + B.Wb + 2.0 * B.nb) * 16.0;
  static int capacity[kMaxDevices] = {};
  int dev = 0;
  cudaGetDevice(&dev);
  if (dev >= 0 && dev < kMaxDevices && capacity[dev] == 0) {
    int per_sm = 0, sms = 0;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_band_coop_df<T>, 256, 0);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    capacity[dev] = std::max(1, std::min(per_sm, 4)) * std::max(1, sms);
  }
  const int grid = (dev >= 0 && dev < kMaxDevices) ? capacity[dev] : kSMs;
  static thread_local int id = -1;
  if (id < 0 || (size_t)id >= ctx.names.size() || ctx.names[id] != "band_solve") id = ctx.name_id("band_solve");
  cudaEvent_t ev = nullptr;
  ctx.before(id, &ev);
  const BandBlock* blk = op.dblocks;
  const float4* Tp = reinterpret_cast<const float4*>(op.T);
  const float4* Gp = reinterpret_cast<const float4*>(op.G);
  long long ldb = ld, ldx = ld;
  void* args[] = {(void*)&N,    (void*)&nbk,  (void*)&blk,   (void*)&Tp,   (void*)&Gp, (void*)&b,
                  (void*)&ldb,  (void*)&cols, (void*)&ncols, (void*)&work, (void*)&x,  (void*)&ldx};
  const cudaError_t e =
      cudaLaunchCooperativeKernel((const void*)k_band_coop_df<T>, dim3(grid), dim3(256), args, 0, ctx.stream);
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw std::runtime_error(std::string("band_solve (emulated FP64) cooperative launch failed: ") +
                             cudaGetErrorString(e));
  }
  ctx.after(id, ev, bytes);
}
template void launch_band_solve_df<float>(Ctx&, const BandSolveOps&, const float2*, float2*, long long, const int*,
                                          int, float4*);

// ---- solution update x += sum_i y_i Z_i (Z complex FP32, x FP64) -----------------
// Bound by the wait for Z with one vector's load at a time (2.0 TB/s): kUx vectors' loads are
// issued together.  193 x 161 x 97 nodes, 16 columns, 10 vectors: 2706 -> 1324 us.
static constexpr int kUx = 5;
__global__ void __launch_bounds__(256, 4) k_update_x_df(long long N, const float2* __restrict__ Z, long long zstride,
                                                     long long ld, const int* __restrict__ kcol,
                                                     const double2* __restrict__ y, int ystride,
                                                     double2* __restrict__ x, long long xld,
                                                     const int* __restrict__ cols) {
  const int c = cols[blockIdx.y];
  const int k = kcol[c];
  // the coefficients of this column, split into FP32 pairs once per block and
  // read from shared memory (broadcast): registers stay free for occupancy
  __shared__ float4 sy[64 + kUx];  // Re hi, Re lo, Im hi, Im lo; restart length <= 64; zeros fill the last group
  for (int s = threadIdx.x; s < 64 + kUx; s += blockDim.x) {
    const double2 v = s < k ? y[(long long)c * ystride + s] : mk<double>(0, 0);
    float4 p;
    split(v.x, p.x, p.y);
    split(v.y, p.z, p.w);
    sy[s] = p;
  }
  __syncthreads();
  double2* xc = x + (long long)c * xld;
  const float2* zc = Z + (long long)c * ld;
  const long long zs = zstride * ld;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (long long)gridDim.x * blockDim.x) {
    DAcc re, im;
    re.init(0.f, 0.f);
    im.init(0.f, 0.f);
    const double2 xv = xc[p];
    for (int s0 = 0; s0 < k; s0 += kUx) {
      float2 z[kUx];
#pragma unroll
      for (int s = 0; s < kUx; ++s) z[s] = s0 + s < k ? __ldcs(zc + (s0 + s) * zs + p) : make_float2(0.f, 0.f);
#pragma unroll
      for (int s = 0; s < kUx; ++s) {
        const float4 q = sy[s0 + s];
        // (yr + i yi)(zr + i zi)
        re.mac1(q.x, q.y, z[s].x);
        re.mac1(-q.z, -q.w, z[s].y);
        im.mac1(q.x, q.y, z[s].y);
        im.mac1(q.z, q.w, z[s].x);
      }
    }
    xc[p] = mk<double>(xv.x + re.to_double(), xv.y + im.to_double());
  }
}

void launch_update_x_df(Ctx& ctx, long long N, const float2* Z, long long zstride, long long ld, const int* kcol,
                        const double2* y, int ystride, double2* x, long long xld, const int* cols, int ncols,
                        long long zcols) {
  if (ncols <= 0) return;
  const int nb = std::max(1, std::min((int)((N + 255) / 256), 8 * kSMs / std::max(ncols, 1) + 1));
  const double bytes = (double)N * (ncols * 2.0 * 16.0 + zcols * 8.0);
  HZ_LAUNCH(ctx, "update_x", bytes, k_update_x_df, dim3(nb, ncols), 256, 0, N, Z, zstride, ld, kcol, y, ystride, x,
            xld, cols);
}

// ---- conversions and scaling -------------------------------------------------
// y[:, c] = s[c] * x[:, c]: FP64 x into a df64 y (the start vector of a cycle)
__global__ void __launch_bounds__(256) k_to_df(long long N, const double2* __restrict__ x, long long xld,
                                               float4* __restrict__ y, long long yld, const double* __restrict__ s,
                                               const int* __restrict__ cols) {
  const int c = cols[blockIdx.y];
  const double sc = s[c];
  const double2* xc = x + (long long)c * xld;
  float4* yc = y + (long long)c * yld;
  // elements are independent (in place: each is read before it is written)
#pragma unroll 4
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (long long)gridDim.x * blockDim.x) {
    const double2 v = __ldcs(&xc[p]);
    float rh, rl, ih, il;
    split(sc * v.x, rh, rl);
    split(sc * v.y, ih, il);
    __stcs(&yc[p], make_float4(rh, ih, rl, il));
  }
}

void launch_to_df(Ctx& ctx, long long N, const double2* x, long long xld, float4* y, long long yld, const double* s,
                  const int* cols, int ncols) {
  if (ncols <= 0) return;
  const int nb = std::max(1, std::min((int)((N + 255) / 256), 8 * kSMs / std::max(ncols, 1) + 1));
  HZ_LAUNCH(ctx, "scale_cols", (double)N * ncols * 32.0, k_to_df, dim3(nb, ncols), 256, 0, N, x, xld, y, yld, s,
            cols);
}

// df64 diag(H) from the FP64 array (once per handle)
__global__ void k_diag_to_df(long long N, const double2* __restrict__ d, float4* __restrict__ out) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (long long)gridDim.x * blockDim.x) {
    float rh, rl, ih, il;
    split(d[p].x, rh, rl);
    split(d[p].y, ih, il);
    out[p] = make_float4(rh, ih, rl, il);
  }
}

void launch_diag_to_df(Ctx& ctx, long long N, const double2* d, float4* out) {
  const long long nb = std::min<long long>((N + 255) / 256, 16LL * kSMs);
  HZ_LAUNCH(ctx, "cast", (double)N * 32.0, k_diag_to_df, (unsigned)nb, 256, 0, N, d, out);
}

}  // namespace hz
