// Folding of the Gram-Schmidt sums and the per-column scalar steps of FGMRES, shared
// by the FP64 (hz_krylov.cu) and the double-float (hz_df64.cu) kernels.
//
// A pass is two launches, dots and update (the double-float form's first update carries the
// second pass's dots).  The last block of a column to finish folds the
// blocks' partial sums in block order (deterministic) and does the column's scalar work
// there: the update coefficients after the dots, the DGKS test and, when no second pass is
// due, the Hessenberg column, Givens rotation and residual estimate after the update.
// These were 14 launches per iteration with the host reading two copies; small problems
// spent most of an iteration in them.
#pragma once

#include "hz_launch.cuh"

namespace hz {

// Totals over a warp of P (a power of two up to 32) values per lane, each in the order of a
// full exchange (xor 16, 8, 4, 2, 1), P - 1 + log2(32 / P) additions instead of 5 P: every
// step halves the values a lane carries.  Lane l returns the total of value
// warp_total_index<P>(l).
template <int P>
__device__ __forceinline__ double warp_totals(double (&v)[P], int lane) {
  int cnt = P;
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    if (cnt > 1) {
      cnt >>= 1;
      const bool up = lane & o;
#pragma unroll
      for (int i = 0; i < P / 2; ++i)
        if (i < cnt) {
          const double give = up ? v[i] : v[i + cnt], keep = up ? v[i + cnt] : v[i];
          v[i] = keep + __shfl_xor_sync(0xffffffffu, give, o);
        }
    } else {
      v[0] += __shfl_xor_sync(0xffffffffu, v[0], o);
    }
  }
  return v[0];
}
template <int P>
__device__ __forceinline__ int warp_total_index(int lane) {
  int idx = 0;
#pragma unroll
  for (int o = 16, c = P / 2; c > 0; o >>= 1, c >>= 1) idx += (lane & o) ? c : 0;
  return idx;
}
__host__ __device__ constexpr int pow2_at_least(int n) { return n <= 1 ? 1 : 2 * pow2_at_least((n + 1) / 2); }

// A block's sums of nv complex values and a norm (slot nv), 8 warps, as doubles in
// part[(slot * 2 + (0 | 1)) * nblk + blk]; sh holds 8 * (2 NV + 2) doubles.
template <int NV>
__device__ __forceinline__ void block_partials(const double2 (&acc)[NV], int nv, double nrm, int want_norm,
                                               double* part, int nblk) {
  constexpr int P = pow2_at_least(2 * NV);
  static_assert(P <= 32, "up to 16 complex sums");
  __shared__ double sh[8][P + 1];
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double v[P];
#pragma unroll
  for (int s = 0; s < P / 2; ++s) {
    v[2 * s] = s < NV ? acc[s < NV ? s : 0].x : 0.0;
    v[2 * s + 1] = s < NV ? acc[s < NV ? s : 0].y : 0.0;
  }
  const double t = warp_totals<P>(v, lane);
  if ((lane & (32 / P - 1)) == 0) sh[warp][warp_total_index<P>(lane)] = t;
  if (want_norm) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
    if (lane == 0) sh[warp][P] = nrm;
  }
  __syncthreads();
  const int tot = 2 * nv + want_norm;
  if ((int)threadIdx.x < tot) {
    const int src = (int)threadIdx.x < 2 * nv ? (int)threadIdx.x : P;
    double a = 0.0;
#pragma unroll
    for (int w = 0; w < 8; ++w) a += sh[w][src];
    __stcg(&part[(long long)threadIdx.x * nblk + blockIdx.x], a);
    __threadfence();
  }
}

// True in the last block of column c to come here; its threads then see every
// block's partials.  count[c] is left at 0.
__device__ __forceinline__ bool last_of_column(int* count, int c, int nblk) {
  __shared__ int last;
  __syncthreads();
  if (threadIdx.x == 0)
    last = atomicInc(reinterpret_cast<unsigned*>(&count[c]), (unsigned)nblk - 1) == (unsigned)nblk - 1;
  __syncthreads();
  if (last) __threadfence();
  return last;
}

// out[i] = sum of partial i over the blocks, i < tot (shared memory; all threads may read it after)
__device__ __forceinline__ void fold_partials(const double* part, int nblk, int tot, double* out) {
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  for (int i = warp; i < tot; i += 8) {
    double a = 0.0;
    for (int b = lane; b < nblk; b += 32) a += __ldcg(&part[(long long)i * nblk + b]);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) a += __shfl_xor_sync(0xffffffffu, a, o);
    if (lane == 0) out[i] = a;
  }
  __syncthreads();
}

// sqrt of a reduced sum of squares: rounding can leave it a hair below zero;
// NaN and Inf pass through so the host sees a corrupted column.
__device__ __forceinline__ double gs_sqrt(double v) { return (v > 0.0 || v != v) ? sqrt(v) : 0.0; }

// After the dots of one launch (K vectors from i0): the dots into out, the update
// coefficients sig_i^2 d_i into coef, ||w||^2 (want_norm) into slot i0 + K.
__device__ __forceinline__ void gs_after_dots(const GsColumn& g, int c, int i0, int K, int want_norm, int pass,
                                              const double* tot) {
  double2* out = (pass ? g.hB : g.hA) + (long long)c * g.hstride + i0;
  for (int i = threadIdx.x; i < K; i += blockDim.x) {
    const double s = g.sig[(long long)c * g.sstride + i0 + i];
    out[i] = mk<double>(tot[2 * i], tot[2 * i + 1]);
    g.coef[(long long)c * g.hstride + i0 + i] = mk<double>(s * s * tot[2 * i], s * s * tot[2 * i + 1]);
  }
  if (want_norm && threadIdx.x == 0) out[K] = mk<double>(tot[2 * K], 0.0);
}

// Step j of column c is complete: Hessenberg entries of the normalised basis (sig_i tau_j d_i,
// h_{j+1,j} = tau_j ||w''||), Givens rotations (u, v) -> (conj(c) u + conj(s) v, -s u + c v),
// residual estimate (to the device and to pinned host memory) and the next scale.
// Called by one warp.
__device__ __forceinline__ void gs_finish(const GsColumn& g, int c, int j, bool second, double n2) {
  const int lane = threadIdx.x & 31, m = g.m;
  const double* sc = g.sig + (long long)c * g.sstride;
  double2* H = g.Hh + (long long)c * (m + 1) * m + (long long)j * (m + 1);
  const double2 *csc = g.cs + (long long)c * m, *snc = g.sn + (long long)c * m;
  const double sj = basis_tau(sc[j]);  // the candidate's scale
  for (int i = lane; i <= j; i += 32) {
    double2 v = g.hA[(long long)c * g.hstride + i];
    const double f = sc[i] * sj;
    v = mk<double>(f * v.x, f * v.y);
    if (second) {
      const double2 u = g.hB[(long long)c * g.hstride + i];
      v = mk<double>(v.x + f * u.x, v.y + f * u.y);
    }
    H[i] = v;
  }
  __syncwarp();
  if (lane) return;
  const double hn = gs_sqrt(n2 * sj * sj);
  double2 u = H[0];
  for (int i = 0; i < j; ++i) {
    const double2 v = H[i + 1], ci = csc[i], si = snc[i];
    H[i] = cadd<double>(cmul<double>(cconj<double>(ci), u), cmul<double>(cconj<double>(si), v));
    u = csub<double>(cmul<double>(ci, v), cmul<double>(si, u));
  }
  double den = sqrt(u.x * u.x + u.y * u.y + hn * hn);
  double2 cj = mk<double>(1.0, 0.0), sn = mk<double>(0.0, 0.0);
  if (den > 0) {
    cj = mk<double>(u.x / den, u.y / den);
    sn = mk<double>(hn / den, 0.0);
  } else {
    den = 0.0;
  }
  g.cs[(long long)c * m + j] = cj;
  g.sn[(long long)c * m + j] = sn;
  H[j] = mk<double>(den, 0.0);
  H[j + 1] = mk<double>(0.0, 0.0);
  double2* gc = g.g + (long long)c * (m + 1);
  const double2 gj = gc[j];
  gc[j] = cmul<double>(cconj<double>(cj), gj);
  const double2 gn = cmul<double>(sn, gj);
  gc[j + 1] = mk<double>(-gn.x, -gn.y);
  g.host_est[c] = sqrt(gn.x * gn.x + gn.y * gn.y);
  g.sig[(long long)c * g.sstride + j + 1] = sj * (hn > 0 ? 1.0 / hn : 0.0);
}

// After the update of a pass: ||w'||^2 = n2.  Pass 0: the DGKS test (a second pass when
// the first removed more than half of the squared norm).
__device__ __forceinline__ void gs_after_update(const GsColumn& g, int c, int j, int pass, double n2) {
  if (threadIdx.x >= 32) return;
  bool second = pass != 0;
  if (!pass) {
    const bool again = n2 < 0.5 * g.hA[(long long)c * g.hstride + j + 1].x;
    if (threadIdx.x == 0) {
      g.flag[c] = again ? 1 : 0;
      g.host_flag[c] = again ? 1 : 0;
    }
    if (again) return;
  }
  gs_finish(g, c, j, second, n2);
}

}  // namespace hz
