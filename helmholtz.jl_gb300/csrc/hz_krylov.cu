// FP64 FGMRES kernels (Arnoldi with classical Gram-Schmidt, Givens rotations,
// least squares, solution update) batched over the active right-hand-side
// columns, plus the multigrid setup kernels (Galerkin probing, coefficient
// transpose, casts).
//
// Replaces solveGMRES_MG of Multigrid.jl / KrylovMethods.jl called at
// src/ShiftedLaplacianMultigridSolver.jl:89 and the RAP products of MGsetup
// (src/ShiftedLaplacianMultigridSolver.jl:64-65).
#include <algorithm>

#include "hz_fixed.cuh"
#include "hz_gs.cuh"
#include "hz_launch.cuh"

namespace hz {


static constexpr int RT = 256; // threads per reduction CTA

int krylov_nblk(long long N, int ncols) {
  long long target = 4LL * kSMs * 2;  // ~8 CTAs of 256 threads per SM in total
  long long nb = (target + ncols - 1) / std::max(ncols, 1);
  long long maxb = (N + RT - 1) / RT;
  nb = std::max(1LL, std::min(nb, maxb));
  return (int)nb;
}

// KT (0 or 1) dots and the norm of w: native FP64, its rounding order is part of the
// BiCGSTAB iteration.  Block totals in part[(pos * K1 + slot) * nblk + blk].
template <int KT>
__global__ void __launch_bounds__(RT, 2) k_dots(long long N, const double2* __restrict__ V, long long ld,
                                                const double2* __restrict__ w, long long wld,
                                                const int* __restrict__ cols, int nblk, int want_norm,
                                                double2* __restrict__ part) {
  __shared__ double sh[RT / 32][4];
  const int pos = blockIdx.y;
  const int c = cols[pos];
  const int K1 = KT + want_norm;
  double2* pp = part + (long long)pos * K1 * nblk;
  const double2* wc = w + (long long)c * wld;
  const double2* vc = V + (long long)c * ld;
  double2 acc = mk<double>(0, 0);
  double nrm = 0.0;
  const long long stride = (long long)nblk * RT;
#pragma unroll 4
  for (long long p = (long long)blockIdx.x * RT + threadIdx.x; p < N; p += stride) {
    const double2 wv = wc[p];
    if (KT) acc = cfma_conj<double>(vc[p], wv, acc);
    if (want_norm) nrm = fma(wv.x, wv.x, fma(wv.y, wv.y, nrm));
  }
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  double v[4] = {acc.x, acc.y, nrm, 0.0};
  const double t = warp_totals<4>(v, lane);
  if ((lane & 7) == 0) sh[warp][warp_total_index<4>(lane)] = t;
  __syncthreads();
  if ((int)threadIdx.x < K1) {
    const int i = (int)threadIdx.x < KT ? 0 : 2;
    double a = 0, b = 0;
    for (int q = 0; q < RT / 32; ++q) {
      a += sh[q][i];
      b += sh[q][i + 1];
    }
    pp[(long long)threadIdx.x * nblk + blockIdx.x] = mk<double>(a, b);
  }
}

void launch_dots(Ctx& ctx, long long N, const double2* V, long long ld, int K, const double2* w, long long wld,
                 const int* cols, int ncols, int nblk, int want_norm, double2* part) {
  if (ncols <= 0) return;
  const dim3 grid(nblk, ncols);
  const double bytes = (double)N * ncols * (K + 1) * sizeof(double2);
  // FP64 arithmetic: a complex multiply-add (8 flops) per vector and node, 4 for ||w||^2
  ctx.add_flops("krylov_dots", (double)N * ncols * (8.0 * K + (want_norm ? 4.0 : 0.0)));
  if (K == 0)
    HZ_LAUNCH(ctx, "krylov_dots", bytes, k_dots<0>, grid, RT, 0, N, V, ld, w, wld, cols, nblk, want_norm, part);
  else if (K == 1)
    HZ_LAUNCH(ctx, "krylov_dots", bytes, k_dots<1>, grid, RT, 0, N, V, ld, w, wld, cols, nblk, want_norm, part);
  else
    throw std::runtime_error("launch_dots: 0 or 1 vectors");
}

// ---------------------------------------------------------------------------
// Gram-Schmidt in FP64 on the integer pipe (hz_fixed.cuh)
// ---------------------------------------------------------------------------
// Native FP64 takes four FMAs per 16-byte basis element, two clocks of an SM; HBM delivers
// the element in 0.7.  So the basis is kept as fixed-point words (58 bits, hz_fixed.cuh) with one
// reference per 128 nodes, the largest value's exponent: the first dots of step j, which read the
// newest vector v_j as the preconditioner did, write it back so, in place.  Dots: a warp takes
// such a group, four nodes per lane, relates w to the largest of a lane's four, sums the
// products in integers and adds the exact total to its FP64 accumulator.  Update: the
// coefficients are related to the group's largest term instead of the basis values; the exact sum
// is subtracted from w with one rounding.  Groups outside the range of hz_fixed.cuh stay FP64
// (kGsRaw) and take the native steps, as do values of w.
// Measured per pass averaged over the steps of restart 10 (the second pass included, which most
// columns take), native / converting every value in every pass / words: 129^3 x 8: dots 632 / 461 /
// 301 us, update 642 / 427 / 359 us; 1025 x 513 x 16: 333 / 235 / 157, 320 / 215 / 181 us: 5.0 to
// 5.4 TB/s.  What bounds them is latency: 16 warps per SM at 113 to 128 registers, dots with one
// vector on its way (352 us without), update with all of a node's.  Errors against quadruple
// precision, 4,096 to 200,000 nodes, waves, a point source's peak and noise: dots 5e-17 to
// 1.1e-16 of |V||w| (native 5e-17 to 2.5e-16), update 5e-17 to 7e-17 of |w'| rms (2.4e-16).
static constexpr int kGsNodes = 4;
static constexpr int kGsGroup = 32 * kGsNodes;
enum { kGsZero = -1, kGsRaw = -2 };  // exponents of a group without a reference

size_t gs_exponents(long long N, int vectors) { return (size_t)vectors * ((N + kGsGroup - 1) / kGsGroup) * sizeof(int); }

// FP64 value of stored words (kept raw: their bits)
__device__ __forceinline__ double gs_value(int hi, int lo, int e) {
  if (e == kGsRaw) return __hiloint2double(lo, hi);
  if (e < 0) return 0.0;
  const double v = fma((double)hi, 536870912.0, (double)lo);  // 2^29
  return v * __hiloint2double((e - 1080 + 1023) << 20, 0);
}
__device__ __forceinline__ double2 gs_value(int4 r, int e) { return mk<double>(gs_value(r.x, r.y, e), gs_value(r.z, r.w, e)); }

template <int KT>
__global__ void __launch_bounds__(RT, 2) k_gs_dots(long long N, double2* __restrict__ V, long long vstride,
                                                   long long ld, int i0, const double2* __restrict__ w,
                                                   const int* __restrict__ cols, int pass, int want_norm, int fresh,
                                                   GsColumn g) {
  __shared__ double tot[2 * KT + 1];
  const int c = cols[blockIdx.y];
  if (pass && !g.flag[c]) return;
  const int nblk = gridDim.x;
  const int lane = threadIdx.x & 31;
  const double2* wc = w + (long long)c * ld;
  int4* vb = reinterpret_cast<int4*>(V + ((long long)i0 * vstride + c) * ld);
  const long long vs = vstride * ld;  // distance between consecutive basis vectors
  const long long groups = (N + kGsGroup - 1) / kGsGroup, es = vstride * groups;
  int* eb = g.vexp + ((long long)i0 * vstride + c) * groups;
  // lanes below 16 carry the sums' real parts, the others the imaginary ones: a pair of lanes
  // exchanges its exact totals, so that each converts one of them (the conversion takes two and
  // a half slots of the FP64 pipe)
  const bool upper = lane & 16;
  double acc[KT];
#pragma unroll
  for (int s = 0; s < KT; ++s) acc[s] = 0.0;
  double nrm = 0.0;
  // one vector's nodes and the next group's references (lane s: vector s's) are on their way while
  // the vector before is worked on
  const long long first = (long long)blockIdx.x * (RT / 32) + (threadIdx.x >> 5), round = (long long)nblk * (RT / 32);
  int4 next[kGsNodes];
  auto fetch = [&](int s, long long gi) {
    const long long p = gi * kGsGroup + lane;
#pragma unroll
    for (int q = 0; q < kGsNodes; ++q)
      next[q] = gi < groups && p + q * 32 < N ? vb[s * vs + p + q * 32] : make_int4(0, 0, 0, 0);
  };
  const int* el = eb + (lane < KT ? lane : 0) * es;
  int ahead = first < groups ? el[first] : kGsZero;
  fetch(0, first);
  for (long long gi = first; gi < groups; gi += round) {
    const long long p = gi * kGsGroup + lane;
    const int e = ahead;
    if (gi + round < groups) ahead = el[gi + round];
    double2 wv[kGsNodes];
    Fixed wx[kGsNodes], wy[kGsNodes];
    int ew = 0;
#pragma unroll
    for (int q = 0; q < kGsNodes; ++q) {
      wv[q] = p + q * 32 < N ? wc[p + q * 32] : mk<double>(0, 0);
      ew = max(ew, max(fixed_exponent((uint32_t)__double2hiint(wv[q].x)), fixed_exponent((uint32_t)__double2hiint(wv[q].y))));
    }
    ew = __reduce_max_sync(0xffffffffu, ew);
    const bool wok = fixed_ref_ok(ew);
#pragma unroll
    for (int q = 0; q < kGsNodes; ++q) {
      wx[q] = fixed_from<6>((uint32_t)__double2hiint(wv[q].x), (uint32_t)__double2loint(wv[q].x), ew);
      wy[q] = fixed_from<6>((uint32_t)__double2hiint(wv[q].y), (uint32_t)__double2loint(wv[q].y), ew);
      if (want_norm) nrm = fma(wv[q].x, wv[q].x, fma(wv[q].y, wv[q].y, nrm));
    }
#pragma unroll
    for (int s = 0; s < KT; ++s) {
      int4 v[kGsNodes];
#pragma unroll
      for (int q = 0; q < kGsNodes; ++q) v[q] = next[q];
      if (s + 1 < KT)
        fetch(s + 1, gi);
      else
        fetch(0, gi + round);
      int ev;
      if (s == KT - 1 && fresh) {  // FP64 still: to words, in place
        uint32_t top = 0, any = 0;
#pragma unroll
        for (int q = 0; q < kGsNodes; ++q) {
          top = max(top, max((uint32_t)v[q].y & 0x7fffffffu, (uint32_t)v[q].w & 0x7fffffffu));
          any |= (uint32_t)v[q].x | (uint32_t)v[q].z;
        }
        top = __reduce_max_sync(0xffffffffu, top);
        any = __reduce_or_sync(0xffffffffu, any);
        ev = (int)(top >> 20);
        if (fixed_ref_ok(ev)) {
#pragma unroll
          for (int q = 0; q < kGsNodes; ++q) {
            const Fixed a = fixed_from<6>((uint32_t)v[q].y, (uint32_t)v[q].x, ev);
            const Fixed b = fixed_from<6>((uint32_t)v[q].w, (uint32_t)v[q].z, ev);
            v[q] = make_int4(a.hi, a.lo, b.hi, b.lo);
            if (p + q * 32 < N) vb[s * vs + p + q * 32] = v[q];
          }
        } else {
          ev = (top | any) ? kGsRaw : kGsZero;
        }
        if (lane == 0) eb[s * es + gi] = ev;
      } else {
        ev = __shfl_sync(0xffffffffu, e, s);
      }
      if (ev >= 0 && wok && fixed_ok(ev + ew)) {
        FixedSum f{0, 0, 0, 0};
#pragma unroll
        for (int q = 0; q < kGsNodes; ++q)
          fixed_conj_mac(f, Fixed{v[q].x, v[q].y}, Fixed{v[q].z, v[q].w}, wx[q], wy[q]);
        const long long re = fixed_total(f.rh, f.rl), im = fixed_total(f.ih, f.il);
        const long long t = (upper ? im : re) + __shfl_xor_sync(0xffffffffu, upper ? re : im, 16);
        acc[s] = fma((double)t, __hiloint2double((int)fixed_scale_hi(ev + ew, 0), 0), acc[s]);
      } else if (ev != kGsZero) {
        double2 t = mk<double>(0, 0);
#pragma unroll
        for (int q = 0; q < kGsNodes; ++q) t = cfma_conj<double>(gs_value(v[q], ev), wv[q], t);
        acc[s] += (upper ? t.y : t.x) + __shfl_xor_sync(0xffffffffu, upper ? t.x : t.y, 16);
      }
    }
  }
  double2 sums[KT];
#pragma unroll
  for (int s = 0; s < KT; ++s) sums[s] = upper ? mk<double>(0, acc[s]) : mk<double>(acc[s], 0);
  double* part = g.part + (long long)blockIdx.y * (2 * KT + 1) * nblk;
  block_partials<KT>(sums, KT, nrm, want_norm, part, nblk);
  if (!last_of_column(g.count, c, nblk)) return;
  fold_partials(part, nblk, 2 * KT + want_norm, tot);
  gs_after_dots(g, c, i0, KT, want_norm, pass, tot);
}

template <int KT>
__global__ void __launch_bounds__(RT, 2) k_gs_update(long long N, const double2* __restrict__ V, long long vstride,
                                                     long long ld, int i0, double2* __restrict__ w,
                                                     const int* __restrict__ cols, int j, int pass, int last,
                                                     GsColumn g) {
  __shared__ int4 hl[RT / 32][KT];
  __shared__ double tot[1];
  const int c = cols[blockIdx.y];
  if (pass && !g.flag[c]) return;
  const int nblk = gridDim.x;
  const double2* h = g.coef + (long long)c * g.hstride + i0;
  constexpr int kNone = -(1 << 20);  // exponent of a zero coefficient
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  // lane s holds the coefficient of vector s
  const uint4 hr = lane < KT ? *reinterpret_cast<const uint4*>(h + lane) : make_uint4(0, 0, 0, 0);
  const bool hzero = ((hr.x | hr.z) == 0) && (((hr.y | hr.w) & 0x7fffffffu) == 0);
  const int he = max(fixed_exponent(hr.y), fixed_exponent(hr.w));
  const bool bad = __any_sync(0xffffffffu, !hzero && !fixed_ref_ok(he));
  const int4* vb = reinterpret_cast<const int4*>(V + ((long long)i0 * vstride + c) * ld);
  const long long vs = vstride * ld;
  const long long groups = (N + kGsGroup - 1) / kGsGroup;
  const int* el = g.vexp + ((long long)(i0 + (lane < KT ? lane : 0)) * vstride + c) * groups;  // lane s: vector s's
  double2* wc = w + (long long)c * ld;
  double nrm = 0.0;
  // a warp's 32 nodes, a quarter of a group; their references one round ahead
  const long long first = (long long)blockIdx.x * (RT / 32) + warp, round = (long long)nblk * (RT / 32);
  const long long units = (N + 31) / 32;
  int ahead = first < units ? el[first / kGsNodes] : kGsZero;
  for (long long u = first; u < units; u += round) {
    const long long p = u * 32 + lane;
    int4 v[KT];
#pragma unroll
    for (int s = 0; s < KT; ++s) v[s] = p < N ? vb[s * vs + p] : make_int4(0, 0, 0, 0);
    double2 wv = p < N ? wc[p] : mk<double>(0, 0);
    const int e = lane < KT ? ahead : kGsZero;
    if (u + round < units) ahead = el[(u + round) / kGsNodes];
    // the coefficients' words, related to the largest term of the group
    const bool term = e >= 0 && !hzero;
    const int T = __reduce_max_sync(0xffffffffu, term ? e + he : kNone);
    const bool ok = !bad && (T == kNone || fixed_ok(T)) &&
                    __all_sync(0xffffffffu, e != kGsRaw && (!term || T - e >= kFixedMin));
    if (ok) {
      const Fixed a = fixed_from<7>(hr.y, hr.x, term ? T - e : 2047), b = fixed_from<7>(hr.w, hr.z, term ? T - e : 2047);
      __syncwarp();
      if (lane < KT) hl[warp][lane] = term ? make_int4(a.hi, a.lo, b.hi, b.lo) : make_int4(0, 0, 0, 0);
      __syncwarp();
      FixedSum f{0, 0, 0, 0};
#pragma unroll
      for (int s = 0; s < KT; ++s) {
        const int4 k = hl[warp][s];
        fixed_cmac(f, Fixed{v[s].x, v[s].y}, Fixed{v[s].z, v[s].w}, Fixed{k.x, k.y}, Fixed{k.z, k.w});
      }
      const double sc = T == kNone ? 0.0 : __hiloint2double((int)fixed_scale_hi(T, 1), 0);
      wv.x = fma((double)-fixed_total(f.rh, f.rl), sc, wv.x);
      wv.y = fma((double)-fixed_total(f.ih, f.il), sc, wv.y);
    } else {
#pragma unroll
      for (int s = 0; s < KT; ++s)
        wv = cfms<double>(h[s], gs_value(v[s], __shfl_sync(0xffffffffu, e, s)), wv);
    }
    if (p < N) wc[p] = wv;
    if (last) nrm = fma(wv.x, wv.x, fma(wv.y, wv.y, nrm));
  }
  if (!last) return;
  double* part = g.part + (long long)blockIdx.y * nblk;
  const double2 none[1] = {mk<double>(0, 0)};
  block_partials<1>(none, 0, nrm, 1, part, nblk);
  if (!last_of_column(g.count, c, nblk)) return;
  fold_partials(part, nblk, 1, tot);
  gs_after_update(g, c, j, pass, tot[0]);
}

#define HZ_K_CASES(X) X(1) X(2) X(3) X(4) X(5) X(6) X(7) X(8) X(9) X(10) X(11) X(12) X(13) X(14) X(15) X(16)

// Blocks per column: two blocks fit an SM.  Four waves of them where a thread still has 64
// nodes, else one wave, or as many as leave less than a tenth of the last one's slots empty:
// a block's reduction costs as much as several nodes per thread.
int gs_nblk(long long N, int ncols) {
  const int slots = 2 * kSMs, cols = std::max(ncols, 1);
  const long long most = std::max<long long>(1, (N + RT - 1) / RT);
  auto blocks = [&](int waves) { return std::min<long long>(most, std::max(1, waves * slots / cols)); };
  if (N >= 64 * RT * blocks(4)) return (int)blocks(4);
  long long best = 1;
  double eff = 0.0;
  for (int waves = 1; waves <= 4; ++waves) {
    const long long ctas = blocks(waves) * cols;
    const double e = (double)ctas / (double)((ctas + slots - 1) / slots * slots);
    if (e > eff + 0.1) {
      best = blocks(waves);
      eff = e;
    }
  }
  return (int)best;
}

size_t gs_part_bytes(long long N, int R) { return (size_t)R * krylov_nblk(N, 1) * 33 * sizeof(double); }

void launch_gs_pass(Ctx& ctx, long long N, double2* V, long long vstride, long long ld, int j, int pass,
                    const int* cols, int ncols, const GsColumn& g) {
  if (ncols <= 0) return;
  double2* w = V + (long long)(j + 1) * vstride * ld;
  const int K = j + 1;
  const dim3 grid(gs_nblk(N, ncols), ncols);
  // a masked pass is charged by the host once it knows which columns took it
  const double el = pass ? 0.0 : (double)N * ncols;
  for (int i0 = 0; i0 < K; i0 += 16) {
    const int k = std::min(16, K - i0);
    const int wn = (pass == 0 && i0 + 16 >= K) ? 1 : 0;  // ||w||^2 before the update (slot K)
    const int fresh = wn;                                // v_j's first use here
    ctx.add_flops("krylov_dots", el * (8.0 * k + (wn ? 4.0 : 0.0)));
    switch (k) {
#define HZ_GS_CASE(q)                                                                                             \
  case q:                                                                                                         \
    HZ_LAUNCH(ctx, "krylov_dots", el * (k + 1) * 16.0, k_gs_dots<q>, grid, RT, 0, N, V, vstride, ld, i0, w, cols, \
              pass, wn, fresh, g);                                                                                \
    break;
      HZ_K_CASES(HZ_GS_CASE)
#undef HZ_GS_CASE
    }
  }
  for (int i0 = 0; i0 < K; i0 += 16) {
    const int k = std::min(16, K - i0);
    const int last = i0 + 16 >= K ? 1 : 0;
    ctx.add_flops("krylov_update", el * (8.0 * k + (last ? 4.0 : 0.0)));
    switch (k) {
#define HZ_GS_CASE(q)                                                                                               \
  case q:                                                                                                           \
    HZ_LAUNCH(ctx, "krylov_update", el * (k + 2) * 16.0, k_gs_update<q>, grid, RT, 0, N, V, vstride, ld, i0, w, cols, \
              j, pass, last, g);                                                                                    \
    break;
      HZ_K_CASES(HZ_GS_CASE)
#undef HZ_GS_CASE
    }
  }
}

// One warp per (column, slot): fixed-order sum over the nblk partials.
__global__ void k_reduce(const double2* __restrict__ part, const int* __restrict__ cols, int ncols, int K1, int nblk,
                         double2* __restrict__ out, int ostride, int accum) {
  const int gw = (blockIdx.x * blockDim.x + threadIdx.x) >> 5;
  const int lane = threadIdx.x & 31;
  if (gw >= ncols * K1) return;
  const int pos = gw / K1, slot = gw % K1;
  const double2* pp = part + ((long long)pos * K1 + slot) * nblk;
  double a = 0, b = 0;
  for (int i = lane; i < nblk; i += 32) {
    a += pp[i].x;
    b += pp[i].y;
  }
#pragma unroll
  for (int o = 16; o > 0; o >>= 1) {
    a += __shfl_xor_sync(0xffffffffu, a, o);
    b += __shfl_xor_sync(0xffffffffu, b, o);
  }
  if (lane == 0) {
    double2* dst = out + (long long)cols[pos] * ostride + slot;
    if (accum) {
      a += dst->x;
      b += dst->y;
    }
    *dst = mk<double>(a, b);
  }
}

void launch_reduce(Ctx& ctx, const double2* part, const int* cols, int ncols, int K1, int nblk, double2* out,
                   int ostride, int accum) {
  if (ncols <= 0 || K1 <= 0) return;
  long long warps = (long long)ncols * K1;
  int blocks = (int)((warps * 32 + 255) / 256);
  HZ_LAUNCH(ctx, "krylov_reduce", (double)ncols * K1 * (nblk + 1) * sizeof(double2), k_reduce, blocks, 256, 0, part, cols, ncols, K1, nblk, out, ostride, accum);
}

// ---- deferred normalisation of the FGMRES basis --------------------------------
// The stored basis vector v_i of column c stands for V_i = sig_i v_i with
// sig_i = sig[c*sstride + i] > 0, so no pass over the vector is spent on
// normalising it.  From the stored dots d_i = conj(v_i) . w' of the stored
// candidate w' (= 2^k H Z'_j, Z'_j the cycle applied to v_j, tau_j = 2^-k sig_j in [1, 2)): the
// update uses the coefficients sig_i^2 d_i, the Hessenberg entries are sig_i tau_j d_i,
// h_{j+1,j} = tau_j ||w''|| and sig_{j+1} = tau_j / h_{j+1,j} (hz_gs.cuh).  Without the power of
// two the scale is the product of all h: a cycle that amplifies took the FP32 levels' sums of squares
// out of range within a restart.  It changes no bit inside it.
__global__ void k_sig_init(const int* __restrict__ cols, int ncols, double* __restrict__ sig, int sstride) {
  const int i = blockIdx.x * blockDim.x + threadIdx.x;
  if (i < ncols) sig[(long long)cols[i] * sstride] = 1.0;
}

__global__ void k_sig_y(const int* __restrict__ cols, int ncols, const int* __restrict__ kcol,
                        const double* __restrict__ sig, int sstride, double2* __restrict__ y, int ystride) {
  const int pos = blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= ncols) return;
  const int c = cols[pos];
  for (int i = 0; i < kcol[c]; ++i) {
    const double s = sig[(long long)c * sstride + i];
    double2& v = y[(long long)c * ystride + i];
    v = mk<double>(s * v.x, s * v.y);
  }
}

void launch_sig_init(Ctx& ctx, const int* cols, int ncols, double* sig, int sstride) {
  if (ncols <= 0) return;
  HZ_LAUNCH(ctx, "basis_scale", 0.0, k_sig_init, (ncols + 127) / 128, 128, 0, cols, ncols, sig, sstride);
}
void launch_sig_y(Ctx& ctx, const int* cols, int ncols, const int* kcol, const double* sig, int sstride, double2* y,
                  int ystride) {
  if (ncols <= 0) return;
  HZ_LAUNCH(ctx, "basis_scale", 0.0, k_sig_y, (ncols + 127) / 128, 128, 0, cols, ncols, kcol, sig, sstride, y,
            ystride);
}

__global__ void __launch_bounds__(256) k_scale_cols(long long N, const double2* __restrict__ x, long long xld,
                                                    double2* __restrict__ y, long long yld,
                                                    const double* __restrict__ s, const int* __restrict__ cols) {
  const int c = cols[blockIdx.y];
  const double sc = s[c];
  const double2* xc = x + (long long)c * xld;
  double2* yc = y + (long long)c * yld;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (long long)gridDim.x * blockDim.x) {
    const double2 v = __ldcs(&xc[p]);  // streamed once
    __stcs(&yc[p], mk<double>(sc * v.x, sc * v.y));
  }
}

void launch_scale_cols(Ctx& ctx, long long N, const double2* x, long long xld, double2* y, long long yld,
                       const double* s, const int* cols, int ncols) {
  if (ncols <= 0) return;
  int nb = krylov_nblk(N, ncols);
  dim3 grid(nb, ncols);
  HZ_LAUNCH(ctx, "scale_cols", (double)N * ncols * 2 * sizeof(double2), k_scale_cols, grid, 256, 0, N, x, xld, y, yld, s, cols);
}

// kUx vectors' loads are issued together; four FP64 operations per value of Z are the bound then:
// 129^3 x 8, 10 FP32 vectors 1419 -> 1045 us, 65 x 65 x 33 x 8, 10 FP64 vectors 142 -> 90.
static constexpr int kUx = 5;
template <typename TZ>
__global__ void __launch_bounds__(256) k_update_x(long long N, const cplx<TZ>* __restrict__ Z, long long zstride,
                                                  long long ld, const int* __restrict__ kcol,
                                                  const double2* __restrict__ y, int ystride, double2* __restrict__ x,
                                                  long long xld, const int* __restrict__ cols) {
  const int c = cols[blockIdx.y];
  const int k = kcol[c];
  __shared__ double2 yv[64];  // restart length <= 64
  for (int s = threadIdx.x; s < k; s += blockDim.x) yv[s] = y[(long long)c * ystride + s];
  __syncthreads();
  double2* xc = x + (long long)c * xld;
  const cplx<TZ>* zc = Z + (long long)c * ld;
  const long long zs = zstride * ld;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (long long)gridDim.x * blockDim.x) {
    double2 acc = xc[p];
    for (int s0 = 0; s0 < k; s0 += kUx) {
      cplx<TZ> z[kUx];
#pragma unroll
      for (int s = 0; s < kUx; ++s) z[s] = s0 + s < k ? __ldcs(zc + (s0 + s) * zs + p) : mk<TZ>(0, 0);
#pragma unroll
      for (int s = 0; s < kUx; ++s)
        if (s0 + s < k) acc = cfma<double>(yv[s0 + s], ccast<double, TZ>(z[s]), acc);
    }
    xc[p] = acc;
  }
}

template <typename TZ>
void launch_update_x(Ctx& ctx, long long N, const cplx<TZ>* Z, long long zstride, long long ld, const int* kcol,
                     const double2* y, int ystride, double2* x, long long xld, const int* cols, int ncols,
                     long long zcols) {
  if (ncols <= 0) return;
  int nb = krylov_nblk(N, ncols);
  dim3 grid(nb, ncols);
  const double bytes = (double)N * (ncols * 2.0 * sizeof(double2) + zcols * sizeof(cplx<TZ>));
  ctx.add_flops("update_x", 8.0 * N * zcols);  // FP64: a complex multiply-add per stored Z vector and node
  HZ_LAUNCH(ctx, "update_x", bytes, k_update_x<TZ>, grid, 256, 0, N, Z, zstride, ld, kcol, y, ystride, x, xld, cols);
}

__global__ void k_norms(const double2* __restrict__ red, int stride, int slot, const int* __restrict__ cols, int ncols,
                        double* __restrict__ nrm, double* __restrict__ inv) {
  const int pos = blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= ncols) return;
  const int c = cols[pos];
  const double v = gs_sqrt(red[(long long)c * stride + slot].x);
  nrm[c] = v;
  if (inv) inv[c] = (v > 0) ? 1.0 / v : 0.0;
}

void launch_norms(Ctx& ctx, const double2* red, int stride, int slot, const int* cols, int ncols, double* nrm,
                  double* inv) {
  if (ncols <= 0) return;
  HZ_LAUNCH(ctx, "krylov_norms", 0.0, k_norms, (ncols + 127) / 128, 128, 0, red, stride, slot, cols, ncols, nrm, inv);
}

__global__ void k_cycle_init(int m, const int* __restrict__ cols, int ncols, const double* __restrict__ beta,
                             double2* __restrict__ g) {
  const int pos = blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= ncols) return;
  const int c = cols[pos];
  for (int i = 0; i <= m; ++i) g[(long long)c * (m + 1) + i] = mk<double>(i == 0 ? beta[c] : 0.0, 0.0);
}

void launch_cycle_init(Ctx& ctx, int m, const int* cols, int ncols, const double* beta, double2* g) {
  if (ncols <= 0) return;
  HZ_LAUNCH(ctx, "cycle_init", 0.0, k_cycle_init, (ncols + 127) / 128, 128, 0, m, cols, ncols, beta, g);
}

__global__ void k_lsq(int m, const int* __restrict__ cols, int ncols, const int* __restrict__ kcol,
                      const double2* __restrict__ Hh, const double2* __restrict__ g, double2* __restrict__ y) {
  const int pos = blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= ncols) return;
  const int c = cols[pos];
  const int k = kcol[c];
  const double2* H = Hh + (long long)c * (m + 1) * m;
  const double2* gc = g + (long long)c * (m + 1);
  double2* yc = y + (long long)c * m;
  for (int i = k - 1; i >= 0; --i) {
    double2 s = gc[i];
    for (int l = i + 1; l < k; ++l) s = cfms<double>(H[(long long)l * (m + 1) + i], yc[l], s);
    const double2 d = H[(long long)i * (m + 1) + i];
    const double den = d.x * d.x + d.y * d.y;
    yc[i] = (den > 0) ? mk<double>((s.x * d.x + s.y * d.y) / den, (s.y * d.x - s.x * d.y) / den) : mk<double>(0, 0);
  }
}

void launch_lsq(Ctx& ctx, int m, const int* cols, int ncols, const int* kcol, const double2* Hh, const double2* g,
                double2* y) {
  if (ncols <= 0) return;
  HZ_LAUNCH(ctx, "lsq", 0.0, k_lsq, (ncols + 63) / 64, 64, 0, m, cols, ncols, kcol, Hh, g, y);
}

// ---------------------------------------------------------------------------
// BiCGSTAB (right preconditioned) per-column vector updates and scalars
// ---------------------------------------------------------------------------
// Scalars per column c (complex, sc[c*8 + k]): 0 rho, 1 rho_prev, 2 alpha,
// 3 omega, 4 beta.  red[c*rstride + slot] hold the reduced dot products.
__global__ void k_bicg_scalars(int stage, const int* __restrict__ cols, int ncols, const double2* __restrict__ red,
                               int rstride, double2* __restrict__ sc) {
  const int pos = blockIdx.x * blockDim.x + threadIdx.x;
  if (pos >= ncols) return;
  const int c = cols[pos];
  double2* q = sc + (long long)c * 8;
  const double2* d = red + (long long)c * rstride;
  auto cdiv = [](double2 a, double2 b) {
    const double den = b.x * b.x + b.y * b.y;
    return mk<double>((a.x * b.x + a.y * b.y) / den, (a.y * b.x - a.x * b.y) / den);
  };
  if (stage == -1) {  // start: rho_prev = alpha = omega = 1
    q[1] = mk<double>(1, 0);
    q[2] = mk<double>(1, 0);
    q[3] = mk<double>(1, 0);
  } else if (stage == 0) {  // d[0] = <rh, r>: beta = (rho/rho_prev)(alpha/omega)
    const double2 rho = d[0];
    q[4] = cmul<double>(cdiv(rho, q[1]), cdiv(q[2], q[3]));
    q[0] = rho;
    q[1] = rho;
  } else if (stage == 1) {  // d[0] = <rh, v>: alpha = rho / <rh, v>
    q[2] = cdiv(q[0], d[0]);
  } else {  // d[0] = sum conj(s) t = conj(<t, s>), d[1] = ||t||^2: omega = <t, s> / ||t||^2
    q[3] = mk<double>(d[0].x / d[1].x, -d[0].y / d[1].x);
  }
}

void launch_bicg_scalars(Ctx& ctx, int stage, const int* cols, int ncols, const double2* red, int rstride,
                         double2* sc) {
  if (ncols <= 0) return;
  HZ_LAUNCH(ctx, "bicg_scalars", 0.0, k_bicg_scalars, (ncols + 127) / 128, 128, 0, stage, cols, ncols, red, rstride,
            sc);
}

// mode 0: p = r + beta (p - omega v);  mode 1: s = r - alpha v (into out)
__global__ void __launch_bounds__(256) k_bicg_vec(int mode, long long N, const double2* __restrict__ r,
                                                  double2* __restrict__ p, const double2* __restrict__ v,
                                                  double2* __restrict__ out, const double2* __restrict__ sc,
                                                  const int* __restrict__ cols) {
  const int c = cols[blockIdx.y];
  const double2* q = sc + (long long)c * 8;
  const long long off = (long long)c * N;
  const double2 beta = q[4], omega = q[3], alpha = q[2];
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const double2 ri = r[off + i], vi = v[off + i];
    if (mode == 0) {
      const double2 t = cfms<double>(omega, vi, p[off + i]);  // p - omega v
      p[off + i] = cfma<double>(beta, t, ri);
    } else {
      out[off + i] = cfms<double>(alpha, vi, ri);
    }
  }
}

void launch_bicg_vec(Ctx& ctx, int mode, long long N, const double2* r, double2* p, const double2* v, double2* out,
                     const double2* sc, const int* cols, int ncols) {
  if (ncols <= 0) return;
  const int nb = krylov_nblk(N, ncols);
  const double bytes = (double)N * ncols * (mode == 0 ? 4 : 3) * sizeof(double2);
  HZ_LAUNCH(ctx, mode == 0 ? "bicg_p" : "bicg_s", bytes, k_bicg_vec, dim3(nb, ncols), 256, 0, mode, N, r, p, v, out,
            sc, cols);
}

// x += alpha ph + omega sh ;  r = s - omega t   (ph, sh in the cycle precision)
template <typename TZ>
__global__ void __launch_bounds__(256) k_bicg_xr(long long N, double2* __restrict__ x, const cplx<TZ>* __restrict__ ph,
                                                 const cplx<TZ>* __restrict__ sh, const double2* __restrict__ s,
                                                 const double2* __restrict__ t, double2* __restrict__ r,
                                                 const double2* __restrict__ sc, const int* __restrict__ cols) {
  const int c = cols[blockIdx.y];
  const double2* q = sc + (long long)c * 8;
  const long long off = (long long)c * N;
  const double2 alpha = q[2], omega = q[3];
  for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < N; i += (long long)gridDim.x * blockDim.x) {
    const cplx<TZ> a = ph[off + i], b = sh[off + i];
    double2 xi = x[off + i];
    xi = cfma<double>(alpha, mk<double>((double)a.x, (double)a.y), xi);
    xi = cfma<double>(omega, mk<double>((double)b.x, (double)b.y), xi);
    x[off + i] = xi;
    r[off + i] = cfms<double>(omega, t[off + i], s[off + i]);
  }
}

template <typename TZ>
void launch_bicg_xr(Ctx& ctx, long long N, double2* x, const cplx<TZ>* ph, const cplx<TZ>* sh, const double2* s,
                    const double2* t, double2* r, const double2* sc, const int* cols, int ncols) {
  if (ncols <= 0) return;
  const int nb = krylov_nblk(N, ncols);
  const double bytes = (double)N * ncols * (5 * sizeof(double2) + 2 * sizeof(cplx<TZ>));
  HZ_LAUNCH(ctx, "bicg_xr", bytes, k_bicg_xr<TZ>, dim3(nb, ncols), 256, 0, N, x, ph, sh, s, t, r, sc, cols);
}
template void launch_bicg_xr<double>(Ctx&, long long, double2*, const double2*, const double2*, const double2*,
                                     const double2*, double2*, const double2*, const int*, int);
template void launch_bicg_xr<float>(Ctx&, long long, double2*, const float2*, const float2*, const double2*,
                                    const double2*, double2*, const double2*, const int*, int);

// ---------------------------------------------------------------------------
// Operator setup on the device (src/GetHelmholtz.jl:33-50, 81-83, 222-247)
// ---------------------------------------------------------------------------
// Per node: Sommerfeld term summed over the boundary faces the node lies on
// (top face skipped when NeumannOnTop; same face order as the host helper),
// mass = -w^2 m (1 - i gamma / Re w) - Somm, diag(H) = Laplacian diagonal + mass,
// diag(SH) = diag(H) + i s (Re w)^2 m, and 1/diag(SH).  BC is the Laplacian's
// boundary-row factor (orderNeumannBC); the Sommerfeld term always takes the
// factor 2, because src/GetHelmholtz.jl:45 calls getSommerfeldBC without the
// order and its default is 2 (:222).
__global__ void k_fine_setup(Grid g, int dim, double h0, double h1, double h2, double wr, double wi, double s,
                             double BC, int neumann_on_top, int sommerfeld, const double* __restrict__ m,
                             const double* __restrict__ gamma, double2* __restrict__ dH, double2* __restrict__ dSH,
                             double2* __restrict__ iSH, FixedRefs* __restrict__ refs) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  const unsigned lanes = __ballot_sync(0xffffffffu, p < g.N);  // the lanes that take part in the maxima below
  if (p >= g.N) return;
  const int i = (int)(p % g.nx);
  const long long t = p / g.nx;
  const int j = (int)(t % g.ny);
  const int k = (int)(t / g.ny);
  const double mp = m[p], gp = gamma[p];
  // -w^2 m (1 - i gamma / Re w), w complex
  const double w2r = wr * wr - wi * wi, w2i = 2.0 * wr * wi;
  const double a = 1.0, b = -gp / wr;  // (1 + i b)
  double mr = -(w2r * a - w2i * b) * mp;
  double mi = -(w2r * b + w2i * a) * mp;
  if (sommerfeld) {
    // Somm += -i w (SB/h_d) sqrt(m) on each face, SB = 2; host order: 2D top, bottom,
    // x-high, x-low; 3D top, bottom, y-low, y-high, x-low, x-high
    const double SB = 2.0;
    const double sq = sqrt(mp);
    double si = 0.0;
    if (dim == 2) {
      if (!neumann_on_top && j == 0) si += -wr * (SB / h1) * sq;
      if (j == g.ny - 1) si += -wr * (SB / h1) * sq;
      if (i == g.nx - 1) si += -wr * (SB / h0) * sq;
      if (i == 0) si += -wr * (SB / h0) * sq;
    } else {
      if (!neumann_on_top && k == 0) si += -wr * (SB / h2) * sq;
      if (k == g.nz - 1) si += -wr * (SB / h2) * sq;
      if (j == 0) si += -wr * (SB / h1) * sq;
      if (j == g.ny - 1) si += -wr * (SB / h1) * sq;
      if (i == 0) si += -wr * (SB / h0) * sq;
      if (i == g.nx - 1) si += -wr * (SB / h0) * sq;
    }
    mi -= si;
  }
  double lap = ((i == 0 || i == g.nx - 1) ? BC : 2.0) / (h0 * h0) + ((j == 0 || j == g.ny - 1) ? BC : 2.0) / (h1 * h1);
  if (dim == 3) lap += ((k == 0 || k == g.nz - 1) ? BC : 2.0) / (h2 * h2);
  const double hr = lap + mr, hi = mi;
  dH[p] = mk<double>(hr, hi);
  const double sr = hr, shi = hi + s * wr * wr * mp;
  dSH[p] = mk<double>(sr, shi);
  const double den = sr * sr + shi * shi;
  iSH[p] = mk<double>(sr / den, -shi / den);
  // the largest exponents of each operator's coefficients
  auto ex = [](double v) { return __double2hiint(v) >> 20 & 0x7ff; };
  int off = max(ex(1.0 / (h0 * h0)), ex(1.0 / (h1 * h1)));
  if (dim == 3) off = max(off, ex(1.0 / (h2 * h2)));
  const int eH = __reduce_max_sync(lanes, max(off, max(ex(hr), ex(hi))));
  const int eSH = __reduce_max_sync(lanes, max(off, max(ex(sr), ex(shi))));
  if ((threadIdx.x & 31) == 0) {
    if (eH > *(volatile int*)&refs[0].exponent) atomicMax(&refs[0].exponent, eH);
    if (eSH > *(volatile int*)&refs[1].exponent) atomicMax(&refs[1].exponent, eSH);
  }
}

void launch_fine_setup(Ctx& ctx, const Grid& g, int dim, const double* h, double wr, double wi, double shift, double BC,
                       int neumann_on_top, int sommerfeld, const double* m, const double* gamma, double2* dH,
                       double2* dSH, double2* iSH, FixedRefs* refs) {
  const long long nb = (g.N + 255) / 256;
  if (cudaMemsetAsync(refs, 0, 2 * sizeof(FixedRefs), ctx.stream) != cudaSuccess)
    throw std::runtime_error("fine setup: clear");
  HZ_LAUNCH(ctx, "fine_setup", (double)g.N * (2 * 8 + 3 * 16), k_fine_setup, (unsigned)nb, 256, 0, g, dim, h[0], h[1],
            dim == 3 ? h[2] : 1.0, wr, wi, shift, BC, neumann_on_top, sommerfeld, m, gamma, dH, dSH, iSH,
            refs);
}

// ---------------------------------------------------------------------------
// Setup kernels
// ---------------------------------------------------------------------------
// Galerkin probing: column k of the probe block is the indicator of the
// coarse nodes whose subscripts are congruent to pattern(k) modulo 3.  Within
// a 3^d neighbourhood exactly one node of each class exists, so R A P applied
// to probe k yields, at node I, the entry A_c(I, J) for that unique J.
__global__ void k_probe_init(Grid g, int dim, double2* out, long long ld) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= g.N) return;
  const int i = (int)(p % g.nx);
  const long long t = p / g.nx;
  const int j = (int)(t % g.ny);
  const int k = (int)(t / g.ny);
  const int cls = (i % 3) + 3 * (j % 3) + (dim == 3 ? 9 * (k % 3) : 0);
  const int ns = dim == 3 ? 27 : 9;
  for (int s = 0; s < ns; ++s) out[(long long)s * ld + p] = mk<double>(s == cls ? 1.0 : 0.0, 0.0);
}

void launch_probe_init(Ctx& ctx, const Grid& gc, int dim, double2* out, long long ld) {
  long long nb = (gc.N + 255) / 256;
  HZ_LAUNCH(ctx, "probe_init", (double)gc.N * (dim == 3 ? 27 : 9) * sizeof(double2), k_probe_init, (unsigned)nb, 256, 0, gc, dim, out, ld);
}

__device__ __forceinline__ int off3(int cls_d, int I) {
  // offset o in {-1,0,1} with (I + o) = cls_d (mod 3)
  int o = ((cls_d - I) % 3 + 3) % 3;
  return o == 2 ? -1 : o;
}

__global__ void k_probe_scatter(Grid g, int dim, const double2* __restrict__ y, long long ld, double2* coef,
                                long long cld) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= g.N) return;
  const int i = (int)(p % g.nx);
  const long long t = p / g.nx;
  const int j = (int)(t % g.ny);
  const int k = (int)(t / g.ny);
  const int ns = dim == 3 ? 27 : 9;
  for (int s = 0; s < ns; ++s) {
    const int ox = off3(s % 3, i), oy = off3((s / 3) % 3, j), oz = dim == 3 ? off3(s / 9, k) : 0;
    const int slot = (ox + 1) + 3 * (oy + 1) + (dim == 3 ? 9 * (oz + 1) : 0);
    coef[(long long)slot * cld + p] = y[(long long)s * ld + p];
  }
}

void launch_probe_scatter(Ctx& ctx, const Grid& gc, int dim, const double2* y, long long ld, double2* coef,
                          long long cld) {
  long long nb = (gc.N + 255) / 256;
  HZ_LAUNCH(ctx, "probe_scatter", 2.0 * gc.N * (dim == 3 ? 27 : 9) * sizeof(double2), k_probe_scatter, (unsigned)nb, 256, 0, gc, dim, y, ld, coef, cld);
}

// coefT[o][I] = conj(coef[-o][I + o]) (zero where I + o is outside the grid).
__global__ void k_coef_transpose(Grid g, int dim, const double2* __restrict__ coef, double2* __restrict__ coefT,
                                 long long cld) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= g.N) return;
  const int i = (int)(p % g.nx);
  const long long t = p / g.nx;
  const int j = (int)(t % g.ny);
  const int k = (int)(t / g.ny);
  const int ns = dim == 3 ? 27 : 9;
  for (int s = 0; s < ns; ++s) {
    const int ox = s % 3 - 1, oy = (s / 3) % 3 - 1, oz = dim == 3 ? s / 9 - 1 : 0;
    const int ii = i + ox, jj = j + oy, kk = k + oz;
    double2 v = mk<double>(0, 0);
    if (ii >= 0 && ii < g.nx && jj >= 0 && jj < g.ny && kk >= 0 && kk < g.nz) {
      const long long q = ii + (long long)g.nx * (jj + (long long)g.ny * kk);
      const int ms = (1 - ox) + 3 * (1 - oy) + (dim == 3 ? 9 * (1 - oz) : 0);
      v = coef[(long long)ms * cld + q];
      v.y = -v.y;
    }
    coefT[(long long)s * cld + p] = v;
  }
}

void launch_coef_transpose(Ctx& ctx, const Grid& g, int dim, const double2* coef, double2* coefT, long long cld) {
  long long nb = (g.N + 255) / 256;
  HZ_LAUNCH(ctx, "coef_transpose", 2.0 * g.N * (dim == 3 ? 27 : 9) * sizeof(double2), k_coef_transpose, (unsigned)nb, 256, 0, g, dim, coef, coefT, cld);
}

template <typename T>
__global__ void k_center_inverse(long long N, int center, const double2* __restrict__ coef, long long cld,
                                 cplx<T>* __restrict__ dinv) {
  const long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (p >= N) return;
  const double2 d = coef[(long long)center * cld + p];
  const double den = d.x * d.x + d.y * d.y;
  dinv[p] = mk<T>((T)(d.x / den), (T)(-d.y / den));
}

template <typename T>
void launch_center_inverse(Ctx& ctx, const Grid& g, int dim, const double2* coef, long long cld, cplx<T>* dinv) {
  long long nb = (g.N + 255) / 256;
  HZ_LAUNCH(ctx, "center_inverse", (double)g.N * (sizeof(double2) + sizeof(cplx<T>)), k_center_inverse<T>, (unsigned)nb, 256, 0, g.N, dim == 3 ? 13 : 4, coef, cld,
            dinv);
}

template <typename To, typename From>
__global__ void k_cast(const cplx<From>* __restrict__ in, cplx<To>* __restrict__ out, long long n) {
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < n; p += (long long)gridDim.x * blockDim.x)
    out[p] = mk<To>((To)in[p].x, (To)in[p].y);
}

template <typename To, typename From>
void launch_cast(Ctx& ctx, const cplx<From>* in, cplx<To>* out, long long n) {
  if (n <= 0) return;
  long long nb = std::min<long long>((n + 255) / 256, 16LL * kSMs);
  HZ_LAUNCH(ctx, "cast", (double)n * (sizeof(cplx<To>) + sizeof(cplx<From>)), (k_cast<To, From>), (unsigned)nb, 256, 0, in, out, n);
}

template <typename To, typename From>
__global__ void k_cast_cols(long long N, const cplx<From>* __restrict__ in, long long ldi, cplx<To>* __restrict__ out,
                            long long ldo, const int* __restrict__ cols) {
  const int c = cols[blockIdx.y];
  const cplx<From>* ic = in + (long long)c * ldi;
  cplx<To>* oc = out + (long long)c * ldo;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (long long)gridDim.x * blockDim.x)
    oc[p] = mk<To>((To)ic[p].x, (To)ic[p].y);
}

template <typename To, typename From>
void launch_cast_cols(Ctx& ctx, long long N, const cplx<From>* in, long long ldi, cplx<To>* out, long long ldo,
                      const int* cols, int ncols) {
  if (ncols <= 0) return;
  int nb = krylov_nblk(N, ncols);
  dim3 grid(nb, ncols);
  HZ_LAUNCH(ctx, "cast_cols", (double)N * ncols * (sizeof(cplx<To>) + sizeof(cplx<From>)), (k_cast_cols<To, From>), grid, 256, 0, N, in, ldi, out, ldo, cols);
}

template <typename T>
__global__ void k_zero_cols(long long N, cplx<T>* __restrict__ x, long long ld, const int* __restrict__ cols) {
  const int c = cols[blockIdx.y];
  cplx<T>* xc = x + (long long)c * ld;
  for (long long p = (long long)blockIdx.x * blockDim.x + threadIdx.x; p < N; p += (long long)gridDim.x * blockDim.x)
    xc[p] = mk<T>(0, 0);
}

template <typename T>
void launch_zero_cols(Ctx& ctx, long long N, cplx<T>* x, long long ld, const int* cols, int ncols) {
  if (ncols <= 0) return;
  int nb = krylov_nblk(N, ncols);
  dim3 grid(nb, ncols);
  HZ_LAUNCH(ctx, "zero_cols", (double)N * ncols * sizeof(cplx<T>), k_zero_cols<T>, grid, 256, 0, N, x, ld, cols);
}

// explicit instantiations
template void launch_update_x<double>(Ctx&, long long, const double2*, long long, long long, const int*,
                                      const double2*, int, double2*, long long, const int*, int, long long);
template void launch_update_x<float>(Ctx&, long long, const float2*, long long, long long, const int*, const double2*,
                                     int, double2*, long long, const int*, int, long long);
template void launch_center_inverse<double>(Ctx&, const Grid&, int, const double2*, long long, double2*);
template void launch_center_inverse<float>(Ctx&, const Grid&, int, const double2*, long long, float2*);
template void launch_cast<float, double>(Ctx&, const double2*, float2*, long long);
template void launch_cast<double, float>(Ctx&, const float2*, double2*, long long);
template void launch_cast_cols<float, double>(Ctx&, long long, const double2*, long long, float2*, long long,
                                              const int*, int);
template void launch_cast_cols<double, float>(Ctx&, long long, const float2*, long long, double2*, long long,
                                              const int*, int);
template void launch_cast_cols<double, double>(Ctx&, long long, const double2*, long long, double2*, long long,
                                               const int*, int);
template void launch_cast_cols<float, float>(Ctx&, long long, const float2*, long long, float2*, long long, const int*,
                                             int);
template void launch_cast_cols<float, df64_tag>(Ctx&, long long, const float4*, long long, float2*, long long,
                                                const int*, int);
template void launch_zero_cols<double>(Ctx&, long long, double2*, long long, const int*, int);
template void launch_zero_cols<float>(Ctx&, long long, float2*, long long, const int*, int);

}  // namespace hz
