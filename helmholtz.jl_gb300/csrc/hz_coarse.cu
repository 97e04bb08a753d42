// Coarsest multigrid level: x = A^{-1} b as one tensor-core product.
//
// Setup (FP64, once per hierarchy): the level's operator is block tridiagonal
// in slabs of nodes along its longest axis.  A block elimination with pivoted
// slab inverses gives the dense A^{-1} by the block recurrences
//   S_0 = A_00,  G_k = S_k^{-1},  E_k = -G_k A_{k,k+1},  F_k = -A_{k+1,k} G_k,
//   S_{k+1} = A_{k+1,k+1} + F_k A_{k,k+1},
//   X_{k,j} = E_k X_{k+1,j},  X_{j,k} = X_{j,k+1} F_k  (j > k),
//   X_{k,k} = G_k + E_k X_{k+1,k},
// N^2 M complex multiply-adds for slabs of M nodes.
//
// Solve: every row of A^{-1} and every column of b is split, relative to the
// power of two above its largest component, into S signed base-256 digits.  A
// digit is exact in BF16, a product of two digits is an integer below 2^14, and
// the FP32 accumulators of the tensor core stay exact integers for kFlush steps
// (below 2^24); they are then folded into 64-bit integers.  Digit pairs (i, j)
// with i + j < S are kept.  S = 8 (64 bits below the row's and the column's largest), or S = 6
// (48 bits) in the emulated mode, whose double-float pairs hold no more.
//
// Why: GB300 has two FP64 FMA lanes per clock and SM, so a band substitution in
// FP64 is bound by that pipe and by its chain of grid barriers, two per kl rows.
// Band substitution -> digits + product, event-timed per solve:
//   FP64 columns:  289 nodes x 1:  131 -> 7 + 10 us;   2601 x 8: 573 -> 9 + 76 us
//   FP32 columns: 2145 nodes x 16: 839 -> 10 + 63 us;  4913 x 8: 1425 -> 14 + 192 us
// (with 6 digits 43 and 136 us, but then the residual is 1e-12 of the right-hand side, the LU's 1e-16)
// and against a dense double-float product on the FP32 pipe (861 nodes x 33):
// 45 -> 8 + 23 us.  The setup (slab elimination on the GPU) takes 10 to 140 ms
// over those sizes, as the banded LU on the host did.
#include <algorithm>
#include <stdexcept>
#include <string>
#include <type_traits>

#include <cooperative_groups.h>

#include "hz_coarse.h"
#include "hz_launch.cuh"

namespace cg = cooperative_groups;

namespace hz {

// ---------------------------------------------------------------------------
// Setup
// ---------------------------------------------------------------------------
// Slab order: index q = s * M + r, s along the longest axis; -> node number.
struct SlabOrder {
  int ns, n0, n1;              // nodes along the slab axis and the two others
  long long ss, s0, s1;        // their strides in the node numbering
  __device__ __forceinline__ void coords(long long q, int& s, int& a, int& b) const {
    const long long M = (long long)n0 * n1;
    s = (int)(q / M);
    const int r = (int)(q % M);
    a = r % n0;
    b = r / n0;
  }
  __device__ __forceinline__ long long node(int s, int a, int b) const { return s * ss + a * s0 + b * s1; }
};

// Dense block of the level operator, rows r0.. and columns c0.. in slab order;
// coef[k * N + p] = A(p, p + offset_k).  t_s, t_0, t_1: the axes' offset strides
// in k (1, 3, 9), so that k = center + ds t_s + d0 t_0 + d1 t_1.
__global__ void k_coarse_block(SlabOrder o, int center, int ts, int t0, int t1, const double2* __restrict__ coef,
                               long long N, long long r0, int nr, long long c0, int nc, double2* __restrict__ out,
                               int ld) {
  const long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x;
  if (e >= (long long)nr * nc) return;
  const int i = (int)(e / nc), j = (int)(e % nc);
  int si, ai, bi, sj, aj, bj;
  o.coords(r0 + i, si, ai, bi);
  o.coords(c0 + j, sj, aj, bj);
  const int ds = sj - si, d0 = aj - ai, d1 = bj - bi;
  double2 v = mk<double>(0, 0);
  if (abs(ds) <= 1 && abs(d0) <= 1 && abs(d1) <= 1)
    v = coef[(long long)(center + ds * ts + d0 * t0 + d1 * t1) * N + o.node(si, ai, bi)];
  out[(long long)i * ld + j] = v;
}

// C = sgn A B + D (row-major, D may be null), FP64 complex.  32 x 32 tiles, four
// outputs per thread: bound by the FP64 pipe.
__global__ void __launch_bounds__(256) k_coarse_gemm(int m, int n, int k, const double2* __restrict__ A, long long lda,
                                                     const double2* __restrict__ B, long long ldb,
                                                     const double2* __restrict__ D, long long ldd, double sgn,
                                                     double2* __restrict__ C, long long ldc) {
  __shared__ double2 As[32][17], Bs[16][33];
  const int tx = threadIdx.x & 15, ty = threadIdx.x >> 4;
  const int i0 = blockIdx.y * 32, j0 = blockIdx.x * 32;
  double2 acc[2][2];
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) acc[a][b] = mk<double>(0, 0);
  for (int k0 = 0; k0 < k; k0 += 16) {
    for (int e = threadIdx.x; e < 512; e += 256) {
      const int ar = e >> 4, ac = e & 15, br = e >> 5, bc = e & 31;
      As[ar][ac] = (i0 + ar < m && k0 + ac < k) ? A[(i0 + ar) * lda + k0 + ac] : mk<double>(0, 0);
      Bs[br][bc] = (k0 + br < k && j0 + bc < n) ? B[(k0 + br) * ldb + j0 + bc] : mk<double>(0, 0);
    }
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 16; ++q) {
      const double2 a0 = As[ty][q], a1 = As[ty + 16][q], b0 = Bs[q][tx], b1 = Bs[q][tx + 16];
      acc[0][0] = cfma<double>(a0, b0, acc[0][0]);
      acc[0][1] = cfma<double>(a0, b1, acc[0][1]);
      acc[1][0] = cfma<double>(a1, b0, acc[1][0]);
      acc[1][1] = cfma<double>(a1, b1, acc[1][1]);
    }
    __syncthreads();
  }
#pragma unroll
  for (int a = 0; a < 2; ++a)
#pragma unroll
    for (int b = 0; b < 2; ++b) {
      const int i = i0 + ty + 16 * a, j = j0 + tx + 16 * b;
      if (i < m && j < n) {
        double2 v = mk<double>(sgn * acc[a][b].x, sgn * acc[a][b].y);
        if (D) v = cadd<double>(v, D[i * ldd + j]);
        C[i * ldc + j] = v;
      }
    }
}

// In-place Gauss-Jordan inverse of one m x m slab operator with partial pivoting
// (rows stay where they are; step p eliminates with the unused row of largest
// pivot).  One cooperative launch: every CTA finds the same pivot from the shared
// column and updates its share of the matrix into the other buffer; one grid
// barrier per step.  The result (rows and columns put back in order) goes to
// out; *bad counts steps without a usable pivot.
static constexpr int kSlabMax = 1024;  // rows of a slab block (pivot flags in shared memory)

__global__ void __launch_bounds__(256) k_coarse_inverse(int m, double2* __restrict__ b0, double2* __restrict__ b1,
                                                        double2* __restrict__ out, int* __restrict__ bad) {
  cg::grid_group grid = cg::this_grid();
  __shared__ unsigned char used[kSlabMax];
  __shared__ short piv[kSlabMax];
  __shared__ double wmag[8];
  __shared__ int wrow[8];
  __shared__ int prow;
  for (int i = threadIdx.x; i < m; i += 256) used[i] = 0;
  __syncthreads();
  const long long gt = (long long)blockIdx.x * 256 + threadIdx.x, gn = (long long)gridDim.x * 256;
  for (int p = 0; p < m; ++p) {
    const double2* src = (p & 1) ? b1 : b0;
    double2* dst = (p & 1) ? b0 : b1;
    double best = -1.0;
    int row = m;
    for (int i = threadIdx.x; i < m; i += 256) {
      if (used[i]) continue;
      const double2 v = src[(long long)i * m + p];
      const double mag = fabs(v.x) + fabs(v.y);
      if (mag > best) {
        best = mag;
        row = i;
      }
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
      const double bm = __shfl_xor_sync(0xffffffffu, best, o);
      const int br = __shfl_xor_sync(0xffffffffu, row, o);
      if (bm > best || (bm == best && br < row)) {
        best = bm;
        row = br;
      }
    }
    if ((threadIdx.x & 31) == 0) {
      wmag[threadIdx.x >> 5] = best;
      wrow[threadIdx.x >> 5] = row;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
      for (int w = 1; w < 8; ++w)
        if (wmag[w] > best || (wmag[w] == best && wrow[w] < row)) {
          best = wmag[w];
          row = wrow[w];
        }
      if (!(best > 0.0) || !(best < 1e300)) {  // no pivot, or a NaN / Inf column: any unused row, reported
        if (blockIdx.x == 0) atomicAdd(bad, 1);
        for (row = 0; row < m - 1 && used[row]; ++row) {
        }
      }
      used[row] = 1;
      piv[p] = (short)row;
      prow = row;
    }
    __syncthreads();
    const int r = prow;
    const double2 d = src[(long long)r * m + p];
    const double den = d.x * d.x + d.y * d.y;
    const double2 inv = mk<double>(d.x / den, -d.y / den);
    for (long long e = gt; e < (long long)m * m; e += gn) {
      const int i = (int)(e / m), j = (int)(e % m);
      double2 v;
      if (i == r) {
        v = (j == p) ? inv : cmul<double>(src[(long long)r * m + j], inv);
      } else {
        const double2 f = src[(long long)i * m + p];
        if (j == p) {
          const double2 t = cmul<double>(f, inv);
          v = mk<double>(-t.x, -t.y);
        } else {
          v = cfms<double>(f, cmul<double>(src[(long long)r * m + j], inv), src[e]);
        }
      }
      dst[e] = v;
    }
    grid.sync();
  }
  // inverse(p, piv[q]) = R(piv[p], q)
  const double2* R = (m & 1) ? b1 : b0;
  for (long long e = gt; e < (long long)m * m; e += gn) {
    const int p = (int)(e / m), q = (int)(e % m);
    out[(long long)p * m + piv[q]] = R[(long long)piv[p] * m + q];
  }
}

// ---------------------------------------------------------------------------
// Digits
// ---------------------------------------------------------------------------
// v 2^-e with |v| < 2^e / 4 as S balanced base-256 digits (most significant
// first), v 2^-e = sum_s d_s 2^{-8 (s + 1)} up to half a last digit.  From the bits
// of v: the FP64 pipe takes no part.
template <int S>
__device__ __forceinline__ void digits(uint64_t v, int e, int (&d)[S]) {
  int E = (int)(v >> 52) & 0x7ff;
  long long X = (long long)(v & 0xfffffffffffffull);
  if (E)
    X |= 1ll << 52;
  else
    E = 1;
  const int sh = E - 1075 + 8 * S - e;  // at most 9
  if (sh >= 0)
    X <<= sh;
  else
    X = sh > -55 ? (X + (1ll << (-sh - 1))) >> -sh : 0;
  if (v >> 63) X = -X;
#pragma unroll
  for (int s = S - 1; s >= 0; --s) {
    const int q = (int)(signed char)(X & 255);
    d[s] = q;
    X = (X - q) >> 8;
  }
}
__device__ __forceinline__ uint64_t bits64(double v) { return (uint64_t)__double_as_longlong(v); }
__device__ __forceinline__ uint64_t bits64(float v) { return widen_f32_bits(__float_as_uint(v)); }
// biased FP64 exponent of a value (0x7ff: NaN or Inf)
__device__ __forceinline__ int exponent64(uint64_t v) { return (int)(v >> 52) & 0x7ff; }
// two digits as packed BF16 (low half: first argument); |d| <= 128 is exact
__device__ __forceinline__ uint32_t pack_digits(int a, int b) {
  return (__float_as_uint((float)a) >> 16) | (__float_as_uint((float)b) & 0xffff0000u);
}
// e with |v| < 2^e / 4 for every v of biased exponent E or less
__device__ __forceinline__ int digit_exponent(int E) { return max(E, 1) - 1020; }

// Rows of X (slab order, row-major) into the operand image: for the row tile t
// of 16 nodes and the step ks of 8 columns, slice s, lane l holds the four
// registers of the m16n8k16 A fragment: register r = digits (re, im) of entry
// (16 t + l / 4 + 8 (r & 1), 8 ks + l % 4 + 4 (r >> 1)).  One warp per row; scale[row] = e.
template <int S>
__global__ void __launch_bounds__(256) k_coarse_image(SlabOrder o, long long N, int KS, const double2* __restrict__ X,
                                                      uint32_t* __restrict__ img, int* __restrict__ scale) {
  const int lane = threadIdx.x & 31;
  const long long q = (long long)blockIdx.x * 8 + (threadIdx.x >> 5);  // row in slab order
  if (q >= N) return;
  int s, a, b;
  o.coords(q, s, a, b);
  const long long row = o.node(s, a, b);
  int mx = 0;
  for (long long k = lane; k < N; k += 32) {
    const double2 v = X[q * N + k];
    mx = max(mx, max(exponent64(bits64(v.x)), exponent64(bits64(v.y))));
  }
  const int e = digit_exponent(__reduce_max_sync(0xffffffffu, mx));
  if (lane == 0) scale[row] = e;
  const long long t = row >> 4;
  const int ri = (int)(row & 15);
  for (long long kq = lane; kq < N; kq += 32) {
    const double2 v = X[q * N + kq];
    o.coords(kq, s, a, b);
    const long long k = o.node(s, a, b);
    int dr[S], di[S];
    digits<S>(bits64(v.x), e, dr);
    digits<S>(bits64(v.y), e, di);
    const int kk = (int)(k & 7);
    const int l = (ri & 7) * 4 + (kk & 3), r = (ri >> 3) + 2 * (kk >> 2);
    const long long base = (t * KS + (k >> 3)) * S;
#pragma unroll
    for (int c = 0; c < S; ++c) img[((base + c) * 32 + l) * 4 + r] = pack_digits(dr[c], di[c]);
  }
}

// Columns of b into digit words [column / 4][step][column % 4][k % 8][8 slices];
// scale = e.  A column with a NaN or Inf is marked with kNotFinite: its solution is
// NaN.  kSliceParts CTAs per active column, each of which finds the column's
// exponent (a few loads per thread) and converts its share: integer work on one SM
// per column took 18 us for 16 columns of 2145, ahead of a product of 43 us.
static constexpr int kNotFinite = 1 << 30;
static constexpr int kSliceParts = 8;

template <typename T, int S>
__global__ void __launch_bounds__(256) k_coarse_slice(long long N, int KS, const cplx<T>* __restrict__ b, long long ldb,
                                                      const int* __restrict__ cols, uint4* __restrict__ words,
                                                      int* __restrict__ scale) {
  __shared__ int red[8];
  const int ci = blockIdx.x;
  const cplx<T>* bc = b + (long long)cols[ci] * ldb;
  int mx = 0;
#pragma unroll 4
  for (long long k = threadIdx.x; k < N; k += 256) {
    const cplx<T> v = bc[k];
    mx = max(mx, max(exponent64(bits64(v.x)), exponent64(bits64(v.y))));
  }
  mx = __reduce_max_sync(0xffffffffu, mx);
  if ((threadIdx.x & 31) == 0) red[threadIdx.x >> 5] = mx;
  __syncthreads();
#pragma unroll
  for (int w = 0; w < 8; ++w) mx = max(mx, red[w]);
  const bool bad = mx == 0x7ff;
  const int e = digit_exponent(mx);
  if (threadIdx.x == 0 && blockIdx.y == 0) scale[ci] = bad ? kNotFinite : e;
  uint4* wc = words + ((long long)(ci >> 2) * KS * 32 + (ci & 3) * 8) * 2;
  for (long long k = blockIdx.y * 256 + threadIdx.x; k < 8LL * KS; k += 256 * kSliceParts) {
    uint32_t w[8];
#pragma unroll
    for (int s = 0; s < 8; ++s) w[s] = 0;
    if (k < N && !bad) {
      const cplx<T> v = bc[k];
      int dr[S], di[S];
      digits<S>(bits64(v.x), e, dr);
      digits<S>(bits64(v.y), e, di);
#pragma unroll
      for (int s = 0; s < S; ++s) w[s] = pack_digits(dr[s], di[s]);
    }
    uint4* p = wc + ((k >> 3) * 32 + (k & 7)) * 2;
    p[0] = make_uint4(w[0], w[1], w[2], w[3]);
    p[1] = make_uint4(w[4], w[5], w[6], w[7]);
  }
}

// ---------------------------------------------------------------------------
// Product
// ---------------------------------------------------------------------------
static constexpr int kFlush = 8;  // steps of exact FP32 accumulation: 8 pairs x 16 products x 8 steps x 2^14 = 2^24

__device__ __forceinline__ void mma_digits(float (&c)[4], const uint4& a, uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a.x), "r"(a.y), "r"(a.z), "r"(a.w), "r"(b0), "r"(b1));
}

// 16 bytes from global to shared memory, asynchronously
__device__ __forceinline__ void copy16(void* smem, const void* gmem) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)), "l"(gmem));
}

// A CTA owns 16 rows and 4 NT columns; its 8 warps share the steps of the sum and
// meet once, in shared memory, in a fixed order.  Each warp keeps the operands of
// its next step in flight through a private two-slot ring of shared memory
// (cp.async; no CTA barrier in the loop): the operand image is in fragment order,
// so a lane copies and reads back its own 16 bytes per slice.  The slots of the
// two CTAs of an SM hold up to 96 KB in flight.  Bound by reading the image (4 S
// bytes per entry) up to about 8 columns, by the tensor pipe above.
template <int S, int NT> struct ProductRing {
  uint4 a[S][32];
  uint4 b[NT][64];
};
template <int S, int NT> constexpr size_t product_smem() { return 16 * sizeof(ProductRing<S, NT>); }

template <typename T, int S, int NT>
__global__ void __launch_bounds__(256, 2) k_coarse_product(long long N, int KS, const uint4* __restrict__ img,
                                                           const int* __restrict__ rscale,
                                                           const uint4* __restrict__ words,
                                                           const int* __restrict__ cscale,
                                                           const int* __restrict__ cols, int ncols,
                                                           cplx<T>* __restrict__ x, long long ldx) {
  extern __shared__ __align__(16) unsigned char smem[];
  static_assert(sizeof(double2) * 8 * 16 * 4 * NT <= product_smem<S, NT>(), "the reduction reuses the rings");
  double2 (*red)[16][4 * NT] = reinterpret_cast<double2 (*)[16][4 * NT]>(smem);
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  ProductRing<S, NT>* ring = reinterpret_cast<ProductRing<S, NT>*>(smem) + 2 * warp;
  const long long rt = blockIdx.y;
  const int g0 = blockIdx.x * NT;  // first group of four columns
  const int groups = (ncols + 3) >> 2;
  float acc[NT][S][4];
  long long hi[NT][4], lo[NT][4];
#pragma unroll
  for (int t = 0; t < NT; ++t)
#pragma unroll
    for (int c = 0; c < 4; ++c) {
      hi[t][c] = lo[t][c] = 0;
#pragma unroll
      for (int g = 0; g < S; ++g) acc[t][g][c] = 0.f;
    }
  // column n = lane / 4 of a tile is Re (even) or Im (odd) of column n / 2:
  // (b_re, -b_im) against (a_re, a_im) sums Re, (b_im, b_re) sums Im
  const bool im = (lane >> 2) & 1;
  const uint4* ap = img + rt * KS * S * 32 + lane;
  auto fetch = [&](int ks, int slot) {
    if (ks < KS) {
#pragma unroll
      for (int s = 0; s < S; ++s) copy16(&ring[slot].a[s][lane], ap + ((long long)ks * S + s) * 32);
#pragma unroll
      for (int t = 0; t < NT; ++t) {
        const uint4* p = words + ((long long)min(g0 + t, groups - 1) * KS + ks) * 64 + lane;
        copy16(&ring[slot].b[t][lane], p);
        copy16(&ring[slot].b[t][lane + 32], p + 32);
      }
    }
    asm volatile("cp.async.commit_group;");
  };
  int steps = 0;
  auto flush = [&] {
#pragma unroll
    for (int t = 0; t < NT; ++t)
#pragma unroll
      for (int c = 0; c < 4; ++c) {
#pragma unroll
        for (int g = 0; g < S; ++g) {
          const int v = __float2int_rn(acc[t][g][c]);
          if (g < 4)
            hi[t][c] += (long long)v * (1 << (24 - 8 * g));
          else
            lo[t][c] += (long long)v * (1 << (56 - 8 * g));
          acc[t][g][c] = 0.f;
        }
      }
  };
  fetch(warp, 0);
  int slot = 0;
  for (int ks = warp; ks < KS; ks += 8, slot ^= 1) {
    fetch(ks + 8, slot ^ 1);
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncwarp();
#pragma unroll
    for (int t = 0; t < NT; ++t) {
      const uint4* p = &ring[slot].b[t][((lane >> 3) * 8 + (lane & 3)) * 2];
      const uint4 w0 = p[0], w1 = p[1], w2 = p[8], w3 = p[9];
      uint32_t v0[8] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z, w1.w};
      uint32_t v1[8] = {w2.x, w2.y, w2.z, w2.w, w3.x, w3.y, w3.z, w3.w};
#pragma unroll
      for (int j = 0; j < S; ++j) {
        v0[j] = im ? __byte_perm(v0[j], 0, 0x1032) : (v0[j] ^ 0x80000000u);
        v1[j] = im ? __byte_perm(v1[j], 0, 0x1032) : (v1[j] ^ 0x80000000u);
      }
#pragma unroll
      for (int i = 0; i < S; ++i) {
        const uint4 a = ring[slot].a[i][lane];
#pragma unroll
        for (int j = 0; i + j < S; ++j) mma_digits(acc[t][i + j], a, v0[j], v1[j]);
      }
    }
    __syncwarp();  // the slot is refilled in the next step
    if (++steps == kFlush) {
      flush();
      steps = 0;
    }
  }
  flush();
  __syncthreads();  // every warp has left its ring
  const int r = lane >> 2, c = lane & 3;
#pragma unroll
  for (int t = 0; t < NT; ++t) {
    // sum_g acc_g 2^{-8 g - 16}: hi carries 2^-40, lo 2^-72
    double v[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) v[q] = fma((double)lo[t][q], 0x1p-72, (double)hi[t][q] * 0x1p-40);
    red[warp][r][4 * t + c] = mk<double>(v[0], v[1]);
    red[warp][r + 8][4 * t + c] = mk<double>(v[2], v[3]);
  }
  __syncthreads();
  for (int e = threadIdx.x; e < 64 * NT; e += 256) {
    const int rr = e / (4 * NT), cc = e % (4 * NT);
    const long long row = rt * 16 + rr;
    const int ci = 4 * g0 + cc;
    if (row >= N || ci >= ncols) continue;
    double2 v = red[0][rr][cc];
#pragma unroll
    for (int w = 1; w < 8; ++w) v = cadd<double>(v, red[w][rr][cc]);
    const int sc = cscale[ci], sh = rscale[row] + sc;
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    x[(long long)cols[ci] * ldx + row] =
        sc == kNotFinite ? mk<T>((T)nan, (T)nan) : mk<T>((T)ldexp(v.x, sh), (T)ldexp(v.y, sh));
  }
}

// ---------------------------------------------------------------------------
// Host side
// ---------------------------------------------------------------------------
size_t CoarseOp::image_bytes() const { return (size_t)((N + 15) / 16) * steps() * slices * 512; }
size_t CoarseOp::work_bytes(int ncols) const {
  const size_t groups = (size_t)(ncols + 3) / 4;
  return groups * steps() * 1024 + groups * 4 * sizeof(int);
}

namespace {
SlabOrder slab_order(const Grid& g, int (&tap)[3]) {
  const int n[3] = {g.nx, g.ny, g.nz};
  const long long st[3] = {1, g.nx, (long long)g.nx * g.ny};
  const int tp[3] = {1, 3, 9};
  int s = 0;
  for (int d = 1; d < 3; ++d)
    if (n[d] >= n[s]) s = d;
  const int a = s == 0 ? 1 : 0, b = s == 2 ? 1 : 2;
  tap[0] = tp[s];
  tap[1] = tp[a];
  tap[2] = tp[b];
  return SlabOrder{n[s], n[a], n[b], st[s], st[a], st[b]};
}
unsigned blocks_for(long long n) { return (unsigned)((n + 255) / 256); }
void allow_smem(const void* kernel, size_t bytes) {
  const cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)bytes);
  if (e != cudaSuccess) {
    cudaGetLastError();
    throw std::runtime_error(std::string("coarse product shared memory: ") + cudaGetErrorString(e));
  }
}
}  // namespace

int coarse_slab_rows(const Grid& g) {
  int tap[3];
  const SlabOrder o = slab_order(g, tap);
  const long long M = (long long)o.n0 * o.n1;
  // a block holds enough planes for 32 rows: fewer steps of the recurrence on narrow grids
  return (int)std::min<long long>(g.N, M * ((31 + M) / M));
}

bool coarse_supported(const Grid& g) { return g.N <= kCoarseDenseMax && coarse_slab_rows(g) <= kSlabMax; }

size_t coarse_setup_bytes(const Grid& g) {
  const size_t M = (size_t)coarse_slab_rows(g), nb = ((size_t)g.N + M - 1) / M;
  return ((size_t)g.N * g.N + M * M * (5 + 3 * nb)) * sizeof(double2);
}

void launch_coarse_setup(Ctx& ctx, const Grid& g, bool is3d, const double2* coef, CoarseOp& op, double2* scratch,
                         int* bad) {
  int tap[3];
  const SlabOrder o = slab_order(g, tap);
  const long long N = g.N;
  const int Mb = coarse_slab_rows(g);
  const int nb = (int)((N + Mb - 1) / Mb);
  const int center = is3d ? 13 : 4;
  const size_t MM = (size_t)Mb * Mb;
  double2* X = scratch;
  double2* S0 = X + (size_t)N * N;
  double2* S1 = S0 + MM;
  double2* Bk = S1 + MM;
  double2* Ck = Bk + MM;
  double2* Sn = Ck + MM;
  double2* G = Sn + MM;
  double2* E = G + MM * nb;
  double2* F = E + MM * nb;
  auto rows = [&](int k) { return (int)std::min<long long>(Mb, N - (long long)k * Mb); };
  auto block = [&](int i, int j, double2* out, int ld) {
    const int nr = rows(i), nc = rows(j);
    HZ_LAUNCH(ctx, "coarse_setup", 0.0, k_coarse_block, blocks_for((long long)nr * nc), 256, 0, o, center, tap[0],
              tap[1], tap[2], coef, N, (long long)i * Mb, nr, (long long)j * Mb, nc, out, ld);
  };
  auto gemm = [&](long long m, long long n, int k, const double2* A, long long lda, const double2* B, long long ldb,
                  const double2* D, long long ldd, double sgn, double2* C, long long ldc) {
    const dim3 grid((unsigned)((n + 31) / 32), (unsigned)((m + 31) / 32));
    HZ_LAUNCH(ctx, "coarse_setup", 0.0, k_coarse_gemm, grid, 256, 0, (int)m, (int)n, k, A, lda, B, ldb, D, ldd, sgn, C,
              ldc);
  };
  int dev = 0, per_sm = 0, sms = 0;
  cudaGetDevice(&dev);
  cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_coarse_inverse, 256, 0);
  cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
  const int capacity = std::max(1, std::min(per_sm, 2)) * std::max(1, sms);
  block(0, 0, S0, rows(0));
  for (int k = 0; k < nb; ++k) {
    int m = rows(k);
    double2* Gk = G + MM * k;
    {
      const int ctas = (int)std::min<long long>(capacity, std::max<long long>(1, ((long long)m * m + 1023) / 1024));
      void* args[] = {(void*)&m, (void*)&S0, (void*)&S1, (void*)&Gk, (void*)&bad};
      const cudaError_t e = cudaLaunchCooperativeKernel((const void*)k_coarse_inverse, dim3((unsigned)ctas), dim3(256),
                                                        args, 0, ctx.stream);
      if (e != cudaSuccess) {
        cudaGetLastError();
        throw std::runtime_error(std::string("coarse inverse cooperative launch failed: ") + cudaGetErrorString(e));
      }
      ++ctx.launches;
    }
    if (k + 1 == nb) break;
    const int mn = rows(k + 1);
    block(k + 1, k, Bk, m);
    block(k, k + 1, Ck, mn);
    gemm(mn, m, m, Bk, m, Gk, m, nullptr, 0, -1.0, F + MM * k, m);
    gemm(m, mn, m, Gk, m, Ck, mn, nullptr, 0, -1.0, E + MM * k, mn);
    block(k + 1, k + 1, Sn, mn);
    gemm(mn, mn, m, F + MM * k, m, Ck, mn, Sn, mn, 1.0, S0, mn);
  }
  auto at = [&](int i, int j) { return X + (long long)i * Mb * N + (long long)j * Mb; };
  {
    const int m = rows(nb - 1);
    cudaMemcpy2DAsync(at(nb - 1, nb - 1), (size_t)N * 16, G + MM * (nb - 1), (size_t)m * 16, (size_t)m * 16, m,
                      cudaMemcpyDeviceToDevice, ctx.stream);
  }
  for (int k = nb - 2; k >= 0; --k) {
    const int m = rows(k), mn = rows(k + 1);
    const long long rest = N - (long long)(k + 1) * Mb;
    gemm(m, rest, mn, E + MM * k, mn, at(k + 1, k + 1), N, nullptr, 0, 1.0, at(k, k + 1), N);
    gemm(rest, m, mn, at(k + 1, k + 1), N, F + MM * k, m, nullptr, 0, 1.0, at(k + 1, k), N);
    gemm(m, m, mn, E + MM * k, mn, at(k + 1, k), N, G + MM * k, m, 1.0, at(k, k), N);
  }
  const unsigned gr = (unsigned)((N + 7) / 8);
  if (op.slices == 8)
    HZ_LAUNCH(ctx, "coarse_setup", 0.0, k_coarse_image<8>, gr, 256, 0, o, N, op.steps(), X, (uint32_t*)op.image,
              op.rscale);
  else
    HZ_LAUNCH(ctx, "coarse_setup", 0.0, k_coarse_image<6>, gr, 256, 0, o, N, op.steps(), X, (uint32_t*)op.image,
              op.rscale);
}

template <typename T, int S>
static void coarse_solve(Ctx& ctx, const CoarseOp& op, const cplx<T>* b, cplx<T>* x, long long ld, const int* cols,
                         int ncols, void* work) {
  const int KS = op.steps();
  const size_t groups = (size_t)(ncols + 3) / 4;
  uint4* words = (uint4*)work;
  int* cscale = (int*)((char*)work + groups * KS * 1024);
  HZ_LAUNCH(ctx, "coarse_slice", (double)ncols * op.N * (sizeof(cplx<T>) + 32.0), (k_coarse_slice<T, S>),
            dim3((unsigned)ncols, kSliceParts), 256, 0, op.N, KS, b, ld, cols, words, cscale);
  const double bytes = (double)op.N * op.N * 4.0 * S + (double)ncols * op.N * (32.0 + sizeof(cplx<T>));
  const unsigned rt = (unsigned)((op.N + 15) / 16);
  // one tile of four columns per CTA, or two that share the image's bytes
  auto launch = [&](auto nt) {
    constexpr int NT = decltype(nt)::value;
    constexpr size_t sm = product_smem<S, NT>();
    allow_smem((const void*)k_coarse_product<T, S, NT>, sm);
    HZ_LAUNCH(ctx, "coarse_product", bytes, (k_coarse_product<T, S, NT>),
              dim3((unsigned)((ncols + 4 * NT - 1) / (4 * NT)), rt), 256, sm, op.N, KS, (const uint4*)op.image,
              op.rscale, words, cscale, cols, ncols, x, ld);
  };
  if (ncols <= 4)
    launch(std::integral_constant<int, 1>());
  else
    launch(std::integral_constant<int, 2>());
}

template <>
void launch_coarse<double>(Ctx& ctx, const CoarseOp& op, const double2* b, double2* x, long long ld, const int* cols,
                           int ncols, void* work) {
  if (ncols <= 0) return;
  if (op.slices == 8)
    coarse_solve<double, 8>(ctx, op, b, x, ld, cols, ncols, work);
  else
    coarse_solve<double, 6>(ctx, op, b, x, ld, cols, ncols, work);
}
template <>
void launch_coarse<float>(Ctx& ctx, const CoarseOp& op, const float2* b, float2* x, long long ld, const int* cols,
                          int ncols, void* work) {
  if (ncols <= 0) return;
  if (op.slices == 8)
    coarse_solve<float, 8>(ctx, op, b, x, ld, cols, ncols, work);
  else
    coarse_solve<float, 6>(ctx, op, b, x, ld, cols, ncols, work);
}

}  // namespace hz
