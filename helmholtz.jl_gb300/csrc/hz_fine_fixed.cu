// The fine-level operator with FP64 results on the integer pipe (hz_fixed.cuh).
//
// Native FP64 takes 16 operations per node and column in 3D (12 in 2D), 8 clocks of an SM
// with its two FP64 lanes; HBM delivers the operands in 1.4.  Here the neighbours are summed
// as integers: a block takes a brick of one column, loads it with its halo in one go, relates
// all values to the brick's largest, converts each once (57 bits in two words whose sums over
// six neighbours still fit) and shares it through shared memory.  The Laplacian's
// coefficients and the diagonal are fixed-point numbers of 58 bits, so a node is one
// integer sum, rounded once.
//
// Boundary rows need no case of their own: with second-order rows (2 u_0 - 2 u_1) / h^2 the
// missing neighbour is the mirrored one, with first-order rows it is zero.  The adjoint
// of the mirrored operator A is W A W^-1 with W = 1/2 per boundary the node lies on:
// values are shifted up by that many bits when converted and results down.
//
// A value is off by at most 2^-56 of the brick's reference.  A node with no value, its own or a
// neighbour's, above 2^-5 of it takes the native steps; so do bricks whose exponents are out of
// range and values that are NaN or Inf.  Zeros (a brick's, a node's with its neighbours) are not
// worked on: a sparse column has little else.  Against quad precision the product's error is
// 5.1e-17 of its norm on noise (native 7.5e-17), 9.2e-17 on plane waves (5.4e-16) and 6.0e-17 to
// 7.4e-17 on noise that decays or spreads over 2^6 (7.4e-17 to 7.6e-17).  At a single node, one
// 2^-5 below its brick, up to 3.8 u of the row's sum of magnitudes was measured on these inputs,
// u = 2^-53 (native 1.7 u).  The bound is 48 u of the row's sum of coefficients times the largest
// value around the node (tests/test_gpu_fine_fixed.py): coefficients are rounded relative to the
// operator's largest, so where the diagonal is far below it and the neighbours are zeros the
// error can be more of the node's own row.
//
// Measured: 157 x 131 x 101 nodes, 13 columns, adjoint: 887 us native, 434; 129^3 nodes, 8 columns of
// FP32 537 and 355; 1025 x 513 nodes, 16 columns of FP32 176 and 114; the FP64 cycle's residual
// and Jacobi sweep, 65 x 65 x 33 nodes, 8 columns, 48 and 34, 59 and 49.  What bounds it is
// instructions (36 per cell converted, 1.75 cells per node in 3D; 106 per sum; 4 additions of the
// FP64 pipe) at half the issue rate: the rest is the wait for a brick's loads, with four
// bricks in flight per SM.  Bringing a block's next column by asynchronous copies, 2 or 3
// bricks per SM, took 326 to 330 instead of 355 in that one case and 2% to 8% longer in the other
// two; giving every third or fourth brick to the native steps took a quarter longer.
#include <algorithm>
#include <cstring>
#include <stdexcept>
#include <type_traits>

#include "hz_fixed.cuh"
#include "hz_kernels.cuh"
#include "hz_launch.cuh"

namespace hz {

namespace {
constexpr int kN = 4;         // nodes per thread: planes (3D), rows one tile height apart (2D)
constexpr int kThreads = 256;
constexpr int kHalo = 2;      // halo cells per thread, at most
constexpr int kBits = 57;     // bits of a value below its reference
constexpr int kLow = 29;      // of them in the low word
constexpr int kGuard = 4;     // exponents below the reference a node's largest value may lie
constexpr int kRange = 3;     // exponents the neighbours' coefficients may lie below the diagonal's
// Nodes times columns from which the integer sums pay.  us per product, native / integer:
// 129 x 129 nodes 8 columns (2^17) 9.9 / 9.9, 16 columns 12.8 / 11.2; 25^3 nodes 8 columns (2^17)
// 11.6 / 9.1; 65^3 1 column (2^18) 16.6 / 12.5; 101^3 2 columns 73 / 35; below 2^16 native is ahead.
constexpr long long kFineFixedMin = 1 << 17;

struct FixOp {
  int nx, ny, nz;
  int adj;
  int uniform;  // the same spacing on every axis
  double o[3], b[3];
  int w, h;     // tile: w x h nodes (3D), w x kN h (2D)
  int tiles_x, tiles;
  const double* sig;
  int sig_stride;
  unsigned inv_w, inv_ring;  // 2^16 / w and 2^16 / ring, rounded up: quotients of numbers below 2 kThreads
};
// boundary rows: first order, second order, the second order's adjoint
enum { kPlain, kMirror, kMirrorAdj };

// raw words of a value, exponent field as in FP64
template <typename TX> struct Raw;
template <> struct Raw<double> {
  using type = uint4;
  static __device__ __forceinline__ uint4 widen(uint4 r) { return r; }
  static __device__ __forceinline__ uint32_t any(uint4 r) { return r.x | r.z | (r.y | r.w) << 1; }
};
template <> struct Raw<float> {
  using type = uint2;
  static __device__ __forceinline__ uint4 widen(uint2 r) {
    uint4 w;
    widen_f32_hilo(r.x, w.y, w.x);
    widen_f32_hilo(r.y, w.w, w.z);
    return w;
  }
  static __device__ __forceinline__ uint32_t any(uint2 r) { return (r.x | r.y) << 1; }
};

// |v| in units of 2^(E - 1022 - kBits), truncated; s = E - exponent field (a zero or
// subnormal's field reads as 0 and E is at least kFixedMin - 3: it is shifted out)
__device__ __forceinline__ long long to_fixed(uint32_t vhi, uint32_t vlo, int s) {
  const uint32_t mh = (vhi & 0xfffffu) | 0x100000u;
  const uint64_t m = (((uint64_t)mh << 32 | vlo) << (kBits - 53)) >> min(s, 63);
  return (int32_t)vhi < 0 ? -(long long)m : (long long)m;
}
// A value's cell: high (signed) and low words of both components.  Bit 0 of the first
// low word says that one of them lies within kGuard exponents of the reference; it counts
// as part of the value.  top: the reference's exponent field in place, all below it set.
__device__ __forceinline__ int4 to_cell(uint4 r, uint32_t top) {
  const int sx = (int)((top - (r.y & 0x7fffffffu)) >> 20), sy = (int)((top - (r.w & 0x7fffffffu)) >> 20);
  const long long x = to_fixed(r.y, r.x, sx), y = to_fixed(r.w, r.z, sy);
  constexpr int mask = (1 << kLow) - 1;
  return make_int4((int)(x >> kLow), ((int)x & (mask - 1)) | (min(sx, sy) <= kGuard ? 1 : 0), (int)(y >> kLow),
                   (int)y & mask);
}
// The words of a sum of up to six cells, the low one's carry moved up
__device__ __forceinline__ Fixed carried(int hi, uint32_t lo) {
  return Fixed{hi + (int)(lo >> kLow), (int)(lo & ((1u << kLow) - 1))};
}
__device__ __forceinline__ Fixed coefficient(double v, int E) {
  return fixed_from<6>((uint32_t)__double2hiint(v), (uint32_t)__double2loint(v), E);
}
__device__ __forceinline__ Fixed negative(Fixed a) { return Fixed{-a.hi, -a.lo}; }

// Totals to FP64, scaled by 2^e and rounded once, with two additions: the halves of the integer
// are the low mantissa words of 2^(52+e) and 2^(84+e).
struct Assemble {
  uint32_t lo, hi;  // high words
  double bias;      // 2^e (2^84 + 2^63 + 2^52)
  __device__ __forceinline__ explicit Assemble(int e) {
    lo = (uint32_t)(52 + e + 1023) << 20;
    hi = (uint32_t)(84 + e + 1023) << 20;
    bias = __hiloint2double((int)hi, (int)0x80100000u);
  }
  __device__ __forceinline__ double operator()(long long t) const {
    const double a = __hiloint2double((int)hi, (int)((uint32_t)(t >> 32) ^ 0x80000000u));
    const double c = __hiloint2double((int)lo, (int)(uint32_t)t);
    return (a - bias) + c;
  }
};

template <typename TX, bool IS3D>
__device__ __forceinline__ double2 native_node(const FixOp& op, double2 d, const cplx<TX>* xc, int i, int j, int k) {
  const long long sy = op.nx, sz = (long long)op.nx * op.ny;
  const long long p = i + sy * j + sz * k;
  const int at[3] = {i, j, k}, n[3] = {op.nx, op.ny, op.nz};
  const long long st[3] = {1, sy, sz};
  double sr = 0.0, si = 0.0;
#pragma unroll
  for (int a = 0; a < (IS3D ? 3 : 2); ++a) {
    double cl, cr;
    if (!op.adj) {
      cl = (at[a] > 0) ? ((at[a] == n[a] - 1) ? op.b[a] : op.o[a]) : 0.0;
      cr = (at[a] < n[a] - 1) ? ((at[a] == 0) ? op.b[a] : op.o[a]) : 0.0;
    } else {
      cl = (at[a] > 0) ? ((at[a] - 1 == 0) ? op.b[a] : op.o[a]) : 0.0;
      cr = (at[a] < n[a] - 1) ? ((at[a] + 1 == n[a] - 1) ? op.b[a] : op.o[a]) : 0.0;
    }
    const double2 l = ccast<double, TX>(xc[p - (at[a] > 0 ? st[a] : 0)]);
    const double2 r = ccast<double, TX>(xc[p + (at[a] < n[a] - 1 ? st[a] : 0)]);
    sr += cl * l.x + cr * r.x;
    si += cl * l.y + cr * r.y;
  }
  if (op.adj) d.y = -d.y;
  return cfma<double>(d, ccast<double, TX>(xc[p]), mk<double>(-sr, -si));
}

// Whether a node and its neighbours are zeros
template <typename TX, bool IS3D>
__device__ __forceinline__ bool no_value(const FixOp& op, const cplx<TX>* xc, int i, int j, int k) {
  const long long sy = op.nx, sz = (long long)op.nx * op.ny;
  const typename Raw<TX>::type* x = reinterpret_cast<const typename Raw<TX>::type*>(xc) + (i + sy * j + sz * k);
  const int at[3] = {i, j, k}, n[3] = {op.nx, op.ny, op.nz};
  const long long st[3] = {1, sy, sz};
  uint32_t any = Raw<TX>::any(__ldg(x));
#pragma unroll
  for (int a = 0; a < (IS3D ? 3 : 2); ++a)
    any |= Raw<TX>::any(__ldg(x - (at[a] > 0 ? st[a] : 0))) | Raw<TX>::any(__ldg(x + (at[a] < n[a] - 1 ? st[a] : 0)));
  return any == 0;
}

struct Acc {
  long long h = 0, l = 0;
  __device__ __forceinline__ void add(Fixed a, Fixed b) { fixed_mac(h, l, a, b); }
  __device__ __forceinline__ long long total() const { return fixed_total(h, l); }
};

template <typename TX, int MODE, bool IS3D, int ROWS>
__global__ void __launch_bounds__(kThreads, IS3D ? 4 : 5)
    k_fine_fixed(const __grid_constant__ FixOp op, const FixedRefs* __restrict__ refs,
                 const int4* __restrict__ dfix, const double2* __restrict__ diag, const cplx<TX>* __restrict__ x,
                 const double2* __restrict__ b, double2* __restrict__ y, long long ld, const int* __restrict__ cols,
                 const double2* __restrict__ dinv, double weight) {
  using R = Raw<TX>;
  using RT = typename R::type;
  constexpr int ZH = IS3D ? 1 : 0, NL = kN + 2 * ZH;
  constexpr bool WEIGH = ROWS == kMirrorAdj;  // values carry 2^(boundaries of their node)
  extern __shared__ int4 cell[];  // 3D: [kN + 2][h + 2][w + 2], 2D: [kN h + 2][w + 2]
  __shared__ uint32_t largest;
  const int tid = threadIdx.x;
  const int w = op.w, h = op.h, pitch = w + 2;
  const int ty = (int)(tid * op.inv_w >> 16), tx = tid - ty * w;
  const bool mine = ty < h;
  const int rows = IS3D ? h : kN * h;                   // of a tile's plane
  const int step = IS3D ? pitch * (h + 2) : pitch * h;  // between a thread's cells
  const int x0 = (int)(blockIdx.x % op.tiles_x) * w, y0 = (int)(blockIdx.x / op.tiles_x) * rows;
  const int z0 = IS3D ? (int)blockIdx.y * kN : 0;
  const long long off = (long long)cols[blockIdx.z] * ld;
  const RT* xr = reinterpret_cast<const RT*>(x + off);
  const int sy = op.nx, sz = op.nx * op.ny;  // a column has less than 2^31 nodes
  const int Ec = refs->exponent;
  const int base = (ty + 1) * pitch + tx + 1;
  if (tid == 0) largest = 0;
  // Node of a cell.  Mirrored rows: its reflection, some node for cells further outside; else
  // negative for none.
  auto fold = [&](int q, int n) {
    if (ROWS != kPlain) {
      q = abs(q);
      return max(min(q, 2 * (n - 1) - q), 0);
    }
    return q < n ? q : -1;
  };
  auto edge = [&](int q, int n) { return (q == 0 || q == n - 1) ? 1 : 0; };
  auto fetch = [&](int i, int j, int k, int& power) {
    power = WEIGH ? edge(i, op.nx) + edge(j, op.ny) + (IS3D ? edge(k, op.nz) : 0) : 0;
    if (ROWS == kPlain && (i | j | k) < 0) return make_uint4(0, 0, 0, 0);
    return R::widen(__ldg(xr + (k * sz + (j * sy + i))));
  };
  uint4 own[NL], halo[kHalo];
  int pown[NL], phalo[kHalo], at[kHalo];
  const int fi = fold(x0 + tx, op.nx);
  const int fj = IS3D ? fold(y0 + ty, op.ny) : 0;
#pragma unroll
  for (int q = 0; q < NL; ++q)
    own[q] = IS3D ? fetch(fi, fj, fold(z0 + q - 1, op.nz), pown[q]) : fetch(fi, fold(y0 + ty + q * h, op.ny), 0, pown[q]);
  // the halo: rows above and below, columns left and right, no corners
  const int ring = 2 * (w + rows), cells = IS3D ? kN * ring : ring;
#pragma unroll
  for (int q = 0; q < kHalo; ++q) {
    const int m = tid + q * (int)blockDim.x;
    at[q] = -1;
    halo[q] = make_uint4(0, 0, 0, 0);
    phalo[q] = 0;
    if (m < cells) {
      const int k = IS3D ? (int)(m * op.inv_ring >> 16) : 0, r = m - k * ring;
      const int e = r - 2 * w;
      const int ci = e < 0 ? (r < w ? r : r - w) : (e < rows ? -1 : w);
      const int cj = e < 0 ? (r < w ? -1 : rows) : (e < rows ? e : e - rows);
      at[q] = (IS3D ? (k + 1) * step : 0) + (cj + 1) * pitch + ci + 1;
      halo[q] = fetch(fold(x0 + ci, op.nx), fold(y0 + cj, op.ny), IS3D ? fold(z0 + k, op.nz) : 0, phalo[q]);
    }
  }
  uint32_t t = 0;  // largest magnitude's high word
  auto over = [&](uint4 r, int power) {
    t = max(t, max(r.y & 0x7fffffffu, r.w & 0x7fffffffu) + ((uint32_t)power << 20));
  };
#pragma unroll
  for (int q = 0; q < NL; ++q) over(own[q], pown[q]);
#pragma unroll
  for (int q = 0; q < kHalo; ++q) over(halo[q], phalo[q]);
  t = __reduce_max_sync(0xffffffffu, t);
  __syncthreads();
  if ((tid & 31) == 0) atomicMax(&largest, t);
  __syncthreads();
  const int E = (int)(largest >> 20);
  // the power of two that the results are scaled by
  const int power =
      MODE == MODE_APPLY && op.sig ? basis_exponent(op.sig[(long long)cols[blockIdx.z] * op.sig_stride]) : 0;
  const bool ok = fixed_ref_ok(E) && fixed_ok(E + Ec) && fixed_ok(E + Ec + power);
  // a brick without a value; its zeros may stand with their powers in E
  bool empty = false;
  if (E < kFixedMin) {
    uint32_t any = 0;
#pragma unroll
    for (int q = 0; q < NL; ++q) any |= Raw<double>::any(own[q]);
#pragma unroll
    for (int q = 0; q < kHalo; ++q) any |= Raw<double>::any(halo[q]);
    empty = !__syncthreads_or((int)any);
  }
  if (ok) {
    const uint32_t top = largest | 0xfffffu;
    if (mine) {
#pragma unroll
      for (int q = 0; q < NL; ++q) cell[base + q * step] = to_cell(own[q], top - ((uint32_t)pown[q] << 20));
    }
#pragma unroll
    for (int q = 0; q < kHalo; ++q)
      if (at[q] >= 0) cell[at[q]] = to_cell(halo[q], top - ((uint32_t)phalo[q] << 20));
  }
  __syncthreads();
  // this thread's nodes
  const int i = x0 + tx, j = y0 + ty;
  const int nk = !mine || i >= op.nx ? 0 : IS3D ? (j < op.ny ? op.nz - z0 : 0) : op.ny - j;  // 2D: rows below
  const int gs = IS3D ? sz : h * sy;  // a plane or h rows
  const int p0 = z0 * sz + (j * sy + i);
  const int e0 = E + Ec + power + 1 - kFixedScale;  // exponent of a total's unit
  const int4* c = cell + base + (IS3D ? step : 0);
  const double2* bc = b + off;
  double2* yc = y + off;
  const Fixed ox = refs->o[0], oy = refs->o[1], oz = refs->o[2];
  // a = (op x) of node p to the mode's result
  auto result = [&](double2 a, int p, double2 bb) {
    if (MODE == MODE_APPLY) return a;
    const double2 r = mk<double>(bb.x - a.x, bb.y - a.y);
    if (MODE == MODE_RESID) return r;
    double2 di = dinv[p];
    if (op.adj) di.y = -di.y;
    const double2 dr = cmul<double>(di, r), xp = ccast<double, TX>(x[off + p]);
    return mk<double>(xp.x + weight * dr.x, xp.y + weight * dr.y);
  };
  uint32_t native = 0;  // nodes left to the native steps
#pragma unroll
  for (int k = 0; k < kN; ++k) {
    if ((IS3D ? k : k * h) >= nk) break;
    const int p = p0 + k * gs;
    double2 bb = mk<double>(0, 0);
    if (MODE != MODE_APPLY) bb = __ldcs(bc + p);
    if (empty) {
      __stcs(yc + p, result(mk<double>(0, 0), p, bb));
      continue;
    }
    const int4 d = __ldg(dfix + p);
    const int4* ck = c + k * step;
    const int4 n0 = ck[0], nl = ck[-1], nr = ck[1], nu = ck[-pitch], nd = ck[pitch];
    const int4 zero = make_int4(0, 0, 0, 0);
    const int4 nf = IS3D ? ck[-step] : zero, nb = IS3D ? ck[step] : zero;
    const int flags = n0.y | nl.y | nr.y | nu.y | nd.y | nf.y | nb.y;
    if (ok && (flags & 1)) {
      const Fixed dr{d.x, d.y}, di{d.z, d.w}, dn = negative(di);
      const Fixed vr{n0.x, n0.y}, vi{n0.z, n0.w};
      Acc re, im;
      re.add(dr, vr);
      re.add(op.adj ? di : dn, vi);
      im.add(dr, vi);
      im.add(op.adj ? dn : di, vr);
      if (op.uniform) {
        re.add(ox, carried((nl.x + nr.x + nu.x) + (nd.x + nf.x + nb.x),
                           ((uint32_t)nl.y + nr.y + nu.y) + ((uint32_t)nd.y + nf.y + nb.y)));
        im.add(ox, carried((nl.z + nr.z + nu.z) + (nd.z + nf.z + nb.z),
                           ((uint32_t)nl.w + nr.w + nu.w) + ((uint32_t)nd.w + nf.w + nb.w)));
      } else {
        re.add(ox, carried(nl.x + nr.x, (uint32_t)nl.y + nr.y));
        im.add(ox, carried(nl.z + nr.z, (uint32_t)nl.w + nr.w));
        re.add(oy, carried(nu.x + nd.x, (uint32_t)nu.y + nd.y));
        im.add(oy, carried(nu.z + nd.z, (uint32_t)nu.w + nd.w));
        if (IS3D) {
          re.add(oz, carried(nf.x + nb.x, (uint32_t)nf.y + nb.y));
          im.add(oz, carried(nf.z + nb.z, (uint32_t)nf.w + nb.w));
        }
      }
      const Assemble out(e0 - pown[k + ZH]);
      const double2 a = mk<double>(out(re.total()), out(im.total()));
      __stcs(yc + p, result(a, p, bb));
    } else if (ok && no_value<TX, IS3D>(op, x + off, i, IS3D ? j : j + k * h, IS3D ? z0 + k : 0)) {
      __stcs(yc + p, result(mk<double>(0, 0), p, bb));
    } else {
      native |= 1u << k;
    }
  }
  while (native) {
    const int k = __ffs((int)native) - 1;
    native &= native - 1;
    const int p = p0 + k * gs;
    double2 a = IS3D ? native_node<TX, IS3D>(op, diag[p], x + off, i, j, z0 + k)
                     : native_node<TX, IS3D>(op, diag[p], x + off, i, j + k * h, 0);
    if (power) a = cscale<double>(basis_power(power), a);
    yc[p] = result(a, p, MODE == MODE_APPLY ? a : bc[p]);
  }
}

__global__ void __launch_bounds__(256) k_diag_fixed(long long N, const double2* __restrict__ d, int dim, double o0,
                                                    double o1, double o2, FixedRefs* refs, int4* __restrict__ out) {
  const long long p = (long long)blockIdx.x * 256 + threadIdx.x;
  const int E = refs->exponent;
  if (p == 0) {
    refs->o[0] = negative(coefficient(o0, E));
    refs->o[1] = negative(coefficient(o1, E));
    refs->o[2] = dim == 3 ? negative(coefficient(o2, E)) : Fixed{0, 0};
  }
  if (p >= N) return;
  const double2 v = d[p];
  const Fixed a = coefficient(v.x, E), c = coefficient(v.y, E);
  out[p] = make_int4(a.hi, a.lo, c.hi, c.lo);
}

// The tile whose blocks take the fewest instructions over the grid: a thread's nodes 106 each, its
// cells 36, a block 400 per warp.  (Grids of 2^k + 1 nodes leave a third of fixed 16 x 16 x 8
// bricks empty.)
void choose_tile(FixOp& op, bool is3d) {
  double best = 0.0;
  for (int w = 8; w <= 64; ++w)
    for (int h = 2; w * h <= kThreads; ++h) {
      const int rows = is3d ? h : kN * h, threads = (w * h + 31) / 32 * 32;
      const int ring = (is3d ? kN : 1) * 2 * (w + rows);
      if (ring > kHalo * threads) continue;
      const double tiles = (double)((op.nx + w - 1) / w) * ((op.ny + rows - 1) / rows);
      const double cost = tiles * (threads * (106.0 * kN + 36.0 * (is3d ? kN + 2 : kN)) + 36.0 * ((ring + 31) / 32 * 32) +
                                   32.0 * 400.0);
      if (best == 0.0 || cost < best) {
        best = cost;
        op.w = w;
        op.h = h;
      }
    }
  const int rows = is3d ? op.h : kN * op.h, ring = 2 * (op.w + rows);
  op.tiles_x = (op.nx + op.w - 1) / op.w;
  op.tiles = op.tiles_x * ((op.ny + rows - 1) / rows);
  op.inv_w = (65536 + op.w - 1) / op.w;
  op.inv_ring = (65536 + ring - 1) / ring;
}
}  // namespace

void launch_diag_fixed(Ctx& ctx, const FineOp& op, const double2* d, FixedRefs* refs, int4* out) {
  HZ_LAUNCH(ctx, "fine_setup", (double)op.g.N * 32.0, k_diag_fixed, (unsigned)((op.g.N + 255) / 256), 256, 0, op.g.N, d,
            op.g.nz > 1 ? 3 : 2, op.o[0], op.o[1], op.o[2], refs, out);
}

// The neighbours' coefficients within kRange exponents of the largest coefficient, the diagonal:
// 8 to 16 times the smallest of them, as they lie in their binades.  Spacings more unequal (one axis
// of three stretched by 1.4 to 2.4, one of two by 1.7 to 2.6) and diagonals far above the
// Laplacian's stay with the native kernel.  157 x 131 x 101 nodes, 13 columns, ratio 4: 890 us
// there, 1,166 with every node of every brick left to the native steps.
bool fine_fixed_fits(const FineOp& op, int exponent) {
  double least = std::min(op.o[0], op.o[1]);
  if (op.g.nz > 1) least = std::min(least, op.o[2]);
  uint64_t bits;
  std::memcpy(&bits, &least, sizeof(bits));
  return fixed_ref_ok(exponent) && exponent - fixed_exponent((uint32_t)(bits >> 32)) <= kRange;
}

bool fine_fixed_pays(const FineOp& op, int ncols) {
  const bool is3d = op.g.nz > 1;
  if (op.g.N >= (1ll << 30)) return false;
  bool same = true, twice = true;
  for (int a = 0; a < (is3d ? 3 : 2); ++a) {
    same = same && op.b[a] == op.o[a];
    twice = twice && op.b[a] == 2.0 * op.o[a];
  }
  if (!same && !twice) return false;
  if (op.g.nx < 2 || op.g.ny < 2) return false;
  if (ncols > 65535 || (is3d && (op.g.nz + kN - 1) / kN > 65535)) return false;
  return op.g.N * (long long)ncols >= kFineFixedMin;
}

template <typename TX>
void launch_fine_fixed(Ctx& ctx, int mode, const FineOp& op, const double2* diag, const FixedDiag& fd,
                       const cplx<TX>* x, const double2* b, double2* y, long long ld, const int* cols, int ncols,
                       const double2* dinv, double weight) {
  if (ncols <= 0) return;
  const bool is3d = op.g.nz > 1;
  FixOp o{};
  o.nx = op.g.nx;
  o.ny = op.g.ny;
  o.nz = op.g.nz;
  o.adj = op.adj;
  o.sig = op.sig;
  o.sig_stride = op.sig_stride;
  o.uniform = op.o[0] == op.o[1] && (!is3d || op.o[0] == op.o[2]);
  for (int a = 0; a < 3; ++a) {
    o.o[a] = op.o[a];
    o.b[a] = op.b[a];
  }
  choose_tile(o, is3d);
  const int rows = is3d ? o.h : kN * o.h;
  const dim3 grid((unsigned)o.tiles, (unsigned)(is3d ? (o.nz + kN - 1) / kN : 1),
                  (unsigned)ncols);
  const int threads = (o.w * o.h + 31) / 32 * 32;
  const size_t smem = (size_t)(is3d ? kN + 2 : 1) * (rows + 2) * (o.w + 2) * sizeof(int4);
  const double nn = (double)op.g.N * ncols;
  const double bytes = nn * (sizeof(cplx<TX>) + 16.0 + (mode == MODE_APPLY ? 0.0 : 16.0)) +
                       op.g.N * (mode == MODE_JACOBI ? 32.0 : 16.0);
  const char* name = mode == MODE_APPLY   ? (op.outer ? "outer_apply" : "fine_apply")
                     : mode == MODE_RESID ? (op.outer ? "outer_resid" : "fine_resid")
                                          : "fine_jacobi";
  if (op.outer) ctx.add_flops(name, (8.0 * (is3d ? 3 : 2) + 8.0 + (mode == MODE_RESID ? 2.0 : 0.0)) * nn);
#define HZ_FF(M, D, W)                                                                                               \
  HZ_LAUNCH(ctx, name, bytes, (k_fine_fixed<TX, M, D, W>), grid, threads, smem, o, fd.refs, fd.d, diag, x, b, y, \
            ld, cols, dinv, weight)
#define HZ_FF_FORMS(M)                                   \
  do {                                                   \
    if (is3d && plain) HZ_FF(M, true, kPlain);           \
    else if (is3d && o.adj) HZ_FF(M, true, kMirrorAdj);  \
    else if (is3d) HZ_FF(M, true, kMirror);              \
    else if (plain) HZ_FF(M, false, kPlain);             \
    else if (o.adj) HZ_FF(M, false, kMirrorAdj);         \
    else HZ_FF(M, false, kMirror);                       \
  } while (0)
  const bool plain = op.b[0] == op.o[0];
  if (mode == MODE_APPLY) HZ_FF_FORMS(MODE_APPLY);
  else if (mode == MODE_RESID) HZ_FF_FORMS(MODE_RESID);
  else if constexpr (std::is_same<TX, double>::value) HZ_FF_FORMS(MODE_JACOBI);
  else throw std::runtime_error("fine operator: FP64 sweeps only");
#undef HZ_FF_FORMS
#undef HZ_FF
}
template void launch_fine_fixed<double>(Ctx&, int, const FineOp&, const double2*, const FixedDiag&, const double2*,
                                        const double2*, double2*, long long, const int*, int, const double2*, double);
template void launch_fine_fixed<float>(Ctx&, int, const FineOp&, const double2*, const FixedDiag&, const float2*,
                                       const double2*, double2*, long long, const int*, int, const double2*, double);

}  // namespace hz
