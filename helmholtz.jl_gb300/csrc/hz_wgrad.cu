// Weight gradient of the networks' convolutions on warp-level tensor cores:
// dw[co][t][ci] = sum over nodes p of dout[p][co] in[p + offset_t][ci], a GEMM with
// M = Cout, N = taps x Cin and K = the nodes.
//
// A CTA marches along y over a chunk of grid rows of one sample (and z-plane).  Each
// input row is staged once, with its x halo and zeros outside the grid, into a ring
// of four rows per z-plane, and serves all its taps: tap (dx, dy, dz) is another
// ring row and a shift by one node.  Rows are fetched with cp.async one step
// ahead.  Fragments come from ldmatrix.trans (nodes are the K dimension, channels lie
// contiguous).  K runs over a row in steps of 16 nodes and one of 8: the networks'
// 8k + 1 and 4k + 1 node rows waste 5 to 18 % of the products.
// A warp owns NC (tap, 16 input channels) pairs for all output channels, so an input
// fragment feeds 2 CO products and an output-gradient fragment 2 NC.
//
// Before, one CTA per tap re-staged every row 9 or 27 times and assembled fragments
// from 16-bit shared-memory loads, 12 per product: 1.95 ms of a 2.7 ms step at 129^2 x
// 32, 1.84 of 2.7 ms at 33^3 x 8.
#include <algorithm>
#include <stdexcept>

#include <cuda_bf16.h>

#include "hz_launch.cuh"
#include "hz_learn.h"

namespace hz {

namespace {
constexpr int kThreads = 256, kWarps = 8;
constexpr int kSegBlocks = 18;  // 8-node blocks of a row segment: 144 nodes
constexpr int kRing = 4;        // staged input rows per z-plane: three in use, one in flight
constexpr size_t kSmemMax = 227 * 1024;

struct WgShape {
  int nx, ny, nz, planes;  // planes: 1 (3 x 3 taps) or 3 (3 x 3 x 3)
  int Cin, Cout, C16;      // C16: Cout rounded up to 16
  int ldi, ldd, d_off;
  int seg_blocks, segs;    // row segment: 8-node blocks, segments per row
  int rows, chunks;        // rows per CTA, chunks per plane
  int combos;              // (tap, 16 input channels) pairs
};

__device__ __forceinline__ void copy16_zfill(void* smem, const void* gmem, bool valid) {
  asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"((uint32_t)__cvta_generic_to_shared(smem)),
               "l"(gmem), "r"(valid ? 16 : 0));
}
__device__ __forceinline__ void ldmatrix4t(uint32_t (&r)[4], const void* smem) {
  asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];"
               : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3])
               : "r"((uint32_t)__cvta_generic_to_shared(smem)));
}
__device__ __forceinline__ void mma16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1) {
  asm volatile(
      "mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};"
      : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
      : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void mma8(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t b0) {
  asm volatile("mma.sync.aligned.m16n8k8.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5}, {%6}, {%0,%1,%2,%3};"
               : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
               : "r"(a0), "r"(a1), "r"(b0));
}

template <int CO, int NC>
__global__ void __launch_bounds__(kThreads) k_wgrad(WgShape s, const __nv_bfloat16* __restrict__ in,
                                                    const __nv_bfloat16* __restrict__ dout, float* __restrict__ dw) {
  extern __shared__ __align__(16) unsigned char wg_smem[];
  const int W = s.seg_blocks * 8;
  const int si = s.Cin + 8, sd = s.C16 + 8;   // padded: ldmatrix rows fall into different banks
  const int in_row = (W + 2) * si, d_row = W * sd;  // elements of a staged row
  __nv_bfloat16* s_in = reinterpret_cast<__nv_bfloat16*>(wg_smem);
  __nv_bfloat16* s_d = s_in + s.planes * kRing * in_row;
  const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
  int w = blockIdx.x;
  const int seg = w % s.segs;
  w /= s.segs;
  const int chunk = w % s.chunks;
  w /= s.chunks;
  const int k = w % s.nz;  // z-plane
  const long long sample = w / s.nz;
  const int x0 = seg * W;
  const int j0 = chunk * s.rows, j1 = min(s.ny, j0 + s.rows);
  const long long plane = (long long)s.nx * s.ny;
  const long long base = (sample * s.nz + k) * plane;  // first node of the z-plane
  const int c8 = s.Cin >> 3, d8 = s.C16 >> 3;
  auto stage_in = [&](int j) {
    const int slot = (j + kRing) & (kRing - 1);
    for (int p = 0; p < s.planes; ++p) {
      const int kk = k + (s.planes == 3 ? p - 1 : 0);
      const bool row_ok = j >= 0 && j < s.ny && kk >= 0 && kk < s.nz;
      const __nv_bfloat16* src = in + (base + (long long)(kk - k) * plane + (long long)j * s.nx) * s.ldi;
      __nv_bfloat16* dst = s_in + (p * kRing + slot) * in_row;
      for (int e = threadIdx.x; e < (W + 2) * c8; e += kThreads) {
        const int q = e / c8, c = e - q * c8;
        const int x = x0 + q - 1;
        const bool ok = row_ok && x >= 0 && x < s.nx;
        copy16_zfill(dst + q * si + c * 8, ok ? src + (long long)x * s.ldi + c * 8 : in, ok);
      }
    }
  };
  auto stage_d = [&](int j) {
    const __nv_bfloat16* src = dout + (base + (long long)j * s.nx) * s.ldd + s.d_off;
    __nv_bfloat16* dst = s_d + (j & 1) * d_row;
    for (int e = threadIdx.x; e < W * d8; e += kThreads) {
      const int q = e / d8, c = e - q * d8;
      const bool ok = x0 + q < s.nx && c * 8 < s.Cout;
      copy16_zfill(dst + q * sd + c * 8, ok ? src + (long long)(x0 + q) * s.ldd + c * 8 : dout, ok);
    }
  };
  // this warp's pairs: ring row and element offset of the tap's first node
  int dyp[NC], off[NC];
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    const int combo = ((int)blockIdx.y * NC + c) * kWarps + warp;
    dyp[c] = -9;  // none
    off[c] = 0;
    if (combo < s.combos) {
      const int t = combo / (s.Cin >> 4), c16 = combo % (s.Cin >> 4);
      dyp[c] = (t / 3) % 3 - 1;
      off[c] = (t / 9) * kRing * in_row + (t % 3) * si + c16 * 16;
    }
  }
  float acc[NC][CO][2][4];
#pragma unroll
  for (int c = 0; c < NC; ++c)
#pragma unroll
    for (int o = 0; o < CO; ++o)
#pragma unroll
      for (int n = 0; n < 2; ++n)
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[c][o][n][q] = 0.f;
  // ldmatrix rows: A matrices (k 0-7 | 0-7 | 8-15 | 8-15) x (m 0 | 8 | 0 | 8), B the other way round
  const int a_off = ((lane & 7) + 8 * (lane >> 4)) * sd + 8 * ((lane >> 3) & 1);
  const int b_off = ((lane & 7) + 8 * ((lane >> 3) & 1)) * si + 8 * (lane >> 4);
  stage_in(j0 - 1);
  stage_in(j0);
  stage_in(j0 + 1);
  stage_d(j0);
  asm volatile("cp.async.commit_group;");
  for (int j = j0; j < j1; ++j) {
    if (j + 1 < j1) {
      stage_in(j + 2);
      stage_d(j + 1);
    }
    asm volatile("cp.async.commit_group;");
    asm volatile("cp.async.wait_group 1;" ::: "memory");
    __syncthreads();
    const __nv_bfloat16* dr = s_d + (j & 1) * d_row;
    const __nv_bfloat16* ir[NC];
#pragma unroll
    for (int c = 0; c < NC; ++c) ir[c] = s_in + off[c] + ((j + max(dyp[c], -1) + kRing) & (kRing - 1)) * in_row;
    int q = 0;
    for (; q + 16 <= W; q += 16) {
      uint32_t a[CO][4];
#pragma unroll
      for (int o = 0; o < CO; ++o) ldmatrix4t(a[o], dr + q * sd + a_off + o * 16);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        if (dyp[c] == -9) continue;
        uint32_t b[4];
        ldmatrix4t(b, ir[c] + q * si + b_off);
#pragma unroll
        for (int o = 0; o < CO; ++o) {
          mma16(acc[c][o][0], a[o], b[0], b[1]);
          mma16(acc[c][o][1], a[o], b[2], b[3]);
        }
      }
    }
    if (q < W) {  // the last 8 nodes: the lanes of rows 8-15 read rows 0-7 again, unused
      const int a8 = (lane & 7) * sd + 8 * ((lane >> 3) & 1), b8 = (lane & 7) * si + 8 * (lane >> 4);
      uint32_t a[CO][4];
#pragma unroll
      for (int o = 0; o < CO; ++o) ldmatrix4t(a[o], dr + q * sd + a8 + o * 16);
#pragma unroll
      for (int c = 0; c < NC; ++c) {
        if (dyp[c] == -9) continue;
        uint32_t b[4];
        ldmatrix4t(b, ir[c] + q * si + b8);
#pragma unroll
        for (int o = 0; o < CO; ++o) {
          mma8(acc[c][o][0], a[o][0], a[o][1], b[0]);
          mma8(acc[c][o][1], a[o][0], a[o][1], b[2]);
        }
      }
    }
    __syncthreads();  // the oldest row and this output-gradient row are refilled in the next step
  }
  const int taps = 9 * s.planes;
  const int g = lane >> 2, tq = lane & 3;
#pragma unroll
  for (int c = 0; c < NC; ++c) {
    if (dyp[c] == -9) continue;
    const int combo = ((int)blockIdx.y * NC + c) * kWarps + warp;
    const int t = combo / (s.Cin >> 4), ci = (combo % (s.Cin >> 4)) * 16 + tq * 2;
#pragma unroll
    for (int o = 0; o < CO; ++o) {
      const int co = o * 16 + g;
#pragma unroll
      for (int n = 0; n < 2; ++n) {
        float* d = dw + ((long long)co * taps + t) * s.Cin + ci + 8 * n;
        if (co < s.Cout) atomicAdd(reinterpret_cast<float2*>(d), make_float2(acc[c][o][n][0], acc[c][o][n][1]));
        if (co + 8 < s.Cout)
          atomicAdd(reinterpret_cast<float2*>(d + 8LL * taps * s.Cin), make_float2(acc[c][o][n][2], acc[c][o][n][3]));
      }
    }
  }
}

size_t staged_bytes(const WgShape& s) {
  const size_t W = (size_t)s.seg_blocks * 8;
  return 2 * ((size_t)s.planes * kRing * (W + 2) * (s.Cin + 8) + 2 * W * (s.C16 + 8));
}

template <int CO, int NC>
void wg_launch(Ctx& ctx, const char* name, WgShape s, long long planes_total, const WgradTc& a) {
  const size_t smem = staged_bytes(s);
  if (smem > kSmemMax) throw std::runtime_error("weight gradient: channel counts not supported");
  static SmemLimit limit;
  raise_smem_limit(limit, (const void*)k_wgrad<CO, NC>, kSmemMax, "weight gradient");
  // Rows per CTA: the CTAs that fit at once, times one to four rounds of them, whichever
  // takes the fewest rows one after another (a chunk stages two rows more than it sums).
  int per_sm = 0;
  if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_wgrad<CO, NC>, kThreads, smem) != cudaSuccess) {
    cudaGetLastError();
    throw std::runtime_error("weight gradient: occupancy");
  }
  const long long slots = (long long)std::max(per_sm, 1) * kSMs;
  const long long units = planes_total * s.segs * ((s.combos + NC * kWarps - 1) / (NC * kWarps));
  long long best = 0;
  for (int rounds = 1; rounds <= 4; ++rounds) {
    const long long want = std::max<long long>(1, std::min<long long>(s.ny, rounds * slots / units));
    const int rows = (int)((s.ny + want - 1) / want), chunks = (s.ny + rows - 1) / rows;
    const long long cost = (units * chunks + slots - 1) / slots * (rows + 2);
    if (best == 0 || cost < best) {
      best = cost;
      s.rows = rows;
      s.chunks = chunks;
    }
  }
  const long long ctas = planes_total * s.chunks * s.segs;
  if (ctas >= (1LL << 31)) throw std::runtime_error("weight gradient: batch too large");
  const int taps = 9 * s.planes;
  const dim3 grid((unsigned)ctas, (unsigned)((s.combos + NC * kWarps - 1) / (NC * kWarps)));
  ctx.add_flops(name, 2.0 * taps * a.Cin * a.Cout * (double)a.nodes);
  HZ_LAUNCH(ctx, name, (double)a.nodes * (a.Cin + a.Cout) * 2.0 + 4.0 * taps * a.Cin * a.Cout, (k_wgrad<CO, NC>), grid,
            kThreads, smem, s, a.in, a.dout, a.dw);
}
}  // namespace

void wgrad_launch(Ctx& ctx, const char* name, const WgradTc& a, int taps) {
  WgShape s{};
  s.nx = a.nx;
  s.ny = a.ny;
  s.nz = a.nz;
  s.planes = taps == 27 ? 3 : 1;
  s.Cin = a.Cin;
  s.Cout = a.Cout;
  s.C16 = (a.Cout + 15) / 16 * 16;
  s.ldi = a.ldi;
  s.ldd = a.ldd;
  s.d_off = a.d_off;
  if (a.Cin % 16 || a.Cin > 128 || a.Cout % 8 || s.C16 > 64 || a.ldi % 8 || a.ldd % 8 || a.d_off % 8 ||
      (reinterpret_cast<uintptr_t>(a.in) | reinterpret_cast<uintptr_t>(a.dout)) % 16 ||
      reinterpret_cast<uintptr_t>(a.dw) % 8)
    throw std::runtime_error("weight gradient: layout not supported");
  const int nblk = (s.nx + 7) / 8;
  s.segs = (nblk + kSegBlocks - 1) / kSegBlocks;
  s.seg_blocks = (nblk + s.segs - 1) / s.segs;
  s.segs = (nblk + s.seg_blocks - 1) / s.seg_blocks;
  s.combos = taps * (s.Cin / 16);
  // Pairs per warp: as many as leave two CTAs per SM (64 accumulators), though the rows are
  // staged again for the others.  One CTA with 112 (96 for Cout = 64): 1,010 against 988 us
  // per 129^2 x 32 step.
  const int co = s.C16 / 16, per = (s.combos + kWarps - 1) / kWarps;
  const int cap = co == 1 ? 11 : co == 2 ? 4 : 2;
  const long long planes_total = a.nodes / ((long long)s.nx * s.ny);
  const int splits = (per + cap - 1) / cap, nc = (per + splits - 1) / splits;
#define HZ_WG(C, K)                                          \
  if (co == C && nc <= K) {                                  \
    wg_launch<C, K>(ctx, name, s, planes_total, a);          \
    return;                                                  \
  }
  HZ_WG(1, 2)
  HZ_WG(1, 4)
  HZ_WG(1, 7)
  HZ_WG(1, 11)
  HZ_WG(2, 2)
  HZ_WG(2, 4)
  HZ_WG(4, 2)
#undef HZ_WG
  throw std::runtime_error("weight gradient: channel counts not supported");
}

}  // namespace hz
