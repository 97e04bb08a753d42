// Per-channel grid transfers of the networks (BF16, channels last, 8 channels per
// thread): full weighting (rows normalised inside the grid), bi/trilinear prolongation and
// their adjoints, with the ReLU mask and accumulation of the backward pass folded in.
//
// A block works on one output row, so a thread's node and channels come from one shift of
// its index; all loads of a node are issued before they are summed (taps outside the grid
// read the node's own cell and are left out of the sum).  Before, six integer divisions per
// thread and a load at a time made the small kernels instruction-bound: 129^2 x 32, all
// transfers of a forward pass 83 us at 1.3 TB/s, now 73 us.
#include <stdexcept>

#include <cuda_bf16.h>

#include "hz_launch.cuh"
#include "hz_learn.h"

namespace hz {

namespace {
using bf16 = __nv_bfloat16;

struct Shape {
  int nxf, nyf, nzf, nxc, nyc, nzc;
  int B, C8, shift;  // shift: log2(C8), or -1
  int ldi, i_off, ldo, o_off, ldm, m_off, accum;
};

__device__ __forceinline__ void unpack(uint4 u, float (&v)[8]) {
  const uint32_t w[4] = {u.x, u.y, u.z, u.w};
#pragma unroll
  for (int k = 0; k < 4; ++k) {
    v[2 * k] = __uint_as_float(w[k] << 16);
    v[2 * k + 1] = __uint_as_float(w[k] & 0xffff0000u);
  }
}

// sum of the 1D full-weighting row of coarse node I on an axis of nf fine nodes
__device__ __forceinline__ float fw_sum(int I, int nf) {
  return 1.f + (2 * I - 1 >= 0 ? 0.5f : 0.f) + (2 * I + 1 < nf ? 0.5f : 0.f);
}

// Taps of one axis for output index o: input indices, weights and validity.
// KIND 0: restriction (coarse o from fine 2o - 1 .. 2o + 1), 1: its adjoint (fine o from its
// coarse parents), 2: prolongation (the two parents, equal for an even o), 3: its adjoint.
template <int KIND> struct Taps {
  static constexpr int n = KIND == 0 || KIND == 3 ? 3 : 2;
  int at[n];
  float w[n], s[n];  // s: KIND 1, the parent's row sum
  bool ok[n];
  __device__ __forceinline__ Taps(int o, int nf) {
#pragma unroll
    for (int k = 0; k < n; ++k) {
      s[k] = 1.f;
      if (KIND == 0 || KIND == 3) {
        const int f = 2 * o + k - 1;
        ok[k] = f >= 0 && f < nf;
        at[k] = ok[k] ? f : 2 * o;
        w[k] = k == 1 ? 1.f : 0.5f;
      } else {
        at[k] = (o + k) >> 1;
        ok[k] = KIND == 2 || k == 0 || (o & 1);
        w[k] = (o & 1) ? 0.5f : 1.f;
        if (KIND == 1) s[k] = fw_sum(at[k], nf);
      }
    }
  }
};

template <int KIND, bool D3>
__global__ void __launch_bounds__(128) k_resample(Shape s, const bf16* __restrict__ in, bf16* out,
                                                  const bf16* __restrict__ mask) {
  constexpr bool coarse = KIND == 0 || KIND == 3;  // the output lies on the coarse grid
  const int nxo = coarse ? s.nxc : s.nxf, nyo = coarse ? s.nyc : s.nyf, nzo = coarse ? s.nzc : s.nzf;
  const int nxi = coarse ? s.nxf : s.nxc, nyi = coarse ? s.nyf : s.nyc, nzi = coarse ? s.nzf : s.nzc;
  const int t = blockIdx.y * 128 + threadIdx.x;
  if (t >= nxo * s.C8) return;
  const int i = s.shift >= 0 ? t >> s.shift : t / s.C8;
  const int c = (t - i * s.C8) * 8;
  const int row = blockIdx.x;  // (sample * nzo + k) * nyo + j
  const int j = row % nyo, bk = row / nyo;
  const int k = D3 ? bk % nzo : 0, b = D3 ? bk / nzo : bk;
  const Taps<KIND> X(i, s.nxf), Y(j, s.nyf), Z(D3 ? k : 0, D3 ? s.nzf : 1);
  constexpr int NZ = D3 ? Taps<KIND>::n : 1, n = Taps<KIND>::n;
  constexpr int z1 = KIND == 0 || KIND == 3 ? 1 : 0;  // the one tap of a missing axis
  const bf16* ib = in + (long long)b * nxi * nyi * nzi * s.ldi + s.i_off + c;
  float acc[8] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
#pragma unroll
  for (int z = 0; z < NZ; ++z) {
    const int zz = D3 ? z : z1;
    uint4 u[n][n];
#pragma unroll
    for (int y = 0; y < n; ++y)
#pragma unroll
      for (int x = 0; x < n; ++x)
        u[y][x] = __ldg(reinterpret_cast<const uint4*>(
            ib + (X.at[x] + (long long)nxi * (Y.at[y] + (long long)nyi * (D3 ? Z.at[zz] : 0))) * s.ldi));
#pragma unroll
    for (int y = 0; y < n; ++y)
#pragma unroll
      for (int x = 0; x < n; ++x) {
        if (!(X.ok[x] && Y.ok[y] && (!D3 || Z.ok[zz]))) continue;
        float w;
        if (KIND == 2)
          w = D3 ? 0.125f : 1.f;
        else
          w = X.w[x] * Y.w[y] * (D3 ? Z.w[zz] : 1.f);
        if (KIND == 1) w /= X.s[x] * Y.s[y] * (D3 ? Z.s[zz] : 1.f);
        float v[8];
        unpack(u[y][x], v);
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] = fmaf(w, v[q], acc[q]);
      }
  }
  if (KIND == 0) {
    const float inv = 1.f / (fw_sum(i, s.nxf) * fw_sum(j, s.nyf) * (D3 ? fw_sum(k, s.nzf) : 1.f));
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] *= inv;
  } else if (KIND == 2 && !D3) {
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] *= 0.25f;
  }
  const long long r = (long long)row * nxo + i;
  if (mask) {
    float m[8];
    unpack(__ldg(reinterpret_cast<const uint4*>(mask + r * s.ldm + s.m_off + c)), m);
#pragma unroll
    for (int q = 0; q < 8; ++q)
      if (!(m[q] > 0.f)) acc[q] = 0.f;
  }
  uint4* o = reinterpret_cast<uint4*>(out + r * s.ldo + s.o_off + c);
  if (s.accum) {
    float old[8];
    unpack(*o, old);
#pragma unroll
    for (int q = 0; q < 8; ++q) acc[q] += old[q];
  }
  __align__(16) __nv_bfloat162 p[4];
#pragma unroll
  for (int q = 0; q < 4; ++q) p[q] = __floats2bfloat162_rn(acc[2 * q], acc[2 * q + 1]);
  *o = *reinterpret_cast<const uint4*>(p);
}
}  // namespace

void launch_resample(Ctx& ctx, const char* name, int mode, int transpose, const int* fine, const int* coarse, bool d3,
                     int B, int C, const bf16* in, int ldi, int i_off, bf16* out, int ldo, int o_off, int accum,
                     const bf16* mask, int ldm, int m_off) {
  if (C % 8 || ldi % 8 || i_off % 8 || ldo % 8 || o_off % 8 || (mask && (ldm % 8 || m_off % 8)))
    throw std::runtime_error("resample: channel layout not aligned");
  Shape s{};
  s.nxf = fine[0];
  s.nyf = fine[1];
  s.nzf = d3 ? fine[2] : 1;
  s.nxc = coarse[0];
  s.nyc = coarse[1];
  s.nzc = d3 ? coarse[2] : 1;
  s.B = B;
  s.C8 = C / 8;
  s.shift = -1;
  for (int q = 0; q < 16; ++q)
    if (s.C8 == 1 << q) s.shift = q;
  s.ldi = ldi;
  s.i_off = i_off;
  s.ldo = ldo;
  s.o_off = o_off;
  s.ldm = ldm;
  s.m_off = m_off;
  s.accum = accum;
  const bool to_coarse = (mode == 0) != (transpose != 0);
  const long long nf = (long long)s.nxf * s.nyf * s.nzf, nc = (long long)s.nxc * s.nyc * s.nzc;
  const long long rows = (long long)B * (to_coarse ? (long long)s.nyc * s.nzc : (long long)s.nyf * s.nzf);
  const long long cells = (long long)(to_coarse ? s.nxc : s.nxf) * s.C8;
  if (rows >= (1LL << 31) || cells >= 128LL * 65535) throw std::runtime_error("resample: batch too large");
  const dim3 grid((unsigned)rows, (unsigned)((cells + 127) / 128));
  const double bytes = (double)B * (nf + nc) * C * 2.0;
  const int kind = mode == 0 ? (transpose ? 1 : 0) : (transpose ? 3 : 2);
#define HZ_RESAMPLE(K)                                                                                \
  if (kind == K) {                                                                                    \
    if (d3)                                                                                           \
      HZ_LAUNCH(ctx, name, bytes, (k_resample<K, true>), grid, 128, 0, s, in, out, mask);             \
    else                                                                                              \
      HZ_LAUNCH(ctx, name, bytes, (k_resample<K, false>), grid, 128, 0, s, in, out, mask);            \
  }
  HZ_RESAMPLE(0)
  HZ_RESAMPLE(1)
  HZ_RESAMPLE(2)
  HZ_RESAMPLE(3)
#undef HZ_RESAMPLE
}

}  // namespace hz
