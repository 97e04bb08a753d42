// Checks of single launches of the library against definitions on the host, for
// test_gpu_kernels.py:
//   fine NX NY NZ ORDER ADJOINT HX HY HZ    the integer-pipe operator, all modes and inputs
//   band N BANDWIDTH COLUMNS                the cluster against the cooperative band solve
//   wgrad NX NY NZ BATCH CIN COUT           the weight gradient (NZ > 1: 27 taps)
// Prints what failed; 0 if nothing did.
#include <cmath>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <random>
#include <vector>

#include <cuda_bf16.h>

#include "hz_kernels.cuh"
#include "hz_learn.h"

using namespace hz;
typedef long double real;
static int failed = 0;
static void ok(cudaError_t e, const char* what) {
  if (e == cudaSuccess) return;
  printf("%s: %s\n", what, cudaGetErrorString(e));
  exit(2);
}
template <typename T> static T* up(const std::vector<T>& v) {
  T* p = nullptr;
  ok(cudaMalloc((void**)&p, v.size() * sizeof(T)), "alloc");
  ok(cudaMemcpy(p, v.data(), v.size() * sizeof(T), cudaMemcpyHostToDevice), "upload");
  return p;
}
template <typename T> static std::vector<T> down(const T* p, size_t n) {
  std::vector<T> v(n);
  ok(cudaDeviceSynchronize(), "run");
  ok(cudaMemcpy(v.data(), p, n * sizeof(T), cudaMemcpyDeviceToHost), "download");
  return v;
}

// Bounds as derived in test_gpu_fine_fixed.py: 48 u of the row's |a| times the largest component
// around the node for the product, one rounding more for b - a, and the sweep's own.
static void fine(char** a) {
  const Grid g{atoi(a[0]), atoi(a[1]), atoi(a[2]), (long long)atoi(a[0]) * atoi(a[1]) * atoi(a[2])};
  const int order = atoi(a[3]), dim = g.nz > 1 ? 3 : 2;
  const double h[3] = {atof(a[5]), atof(a[6]), atof(a[7])};
  const double BC = order == 1 ? 1.0 : 2.0, weight = 0.8;
  const long long N = g.N, ld = N + 5;
  const int R = 4;
  FineOp op{};
  op.g = g;
  op.adj = atoi(a[4]);
  for (int d = 0; d < 3; ++d) {
    op.o[d] = 1.0 / (h[d] * h[d]);
    op.b[d] = BC * op.o[d];
  }
  std::mt19937_64 rng(N);
  std::normal_distribution<double> nd;
  std::uniform_real_distribution<double> ud;
  std::vector<double> m(N), ga(N);
  for (auto& v : m) v = 0.1 + 0.2 * ud(rng);
  for (auto& v : ga) v = 0.3 * ud(rng);
  Ctx ctx;
  double2 *dH, *dSH, *iSH;
  FixedRefs* refs;
  int4* words;
  for (double2** p : {&dH, &dSH, &iSH}) ok(cudaMalloc((void**)p, N * 16), "alloc");
  ok(cudaMalloc((void**)&refs, 2 * sizeof(FixedRefs)), "alloc");
  ok(cudaMalloc((void**)&words, N * 16), "alloc");
  launch_fine_setup(ctx, g, dim, h, 1.0 / h[0], 0.0, 0.5, BC, 1, 1, up(m), up(ga), dH, dSH, iSH, refs);
  launch_diag_fixed(ctx, op, dSH, refs + 1, words);
  if (!fine_fixed_fits(op, down(refs, 2)[1].exponent)) {
    printf("the operator does not fit\n");
    failed = 1;
    return;
  }
  const std::vector<double2> d = down(dSH, N), di = down(iSH, N);
  // noise, noise that decays over the grid, a wave, few values
  std::vector<double2> x(ld * R), b(ld * R);
  for (int c = 0; c < R; ++c)
    for (long long p = 0; p < N; ++p) {
      const int i = p % g.nx, j = p / g.nx % g.ny, k = p / ((long long)g.nx * g.ny);
      double2 v = make_double2(nd(rng), nd(rng));
      if (c == 1) v.x *= std::exp2(-60.0 * p / N), v.y *= std::exp2(-60.0 * p / N);
      if (c == 2) v = make_double2(std::cos(0.6 * i + 0.4 * j + 0.5 * k), std::sin(0.6 * i + 0.4 * j + 0.5 * k));
      if (c == 3 && rng() % 50) v = make_double2(0.0, 0.0);
      x[c * ld + p] = v;
      b[c * ld + p] = make_double2(nd(rng), nd(rng));
    }
  std::vector<float2> xf(x.size());
  for (size_t q = 0; q < x.size(); ++q) xf[q] = make_float2((float)x[q].x, (float)x[q].y);
  const int cols[R] = {2, 0, 3, 1};
  const int* dcols = up(std::vector<int>(cols, cols + R));
  std::vector<double> sig{0.7, 3.0e-9, 1.0, 5.0e11};
  const double* dsig = up(sig);
  const double2 *dx = up(x), *db = up(b);
  const float2* dxf = up(xf);
  const double2 mark = make_double2(-7.0, 7.0);
  double2* y = up(std::vector<double2>(ld * R, mark));
  const FixedDiag fd{refs + 1, words};
  const char* names[5] = {"apply", "residual", "jacobi", "apply of FP32", "residual of FP32"};
  for (int t = 0; t < 5; ++t) {
    const bool f32 = t > 2;
    const int mode = t == 2 ? MODE_JACOBI : t % 3 == 0 ? MODE_APPLY : MODE_RESID;
    ok(cudaMemcpy(y, std::vector<double2>(ld * R, mark).data(), ld * R * 16, cudaMemcpyHostToDevice), "clear");
    if (f32)
      launch_fine_fixed<float>(ctx, mode, op, dSH, fd, dxf, db, y, ld, dcols, R);
    else
      launch_fine_fixed<double>(ctx, mode, op, dSH, fd, dx, db, y, ld, dcols, R, iSH, weight);
    const std::vector<double2> got = down(y, ld * R);
    for (int c = 0; c < R; ++c) {
      double worst = 0.0;
      long long at = -1;
      for (long long p = 0; p < ld; ++p) {
        const double2 z = got[c * ld + p];
        if (p >= N) {
          if (memcmp(&z, &mark, 16)) worst = INFINITY, at = p;
          continue;
        }
        const int pos[3] = {(int)(p % g.nx), (int)(p / g.nx % g.ny), (int)(p / ((long long)g.nx * g.ny))};
        const int n[3] = {g.nx, g.ny, g.nz};
        const long long st[3] = {1, g.nx, (long long)g.nx * g.ny};
        auto X = [&](long long q) {
          return f32 ? make_double2(xf[c * ld + q].x, xf[c * ld + q].y) : x[c * ld + q];
        };
        const double dy = op.adj ? -d[p].y : d[p].y;
        const double2 xp = X(p);
        real re = (real)d[p].x * xp.x - (real)dy * xp.y, im = (real)d[p].x * xp.y + (real)dy * xp.x;
        real row = std::hypot((real)d[p].x, (real)d[p].y), largest = std::max(std::fabs(xp.x), std::fabs(xp.y));
        for (int e = 0; e < dim; ++e)
          for (int s = -1; s <= 1; s += 2) {
            const int q = pos[e] + s;
            if (q < 0 || q >= n[e]) continue;
            const int on = op.adj ? q : pos[e];  // the boundary row whose coefficient it is
            const double cf = on == 0 || on == n[e] - 1 ? op.b[e] : op.o[e];
            const double2 v = X(p + s * st[e]);
            re -= (real)cf * v.x;
            im -= (real)cf * v.y;
            row += cf;
            largest = std::max(largest, (real)std::max(std::fabs(v.x), std::fabs(v.y)));
          }
        const real u = std::ldexp((real)1, -53);
        real bound = 48 * u * row * largest;
        if (mode != MODE_APPLY) {
          const double2 bb = b[c * ld + p];
          re = bb.x - re;
          im = bb.y - im;
          bound += u * (std::fabs(re) + std::fabs(im)) + u * bound;
        }
        if (mode == MODE_JACOBI) {
          const real ir = di[p].x, ii = op.adj ? -di[p].y : di[p].y, ad = std::fabs(ir) + std::fabs(ii);
          const real qr = weight * (ir * re - ii * im), qi = weight * (ir * im + ii * re);
          bound = weight * ad * (bound + 4 * u * (std::fabs(re) + std::fabs(im))) +
                  2 * u * (std::fabs(xp.x) + std::fabs(xp.y) + std::fabs(qr) + std::fabs(qi));
          re = xp.x + qr;
          im = xp.y + qi;
        }
        const real err = std::max(std::fabs(z.x - re), std::fabs(z.y - im));
        const double ratio = bound > 0 ? (double)(err / bound) : (err > 0 ? INFINITY : 0.0);
        if (!(ratio <= worst)) worst = ratio, at = p;
      }
      if (!(worst <= 1.0)) {
        printf("%s, column %d: %.3g of the bound at node %lld\n", names[t], c, worst, at);
        failed = 1;
      }
    }
    if (mode != MODE_APPLY) continue;
    // scaled by powers of two: the same bits
    FineOp sop = op;
    sop.sig = dsig;
    sop.sig_stride = 1;
    if (f32)
      launch_fine_fixed<float>(ctx, mode, sop, dSH, fd, dxf, nullptr, y, ld, dcols, R);
    else
      launch_fine_fixed<double>(ctx, mode, sop, dSH, fd, dx, nullptr, y, ld, dcols, R);
    const std::vector<double2> sc = down(y, ld * R);
    for (int c = 0; c < R; ++c)
      for (long long p = 0; p < N; ++p) {
        const int k = std::ilogb(sig[c]);
        const double2 w = make_double2(std::ldexp(got[c * ld + p].x, k), std::ldexp(got[c * ld + p].y, k));
        if (sc[c * ld + p].x != w.x || sc[c * ld + p].y != w.y) {
          printf("%s scaled, column %d, node %lld\n", names[t], c, p);
          failed = 1;
          break;
        }
      }
  }
}

template <typename T> static void band_as(const BandSolveOps& plan, int nrhs) {
  const long long N = plan.N;
  std::mt19937_64 rng(7);
  std::normal_distribution<double> nd;
  std::vector<cplx<T>> b(N * nrhs);
  for (auto& v : b) v = mk<T>((T)nd(rng), (T)nd(rng));
  std::vector<int> cols(nrhs);
  for (int c = 0; c < nrhs; ++c) cols[c] = nrhs - 1 - c;
  const int* dc = up(cols);
  const cplx<T>* db = up(b);
  cplx<T>* x = up(std::vector<cplx<T>>(N * nrhs, mk<T>(9, 9)));
  double2* work = up(std::vector<double2>(3 * N * nrhs));
  Ctx ctx;
  BandSolveOps coop = plan, cluster = plan;
  coop.cluster = coop.resident = 0;
  cluster.resident = 1 << 20;  // whatever the cost rule says
  launch_band_solve<T>(ctx, coop, db, x, N, dc, nrhs, work);
  const auto xa = down(x, N * nrhs);
  ok(cudaMemset(x, 0, N * nrhs * sizeof(cplx<T>)), "clear");
  launch_band_solve<T>(ctx, cluster, db, x, N, dc, nrhs, work);
  const auto xb = down(x, N * nrhs);
  if (memcmp(xa.data(), xb.data(), xa.size() * sizeof(cplx<T>))) {
    printf("%d-byte columns differ\n", (int)sizeof(cplx<T>));
    failed = 1;
  }
}

static void band(char** a) {
  const long long N = atoi(a[0]);
  const int kl = atoi(a[1]), nrhs = atoi(a[2]);
  const long long ldab = 3LL * kl + 1;
  std::mt19937_64 rng(N);
  std::normal_distribution<double> nd;
  std::vector<std::complex<double>> ab(ldab * N, 0.0);
  for (long long j = 0; j < N; ++j)
    for (long long i = std::max(0LL, j - kl); i <= std::min(N - 1, j + kl); ++i)
      if (i == j || rng() % 3) ab[2 * kl + i - j + j * ldab] = {nd(rng) + (i == j ? 2.0 : 0.0), nd(rng)};
  std::vector<int> piv(N);
  if (band_lu_factor(N, kl, kl, ab.data(), piv.data())) {
    printf("singular\n");
    failed = 1;
    return;
  }
  BandSolveOps op;
  std::vector<std::complex<double>> T, G;
  band_block_operators(N, kl, kl, ab.data(), piv.data(), kl, op.blocks, T, G);
  op.N = N;
  op.T = reinterpret_cast<double2*>(up(T));
  op.G = reinterpret_cast<double2*>(up(G));
  op.dblocks = up(op.blocks);
  plan_band_solve<double>(op);
  if (!op.cluster) {
    printf("no clusters\n");
    failed = 1;
    return;
  }
  band_as<double>(op, nrhs);
  plan_band_solve<float>(op);
  band_as<float>(op, nrhs);
}

// Operands are exact BF16 numbers and their products exact in FP32.  The sums take at most one
// rounding per 16 nodes and one per CTA (two segments of a row), each within 2^-23 of a partial
// sum; those are no larger than the result's norm for operands of random sign.
static void wgrad(char** a) {
  const int nx = atoi(a[0]), ny = atoi(a[1]), nz = atoi(a[2]), B = atoi(a[3]), Cin = atoi(a[4]), Cout = atoi(a[5]);
  const int taps = nz > 1 ? 27 : 9, ldi = Cin + 8, ldd = (Cout + 15) / 16 * 16 + 8, off = 8;
  const long long nodes = (long long)nx * ny * nz * B;
  std::mt19937_64 rng(nodes);
  std::normal_distribution<float> nd;
  std::vector<__nv_bfloat16> in(nodes * ldi), dout(nodes * ldd);
  for (auto& v : in) v = __float2bfloat16(nd(rng));
  for (auto& v : dout) v = __float2bfloat16(nd(rng));
  std::vector<float> zero((size_t)Cout * taps * Cin);
  WgradTc w{nx, ny, nz, nodes, Cin, up(in), ldi, Cout, up(dout), ldd, off, up(zero)};
  Ctx ctx;
  wgrad_launch(ctx, "check", w, taps);
  const auto got = down(w.dw, zero.size());
  std::vector<double> fi(in.size()), fo(dout.size());
  for (size_t q = 0; q < in.size(); ++q) fi[q] = __bfloat162float(in[q]);
  for (size_t q = 0; q < dout.size(); ++q) fo[q] = __bfloat162float(dout[q]);
  std::vector<double> ref(zero.size(), 0.0);
  for (int s = 0; s < B; ++s)
    for (int k = 0; k < nz; ++k)
      for (int j = 0; j < ny; ++j)
        for (int i = 0; i < nx; ++i) {
          const long long p = i + (long long)nx * (j + (long long)ny * (k + (long long)nz * s));
          for (int t = 0; t < taps; ++t) {
            const int ii = i + t % 3 - 1, jj = j + t / 3 % 3 - 1, kk = k + (taps == 27 ? t / 9 - 1 : 0);
            if (ii < 0 || ii >= nx || jj < 0 || jj >= ny || kk < 0 || kk >= nz) continue;
            const long long q = ii + (long long)nx * (jj + (long long)ny * (kk + (long long)nz * s));
            for (int co = 0; co < Cout; ++co) {
              const double v = fo[p * ldd + off + co];
              double* r = &ref[((size_t)co * taps + t) * Cin];
              for (int ci = 0; ci < Cin; ++ci) r[ci] += v * fi[q * ldi + ci];
            }
          }
        }
  double e = 0.0, n = 0.0;
  for (size_t q = 0; q < ref.size(); ++q) {
    e += (got[q] - ref[q]) * (got[q] - ref[q]);
    n += ref[q] * ref[q];
  }
  const double bound = (nodes / 16.0 + 2.0 * ny * nz * B) * std::ldexp(1.0, -23);
  if (!(std::sqrt(e) <= bound * std::sqrt(n))) {
    printf("error %.3g of the norm, bound %.3g\n", std::sqrt(e / n), bound);
    failed = 1;
  }
}

int main(int argc, char** argv) {
  if (argc == 10 && !strcmp(argv[1], "fine")) fine(argv + 2);
  else if (argc == 5 && !strcmp(argv[1], "band")) band(argv + 2);
  else if (argc == 8 && !strcmp(argv[1], "wgrad")) wgrad(argv + 2);
  else return 3;
  return failed;
}
