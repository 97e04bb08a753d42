"""The integer-pipe FP64 sums of the Gram-Schmidt kernels (csrc/hz_fixed.cuh) on the
host, against quadruple precision.

Bounds, from the definitions.  With references 2^(E - 1022) above every value, a 58-bit
value is off by less than 2^-58 of its reference (57 bits: 2^-57), the dropped product of
the low limbs is at most 2^-60 (2^-59), and folding the limbs adds half of 2^-58 (2^-57).
So four complex products are within (8 (2 2^-58 + 2^-60) + 2^-59) of the references'
product, and K terms of an update within 2 K (2^-57 + 2^-58 + 2^-59) + 2^-58."""
import shutil
import subprocess
from pathlib import Path

import pytest

CSRC = Path(__file__).resolve().parent.parent / "helmholtz.jl_gb300" / "csrc"

PROGRAM = r"""
#include <cmath>
#include <cstdio>
#include <cstring>
#include <random>
#include "hz_fixed.cuh"
using namespace hz;
#ifdef __aarch64__
typedef long double quad;
#else
typedef __float128 quad;
#endif
static uint32_t hi32(double v) { uint64_t u; memcpy(&u, &v, 8); return (uint32_t)(u >> 32); }
static uint32_t lo32(double v) { uint64_t u; memcpy(&u, &v, 8); return (uint32_t)u; }
static int ex(double v) { return fixed_exponent(hi32(v)); }
static quad q_abs(quad a) { return a < 0 ? -a : a; }
static quad p2(int e) { quad r = 1; for (; e > 0; --e) r *= 2; for (; e < 0; ++e) r /= 2; return r; }
static std::mt19937_64 rng(1);
static double draw(int base, int spread) {
  // every third value has an extreme mantissa; some are zero or subnormal
  const uint64_t k = rng() % 16;
  if (k == 0) return 0.0;
  if (k == 1) return -0.0;
  if (k == 2) return std::ldexp((double)(rng() % 4096), -1074);
  uint64_t m = rng() & 0xfffffffffffffull;
  if (k < 6) m = 0xfffffffffffffull;
  if (k == 6) m = 0;
  const uint64_t e = (uint64_t)(base - (int)(rng() % (spread + 1)));
  const uint64_t u = (rng() & 1) << 63 | e << 52 | m;
  double v; memcpy(&v, &u, 8); return v;
}
int main() {
  long long n = 0, bad = 0;
  const int bases[] = {kFixedMin, 200, 700, 1023, 1040, 1500, 2046};
  for (int ba : bases) for (int bb : bases) for (int spread : {0, 3, 20, 63, 62}) for (int it = 0; it < 400; ++it) {
    if (ba - spread < 1 || bb - spread < 1) continue;
    double v[16], w[16];
    int ev = 0, ew = 0;
    for (int q = 0; q < 8; ++q) { v[q] = draw(ba, spread); w[q] = draw(bb, spread); ev = std::max(ev, ex(v[q])); ew = std::max(ew, ex(w[q])); }
    if (!fixed_ref_ok(ev) || !fixed_ref_ok(ew) || !fixed_ok(ev + ew)) continue;
    FixedSum f{0, 0, 0, 0};
    quad xr = 0, xi = 0;
    for (int q = 0; q < 4; ++q) {
      auto fx = [](double a, int e) { return fixed_from<6>(hi32(a), lo32(a), e); };
      fixed_conj_mac(f, fx(v[2 * q], ev), fx(v[2 * q + 1], ev), fx(w[2 * q], ew), fx(w[2 * q + 1], ew));
      xr += (quad)v[2 * q] * w[2 * q] + (quad)v[2 * q + 1] * w[2 * q + 1];
      xi += (quad)v[2 * q] * w[2 * q + 1] - (quad)v[2 * q + 1] * w[2 * q];
    }
    uint64_t su = (uint64_t)fixed_scale_hi(ev + ew, 0) << 32; double sc; memcpy(&sc, &su, 8);
    const quad bound = (8 * (2 * p2(-58) + p2(-60)) + p2(-59)) * p2(ev - 1022) * p2(ew - 1022);
    const quad er = q_abs((quad)fixed_total(f.rh, f.rl) * sc - xr), ei = q_abs((quad)fixed_total(f.ih, f.il) * sc - xi);
    ++n; if (er > bound || ei > bound) { ++bad; if (bad < 4) printf("dot %d %d %d\n", ba, bb, spread); }
  }
  // update: K terms related to the largest one
  for (int K : {1, 2, 9, 16}) for (int ba : bases) for (int bb : bases) for (int spread : {0, 5, 40}) for (int it = 0; it < 200; ++it) {
    if (ba - spread < 1 || bb - spread < 1) continue;
    double h[32], v[32];
    int he[16], T = -(1 << 20), hm = -(1 << 20), vm = 0; bool ok = true;
    for (int s = 0; s < K; ++s) {
      for (int c = 0; c < 2; ++c) { h[2 * s + c] = draw(ba, spread); v[2 * s + c] = draw(bb, spread); }
      const int e = std::max(ex(h[2 * s]), ex(h[2 * s + 1]));
      const bool zero = h[2 * s] == 0 && h[2 * s + 1] == 0;
      ok = ok && (zero || fixed_ref_ok(e));
      he[s] = zero ? -(1 << 20) : e;
      hm = std::max(hm, he[s]);
      const int evs = std::max(ex(v[2 * s]), ex(v[2 * s + 1]));
      vm = std::max(vm, evs); T = std::max(T, he[s] + evs);
    }
    if (!ok || vm >= 0x7ff || T - hm < kFixedMin || !fixed_ok(T)) continue;
    FixedSum f{0, 0, 0, 0};
    quad xr = 0, xi = 0;
    for (int s = 0; s < K; ++s) {
      const bool zero = he[s] == -(1 << 20);
      const Fixed z{0, 0};
      const Fixed hr = zero ? z : fixed_from<6>(hi32(h[2 * s]), lo32(h[2 * s]), he[s]);
      const Fixed hi = zero ? z : fixed_from<6>(hi32(h[2 * s + 1]), lo32(h[2 * s + 1]), he[s]);
      const int e = T - he[s];
      fixed_cmac(f, hr, hi, fixed_from<7>(hi32(v[2 * s]), lo32(v[2 * s]), e), fixed_from<7>(hi32(v[2 * s + 1]), lo32(v[2 * s + 1]), e));
      xr += (quad)h[2 * s] * v[2 * s] - (quad)h[2 * s + 1] * v[2 * s + 1];
      xi += (quad)h[2 * s] * v[2 * s + 1] + (quad)h[2 * s + 1] * v[2 * s];
    }
    uint64_t su = (uint64_t)fixed_scale_hi(T, 1) << 32; double sc; memcpy(&sc, &su, 8);
    const quad bound = (2 * K * (p2(-57) + p2(-58) + p2(-59)) + p2(-58)) * p2(T - 2044);
    const quad er = q_abs((quad)fixed_total(f.rh, f.rl) * sc - xr), ei = q_abs((quad)fixed_total(f.ih, f.il) * sc - xi);
    ++n; if (er > bound || ei > bound) { ++bad; if (bad < 8) printf("update K %d %d %d %d\n", K, ba, bb, spread); }
  }
  printf("%lld sums, %lld outside\n", n, bad);
  return bad ? 1 : (n > 50000 ? 0 : 2);
}
"""


def test_fixed_sums(tmp_path):
    gxx, cuda = shutil.which("g++"), Path("/usr/local/cuda/include")
    if gxx is None or not cuda.exists():
        pytest.skip("needs g++ and the CUDA headers")
    src, exe = tmp_path / "fixed.cpp", tmp_path / "fixed"
    src.write_text(PROGRAM)
    subprocess.run([gxx, "-std=c++17", "-O2", f"-I{CSRC}", f"-I{cuda}", str(src), "-o", str(exe)], check=True)
    r = subprocess.run([str(exe)], capture_output=True, text=True)
    assert r.returncode == 0, r.stdout
