// FP64 products and sums on the integer pipe.
//
// GB300 issues two FP64 FMAs per clock and SM, 64 integer multiply-adds.  An FP64 value v is
// taken relative to a reference exponent E >= its own as a fixed-point number of 58 bits
// in two signed limbs, v = (hi 2^29 + lo) 2^(E - 1080) up to its 59th bit; a product of two
// values keeps hi hi, hi lo and lo hi (the dropped lo lo lies 60 bits below the product of
// the references, with either sign), and sums of such products are exact in 64-bit integers.
// Used with references local to a neighbourhood (128 nodes in hz_krylov.cu, a brick in
// hz_fine_fixed.cu), so an element's rounding is relative to its neighbours, 2^-58, not to a
// vector's largest element.
//
// Values this does not cover are told by their exponents: fixed_ok().
#pragma once

#include "hz_common.cuh"

namespace hz {

struct Fixed {
  int32_t hi, lo;
};

// exponent field (0: zero or subnormal, 0x7ff: Inf or NaN)
__host__ __device__ __forceinline__ int fixed_exponent(uint32_t vhi) { return (int)(vhi >> 20) & 0x7ff; }

// SHIFT 6: 58 bits, |hi| <= 2^29; SHIFT 7: 57 bits, |hi| <= 2^28, and one less in the scale.
// |lo| <= 2^28.  E is at least the value's exponent and at least kFixedMin, so that
// a subnormal value (its exponent field read as 0) is below the last bit.
static constexpr int kFixedMin = 64;

template <int SHIFT>
__host__ __device__ __forceinline__ Fixed fixed_from(uint32_t vhi, uint32_t vlo, int E) {
  const int e = fixed_exponent(vhi);
  const int sh = E - e + SHIFT;
  const uint64_t m = ((uint64_t)((vhi << 11) | (vlo >> 21) | (e ? 0x80000000u : 0u)) << 32) | (uint64_t)(vlo << 11);
  const uint64_t x = m >> (sh < 63 ? sh : 63);
  int32_t hi = (int32_t)(uint32_t)(x >> 29), lo = (int32_t)((uint32_t)x & 0x1fffffffu);
  const int32_t c = (int32_t)((uint32_t)x >> 28) & 1;
  hi += c;
  lo -= c << 29;
  const int32_t s = (int32_t)vhi >> 31;
  Fixed f;
  f.hi = (hi ^ s) - s;
  f.lo = (lo ^ s) - s;
  return f;
}

// A complex sum of products: h in units of 2^58, l in units of 2^29.
struct FixedSum {
  long long rh, rl, ih, il;
};
__host__ __device__ __forceinline__ void fixed_mac(long long& h, long long& l, Fixed a, Fixed b) {
  h += (long long)a.hi * b.hi;
  l += (long long)a.hi * b.lo;
  l += (long long)a.lo * b.hi;
}
__host__ __device__ __forceinline__ void fixed_msub(long long& h, long long& l, Fixed a, Fixed b) {
  h -= (long long)a.hi * b.hi;
  l -= (long long)a.hi * b.lo;
  l -= (long long)a.lo * b.hi;
}
// += conj(a) b.  Up to 15 of them fit (two products of at most 2^58 each per sum).
__host__ __device__ __forceinline__ void fixed_conj_mac(FixedSum& s, Fixed ar, Fixed ai, Fixed br, Fixed bi) {
  fixed_mac(s.rh, s.rl, ar, br);
  fixed_mac(s.rh, s.rl, ai, bi);
  fixed_mac(s.ih, s.il, ar, bi);
  fixed_msub(s.ih, s.il, ai, br);
}
// += a b.  Up to 31 with one 57-bit factor.
__host__ __device__ __forceinline__ void fixed_cmac(FixedSum& s, Fixed ar, Fixed ai, Fixed br, Fixed bi) {
  fixed_mac(s.rh, s.rl, ar, br);
  fixed_msub(s.rh, s.rl, ai, bi);
  fixed_mac(s.ih, s.il, ar, bi);
  fixed_mac(s.ih, s.il, ai, br);
}
__host__ __device__ __forceinline__ long long fixed_total(long long h, long long l) {
  return h + ((l + (1ll << 28)) >> 29);
}

// The sum's value is fixed_total 2^(Ea + Eb - 2102) for 58-bit factors with references Ea
// and Eb (one more with a 57-bit factor).  fixed_ok: that power of two and every product with
// a 63-bit total are normal FP64 numbers.
static constexpr int kFixedScale = 2102;
__host__ __device__ __forceinline__ bool fixed_ok(int Esum) { return Esum >= 1100 && Esum <= 3000; }
__host__ __device__ __forceinline__ bool fixed_ref_ok(int E) { return E >= kFixedMin && E < 0x7ff; }
// high word of 2^(Esum - kFixedScale + one)
__host__ __device__ __forceinline__ uint32_t fixed_scale_hi(int Esum, int one) {
  return (uint32_t)(Esum - kFixedScale + one + 1023) << 20;
}

}  // namespace hz
