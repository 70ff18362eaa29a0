// IEEE double products on the integer pipe.
//
// GB300 issues one FP64 warp instruction per SM every 16 cycles while the four
// schedulers could issue 64 others in that time, so a kernel whose FP64
// instructions are half products and half sums (the reference's rounding
// allows no fused multiply-add) leaves most issue slots idle.  soft_mul forms
// the correctly rounded (nearest, ties to even) product of two doubles from
// four 32 x 32 -> 64 bit integer products, equal bit for bit to the hardware
// product (1.3e9 random and special pairs), and leaves the FP64 pipe to the
// sums.  Measured in SM cycles per warp instruction: DMUL and DADD 19.1 each,
// soft_mul about 12 alone, soft_mul with a DADD on its result 19.2 against DMUL +
// DADD 38.2: the products cost nothing beside the sums.  The ALU pipe bounds it
// (some 19 operations; the multiplications and one shift, as a product, run
// beside it); more shifts as products (14.7) or additions as multiply-adds
// (13.1) were slower.
//
// The second factor has an exponent in [kSoftLo, kSoftLo + 256) (magnitudes
// 2^-128 .. 2^128: coefficients, fluxes, thicknesses) and the product one from
// 2^-895 to 2^129, which leaves the first factor any normal number that a
// decaying tracer tail runs through; others -- subnormals, infinities, NaN, the
// rest -- set a bit of `bad` and the caller forms the products in hardware.  A
// zero first factor is common (tracer plateaus, still water) and gives +0 in
// line: a branch that single lanes of most warps take would make the warp issue
// the sums behind it twice, once for each side.  The sign of such a zero is
// not kept; the sums it enters start from +0 and cannot tell.
#pragma once

#include <cstdint>

#include "device.cuh"

namespace mpaso {

constexpr uint32_t kExp = 0x7ff00000u;     // exponent field of a high word
constexpr uint32_t kSignExp = 0xfff00000u;
constexpr uint32_t kSoftLo = 895u << 20;   // lowest exponent of a factor, at its place
constexpr uint32_t kSoftMin = 128u << 20;  // lowest exponent of a product, likewise
constexpr uint32_t kSoftOut = 0x40000000u; // set from 1024 exponents above that on, and by a borrow

// A factor prepared once for several products: significand shifted up by 10
// bits (so the cross products cannot overflow 64 bits), and sign and exponent
// fields less the bias and kSoftMin (two sign bits add to the product's).
struct SoftFactor {
  uint32_t h, l, x;
};
// The words of a double, hidden from the optimiser, which would turn tests of
// them back into floating-point comparisons on the FP64 pipe.
__device__ __forceinline__ void soft_words(double x, uint32_t &hi, uint32_t &lo) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
}
__device__ __forceinline__ bool nonfinite(double x) {
  uint32_t hi, lo;
  soft_words(x, hi, lo);
  return (hi & kExp) == kExp;
}
__device__ __forceinline__ SoftFactor soft_factor(double b, uint32_t &bad) {
  uint32_t hi, lo;
  soft_words(b, hi, lo);
  SoftFactor f;
  f.h = (__funnelshift_l(lo, hi, 10) & 0x3fffffffu) | 0x40000000u;
  f.l = lo << 10;
  f.x = (hi & kSignExp) - (1023u << 20) - kSoftMin;
  bad |= ((hi & kExp) - kSoftLo) & 0xf0000000u;  // an exponent outside borrows into or reaches these bits
  return f;
}

__device__ __forceinline__ double soft_mul(double a, const SoftFactor &f, uint32_t &bad) {
  uint32_t hi, al;
  soft_words(a, hi, al);
  const bool zero = ((hi & 0x7fffffffu) | al) == 0;
  // sign and exponent of the product less kSoftMin, valid below 1024.  With the
  // factor's window a subnormal `a` stays below 0, an infinity or NaN above 1024.
  const uint32_t x = (hi & kSignExp) + f.x;
  bad |= zero ? 0u : x & kSoftOut;
  const uint32_t ah = (hi & 0xfffffu) | 0x100000u;
  // P = a f 2^10 = top 2^64 + lo(t2) 2^32 + lo(t0), in [2^114, 2^116)
  const uint64_t t0 = (uint64_t)al * f.l;
  const uint64_t t1 = (uint64_t)ah * f.l + (t0 >> 32);
  const uint64_t t2 = (uint64_t)al * f.h + t1;  // < 2^63 + 2^54
  const uint64_t top = (uint64_t)ah * f.h + (t2 >> 32);
  const uint32_t th = (uint32_t)(top >> 32), tl = (uint32_t)top, tr = (uint32_t)t2;
  const uint32_t n = th >> 19;  // 1 where the significands' product is >= 2
  const uint32_t s = 2 - n;     // brings the leading bit to the implicit bit's place
  const uint32_t mh = __funnelshift_l(tl, th, s), ml = __funnelshift_l(tr, tl, s), r = tr * (4 - 2 * n);
  // round to nearest even: r + 0x7fffffff + (odd | sticky) carries exactly when
  // the discarded part exceeds a half, or equals it and the result is odd
  const uint32_t inc = ((ml | min((uint32_t)t0, 1u)) & 1u) + 0x7fffffffu;
  // to add to the significand, whose leading bit counts one
  const uint32_t e = x + (kSoftMin - (1u << 20)) + n * 0x100000u;
  uint32_t oh, ol;
  asm("{\n\t.reg .u32 t;\n\tadd.cc.u32 t, %2, %3;\n\taddc.cc.u32 %0, %4, 0;\n\taddc.u32 %1, %5, %6;\n\t}"
      : "=r"(ol), "=r"(oh)
      : "r"(r), "r"(inc), "r"(ml), "r"(mh), "r"(e));
  return __hiloint2double(zero ? 0 : (int)oh, zero ? 0 : (int)ol);
}

// a a: the factor is the number itself, which may be zero and anything with a
// normal square (exponents 520 .. 1519).
__device__ __forceinline__ double soft_square(double a, uint32_t &bad) {
  uint32_t hi, lo;
  soft_words(a, hi, lo);
  const bool zero = ((hi & 0x7fffffffu) | lo) == 0;
  bad |= !zero && ((hi & kExp) >> 20) - 520u >= 1000u ? 1u : 0u;
  // the number scaled to an exponent of 1023, whose square's exponent is put back
  const double m = __hiloint2double((int)((hi & 0xfffffu) | (1023u << 20)), (int)lo);
  uint32_t none = 0;
  const double r = soft_mul(m, soft_factor(m, none), none);
  const uint32_t e = ((hi & kExp) - (1023u << 20)) * 2u;
  uint32_t rh, rl;
  soft_words(r, rh, rl);
  return zero ? 0.0 : __hiloint2double((int)(rh + e), (int)rl);
}

// The product where soft_mul's window does not hold.  A call, not inlined:
// few warps need it, and the compiler turns a plain branch around an inlined
// multiplication into a predicated one, which occupies the FP64 pipe for the
// whole warp even where no lane takes it.
// A zero times a finite number, the whole of water at rest, stays off that pipe
// (level-6 ocean at rest, 60 x 3: 7.74 -> 6.55 ms per step, in motion 5.73).
static __device__ __noinline__ double product_hw(double a, double b) { return a * b; }
static __device__ __noinline__ double product_outside(double a, double b) {
  uint32_t ah, al, bh, bl;
  soft_words(a, ah, al);
  soft_words(b, bh, bl);
  const bool zero = ((ah & 0x7fffffffu) | al) == 0 || ((bh & 0x7fffffffu) | bl) == 0;
  if (zero && (ah & kExp) != kExp && (bh & kExp) != kExp) return __hiloint2double((int)((ah ^ bh) & 0x80000000u), 0);
  return product_hw(a, b);
}

// One product on the integer pipe.
__device__ __forceinline__ double mul_int(double a, double b) {
  uint32_t bad = 0;
  const SoftFactor f = soft_factor(b, bad);
  double r = soft_mul(a, f, bad);
  if (bad) r = product_outside(a, b);
  return r;
}

// A sum of up to 15 products on the integer pipe, where it may be rounded as a
// whole: 64-bit fixed point under the largest exponent so far (the accumulator
// is shifted down when a term with a larger one comes).  A term is the
// product's leading 58 bits or more, cut below 2^-57 of the largest term, so the
// sum's error is below that of a chain of fused multiply-adds, which rounds
// every partial sum to 53 bits (random sums of ten, of the largest term: at most
// 6.9e-16 against 2.0e-15; exponents over 2^60: 2.8e-16 against 9.9e-16).
struct FixedFactor {  // one factor of several terms
  uint32_t h, l, hi;
  __device__ __forceinline__ explicit FixedFactor(double b) {
    uint32_t lo;
    soft_words(b, hi, lo);
    h = (__funnelshift_l(lo, hi, 10) & 0x3fffffffu) | 0x40000000u, l = lo << 10;
  }
};
struct FixedSum {
  int64_t acc = 0;
  uint32_t top = 0;  // largest sum of two biased exponents, in units of 2^20
  uint32_t big = 0, low = 0;  // largest high word of an |a|; its low words' bits together
  __device__ __forceinline__ void add(double a, const FixedFactor &b) {
    uint32_t hi, al;
    soft_words(a, hi, al);
    const uint32_t mag = hi & 0x7fffffffu;
    big = max(big, mag), low |= al;
    const uint32_t x = (mag >> 20) + ((b.hi & kExp) >> 20);
    const uint32_t ah = (hi & 0xfffffu) | 0x100000u;
    const uint64_t t0 = (uint64_t)al * b.l;
    const uint64_t t1 = (uint64_t)ah * b.l + (t0 >> 32);
    const uint64_t t2 = (uint64_t)al * b.h + t1;
    const uint64_t t3 = (uint64_t)ah * b.h + (t2 >> 32);
    // a b 2^10 = t3 2^64 + ..; v = significands' product / 2^47, in [2^57, 2^59)
    const uint64_t v = ((uint64_t)__funnelshift_l((uint32_t)t3, (uint32_t)(t3 >> 32), 7) << 32) |
                       __funnelshift_l((uint32_t)t2, (uint32_t)t3, 7);
    const uint32_t m = max(top, x);
    const int64_t s = (int32_t)(hi ^ b.hi) >> 31;
    acc = (acc >> min(m - top, 63u)) + ((int64_t)(v >> min(m - x, 63u)) ^ s) - s;
    top = m;
  }
  // Whether some a is not a zero.
  __device__ __forceinline__ bool any() const { return (big | low) != 0; }
  // Whether the exponents were such that the sum holds: no a is infinite or NaN,
  // and the largest term is far above what zeros and subnormals count as, which
  // is a number of exponent 0 -- as an a beside any b (the first condition), and
  // as a b beside the largest a.
  __device__ __forceinline__ bool valid() const {
    return top - 1280u < 1600u && big < kExp && (big >> 20) + 58u <= top;
  }
  __device__ __forceinline__ double value() const {
    const double r = (double)acc;  // rounded to nearest
    return acc == 0 ? 0.0 : __hiloint2double(__double2hiint(r) + (int)((top - 2103u) << 20), __double2loint(r));
  }
};

// Rare work of the high-order flux, called so that warps without it skip it: inlined, it becomes
// predicated instructions, which occupy the FP64 pipe all the same (11 a
// thread beside the 36 sums of three tracers).
static __device__ __noinline__ double masked_weight(double f, int mask) { return f * (double)mask; }
static __device__ __noinline__ double add_centred_flux(double flx, double dv, double f, double t1, double t2) {
  return flx + (dv * 0.5) * f * (t1 + t2);
}

// num / den where few lanes need it (a call, as product_outside).
static __device__ __noinline__ double rare_quotient(double num, double den) { return num / den; }

// min(1, max(0, num / den)) for den > 0, divided only strictly inside (0, 1):
// num <= 0 gives 0 and num >= den gives 1 exactly as the clamped quotient does.
__device__ __forceinline__ double clamp_quotient(double num, double den) {
  double r = dgt0(num) ? 1.0 : 0.0;
  if (!dgt0(den) || (dgt0(num) && dkey(num) < dkey(den))) r = dclamp01(rare_quotient(num, den));
  return r;
}

}  // namespace mpaso
