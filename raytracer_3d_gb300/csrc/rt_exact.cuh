// rt_exact.cuh -- arithmetic of the bit-exact binary64 step: the reference's
// superbee flux (superbee_fluxes.f90:19-30) and divergence with the same
// rounding sequence as flux_fp64u (rt_step.cuh), but with the correctly
// rounded divisions done on the integer pipes.
//
// GB300 issues about 1.7 binary64 instructions per clock and SM against 64
// integer ones, so one binary64 instruction costs as much time as some 38
// integer instructions, and a correctly rounded binary64 division compiled
// to the binary64 pipe about ten of them.  The quotient here is a two-digit
// long division of the 53-bit significands by an approximate reciprocal
// (Knuth, The Art of Computer Programming vol. 2, 4.3.1, with digits
// estimated from a reciprocal instead of a trial division): the remainder is
// kept exactly, so rounding to nearest even from (quotient digits, remainder
// != 0) is exact -- the same bits as the division instruction sequence, held
// against it in tests/native/exact_div_check.cu.
#pragma once
#include <cstdint>
#include <cstring>

#include "rt_common.cuh"
#include "rt_fast.cuh"

// the host form's float reciprocal, moved by this many units in the last
// place (the check runs it at -1, 0 and 1: the device instruction's error)
#ifndef RT_RECIP_HOST_ULP
#define RT_RECIP_HOST_ULP 0
#endif

namespace rt {

// the reciprocal estimate: 2^32/x rounded down a little for x = 1.f, x in
// [1, 2) given by the top 24 bits of a significand (t in [2^23, 2^24)); at
// most 2^-21 below the true value in relative terms, never above it.  The
// divisor is rounded UP to the next value with 23 fraction bits and the
// float reciprocal (within 1 ulp) lowered by one more unit.
__host__ __device__ __forceinline__ uint32_t recip_estimate(uint32_t t) {
  const uint32_t fb = 0x3f800000u + (t - 0x800000u) + 1u;   // (t + 1) / 2^23 as binary32 bits; 2.0 at the top end
  float f, r;
#ifdef __CUDA_ARCH__
  f = __uint_as_float(fb);
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  const uint32_t rb = __float_as_uint(r) - 2u;
#else
  std::memcpy(&f, &fb, 4);
  r = 1.0f / f;
  uint32_t rb;
  std::memcpy(&rb, &r, 4);
  rb = rb - 2u + RT_RECIP_HOST_ULP;
#endif
  // r in [0.5, 1): significand with the hidden bit, as a 32-bit fraction;
  // r just below 0.5 (x = 2 lowered) has one exponent less
  const uint32_t m = (rb & 0x7fffffu) | 0x800000u;
  return (rb >> 23) >= 126u ? m << 8 : m << 7;
}

__host__ __device__ __forceinline__ uint32_t mulhi32(uint32_t a, uint32_t b) {
#ifdef __CUDA_ARCH__
  return __umulhi(a, b);
#else
  return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}

// significand quotient: for ma, mb in [2^52, 2^53), floor(ma*2^56/mb) in
// (2^55, 2^57) with the lowest bit set when the division leaves a remainder
// (three bits at least lie below the 53 that a result keeps, so the lowest
// one only has to say "not exact")
__host__ __device__ __forceinline__ uint64_t quot_sticky(uint64_t ma, uint64_t mb) {
  // reciprocal of x = mb/2^52 in [1, 2): V ~ 2^32/x, below it by less than
  // 2^-29.5 in relative terms after one Newton step in 32-bit fractions
  const uint32_t bh = (uint32_t)(mb >> 21);                  // x * 2^31, truncated
  uint32_t V = recip_estimate((uint32_t)(mb >> 29));
  const uint32_t e = 0x7ffffffeu - mulhi32(V, bh);           // 2^31 * (1 - V*x/2^32) or up to two less, > 0
  V += mulhi32(V, e << 1);
  // first digit: floor(ma*2^31/mb) or up to a few units less
  const uint32_t q1 = mulhi32((uint32_t)(ma >> 21), V);
  const uint64_t r1 = (ma << 31) - (uint64_t)q1 * mb;        // exact modulo 2^64, in [0, 8*mb)
  // second digit: 25 bits more
  uint32_t q2 = mulhi32((uint32_t)(r1 >> 24), V) >> 3;
  // V low by 1.4e-9 (0.4 units of q2), both truncations (1.3 units): the
  // digit is at most one short
  uint64_t r2 = (r1 << 25) - (uint64_t)q2 * mb;              // in [0, 2*mb)
  const bool more = r2 >= mb;
  r2 = more ? r2 - mb : r2;
  q2 = more ? q2 + 1u : q2;
  const uint64_t Q = ((uint64_t)q1 << 25) + q2;
  return Q | (r2 != 0 ? 1ull : 0ull);
}

// Q in (2^55, 2^57) with its sticky bit -> binary64 bits of Q*2^(E-56),
// rounded to nearest even; E the unbiased exponent, the result normal
__host__ __device__ __forceinline__ uint64_t round_quot(uint64_t Q, int E) {
  const bool big = (Q >> 56) != 0;
  const uint64_t h = big ? Q : Q + Q;                        // [2^56, 2^57): four bits to drop
  const uint64_t m = (h + 7u + ((h >> 4) & 1u)) >> 4;        // sticky and half bits in the low four
  const uint64_t eb = (uint64_t)(uint32_t)(1022 + E - (big ? 0 : 1));
  return (eb << 52) + m;                                     // the hidden bit adds one to the exponent
}

struct Bits64 {
  uint32_t hi, lo;
};
__host__ __device__ __forceinline__ Bits64 split64(double x) {
#ifdef __CUDA_ARCH__
  return Bits64{(uint32_t)__double2hiint(x), (uint32_t)__double2loint(x)};
#else
  uint64_t u;
  std::memcpy(&u, &x, 8);
  return Bits64{(uint32_t)(u >> 32), (uint32_t)u};
#endif
}
__host__ __device__ __forceinline__ double join64(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __hiloint2double((int)(uint32_t)(u >> 32), (int)(uint32_t)u);
#else
  double x;
  std::memcpy(&x, &u, 8);
  return x;
#endif
}
__host__ __device__ __forceinline__ uint64_t significand(Bits64 b) {
  return ((uint64_t)((b.hi & 0xfffffu) | 0x100000u) << 32) | b.lo;
}
// biased exponent, the sign dropped
__host__ __device__ __forceinline__ int expo(Bits64 b) { return (int)((b.hi >> 20) & 0x7ffu); }
__host__ __device__ __forceinline__ bool is_zero(Bits64 b) { return ((b.hi << 1) | b.lo) == 0u; }

#ifdef __CUDA_ARCH__
__device__ __noinline__ static double div_slow(double a, double b) { return __ddiv_rn(a, b); }
#else
inline double div_slow(double a, double b) { return a / b; }
#endif

// a / b, correctly rounded.  Everything whose operands and quotient are
// normal numbers goes through the integer quotient; a zero numerator is
// zero; what is left (denormals, infinities, NaN, division by zero, quotients
// near the ends of the exponent range) takes the division instruction
// sequence.
__host__ __device__ __forceinline__ double div_rn(double a, double b) {
  const Bits64 x = split64(a), y = split64(b);
  const int ea = expo(x), eb = expo(y);
  const bool ok = (unsigned)(ea - 1) < 2046u && (unsigned)(eb - 1) < 2046u && (unsigned)(ea - eb + 1000) < 2000u;
  const uint32_t sgn = (x.hi ^ y.hi) & 0x80000000u;
  const bool zero = is_zero(x) && (unsigned)(eb - 1) < 2046u;
  double r = join64((zero ? 0ull : round_quot(quot_sticky(significand(x), significand(y)), ea - eb)) | ((uint64_t)sgn << 32));
  if (!ok && !zero) r = div_slow(a, b);
  return r;
}

// sqrt(x), correctly rounded, on the integer pipes: two digits of the root of
// the significand from an approximate reciprocal root, the remainder kept
// exactly (the longhand method with large digits).  The root of a binary64
// number is never half-way between two of them, so the 54th bit alone decides
// the rounding.
__host__ __device__ __forceinline__ double sqrt_rn(double x) {
  const Bits64 b = split64(x);
  if (!((int)b.hi >= 0 && (unsigned)(expo(b) - 1) < 2046u)) {   // zero, denormal, negative, infinite, NaN
#ifdef __CUDA_ARCH__
    return __dsqrt_rn(x);
#else
    return __builtin_sqrt(x);
#endif
  }
  const int E = expo(b) - 1023;
  const uint64_t m = significand(b) << (E & 1);               // x = m/2^52 * 4^(E >> 1), m/2^52 in [1, 4)
  // reciprocal root of the first 24 bits, lowered by eight units in the last
  // place (the instruction is within two): below the true one by less than 2^-19.7
  const uint32_t fb = (127u << 23) + ((E & 1) ? (1u << 23) : 0u) + ((b.hi & 0xfffffu) << 3) + (b.lo >> 29);
  float f, r;
#ifdef __CUDA_ARCH__
  f = __uint_as_float(fb);
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(f));
  const uint32_t rb = __float_as_uint(r) - 8u;
#else
  std::memcpy(&f, &fb, 4);
  r = 1.0f / __builtin_sqrtf(f);
  uint32_t rb;
  std::memcpy(&rb, &r, 4);
  rb = rb - 8u + RT_RECIP_HOST_ULP;
#endif
  const uint32_t g = (rb & 0x7fffffu) | 0x800000u;
  uint32_t Y = (rb >> 23) >= 126u ? g << 8 : g << 7;          // y*2^32
  const uint32_t a = (uint32_t)(m >> 22);                     // m/2^52 * 2^30, truncated
  const uint32_t e = 0x3ffffffeu - mulhi32(mulhi32(Y, Y), a); // 2^30*(1 - a*y^2) or up to two less, > 0
  Y += mulhi32(Y, e << 1);
  const uint32_t s1 = mulhi32(a, Y);                          // root*2^30 or up to six less
  const uint64_t R1 = (m << 8) - (uint64_t)s1 * s1;           // < 2^35
  uint64_t T = ((uint64_t)s1 << 23) + (mulhi32((uint32_t)(R1 >> 3), Y) >> 5);   // floor(root*2^53) or up to two less
  uint64_t R2 = (m << 54) - T * T;                            // exact modulo 2^64
  if (R2 > 2 * T) {
    R2 -= 2 * T + 1;
    T++;
  }
  if (R2 > 2 * T) T++;
  return join64(((uint64_t)(uint32_t)(1022 + (E >> 1)) << 52) + ((T + 1) >> 1));
}

// x to binary32, to nearest even, without the conversion instruction (which
// shares the binary64 pipe) where the result is a normal number or zero
__host__ __device__ __forceinline__ float float_rn(double x) {
  const Bits64 b = split64(x);
  const bool zero = is_zero(b);
  const uint32_t low = b.lo & 0x1fffffffu;
  uint32_t r = (uint32_t)((((uint64_t)(b.hi & 0x7fffffffu) << 32) | b.lo) >> 29) - (896u << 23);
  r += low + (r & 1u) > 0x10000000u ? 1u : 0u;
  r = (zero ? 0u : r) | (b.hi & 0x80000000u);
  float f;
#ifdef __CUDA_ARCH__
  f = __uint_as_float(r);
  if ((unsigned)(expo(b) - 897) >= 253u && !zero) f = __double2float_rn(x);
#else
  std::memcpy(&f, &r, 4);
  if ((unsigned)(expo(b) - 897) >= 253u && !zero) f = (float)x;
#endif
  return f;
}

// Limiter(up/Rj) for Rj != 0 of superbee_fluxes.f90:10, :21-25:
// max(0, min(1, 2r), min(2, r)) with r = up/Rj correctly rounded.  r <= 0
// gives 0; r >= 2 gives 2 (also where only the rounded r reaches it); in
// between r is needed: 2r below 1/2, 1 up to 1, r up to 2, compared as bit
// patterns.  Rj = 0 returns 0: the caller multiplies by Rj.  The caller has
// sent infinities and NaN elsewhere (flux_exact).
//
// Straight-line code: a branch per case had the compiler copy the binary64
// instructions after it into every branch, and a warp whose lanes take
// different ones issues them all.
__host__ __device__ __forceinline__ double limited_ratio_normal(double up, double Rj) {   // both zero or normal
  const Bits64 x = split64(up), y = split64(Rj);
  const bool none = is_zero(x) || is_zero(y) || (int)(x.hi ^ y.hi) < 0;
  const uint64_t q = round_quot(quot_sticky(significand(x), significand(y)), expo(x) - expo(y));
  const uint32_t h = (uint32_t)(q >> 32);
  const bool half = h < 0x3fe00000u, one = !half && h < 0x3ff00000u, two = h >= 0x40000000u;
  uint32_t hi = half ? h + 0x00100000u : h, lo = (uint32_t)q;
  hi = one ? 0x3ff00000u : (two ? 0x40000000u : hi);
  hi = none ? 0u : hi;
  lo = one || two || none ? 0u : lo;
  return join64(((uint64_t)hi << 32) | lo);
}
__host__ __device__ __forceinline__ double limited_ratio(double up, double Rj) {
  const Bits64 x = split64(up), y = split64(Rj);
  const int ea = expo(x), eb = expo(y);
  double r = limited_ratio_normal(up, Rj);
  if ((ea == 0 || eb == 0 || ea - eb < -1000) && !(is_zero(x) || is_zero(y) || (int)(x.hi ^ y.hi) < 0)) {
    const double t = div_slow(up, Rj);                       // denormal operands or quotient
    r = t < 0.5 ? t + t : (t <= 1.0 ? 1.0 : (t < 2.0 ? t : 2.0));
  }
  return r;
}

#ifdef __CUDACC__
// flux_fp64u's sequence itself, for operands outside flux_exact's range
__device__ __noinline__ static double flux_slow(double v, double u, double S, double Rj, double up) {
  double Cr = (Rj != 0.0) ? __ddiv_rn(up, Rj) : dmul(up, 1.0000000200408773e20);   // the binary32 literal 1.E20
  Cr = fmax2(0.0, fmax2(fmin2(1.0, dmul(2.0, Cr)), fmin2(2.0, Cr)));
  const double adv = dmul(dmul(v, S), 0.5);
  const double dif = dmul(dmul(dmul(fabs(v), dadd(dsub(1.0, Cr), dmul(u, Cr))), Rj), 0.5);
  return dsub(adv, dif);
}

// |x| in [2^-323, 2^277) or zero
__device__ __forceinline__ bool mid_range(Bits64 b) { return (unsigned)(expo(b) - 700) < 600u || is_zero(b); }

// the flux from its parts, every product in the normal range (flux_exact)
__device__ __forceinline__ double flux_of(double v, double u, double S, double Rj, double Cr) {
  const Bits64 vb = split64(v);
  const uint32_t hh = is_zero(vb) ? vb.hi : vb.hi - 0x00100000u;
  const double vh = __hiloint2double((int)hh, (int)vb.lo);
  const double ah = __hiloint2double((int)(hh & 0x7fffffffu), (int)vb.lo);
  const double W = dadd(dsub(1.0, Cr), dmul(u, Cr));
  return dsub(dmul(vh, S), dmul(dmul(ah, W), Rj));
}

// Face flux of flux_fp64u (same bits; a zero flux may have the other sign,
// which no sum of differences that starts at +0 shows) from E(f-1), E(f),
// E(f+1), E(f+2), u = the cached uCFL: ten binary64 instructions and the
// integer quotient.
// The reference's two factors 0.5 are exact unless a product underflows, so
// they are applied to v once (its exponent lowered by one).  With v, u, S and
// Rj zero or in [2^-323, 2^277) every product of v, W and Rj or S stays in
// the normal range: W = (1-Cr)+u*Cr is u itself where Cr = 1, and otherwise
// zero or a cancellation that leaves at least 2^-110.  Other operands take
// the sequence itself.
__device__ __forceinline__ double flux_exact(double v, double u, double Ea, double Eb, double Ec, double Ed) {
  const Bits64 vb = split64(v);
  const bool pos = (int)vb.hi >= 0 && !is_zero(vb);
  const double Rj = dsub(Ec, Eb);
  const double up = dsub(pos ? Eb : Ed, pos ? Ea : Ec);
  const double S = dadd(Ec, Eb);
  if (!(mid_range(vb) && mid_range(split64(S)) && mid_range(split64(Rj)) && mid_range(split64(u)) && expo(split64(up)) < 1900))
    return flux_slow(v, u, S, Rj, up);
  return flux_of(v, u, S, Rj, limited_ratio(up, Rj));
}

// face 0 of an axis whose lower ghosts copy the edge cell: the reference's
// (v*(E0+E0))*0.5 less a diffusive part of Rj = E0-E0, which is v*E0 in
// mid_range (no sum or product overflows, none is denormal).  With the call
// beside it the multiplication also costs less than bare: the update pass keeps
// the binary64 pipe busy for 32 ps per cell, 38 before (7.57 -> 7.22 ms per step
// at 32x32x32x12^3).
__device__ __noinline__ static double face0_slow(double v, double e0) {
  return dsub(dmul(dmul(v, dadd(e0, e0)), 0.5), dsub(e0, e0));
}
__device__ __forceinline__ double face0_flux(double v, double e0) {
  if (!(mid_range(split64(v)) && mid_range(split64(e0)))) return face0_slow(v, e0);
  return dmul(v, e0);
}

// ---- the flux with its differences on the integer pipes ----
// Where the three E values a face's limiter depends on (its sides b and c,
// and w behind the upwind side) lie within 2^8 of each other, they are
// integers of at most 62 bits in units of the smallest one's last place, and
// Rj, the upwind difference and E_b + E_c are exact integers rounded once:
// the bits of the binary64 instructions, seven of which are left of ten.
// (S by its instruction instead: 8.30 against 8.39 ms per step at
// 32x32x32x12^3 with 4 resident CTAs, but 2D sections 3.5% slower; and 1 - Cr on
// the integer pipes as well: 2% slower everywhere.)
__device__ __forceinline__ double near_value(long long m, unsigned lo) {   // m*2^(lo - 1075), |m| < 2^63
  const uint32_t sgn = (uint32_t)((uint64_t)m >> 32) & 0x80000000u;
  uint64_t a = (uint64_t)(m < 0 ? -m : m);
  const int z = __clzll((long long)a);
  const bool none = a == 0;
  a <<= z & 63;
  const uint64_t r = a >> 11;
  const uint32_t frac = (uint32_t)a & 0x7ffu;
  const uint64_t bits = r + (frac + ((uint32_t)r & 1u) > 0x400u ? 1u : 0u) + ((uint64_t)(lo + 10u - (uint32_t)z) << 52);
  return join64((none ? 0ull : bits) | ((uint64_t)sgn << 32));
}

// positive values within 2^8, in [2^-263, 2^267): every difference of theirs
// is zero or in mid_range
__device__ __forceinline__ bool flux_is_near(double v, double u, double b, double c, double w) {
  const unsigned eb = top12(b), ec = top12(c), ew = top12(w);
  const unsigned hi = eb > ec ? (eb > ew ? eb : ew) : (ec > ew ? ec : ew);
  const unsigned lo = eb < ec ? (eb < ew ? eb : ew) : (ec < ew ? ec : ew);
  return hi - lo <= 8u && lo - 760u < 522u && mid_range(split64(v)) && mid_range(split64(u));
}

// pos: the upwind difference is b - w, else w - c; operands of flux_is_near
__device__ __forceinline__ double flux_near(double v, double u, double b, double c, double w, bool pos) {
  const unsigned eb = top12(b), ec = top12(c), ew = top12(w);
  const unsigned lo = eb < ec ? (eb < ew ? eb : ew) : (ec < ew ? ec : ew);
  const long long B = (long long)(significand(split64(b)) << (eb - lo));
  const long long C = (long long)(significand(split64(c)) << (ec - lo));
  const long long U = (long long)(significand(split64(w)) << (ew - lo));
  const double Rj = near_value(C - B, lo);
  const double up = near_value((pos ? B : U) - (pos ? U : C), lo);
  const double S = near_value(B + C, lo);
  return flux_of(v, u, S, Rj, limited_ratio_normal(up, Rj));
}
#endif

}  // namespace rt
