// Correctly rounded r = sqrt(a) and r^-3 = 1 / (a * r) for the reference-form
// pair (GravityAC, Acceleration.cpp:294-317: rij = sqrt(rij2),
// rijm3 = 1.0 / (rij2 * rij)) with no FP64 instruction besides the product
// a * r, bit-identical to IEEE sqrt and division.
//
// The GPU's FP64 pipe issues one warp instruction per 64 cycles per
// sub-partition; IEEE square root and division take about sixteen of them
// per pair, so they, not the twenty-one additions and multiplications of the
// pair, bound the reference form.  Here the approximations come from the FP32
// pipe and the remainders are measured on the integer pipe:
//
//  1. a = m 4^k with m in [1, 4).  From an FP32 rsqrt seed y and one Newton
//     correction evaluated with exact products (TwoProduct by FMA) come
//     float-float approximations (relative error ~2^-45) of m^-1/2, of
//     m^1/2 and of m^-3/2.
//  2. They become 53-bit integers Q ~ m^1/2 2^52 and Z ~ 1/d (d = RN(a r),
//     scaled), at most ~350 and ~1,150 units from the exact values.
//  3. The remainders m 2^104 - Q^2 and 2^105 - D Z (D the significand of d)
//     are small, so the words of the products in their middle are enough:
//     the remainder over 2 Q (over D), times m^-1/2 (times Z) as 31-bit fixed
//     point, is the distance of the exact result from Q (Z) in units in the
//     last place, to 2^-18 (2^-17) unit; rounding it to the nearest integer
//     and adding that gives the correctly rounded result.  This is the
//     remainder-based rounding decision of Markstein (IA-64 and Elementary
//     Functions, 2000, ch. 8; Tuckerman's test for the square root), with the
//     remainder measured rather than only its sign.
//
// Neither quotient can fall exactly on a midpoint between doubles (a
// midpoint needs 54 significant bits; its square, or its product with a
// 53-bit d, cannot be a double, resp. 1).  Where the measured distance lies
// within 2^-16 ulp of a midpoint (probability 2^-15 per function), where a
// distance exceeds its range, where the result would lie next to a power of
// two, or where a is outside [2^-600, 2^600] (zero, denormal, infinite or NaN
// included) the fast path reports failure and the caller takes IEEE sqrt and
// division, so the result is the correctly rounded one in every case.
//
// With the remainders by FP64 FMA (two of a pair's 14.7 FP64 instructions, and
// their conversions to float-float) an evaluation of 16,411 bodies took 7.96 ms
// for 7.01, of 2,049 173 us for 156.
#pragma once

#include "sol_pair.cuh"

namespace solcr {

// h + l (floats, |l| <= ulp(h)) in units of 2^(e - 52), as an integer; h_units:
// h in units of 2^(e - 23), unit: 2^(52 - e).
__device__ __forceinline__ long long ff_significand(unsigned h_units, float l, float unit) {
  return ((long long)h_units << 29) + (long long)__float2int_rn(l * unit);
}

// t: a distance in units of 2^-B ulp.  The nearest whole number of ulps; ok
// turns false within 2^-16 ulp of a midpoint.
template <int B>
__device__ __forceinline__ int round_distance(int t, bool& ok) {
  const int u = t + (1 << (B - 1));
  ok = ok & ((unsigned)(u & ((1 << B) - 1)) - (1u << (B - 16)) <= (1u << B) - (2u << (B - 16)));
  return u >> B;
}

// The double with significand S (2^52 < S < 2^53) and exponent e; ok turns
// false for a significand outside (a power of two, or a result in the next
// binade, which would round in other units).
__device__ __forceinline__ double from_significand(long long S, int e, bool& ok) {
  const unsigned hi = (unsigned)(S >> 32), lo = (unsigned)S;
  ok = ok & (hi - 0x100000u < 0x100000u) & (((hi ^ 0x100000u) | lo) != 0u);
  return __hiloint2double((int)(hi + ((unsigned)(e + 1022) << 20)), (int)lo);
}

// The correctly rounded 1/d from an approximation Z 2^(ez - 52).  With D the
// significand of d, 2^105 - D Z over D is its distance in units of Z; of the
// product bits 32 to 95 are formed (the rest is known), their 32 from bit 33
// on are the remainder where the distance is below 2^11.
__device__ __forceinline__ double rcp_from_approx(double d, long long Z, int ez, bool& ok) {
  const unsigned dh = (unsigned)__double2hiint(d), dl = (unsigned)__double2loint(d);
  const unsigned Dh = (dh & 0xFFFFFu) | 0x100000u;
  const unsigned Zl = (unsigned)Z, Zh = (unsigned)(Z >> 32);
  const unsigned long long t1 = (unsigned long long)Dh * Zl + __umulhi(dl, Zl);
  const unsigned long long t2 = (unsigned long long)dl * Zh + (unsigned)t1;
  const unsigned t3 = Dh * Zh + (unsigned)(t1 >> 32) + (unsigned)(t2 >> 32);
  const int v = -(int)__funnelshift_r((unsigned)t2, t3, 1);
  // beyond 31 bits of remainder, or an approximation in the wrong binade
  ok = ok & (t3 + 1u <= 1u) & ((int)(dh >> 20) - 1023 + ez == -1);
  const int t = __mulhi(v, (int)(Z >> 22));  // v 2^33 / D = v Z 2^(33 - 105)
  return from_significand(Z + (long long)round_distance<18>(t, ok), ez, ok);
}

}  // namespace solcr

// Fast path: returns false where the caller must use IEEE sqrt and division.
__device__ __forceinline__ bool sol_ref_rinv3_fast(double a, double& rij, double& rijm3) {
  using namespace solcr;
  const unsigned hiA = (unsigned)__double2hiint(a);
  const unsigned loA = (unsigned)__double2loint(a);
  const int E = (int)(hiA >> 20);  // the sign bit of a sum of squares is clear, NaN aside
  bool ok = (unsigned)(E - (1023 - 600)) <= 1200u;
  const int e2 = E - 1023;
  const int k = e2 >> 1;   // floor(e2 / 2)
  const int p = e2 - 2 * k;  // 0 or 1: m = a 4^-k in [1, 4)
  // m as float-float (mh exact to 24 bits, ml the rest rounded)
  const float mh = __uint_as_float(((unsigned)(127 + p) << 23) | ((hiA & 0x000FFFFFu) << 3) | (loA >> 29));
  const float ml = __uint2float_rn(loA & 0x1FFFFFFFu) * __uint_as_float((unsigned)(127 + p - 52) << 23);
  // seed and residual e = 1 - m y^2 from exact products
  const float y = sol_rsqrt_normal(mh);  // mh in [1, 4)
  float y2, y2e, q, qe;
  ff_two_prod(y, y, y2, y2e);
  ff_two_prod(mh, y2, q, qe);
  const float e = ((1.0f - q) - qe) - __fmaf_rn(mh, y2e, ml * y2);
  // m^-1/2 = y (1 - e)^-1/2 = y (1 + e/2 + 3/8 e^2 + ...)
  float yh, yl;
  ff_fast_two_sum(y, y * (e * __fmaf_rn(0.375f, e, 0.5f)), yh, yl);
  // m^1/2 = m m^-1/2
  float sh, sl;
  {
    float sp, spe;
    ff_two_prod(mh, yh, sp, spe);
    ff_fast_two_sum(sp, spe + __fmaf_rn(mh, yl, ml * yh), sh, sl);
  }
  // m^-3/2 = y^3 (1 - e)^-3/2 = y^3 (1 + 3/2 e + 15/8 e^2 + ...)
  float Rh, Rl;
  {
    float y3h, y3e;
    ff_two_prod(y2, y, y3h, y3e);
    y3e = __fmaf_rn(y2e, y, y3e);
    const float c3 = e * __fmaf_rn(1.875f, e, 1.5f);
    ff_fast_two_sum(y3h, __fmaf_rn(y3h, c3, y3e), Rh, Rl);
  }

  // ---- sqrt(a) = q 2^k: Q ~ m^1/2 2^52, (m 2^104 - Q^2) / (2 Q) ----
  // (sh in [1, 2], its bits linear there, 2 included)
  const long long Q = ff_significand(__float_as_uint(sh) - 0x3F000000u, sl, 4503599627370496.0f);
  const unsigned Ql = (unsigned)Q, Qh = (unsigned)(Q >> 32);
  const int R = (int)((loA << (20 + p)) - __umulhi(Ql, Ql) - (Qh << 1) * Ql);  // bits 32 to 63, |R| < 2^31
  // m^-1/2 = yh + yl in units of 2^-31 (not for yh = 1: m within 2^-24 of 1)
  ok = ok & (yh < 1.0f);
  const int yi = (int)(((__float_as_uint(yh) & 0x7FFFFFu) | 0x800000u) << 7) +
                 (__float_as_int(__fmaf_rn(yl, 2147483648.0f, 12582912.0f)) - 0x4B400000);
  const int t = __mulhi(R, yi);  // R 2^32 / (2 Q) = R 2^-21 m^-1/2
  const double r = from_significand(Q + (long long)round_distance<20>(t, ok), k, ok);

  // ---- 1/d, d = RN(a r): Z ~ m^-3/2 2^-3k ----
  const double d = a * r;
  const unsigned Rb = __float_as_uint(Rh);
  const long long Z = ff_significand((Rb & 0x7FFFFFu) | 0x800000u, Rl,
                                     __uint_as_float(((127u + 52u + 127u) << 23) - (Rb & 0x7F800000u)));
  rij = r;
  rijm3 = rcp_from_approx(d, Z, (int)(Rb >> 23) - 127 - 3 * k, ok);
  return ok;
}

static __device__ __noinline__ double2 sol_ref_rinv3_ieee(double a) {
  const double r = __dsqrt_rn(a);
  return make_double2(r, __ddiv_rn(1.0, a * r));
}
__device__ __forceinline__ void sol_ref_rinv3_slow(double a, double& rij, double& rijm3) {
  const double2 v = sol_ref_rinv3_ieee(a);
  rij = v.x;
  rijm3 = v.y;
}

// rij = RN(sqrt(a)), rijm3 = RN(1 / RN(a * rij)), bit-identical to IEEE
// sqrt and division for every a.
__device__ __forceinline__ void sol_ref_rinv3(double a, double& rij, double& rijm3) {
  if (!sol_ref_rinv3_fast(a, rij, rijm3)) sol_ref_rinv3_slow(a, rij, rijm3);
}

// ---- IEEE double multiplication on the integer pipe ----------------------------
// Round-to-nearest-even product of two doubles from 32-bit integer
// multiplies of the significands (the 106-bit product in three words, the
// leading 53 bits, the bits below them compared with one half): the textbook
// IEEE 754 multiply.  It serves operands that are zero or of magnitude
// [2^-423, 2^424), whose product is a normal number, so the product's own
// exponent needs no test; ok turns false elsewhere (the caller then takes the
// FP64 instruction).  The FP64 pipe binds the reference form; the integer
// pipe, which it leaves mostly idle, takes a pair's multiplications.

// (t3, w1, w0): a 106-bit significand product in [2^104, 2^106); its sign
// and the exponent field of its 2^104 binade in place (hi).  The result's
// high and low words, rounded to nearest even; a rounding carry out of the
// significand moves into the exponent field.
__device__ __forceinline__ void exact_round(unsigned long long t3, unsigned w1, unsigned w0, unsigned hi,
                                            unsigned& rh, unsigned& rl) {
  const unsigned t3h = (unsigned)(t3 >> 32), t3l = (unsigned)t3;
  const unsigned n = t3h >> 9;  // product >= 2^105: one more place to drop
  const unsigned s = 20 + n;
  const unsigned ml = __funnelshift_r(w1, t3l, s), mh = __funnelshift_r(t3l, t3h, s);  // the leading 53 bits
  const unsigned rem = (w1 << (12 - n)) | (w0 != 0u ? 1u : 0u);  // the rest, its half at bit 31
  const unsigned up = rem > 0x80000000u - (ml & 1u) ? 1u : 0u;
  const unsigned long long r = (((unsigned long long)(mh + hi + (n << 20) - 0x100000u) << 32) | ml) + up;
  rh = (unsigned)(r >> 32);
  rl = (unsigned)r;
}
// Operand exponent fields this multiply serves: [600, 1447) (high word, sign shifted out)
__device__ __forceinline__ bool exact_range(unsigned h) { return (h << 1) - (600u << 21) < (847u << 21); }

// AZ / BZ: whether a / b may be zero on the fast path (else a zero counts as
// out of range): a component that is zero by symmetry (a planar system's z).
template <bool AZ = true, bool BZ = true>
__device__ __forceinline__ double sol_exact_dmul(double a, double b, bool& ok) {
  const unsigned ah = (unsigned)__double2hiint(a), al = (unsigned)__double2loint(a);
  const unsigned bh = (unsigned)__double2hiint(b), bl = (unsigned)__double2loint(b);
  const unsigned mah = (ah & 0xFFFFFu) | 0x100000u, mbh = (bh & 0xFFFFFu) | 0x100000u;
  const unsigned long long t0 = (unsigned long long)al * bl;
  const unsigned long long t1 = (unsigned long long)mah * bl + (unsigned)(t0 >> 32);
  const unsigned long long t2 = (unsigned long long)al * mbh + (unsigned)t1;
  const unsigned long long t3 = (unsigned long long)mah * mbh + (unsigned)(t1 >> 32) + (unsigned)(t2 >> 32);
  const unsigned sign = (ah ^ bh) & 0x80000000u;
  unsigned rh, rl;
  exact_round(t3, (unsigned)t2, (unsigned)t0, (ah & 0x7FF00000u) + (bh & 0x7FF00000u) - (1023u << 20), rh, rl);
  const bool za = AZ && (ah << 1 | al) == 0u, zb = BZ && (bh << 1 | bl) == 0u;
  const bool zero = za | zb;
  ok = ok & (za | exact_range(ah)) & (zb | exact_range(bh));
  return __hiloint2double((int)((zero ? 0u : rh) | sign), (int)(zero ? 0u : rl));
}

// The square of a double, likewise (three partial products, no sign).
template <bool AZ = true>
__device__ __forceinline__ double sol_exact_dsqr(double a, bool& ok) {
  const unsigned ah = (unsigned)__double2hiint(a), al = (unsigned)__double2loint(a);
  const unsigned mah = (ah & 0xFFFFFu) | 0x100000u;
  const unsigned long long t0 = (unsigned long long)al * al;
  const unsigned long long t1 = (unsigned long long)(mah << 1) * al + (unsigned)(t0 >> 32);
  const unsigned long long t3 = (unsigned long long)mah * mah + (unsigned)(t1 >> 32);
  unsigned rh, rl;
  exact_round(t3, (unsigned)t1, (unsigned)t0, ((ah & 0x7FF00000u) << 1) - (1023u << 20), rh, rl);
  const bool zero = AZ && (ah << 1 | al) == 0u;
  ok = ok & (zero | exact_range(ah));
  return __hiloint2double((int)(zero ? 0u : rh), (int)(zero ? 0u : rl));
}

struct SolVec3 {
  double x, y, z;
};
// (by value: a reference argument of a function that is not inlined would keep its variable in local memory)
static __device__ __noinline__ SolVec3 sol_ref_terms_slow(double gm, double rijm3, double dx, double dy, double dz,
                                                          double px, double py, double pz) {
  return SolVec3{gm * (dx * rijm3 - px), gm * (dy * rijm3 - py), gm * (dz * rijm3 - pz)};
}

// The reference's pair term gm (d rijm3 - p) per component
// (Acceleration.cpp:306-308), its six multiplications on the integer pipe;
// bit-identical to the FP64 expression.
__device__ __forceinline__ void sol_ref_terms(double gm, double rijm3, double dx, double dy, double dz, double px,
                                              double py, double pz, double& tx, double& ty, double& tz) {
  bool ok = true;
  const double ux = sol_exact_dmul<false, false>(dx, rijm3, ok) - px;
  const double uy = sol_exact_dmul<false, false>(dy, rijm3, ok) - py;
  const double uz = sol_exact_dmul<true, false>(dz, rijm3, ok) - pz;
  tx = sol_exact_dmul<false, false>(gm, ux, ok);
  ty = sol_exact_dmul<false, false>(gm, uy, ok);
  tz = sol_exact_dmul<false, true>(gm, uz, ok);
  if (!ok) {
    const SolVec3 t = sol_ref_terms_slow(gm, rijm3, dx, dy, dz, px, py, pz);
    tx = t.x;
    ty = t.y;
    tz = t.z;
  }
}

// IEEE arithmetic for a pair the fast paths hand over: |d| and 1 / (|d|^2 |d|)
static __device__ __noinline__ double2 sol_ref_pair_ieee(double dx, double dy, double dz) {
  return sol_ref_rinv3_ieee(dx * dx + dy * dy + dz * dz);
}
