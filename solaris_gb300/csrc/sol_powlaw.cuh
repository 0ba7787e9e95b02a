// Powers r^p and exponentials of the gas model on the integer pipe.
//
// A library pow is a chain of ~100 FP64 instructions (~5,800 cycles of one
// warp; the FP64 pipe takes a warp instruction per 16 cycles of the SM), and a
// planetesimal's drag takes four of them.  Here both halves are table-driven
// (Tang, ACM TOMS 15 (1989) 144 and 16 (1990) 378) in 64-bit fixed point:
//   log2 x = E + log2(1024 / c) + log2(1 + f), x = 2^E m, c a 10-bit integer
//     near 1024 / m from m's leading 7 bits, f = m c / 1024 - 1 exact and
//     |f| < 2^-7.6, its series to f^8 (truncation below 2^-70);
//   2^y = 2^I 2^(j / 128) 2^g, |g| <= 2^-8, the exponential series of g ln 2 to
//     the sixth power (truncation below 2^-72).
// log2 x carries 59 fractional bits and y = p log2 x at least 56, so the
// result before its one rounding is within 2^-55.5 of itself: 0.6 ulp in all
// (0.29 rms measured over 10^6 samples an exponent, -2.75 to 2.75, the largest
// 0.55, and 0.58 over the whole range taken; the library's pow 0.42 and 1.33).
// ~160 instructions, none of them FP64.
#pragma once

#include <cuda_runtime.h>

namespace solpow {

// round(1024 / m) at the middle of the 128 intervals of m, and log2(1024 / c) in units of 2^-62
static __device__ const unsigned short kC[128] = {
    1020, 1012, 1004, 997, 989, 982, 975, 967, 960, 953, 946, 940, 933, 926, 920, 913, 907, 901, 895, 889, 883, 877,
    871, 865, 859, 854, 848, 843, 838, 832, 827, 822, 817, 812, 807, 802, 797, 792, 787, 783, 778, 773, 769, 764,
    760, 755, 751, 747, 743, 738, 734, 730, 726, 722, 718, 714, 710, 707, 703, 699, 695, 692, 688, 684, 681, 677,
    674, 670, 667, 664, 660, 657, 654, 650, 647, 644, 641, 638, 635, 632, 629, 626, 623, 620, 617, 614, 611, 608,
    605, 603, 600, 597, 594, 592, 589, 586, 584, 581, 579, 576, 574, 571, 569, 566, 564, 561, 559, 557, 554, 552,
    550, 547, 545, 543, 541, 538, 536, 534, 532, 530, 527, 525, 523, 521, 519, 517, 515, 513};
static __device__ const unsigned long long kT[128] = {
    0x5c836701aa0d7bull, 0x116a21e20a0a451ull, 0x1d23afc49139f8aull, 0x2779bb373e01e67ull, 0x3360a071b0812abull,
    0x3ddef24a116d3acull, 0x48707bd57c1b081ull, 0x549c69e188a83daull, 0x5f58125b3eed31aull, 0x6a27d69b726b2fbull,
    0x750c0289493505eull, 0x7e725770744593aull, 0x897d37aa87c4aecull, 0x949d61ee0d33433ull, 0x9e37db2866f2851ull,
    0xa9806bcb6f99ccfull, 0xb33e041385c8284ull, 0xbd0c294b1ac92d3ull, 0xc6eb1410a025485ull, 0xd0dafe2705a326eull,
    0xdadc227da59f78bull, 0xe4eebd38768affcull, 0xef130bb884681b9ull, 0xf9494ca4b544456ull, 0x10391bff2dbcf338ull,
    0x10c318aedff3c076ull, 0x1169c05363f15872ull, 0x11f588973c874718ull, 0x128225bb5e64a3e9ull,
    0x132bfee370ee6866ull, 0x13ba7963fc1f8ef0ull, 0x1449d115ef7d876cull, 0x14da08ac46495a4aull,
    0x156b22e6b578e49dull, 0x15fd2291fc33cef6ull, 0x16900a8836d0d507ull, 0x1723ddb1346b6515ull,
    0x17b89f02cf2aad32ull, 0x184e5181475448f9ull, 0x18c6c335d8b965b2ull, 0x195e2f9b51f04e2full,
    0x19f695efbbd0ee9full, 0x1a713787ad97a4b8ull, 0x1b0b67f4f4680ff5ull, 0x1b877c57b1b06ff0ull,
    0x1c2381c08baf4e9eull, 0x1ca111cb2aa5c544ull, 0x1d1f4d7febf867feull, 0x1d9e36b6b825b0a4ull,
    0x1e3dd1156507ddd9ull, 0x1ebe47960e3c0880ull, 0x1f3f71cc1b629b83ull, 0x1fc151b11b36401cull,
    0x2043e946fd97f5dcull, 0x20c73a98433abf2full, 0x214b47b82ea431acull, 0x21d012c2f68d67f2ull,
    0x223428f74e8ca777ull, 0x22ba458ca455b0f6ull, 0x2341260a447795faull, 0x23c8ccafd2fb087bull,
    0x242f0d16186fcf55ull, 0x24b81408c77d5f5cull, 0x2541e78680e0b71eull, 0x25a9cdd122c8ce9dull,
    0x26350d0eb6705c56ull, 0x269e06fad8bf6473ull, 0x272ab98c4a3c8e55ull, 0x2794ccdfa924feb8ull,
    0x27ff5a9ce9e3abcdull, 0x288e2d458104c41cull, 0x28f9dcfaea92e2b1ull, 0x29660adb732b4797ull,
    0x29f70e4bd6b75269ull, 0x2a64671b21d8e3c4ull, 0x2ad24203b3694c82ull, 0x2b40a03c917a88cdull,
    0x2baf830122b03c6bull, 0x2c1eeb9143600e3dull, 0x2c8edb315b321326ull, 0x2cff532a7344f069ull,
    0x2d7054ca4cd97c9dull, 0x2de1e1637889c727ull, 0x2e53fa4d6e0f8fadull, 0x2ec6a0e4a49e5a42ull,
    0x2f39d68aabd5715bull, 0x2fad9ca6454e4c9eull, 0x3021f4a37ecbfaeeull, 0x3096dff3cd105705ull,
    0x30e524bb196cd583ull, 0x315b08d9e6d3481cull, 0x31d184403cfbecceull, 0x3248987450350b4aull,
    0x329850e92589b608ull, 0x3310673cb9f7159aull, 0x33891a8be56a4a25ull, 0x33d9ea17e87e2681ull,
    0x3453a6a249c24501ull, 0x34a52885aa8c11f0ull, 0x351ff2e30214bc30ull, 0x35722a37c2d1badcull,
    0x35ee071e9f68aed8ull, 0x3640f713a7783bb0ull, 0x36bdeb5a7c2ce039ull, 0x37119734556a4251ull,
    0x378fa7d29bdb897bull, 0x37e412ec386bc7c2ull, 0x3838cb7b6a079d0bull, 0x38b872c7291f496dull,
    0x390def6fd4951167ull, 0x3963bb8832dedb05ull, 0x39e503e2be17ce3aull, 0x3a3b991e25055e81ull,
    0x3a927fd6fd0ac35eull, 0x3ae9b8a73bc9e97full, 0x3b6d29207b2970deull, 0x3bc531d817581953ull,
    0x3c1d8ecf99b58c0cull, 0x3c7640a8deaa9421ull, 0x3ccf480796d5cd74ull, 0x3d5574da88e6550dull,
    0x3daf54df46b1e14full, 0x3e098cb530796a64ull, 0x3e641d088b6533dbull, 0x3ebf0687997a2d6dull,
    0x3f1a49e2a175d53aull, 0x3f75e7cbf6d11790ull, 0x3fd1e0f801eb1536ull};
// 2^(j / 128) in units of 2^-63
static __device__ const unsigned long long kE[128] = {
    0x8000000000000000ull, 0x80b1ed4fd999ab6cull, 0x8164d1f3bc030773ull, 0x8218af4373fc25ecull,
    0x82cd8698ac2ba1d7ull, 0x8383594eefb6ee37ull, 0x843a28c3acde4046ull, 0x84f1f656379c1a29ull,
    0x85aac367cc487b15ull, 0x8664915b923fba04ull, 0x871f61969e8d1010ull, 0x87db357ff698d792ull,
    0x88980e8092da8527ull, 0x8955ee03618e5fddull, 0x8a14d575496efd9aull, 0x8ad4c6452c728924ull,
    0x8b95c1e3ea8bd6e7ull, 0x8c57c9c4646f4ddeull, 0x8d1adf5b7e5ba9e6ull, 0x8ddf042022e69cd6ull,
    0x8ea4398b45cd53c0ull, 0x8f6a8117e6c8e5c4ull, 0x9031dc431466b1dcull, 0x90fa4c8beee4b12bull,
    0x91c3d373ab11c336ull, 0x928e727d9531f9acull, 0x935a2b2f13e6e92cull, 0x9426ff0fab1c04b6ull,
    0x94f4efa8fef70961ull, 0x95c3fe86d6cc7fefull, 0x96942d3720185a00ull, 0x97657d49f17ab08eull,
    0x9837f0518db8a96full, 0x990b87e266c189aaull, 0x99e0459320b7fa65ull, 0x9ab62afc94ff864aull,
    0x9b8d39b9d54e5539ull, 0x9c6573682ec32c2dull, 0x9d3ed9a72cffb751ull, 0x9e196e189d472420ull,
    0x9ef5326091a111aeull, 0x9fd228256400dd06ull, 0xa0b0510fb9714fc2ull, 0xa18faeca8544b6e4ull,
    0xa27043030c496819ull, 0xa3520f68e802bb93ull, 0xa43515ae09e6809eull, 0xa5195786be9ef339ull,
    0xa5fed6a9b15138eaull, 0xa6e594cfeee86b1eull, 0xa7cd93b4e965356aull, 0xa8b6d5167b320e09ull,
    0xa9a15ab4ea7c0ef8ull, 0xaa8d2652ec907629ull, 0xab7a39b5a93ed337ull, 0xac6896a4be3fe929ull,
    0xad583eea42a14ac6ull, 0xae493452ca35b80eull, 0xaf3b78ad690a4375ull, 0xb02f0dcbb6e04584ull,
    0xb123f581d2ac2590ull, 0xb21a31a66618fe3bull, 0xb311c412a9112489ull, 0xb40aaea2654b9841ull,
    0xb504f333f9de6484ull, 0xb60093a85ed5f76cull, 0xb6fd91e328d17791ull, 0xb7fbefca8ca41e7cull,
    0xb8fbaf4762fb9ee9ull, 0xb9fcd2452c0b9debull, 0xbaff5ab2133e45fbull, 0xbc034a7ef2e9fb0dull,
    0xbd08a39f580c36bfull, 0xbe0f6809860993e2ull, 0xbf1799b67a731083ull, 0xc0213aa1f0d08db0ull,
    0xc12c4cca66709456ull, 0xc238d2311e3d6673ull, 0xc346ccda24976407ull, 0xc4563ecc5334cb33ull,
    0xc5672a115506daddull, 0xc67990b5aa245f79ull, 0xc78d74c8abb9b15dull, 0xc8a2d85c8ffe2c45ull,
    0xc9b9bd866e2f27a3ull, 0xcad2265e4290774eull, 0xcbec14fef2727c5dull, 0xcd078b86503dcdd2ull,
    0xce248c151f8480e4ull, 0xcf4318cf191918c1ull, 0xd06333daef2b2595ull, 0xd184df6251699ac6ull,
    0xd2a81d91f12ae45aull, 0xd3ccf099859ac379ull, 0xd4f35aabcfedfa1full, 0xd61b5dfe9f9bce07ull,
    0xd744fccad69d6af4ull, 0xd870394c6db32c84ull, 0xd99d15c278afd7b6ull, 0xdacb946f2ac9cc72ull,
    0xdbfbb797daf23755ull, 0xdd2d818508324c20ull, 0xde60f4825e0e9124ull, 0xdf9612deb8f04420ull,
    0xe0ccdeec2a94e111ull, 0xe2055afffe83d369ull, 0xe33f8972be8a5a51ull, 0xe47b6ca0373da88dull,
    0xe5b906e77c8348a8ull, 0xe6f85aaaee1fce22ull, 0xe8396a503c4bdc68ull, 0xe97c38406c4f8c57ull,
    0xeac0c6e7dd24392full, 0xec0718b64c1cbddcull, 0xed4f301ed9942b84ull, 0xee990f980da3025bull,
    0xefe4b99bdcdaf5cbull, 0xf13230a7ad094509ull, 0xf281773c59ffb13aull, 0xf3d28fde3a641a5bull,
    0xf5257d152486cc2cull, 0xf67a416c733f846eull, 0xf7d0df730ad13bb9ull, 0xf92959bb5dd4ba74ull,
    0xfa83b2db722a033aull, 0xfbdfed6ce5f09c49ull, 0xfd3e0c0cf486c175ull, 0xfe9e115c7b8f884cull};

// 2^(y 2^-sh) for y 2^-sh in (-1000, 1000), 0 < sh < 64
__device__ __forceinline__ double exp2_fixed(long long y, int sh) {
  int I = (int)(y >> sh);
  const unsigned long long frac = (unsigned long long)y << (64 - sh);
  const unsigned long long t = frac + (1ull << 56);  // the nearest of 128 points, g from it
  if (t < frac) ++I;
  const unsigned long long T = kE[t >> 57];
  const long long g = (long long)(t & ((1ull << 57) - 1)) - (1ll << 56);  // units of 2^-64
  const long long z = __mul64hi(g << 7, 0x58b90bfbe8e7bcd6ll);           // g ln 2, units of 2^-70
  // (e^z - 1) / z, units of 2^-62, from 1/720 up
  long long b = 0x88888888888889ll + (__mul64hi(z, 0x16c16c16c16c17ll) >> 6);
  b = 0x2aaaaaaaaaaaaabll + (__mul64hi(z, b) >> 6);
  b = 0xaaaaaaaaaaaaaabll + (__mul64hi(z, b) >> 6);
  b = 0x2000000000000000ll + (__mul64hi(z, b) >> 6);
  b = 0x4000000000000000ll + (__mul64hi(z, b) >> 6);
  const long long e = __mul64hi(z, b) << 3;  // e^z - 1, units of 2^-71
  // T (1 + e), units of 2^-63 (T is below 2^64: halved to multiply as signed)
  unsigned long long R = T + (unsigned long long)(__mul64hi((long long)(T >> 1), e) >> 6);
  const int lz = __clzll((long long)R);  // 1 just below a power of two
  R <<= lz;
  const unsigned long long m = (R >> 11) - (1ull << 52) + ((R >> 10) & 1);
  return __longlong_as_double(((long long)(I - lz + 1023) << 52) + (long long)m);
}

static __device__ __noinline__ double library_pow(double x, double p) { return pow(x, p); }
static __device__ __noinline__ double library_exp(double a) { return exp(a); }

}  // namespace solpow

// log2 x in units of 2^-59 for a normal x in [2^-15, 2^15); ok turns false elsewhere.
__device__ __forceinline__ long long sol_log2_fixed(double x, bool& ok) {
  using namespace solpow;
  const long long b = __double_as_longlong(x);
  const int E = (int)(b >> 52) - 1023;  // (a set sign bit takes it out of range)
  ok = ok && (unsigned)(E + 15) < 30u;
  const unsigned long long M = ((unsigned long long)b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  const int i = (int)(M >> 45) & 127;
  const long long f = (long long)(M * kC[i]) - (1ll << 62);  // units of 2^-62, exact
  const long long F = f << 8;                                  // units of 2^-70
  // the series of log2(1 + f) / f: 32-bit terms (units of 2^-30) from f^7 down to f^4, then 2^-62
  const int f32 = (int)(F >> 32);  // units of 2^-38
  int a = 0xd30bb15 - (__mulhi(f32, 0xb8aa3b3) >> 6);
  a = 0xf6384ee - (__mulhi(f32, a) >> 6);
  a = 0x12776c51 - (__mulhi(f32, a) >> 6);
  long long s = 0x171547652b82fe17ll - (__mul64hi(F, (long long)a << 32) >> 6);
  s = 0x1ec709dc3a03fd75ll - (__mul64hi(F, s) >> 6);
  s = 0x2e2a8eca5705fc2fll - (__mul64hi(F, s) >> 6);
  s = 0x5c551d94ae0bf85ell - (__mul64hi(F, s) >> 6);
  const long long l = (long long)kT[i] + ((__mul64hi(F, s) + 32) >> 6);  // log2 m, units of 2^-62
  return (long long)E * (1ll << 59) + ((l + 4) >> 3);
}

// x^p from l = sol_log2_fixed(x) (ok as it left it); p zero, below 1/16 or from 8 up, and an x out
// of its range take the library's pow.
__device__ __forceinline__ double sol_pow_from_log2(double x, long long l, double p, bool ok) {
  const long long pb = __double_as_longlong(p);
  const int ep = (int)((pb >> 52) & 0x7FF) - 1022;  // |p| < 2^ep
  if (!(ok && ep >= -3 && ep <= 3)) return solpow::library_pow(x, p);
  const unsigned long long P = (((unsigned long long)pb & 0xFFFFFFFFFFFFFull) | (1ull << 52)) << 11;  // |p| 2^(64 - ep)
  const unsigned long long la = (unsigned long long)(l < 0 ? -l : l);
  long long y = (long long)__umul64hi(la, P);  // |y| in units of 2^(ep - 59)
  if ((l < 0) != (pb < 0)) y = -y;
  return solpow::exp2_fixed(y, 59 - ep);
}
// (not inlined: a planetesimal's drag has five powers, and the kernels that
// carry it in their epilogue have no registers to spare)
static __device__ __noinline__ double sol_pow(double x, double p) {
  bool ok = true;
  const long long l = sol_log2_fixed(x, ok);
  return sol_pow_from_log2(x, l, p, ok);
}

// e^-a for a in [0, 16); the library's exp elsewhere
static __device__ __noinline__ double sol_exp_neg(double a) {
  if (!(a >= 0.0 && a < 16.0)) return solpow::library_exp(-a);
  const long long b = __double_as_longlong(a);
  const int e = (int)(b >> 52) - 1023;
  const unsigned long long M = ((unsigned long long)b & 0xFFFFFFFFFFFFFull) | (1ull << 52);
  const unsigned long long A = e >= -7 ? M << (7 + e) : (e > -70 ? M >> (-7 - e) : 0ull);  // units of 2^-59
  return solpow::exp2_fixed(-(long long)__umul64hi(A, 0xb8aa3b295c17f0bcull), 58);
}
