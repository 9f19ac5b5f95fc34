// FP64 division, square root, logarithm, exponential and comparisons on the
// integer pipe.
//
// The GB300's FP64 pipe takes one warp instruction per 20 cycles and SM, while
// its four schedulers issue up to 80 others in that time: an FP64 kernel waits
// for that pipe and leaves the integer units idle.  A division or square root
// costs 146 cycles there, log 578, exp 361, a comparison 20 (measured, per
// warp and SM).  Here they are integer arithmetic on the bits:
//
//  * comparisons: the bits of a double, taken as a signed 64-bit integer with
//    the magnitude of negative ones inverted, have the order of the values;
//  * div, sqrt: a 22-bit float seed, one Newton step and one remainder
//    correction in 64-bit fixed point, then the exact remainder decides the last
//    bit: the correctly rounded result, the same bits as a / b and sqrt(a).  A
//    quotient or root of 53-bit numbers is never half way between two doubles,
//    so 54 bits of the floor round correctly;
//  * log, exp: table and polynomial (Tang's method, ACM TOMS 15 and 16) in
//    64-bit fixed point.  log x = k ln2 - ln c_i + log1p(m c_i - 1) with 10-bit
//    c_i, so that m c_i - 1 is exact; exp x = 2^k 2^(j/128) e^y.  Errors below
//    0.51 ulp (log) and 0.62 ulp (exp) of the result.
//
// Arguments or results outside the normal range (zeros but for a zero
// numerator, subnormals, infinities, NaN, logs below 1/16 in size) take the
// built-in operation, so every result there is what it was.
// Outside nvcc the functions are host code, which a test compares with the
// host's own operations.
#pragma once
#include <stdint.h>
#include <string.h>
#ifdef __CUDACC__
#define I64_FN static __device__ __forceinline__
#define I64_COLD static __device__ __noinline__
#define I64_TABLE(ty, name) static __device__ const ty name[128]
#define I64_AT(t, i) __ldg(&t[i])
#else
#include <math.h>
#define I64_FN static inline
#define I64_COLD static inline
#define I64_TABLE(ty, name) static const ty name[128]
#define I64_AT(t, i) t[i]
#endif

#ifndef I64_SEED_SKEW
#define I64_SEED_SKEW(r) (r)  // a host test perturbs the seeds
#endif

namespace i64f {

// c_i: 2^10 / (1 + i/128), rounded up
I64_TABLE(uint32_t, LOG_C) = {
    1024, 1017, 1009, 1001, 993, 986, 979, 971, 964, 957, 950, 943, 937, 930, 924, 917,
    911, 904, 898, 892, 886, 880, 874, 869, 863, 857, 852, 846, 841, 835, 830, 825,
    820, 815, 810, 805, 800, 795, 790, 785, 781, 776, 772, 767, 763, 758, 754, 749,
    745, 741, 737, 733, 729, 725, 721, 717, 713, 709, 705, 701, 698, 694, 690, 687,
    683, 680, 676, 673, 669, 666, 662, 659, 656, 653, 649, 646, 643, 640, 637, 634,
    631, 628, 625, 622, 619, 616, 613, 610, 607, 605, 602, 599, 596, 594, 591, 588,
    586, 583, 580, 578, 575, 573, 570, 568, 565, 563, 561, 558, 556, 554, 551, 549,
    547, 544, 542, 540, 538, 535, 533, 531, 529, 527, 525, 523, 521, 519, 517, 515};
// -ln(c_i / 2^10), Q0.64
I64_TABLE(unsigned long long, LOG_T) = {
    0x0ull, 0x1c189cbb0e27fabull, 0x3c719c606662177ull, 0x5d0c874f401b4a7ull,
    0x7dea6c59e0a156dull, 0x9ae45fd5098357dull, 0xb8132d2a873bb90ull, 0xd9aeecdac5d5675ull,
    0xf7518e0035c3dd8ull, 0x1152b799bb3cc89bull, 0x1333d7f8183f4b6aull, 0x1518874226130a1eull,
    0x16bad83c1883b5e8ull, 0x18a6477a91dc28c1ull, 0x1a4e7640b1bc37a9ull, 0x1c40d6425a5cb112ull,
    0x1def0d8d466db8b0ull, 0x1fe89139dbd56595ull, 0x219cfd9b9985194bull, 0x235456fc47ee53c7ull,
    0x250ea7782357494eull, 0x26cbf9602b202c5full, 0x288c573b9367b7a7ull, 0x2a0456525ed48a06ull,
    0x2bca6628982e31f4ull, 0x2d93a0fa407f8e30ull, 0x2f131b0a8898e67cull, 0x30e2426ea1d328ebull,
    0x3266bcbab293115cull, 0x343bf881e36fe1f1ull, 0x35c594dece57a8d6ull, 0x37519215c95a32e8ull,
    0x38dff78de01ee139ull, 0x3a70ccd0e3e8c9afull, 0x3c04198c46b56a80ull, 0x3d99e591fd24139cull,
    0x3f3238d96766f2fbull, 0x40cd1b8041818a00ull, 0x426a95cb9b1b50a2ull, 0x440ab028d7307021ull,
    0x45597bb5157f0c53ull, 0x46fe658d69ae5377ull, 0x485115b43ae350fcull, 0x49faebd63632733cull,
    0x4b51980ab733b979ull, 0x4d00784abb2e838dull, 0x4e5b38d66efd4f8cull, 0x500f421b3a9e6ef5ull,
    0x516e30285f7c4ddcull, 0x52cf01dc99fa692eull, 0x5431bc7446e5f195ull, 0x55966541a545317full,
    0x56fd01ad50f6c7eeull, 0x58659736c0b07ba9ull, 0x59d02b74c77a51daull, 0x5b3cc41619c3b0b2ull,
    0x5cab66e1d6318170ull, 0x5e1c19b812457d19ull, 0x5f8ee2926b00155eull, 0x6103c784999fc03cull,
    0x621cd960c9f33b8full, 0x63957e6cd26e0de2ull, 0x651050d280c965c1ull, 0x662de0468fb96d4aull,
    0x67ac91b2d3ba84baull, 0x68cd100893e9e323ull, 0x6a4fb4f22b678dbdull, 0x6b7331bf7daa0437ull,
    0x6cf9df411b5c9da8ull, 0x6e206a9966f24d2aull, 0x6fab36789c6b4537ull, 0x70d4e0f22142bcb7ull,
    0x71ffe71d15532491ull, 0x732c4c2973aebefbull, 0x74befa4c80d31c15ull, 0x75ee9eb679f67eeaull,
    0x771facf46467ac1cull, 0x785228689c9b3653ull, 0x79861481b545b657ull, 0x7abb74bab26430cfull,
    0x7bf24c9b45aae2a1ull, 0x7d2a9fb80c64b379ull, 0x7e6471b2cecde5f6ull, 0x7f9fc63ac0f4f857ull,
    0x80dca10cc52d0757ull, 0x821b05f3b01d6774ull, 0x835af8c88e7a8f47ull, 0x849c7d72ec74d7eeull,
    0x85df97e91eea0740ull, 0x86b7e24f8b749c17ull, 0x87fdaa109d23aef7ull, 0x89451278ecd7f9cfull,
    0x8a8e1fb794b09134ull, 0x8b6a69c608cfd3afull, 0x8cb63de258f9d626ull, 0x8e03c24d7300395aull,
    0x8ee30cef034a20dbull, 0x90336bba039bf32full, 0x918586c5f5e4bf02ull, 0x9267e737c06cd34aull,
    0x93bcf0f649f65233ull, 0x94a14a3845bb985eull, 0x95f94fcc20e1d8a4ull, 0x96dfaabd86fa1647ull,
    0x983ab9a278709be8ull, 0x99231f5ee9a74f79ull, 0x9a0c58d42b116668ull, 0x9b6bbf4e9a7eb5faull,
    0x9c5710b8cbb73a43ull, 0x9d433b392b888970ull, 0x9ea71573dbf15ac9ull, 0x9f956593f6b6355cull,
    0xa084945c7ca87ba0ull, 0xa1ecff97c91e267bull, 0xa2de62326449d0a3ull, 0xa3d0a93f45169a4bull,
    0xa4c3d6706d5d83edull, 0xa6324d7f8770ad8dull, 0xa727c1962b06eb6full, 0xa81e21e6c75b4020ull,
    0xa9157039c51ebe71ull, 0xaa0dae5cbcc048b3ull, 0xab06de228a9e3499ull, 0xac010163639a9787ull,
    0xacfc19fcea147ffaull, 0xadf829d243487034ull, 0xaef532cc2d1a7e8dull, 0xaff336d9144c9071ull};
// 2^(j/128), Q1.63
I64_TABLE(unsigned long long, EXP_T) = {
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

I64_FN uint64_t bits_of(double x) {
#ifdef __CUDACC__
  return (uint64_t)__double_as_longlong(x);
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}
I64_FN double of_bits(uint64_t u) {
#ifdef __CUDACC__
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}
I64_FN uint64_t mulhi(uint64_t a, uint64_t b) {
#ifdef __CUDACC__
  return __umul64hi(a, b);
#else
  return (uint64_t)(((unsigned __int128)a * b) >> 64);
#endif
}
I64_FN uint32_t mulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }
// high 64 bits of the 96-bit product
I64_FN uint64_t mul64x32(uint64_t a, uint32_t b) {
  return (uint64_t)(uint32_t)(a >> 32) * b + (((uint64_t)(uint32_t)a * b) >> 32);
}
I64_FN int clz64(uint64_t a) {
#ifdef __CUDACC__
  return __clzll((long long)a);
#else
  return __builtin_clzll(a);
#endif
}
I64_FN float float_of(uint32_t u) {
#ifdef __CUDACC__
  return __uint_as_float(u);
#else
  float f;
  memcpy(&f, &u, 4);
  return f;
#endif
}
I64_FN uint32_t bits32(float f) {
#ifdef __CUDACC__
  return __float_as_uint(f);
#else
  uint32_t u;
  memcpy(&u, &f, 4);
  return u;
#endif
}
// seeds, relative error below 2^-21 (a normal)
I64_FN float rcp_seed(float a) {
#ifdef __CUDACC__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
#else
  return I64_SEED_SKEW(1.0f / a);
#endif
}
I64_FN float rsqrt_seed(float a) {
#ifdef __CUDACC__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(a));
  return r;
#else
  return I64_SEED_SKEW(1.0f / sqrtf(a));
#endif
}

// ------------------------------------------------------------- comparisons
I64_FN int64_t ord(uint64_t u) { return (int64_t)(u ^ ((uint64_t)((int64_t)u >> 63) >> 1)); }
// a < b, false with a NaN; -0 counts as less than +0
I64_FN bool lt(double a, double b) {
  const int64_t x = ord(bits_of(a)), y = ord(bits_of(b));
  return x < y && (int32_t)(y >> 32) <= 0x7ff00000 && (int32_t)(x >> 32) >= (int32_t)0x800fffff;
}
// (a < b) ? b : a and (b < a) ? b : a: std::max and std::min
I64_FN double max2(double a, double b) { return lt(a, b) ? b : a; }
I64_FN double min2(double a, double b) { return lt(b, a) ? b : a; }
I64_FN bool is_nan(double a) { return (bits_of(a) & 0x7fffffffffffffffull) > 0x7ff0000000000000ull; }
// fmax, fmin: a NaN yields the other argument
I64_FN double fmax2(double a, double b) { return (lt(a, b) || is_nan(a)) ? b : a; }
I64_FN double fmin2(double a, double b) { return (lt(b, a) || is_nan(a)) ? b : a; }

// ------------------------------------------------- exact scaling, conversion
// x / 2 and x / 4
I64_FN double half(double x) {
  const uint64_t u = bits_of(x);
  return ((uint32_t)(u >> 52) & 0x7ff) - 2u < 2045u ? of_bits(u - (1ull << 52)) : 0.5 * x;
}
I64_FN double quarter(double x) {
  const uint64_t u = bits_of(x);
  return ((uint32_t)(u >> 52) & 0x7ff) - 3u < 2044u ? of_bits(u - (2ull << 52)) : 0.25 * x;
}
// the integer part of a v in [1, 2^31), else 0
I64_FN int trunc_pos(double v) {
  const uint64_t u = bits_of(v);
  const uint32_t e = (uint32_t)(u >> 52) - 1023u;
  return e < 31u ? (int)(((u & 0xfffffffffffffull) | 0x10000000000000ull) >> (52 - e)) : 0;
}
I64_FN double from_float(float f) {
  const uint32_t u = bits32(f), e = (u >> 23) & 255u;
  if (e - 1u >= 254u) return (double)f;
  return of_bits(((uint64_t)(u & 0x80000000u) << 32) | (((uint64_t)(u & 0x7fffffffu) << 29) + (896ull << 52)));
}

// ---------------------------------------------------------------- division
I64_COLD double div_any(double a, double b) { return a / b; }
I64_FN double div(double a, double b) {
  const uint64_t ua = bits_of(a), ub = bits_of(b);
  const int ea = (int)(ua >> 52) & 0x7ff, eb = (int)(ub >> 52) & 0x7ff;
  const uint64_t sign = (ua ^ ub) & 0x8000000000000000ull;
  const uint64_t ma = (ua & 0xfffffffffffffull) | 0x10000000000000ull;
  const uint64_t mb = (ub & 0xfffffffffffffull) | 0x10000000000000ull;
  const int ge = ma >= mb;
  const int e = ea - eb + 1022 + ge;  // biased exponent of the quotient
  const bool zero = (ua << 1) == 0;
  if ((unsigned)(eb - 1) >= 2046u || !(zero || ((unsigned)(ea - 1) < 2046u && (unsigned)(e - 1) < 2046u)))
    return div_any(a, b);
  const uint64_t X = ma << 11, B = mb << 11;  // x, b in [1/2, 1), Q0.64
  // r0 ~ 1/b, Q1.31: the float has 24 bits in [1, 2]
  const uint32_t fb = bits32(rcp_seed(float_of(0x3f000000u | ((uint32_t)(mb >> 29) & 0x7fffffu))));
  const uint32_t r0 = fb >= 0x40000000u ? 0xffffffffu : (fb < 0x3f800000u ? 0x80000000u : (fb << 8) | 0x80000000u);
  const int64_t d0 = (int64_t)(0x8000000000000000ull - mul64x32(B, r0));  // 1 - b r0, Q1.63
  const uint64_t r1 = ((uint64_t)r0 << 32) + (uint64_t)(((int64_t)(int32_t)(d0 >> 12) * (int64_t)(uint64_t)r0) >> 19);
  const uint64_t q1 = mulhi(X, r1);  // Q1.63
  const int64_t d1 = (int64_t)((X >> 1) - mulhi(q1, B));  // x - q1 b, Q1.63
  const uint64_t q2 = q1 + (uint64_t)((d1 * (int64_t)(uint64_t)(uint32_t)(r1 >> 32)) >> 31);
  uint64_t q = q2 >> (9 + ge);  // 54 bits
  int64_t rem = (int64_t)((ma << (54 - ge)) - q * mb);
  if (rem < 0) { q -= 1; rem += (int64_t)mb; }
  if (rem >= (int64_t)mb) q += 1;
  const uint64_t r = (q >> 1) + (q & 1);
  return of_bits(sign | (zero ? 0ull : ((uint64_t)(e - 1) << 52) + r));
}

// ------------------------------------------------------------- square root
I64_COLD double sqrt_any(double a) { return sqrt(a); }
I64_FN double sqrt_(double a) {
  const uint64_t u = bits_of(a);
  const uint32_t h = (uint32_t)(u >> 32);
  if (h - 0x00100000u >= 0x7fe00000u) return u == 0 ? a : sqrt_any(a);
  const int ea = (int)(h >> 20);
  const int odd = (ea & 1) ^ 1;  // unbiased exponent ea - 1023 odd
  const uint64_t A = ((u & 0xfffffffffffffull) | 0x10000000000000ull) << (10 + odd);  // [1, 4), Q2.62
  const uint32_t fy = bits32(rsqrt_seed(float_of((uint32_t)(127 + odd) << 23 | ((h << 3) & 0x7fffffu) | ((uint32_t)u >> 29))));
  const uint32_t y = fy >= 0x3f800000u ? 0xffffffffu : (fy < 0x3f000000u ? 0x80000000u : (fy << 8) | 0x80000000u);
  // y ~ 1/sqrt, Q0.32
  const uint64_t t0 = mul64x32(A, y) >> 31;
  const uint32_t s0 = (t0 >> 32) ? 0xffffffffu : (uint32_t)t0;  // Q1.31
  const int64_t d0 = (int64_t)(A - (uint64_t)s0 * s0);                             // a - s0^2, Q2.62
  const uint64_t s1 = ((uint64_t)s0 << 31) + (uint64_t)(((int64_t)(int32_t)(d0 >> 14) * (int64_t)(uint64_t)y) >> 19);
  const int64_t d1 = (int64_t)((A >> 2) - mulhi(s1, s1));                          // Q4.60
  const uint64_t s2 = s1 + (uint64_t)((d1 * (int64_t)(uint64_t)y) >> 31);          // Q2.62
  uint64_t s = s2 >> 9;                                                            // 54 bits
  int64_t rem = (int64_t)((A << 44) - s * s);
  if (rem < 0) { s -= 1; rem += (int64_t)(2 * s + 1); }
  if (rem > (int64_t)(2 * s)) s += 1;
  const uint64_t r = (s >> 1) + (s & 1);
  return of_bits(((uint64_t)(((ea - 1023 - odd) >> 1) + 1022) << 52) + r);
}

// --------------------------------------------------------------- logarithm
I64_COLD double log_any(double x) { return log(x); }
I64_FN double log_(double x) {
  const uint64_t u = bits_of(x);
  const uint32_t h = (uint32_t)(u >> 32);
  if (h - 0x00100000u >= 0x7fe00000u) return log_any(x);
  const int k = (int)(h >> 20) - 1023;
  const uint32_t i = (h >> 13) & 127u;
  const uint64_t m = (u & 0xfffffffffffffull) | 0x10000000000000ull;
  const uint32_t ci = I64_AT(LOG_C, i);
  const uint64_t Ti = I64_AT(LOG_T, i);
  const uint64_t z = (m * ci - 0x4000000000000000ull) << 2;  // exact, [0, 0.0087), Q0.64
  const uint32_t w = (uint32_t)(z >> 26);                      // 64 z, Q0.32
  // log1p(z) = z - z^2 (1/2 - z (1/3 - z/4 + z^2 (1/5 - z/6 + z^2/7 - z^3/8)))
  uint32_t q = 0x24924924u - (mulhi32(w, 0x20000000u) >> 6);
  q = 0x2aaaaaabu - (mulhi32(w, q) >> 6);
  q = 0x33333333u - (mulhi32(w, q) >> 6);
  const uint64_t z2 = mulhi(z, z);
  const uint64_t p = 0x5555555555555555ull - (z >> 2) + mul64x32(z2, q);
  const uint64_t r = z - mulhi(z2, 0x8000000000000000ull - mulhi(z, p));
  // k ln2 + T + r as (hi, lo), lo a fraction
  const uint64_t ak = (uint64_t)(uint32_t)(k < 0 ? -k : k);
  uint64_t lo = ak * 0xb17217f7d1cf79acull, hi = mulhi(ak, 0xb17217f7d1cf79acull);
  if (k < 0) { hi = ~hi + (lo == 0); lo = 0 - lo; }
  const uint64_t add = Ti + r;
  lo += add;
  hi += lo < add;
  const bool neg = (int64_t)hi < 0;
  if (neg) { hi = ~hi + (lo == 0); lo = 0 - lo; }
  if (hi == 0 && lo < 0x1000000000000000ull) return log_any(x);
  const int sh = hi ? 64 - clz64(hi) : -clz64(lo);  // |log x| in [2^(sh-1), 2^sh)
  const uint64_t v = sh > 0 ? (hi << (64 - sh)) | (lo >> sh) : lo << -sh;
  return of_bits(((uint64_t)neg << 63) | (((uint64_t)(1021 + sh) << 52) + (v >> 11) + ((v >> 10) & 1)));
}

// ------------------------------------------------------------- exponential
I64_COLD double exp_any(double x) { return exp(x); }
I64_FN double exp_(double x) {
  const uint64_t u = bits_of(x);
  const uint32_t h = (uint32_t)(u >> 32) & 0x7fffffffu;
  if (h >= 0x40862000u) return exp_any(x);  // |x| >= 708, infinities, NaN
  const int s = 51 + 1023 - (int)(h >> 20);  // |x| / ln2 = P 2^-s (integer part above 2^64)
  const uint64_t m = (u & 0xfffffffffffffull) | 0x10000000000000ull;
  const uint64_t plo = m * 0xb8aa3b295c17f0bcull, phi = mulhi(m, 0xb8aa3b295c17f0bcull);
  uint64_t f, I;
  if (s < 64) { f = (phi << (64 - s)) | (plo >> s); I = phi >> s; }
  else { f = s < 128 ? phi >> (s - 64) : 0; I = 0; }
  if (u >> 63) { I = ~I + (f == 0); f = 0 - f; }
  const int k = (int)(int64_t)I;
  const uint32_t j = (uint32_t)(f >> 57);
  const uint64_t Y = mulhi(f << 7, 0xb17217f7d1cf79abull);  // 128 y, Q0.64; y < 2^-7.5
  const uint32_t w = (uint32_t)(Y >> 32);
  // e^y - 1 = y + y^2 (1/2 + y/6 + y^2 (1/24 + y/120 + y^2/720))
  uint32_t q = 0x02222222u + (mulhi32(w, 0x005b05b0u) >> 7);
  q = 0x0aaaaaaau + (mulhi32(w, q) >> 7);
  const uint64_t y2 = mulhi(Y, Y);  // 2^14 y^2
  const uint64_t p = 0x8000000000000000ull + (mulhi(Y, 0x2aaaaaaaaaaaaaaaull) >> 7) + (mul64x32(y2, q) >> 14);
  const uint64_t e1 = (Y >> 7) + (mulhi(y2, p) >> 14);
  const uint64_t T = I64_AT(EXP_T, j);
  const uint64_t v = T + mulhi(T, e1);  // Q1.63, [1, 2)
  return of_bits(((uint64_t)(1022 + k) << 52) + (v >> 11) + ((v >> 10) & 1));
}

}  // namespace i64f
