// Fixed-point arithmetic of the likelihood and prediction blocks
// (sv_loglik_fix.cu, sv_predict_fix.cu) and of the Matern tables: numbers
// of magnitude at most 1 as 64-bit integers in units of 2^-58 ("Q58"), split
// for products into two 30-bit limbs, x = h 2^30 + l with |l| <= 2^29.
//
// GB300 issues a float64 warp instruction every 64 cycles per scheduler and a
// 32 x 32 + 64 bit integer multiply-add every 4 (both measured). A product of
// two split numbers accumulated over a sum takes three of the latter: h h'
// into one 64-bit accumulator, h l' + l h' into another; l l', at most 2^-58 and
// a third of that in the root mean square, is left out (where that adds up with one
// sign or is magnified it is not: pivots, distances, back substitutions). So a
// multiply-add costs 12 cycles instead of 64, the rest of its accumulation is
// exact, and a sum of K products is off by some sqrt(K) / 3 units of 2^-58 of
// the scale and one rounding, where float64 rounds every term to 2^-53 of it. Correlations, their Cholesky
// factor and the whitened columns are bounded by construction, so the scale is
// known; what is not is rescaled or left to the float64 kernels.
//
// Host code may include this header (the tests check it against long double).
#pragma once
#include <stdint.h>
#if !defined(__CUDACC__)
#include <math.h>
#include <string.h>
#endif

#ifndef SV_FX
#if defined(__CUDACC__)
#define SV_FX __host__ __device__ __forceinline__
#else
#define SV_FX inline
#endif
#endif

namespace sv {

// 2^(-i/256), i = 0..255, in units of 2^-63
#if defined(__CUDACC__)
__device__
#endif
const uint64_t kFxExp2[256] = {
    0x8000000000000000ull, 0x7fa765aca88f6453ull, 0x7f4f08ae3dc7c426ull, 0x7ef6e8da4b544f9aull,
    0x7e9f06067a4360baull, 0x7e47600890f223deull, 0x7deff6b672f84e24ull, 0x7d98c9e62113e1faull,
    0x7d41d96db915019dull, 0x7ceb252375c9cf9bull, 0x7c94acddaeea5d3aull, 0x7c3e7072d904a6ceull,
    0x7be86fb985689ddcull, 0x7b92aa886214411cull, 0x7b3d20b6399fc237ull, 0x7ae7d219f329b948ull,
    0x7a92be8a92436616ull, 0x7a3de5df36dcfeefull, 0x79e947ef1d320d2dull, 0x7994e4919db5d74eull,
    0x7940bb9e2cffd89dull, 0x78ecccec5bb84661ull, 0x78991853d684a285ull, 0x78459dac65f45bb5ull,
    0x77f25ccdee6d7ae6ull, 0x779f559070195e36ull, 0x774c87cc06d1812eull, 0x76f9f358ea0c5249ull,
    0x76a7980f6cca15c2ull, 0x765575c7fd81d5a0ull, 0x76038c5b260e5eeeull, 0x75b1dba18b9b4c20ull,
    0x75606373ee921c97ull, 0x750f23ab2a87593eull, 0x74be1c203627c62bull, 0x746d4cac2325a155ull,
    0x741cb5281e25ee34ull, 0x73cc556d6eadce5full, 0x737c2d55770fe711ull, 0x732c3cb9b459d38bull,
    0x72dc8373be41a454ull, 0x728d015d47136b40ull, 0x723db6501b9ed447ull, 0x71eea2262324cb0cull,
    0x719fc4b95f452d29ull, 0x71511de3ebec8913ull, 0x7102ad7fff41e9b4ull, 0x70b47367e994ae92ull,
    0x70666f76154a7089ull, 0x7018a18506ccf314ull, 0x6fcb096f5c782210ull, 0x6f7da70fce881bf9ull,
    0x6f307a412f074892ull, 0x6ee382de69bc7bf8ull, 0x6e96c0c284192610ull, 0x6e4a33c89d278e49ull,
    0x6dfddbcbed791babull, 0x6db1b8a7c714a92bull, 0x6d65ca379564e639ull, 0x6d1a1056dd26c382ull,
    0x6cce8ae13c57ebdbull, 0x6c8339b26a25494eull, 0x6c381ca636d99642ull, 0x6bed33988bcbfab5ull,
    0x6ba27e656b4eb57aull, 0x6b57fce8f09dd17full, 0x6b0daeff4fcde703ull, 0x6ac39484d5bae8c5ull,
    0x6a79ad55e7f6fd10ull, 0x6a2ff94f04b962b0ull, 0x69e6784cc2cd61bdull, 0x699d2a2bd181482aull,
    0x69540ec8f895722dull, 0x690b2601182b5e56ull, 0x68c26fb128b4cd63ull, 0x6879ebb63ae2edc6ull,
    0x683199ed779592caull, 0x67e97a341fca775bull, 0x67a18c678c8c8c61ull, 0x6759d0652ee352afull,
    0x6712460a8fc24072ull, 0x66caed354ff83222ull, 0x6683c5c3281ee6e9ull, 0x663ccf91e88a8873ull,
    0x65f60a7f79393e2eull, 0x65af7669d9c2cbe4ull, 0x6569132f21483ba7ull, 0x6522e0ad7e639312ull,
    0x64dcdec3371793d1ull, 0x64970d4ea8bf8766ull, 0x64516c2e47ff1623ull, 0x640bfb40a0b22959ull,
    0x63c6ba6455dcd8aeull, 0x6381a978219b628full, 0x633cc85ad5122fbdull, 0x62f816eb585de1edull,
    0x62b39508aa836d6full, 0x626f4291e1603dd5ull, 0x622b1f66299a6599ull, 0x61e72b64c690d8afull,
    0x61a3666d124bb204ull, 0x615fd05e7d6c83e4ull, 0x611c69188f1eb339ull, 0x60d9307ae507dd9aull,
    0x6096266533384a2bull, 0x60534ab7441b6546ull, 0x60109d50f86846d8ull, 0x5fce1e124712437cull,
    0x5f8bccdb3d398841ull, 0x5f49a98bfe1bc11cull, 0x5f07b404c304c9f1ull, 0x5ec5ec25db3f6a41ull,
    0x5e8451cfac061b5full, 0x5e42e4e2b073d935ull, 0x5e01a53f7974fd86ull, 0x5dc092c6adb825b8ull,
    0x5d7fad59099f22feull, 0x5d3ef4d75f2ff504ull, 0x5cfe69229605cef5ull, 0x5cbe0a1bab4226dfull,
    0x5c7dd7a3b17dcf75ull, 0x5c3dd19bd0ba1c1aull, 0x5bfdf7e546520f3eull, 0x5bbe4a6164eb92f4ull,
    0x5b7ec8f19468bbc9ull, 0x5b3f737751d915c8ull, 0x5b0049d42f6afbb6ull, 0x5ac14be9d45cf869ull,
    0x5a827999fcef3242ull, 0x5a43d2c67a54e0c0ull, 0x5a05575132a5cc20ull, 0x59c7071c20cfd70cull,
    0x5988e20954889245ull, 0x594ae7faf23eda52ull, 0x590d18d3330c7f1eull, 0x58cf747464a7f584ull,
    0x5891fac0e95612c8ull, 0x5854ab9b37dbd1e5ull, 0x581786e5db7022c2ull, 0x57da8c8373adc331ull,
    0x579dbc56b48521baull, 0x57611642662e4a33ull, 0x57249a29651adc07ull, 0x56e847eea1e80a49ull,
    0x56ac1f752150a563ull, 0x5670209ffc1f2e82ull, 0x56344b525f1ff495ull, 0x55f89f6f8b133af4ull,
    0x55bd1cdad49f699cull, 0x5581c377a44346f0ull, 0x5546932976483b15ull, 0x550b8bd3dab49cbdull,
    0x54d0ad5a753e077cull, 0x5495f7a0fd3bbb8eull, 0x545b6a8b3d990704ull, 0x542105fd14c7b869ull,
    0x53e6c9da74b29ab5ull, 0x53acb60762affaaeull, 0x5372ca67f774358full, 0x533906e05f045106ull,
    0x52ff6b54d8a89c75ull, 0x52c5f7a9b6df5b77ull, 0x528cabc35f4f799dull, 0x525387864abb4762ull,
    0x521a8ad704f3404full, 0x51e1b59a2cc8da3eull, 0x51a907b474015dc9ull, 0x5170810a9f48c7cfull,
    0x513821818624b40cull, 0x50ffe8fe12e750c4ull, 0x50c7d76542a25b72ull, 0x508fec9c251a267cull,
    0x50582887dcb8a7e1ull, 0x50208b0d9e8090dfull, 0x4fe91412b2006e83ull, 0x4fb1c37c7145d328ull,
    0x4f7a993048d088d7ull, 0x4f439513b785cc80ull, 0x4f0cb70c4ea39210ull, 0x4ed5feffb1b3d155ull,
    0x4e9f6cd3967fdba8ull, 0x4e69006dc503ba65ull, 0x4e32b9b417619617ull, 0x4dfc988c79d52661ull,
    0x4dc69cdceaa72a9cull, 0x4d90c68b7a20eb1eull, 0x4d5b157e4a7fc325ull, 0x4d25899b8fe8b365ull,
    0x4cf022c9905bfd32ull, 0x4cbae0eea3a8c63cull, 0x4c85c3f13360c4d5ull, 0x4c50cbb7bacbf4cbull,
    0x4c1bf828c6dc54b8ull, 0x4be7492af621abd6ull, 0x4bb2bea4f8bd5847ull, 0x4b7e587d905625d1ull,
    0x4b4a169b900c2d00ull, 0x4b15f8e5dc6cbab0ull, 0x4ae1ff436b663ff7ull, 0x4aae299b443c4a6bull,
    0x4a7a77d47f7b84b1ull, 0x4a46e9d646edbf6aull, 0x4a137f87d58e025bull, 0x49e038d0777ca5e0ull,
    0x49ad159789f37496ull, 0x497a15c47b39d53eull, 0x4947393eca98fcd6ull, 0x49147fee085028d6ull,
    0x48e1e9b9d588e19bull, 0x48af7689e44b44eaull, 0x487d2645f7725895ull, 0x484af8d5e2a06536ull,
    0x4818ee218a3358eeull, 0x47e70610e3393241ull, 0x47b5408bf36472e2ull, 0x47839d7ad1009a90ull,
    0x47521cc5a2e6a9e0ull, 0x4720be54a071ad01ull, 0x46ef821011734e6bull, 0x46be67e04e28717cull,
    0x468d6fadbf2dd4f3ull, 0x465c9960dd74bd4bull, 0x462be4e23237a6efull, 0x45fb521a56ef0042ull,
    0x45cae0f1f545eb73ull, 0x459a9151c70f0819ull, 0x456a632296394492ull, 0x453a564d3cc4b723ull,
    0x450a6abaa4b77ecdull, 0x44daa053c812abd2ull, 0x44aaf701b0c72feeull, 0x447b6ead78aad636ull,
    0x444c0740496d4294ull, 0x441cc0a35c8cf8eaull, 0x43ed9abffb4c6bc9ull, 0x43be957f7ea712b6ull,
    0x438fb0cb4f468808ull, 0x4360ec8ce577ae44ull, 0x433248adc91fdd02ull, 0x4303c51791b21550ull,
    0x42d561b3e6243d8aull, 0x42a71e6c7ce464afull, 0x4278fb2b1bce0d15ull, 0x424af7d9981f7e98ull,
    0x421d1461d66f2023ull, 0x41ef50adcaa0d899ull, 0x41c1aca777db771bull, 0x41942838f07e22a3ull,
    0x4166c34c5615d0ecull, 0x41397dcbd952c4a6ull, 0x410c57a1b9fe12f6ull, 0x40df50b846ef302bull,
    0x40b268f9de0183baull, 0x4085a050ec0a036aull, 0x4058f6a7ecccd5b6ull, 0x402c6be96af2fb58ull,
};

constexpr uint64_t kFxLn2 = 0x58b90bfbe8e7bcd6ull;    // ln 2, Q63
constexpr uint64_t kFxThird = 0x2aaaaaaaaaaaaaabull;  // 1/3, Q63
constexpr uint64_t kFxA3 = 0x376cf5d0b09954e7ull;     // sqrt 3, Q61
constexpr uint64_t kFxA5 = 0x478dde6e5fd29f05ull;     // sqrt 5, Q61
constexpr uint64_t kFxK3 = 0x4ff657b0991c9270ull;     // sqrt 3 log2 e, Q61
constexpr uint64_t kFxK5 = 0x673b193c97c981c9ull;     // sqrt 5 log2 e, Q61

struct alignas(8) Fx2 {
  int32_t h, l;
};

SV_FX int fx_clz(uint64_t x) {
#if defined(__CUDA_ARCH__)
  return __clzll((long long)x);
#else
  return x ? __builtin_clzll(x) : 64;
#endif
}

SV_FX Fx2 fx_split(int64_t x) {
  Fx2 v;
  v.h = (int32_t)((x + (1ll << 29)) >> 30);
  v.l = (int32_t)((uint32_t)x << 2) >> 2;
  return v;
}
SV_FX int64_t fx_join(Fx2 v) { return (int64_t)v.h * (1ll << 30) + v.l; }

struct FxAcc {
  int64_t h, m;
};
SV_FX void fx_mac(FxAcc& a, Fx2 x, Fx2 y) {
  a.h += (int64_t)x.h * y.h;
  a.m += (int64_t)x.h * y.l;
  a.m += (int64_t)x.l * y.h;
}
// the sum in Q58
SV_FX int64_t fx_val(const FxAcc& a) { return (int64_t)((uint64_t)a.h << 2) + ((a.m + (1ll << 27)) >> 28); }
SV_FX int64_t fx_mul(Fx2 x, Fx2 y) {
  FxAcc a = {0, 0};
  fx_mac(a, x, y);
  return fx_val(a);
}

// the high 64 bits of x y for x, y <= 2^63, low by at most 2 of their units
// (three 32 x 32 bit products)
SV_FX uint64_t fx_mulhi(uint64_t x, uint64_t y) {
  const uint32_t xh = (uint32_t)(x >> 32), xl = (uint32_t)x, yh = (uint32_t)(y >> 32), yl = (uint32_t)y;
  const uint64_t m = (uint64_t)xh * yl + (uint64_t)xl * yh;
  return (uint64_t)xh * yh + (m >> 32);
}
// x y 2^-32 for a 32-bit y
SV_FX uint64_t fx_mul32(uint64_t x, uint32_t y) {
  return (uint64_t)(uint32_t)(x >> 32) * y + (((uint64_t)(uint32_t)x * y) >> 32);
}
SV_FX uint32_t fx_mulhi32(uint32_t x, uint32_t y) { return (uint32_t)(((uint64_t)x * y) >> 32); }

// x >> k for any k >= 0 (0 beyond 63)
SV_FX uint64_t fx_shr(uint64_t x, int k) {
#if defined(__CUDA_ARCH__)
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(x), "r"(k));
  return r;
#else
  return k > 63 ? 0 : x >> k;
#endif
}

// 2^k, 0 beyond 63
SV_FX uint64_t fx_shl1(int k) { return k > 63 ? 0 : 1ull << k; }

// For m 2^-63 in [1/4, 1): the float32 reciprocal square root y0 (Q29),
// g0 = m y0 (Q60), and t with 1/sqrt = y0 (1 + t), sqrt = g0 (1 + t): one
// third-order step t = e/2 + 3 e^2 / 8 (Q61), e = 1 - m y0^2 (|e| < 2^-20; the
// next term is below 2^-61)
SV_FX int64_t fx_rsqrt_step(uint64_t m, uint32_t& y0, uint64_t& g0) {
  const float f = (float)(uint32_t)(m >> 31) * 2.3283064365386963e-10f;
#if defined(__CUDA_ARCH__)
  const float yf = rsqrtf(f);
#else
  const float yf = 1.0f / sqrtf(f);
#endif
  y0 = (uint32_t)(yf * 536870912.0f);                                   // exact
  g0 = fx_mul32(m, y0);                                                 // Q60
  const int64_t e = (int64_t)((1ull << 61) - 8 - (fx_mul32(g0, y0) << 4));  // Q57, in units of Q61; 8: the mean of what the products drop
  const int32_t e10 = (int32_t)(e >> 10);                               // Q51
  const uint32_t ee = (uint32_t)((uint64_t)((int64_t)e10 * e10) >> 32); // Q70
  return (e >> 1) + ((3 * ee) >> 12);
}
// x t for a Q61 t below 2^40 in magnitude, x below 2^62: in x's units
SV_FX int64_t fx_scale_step(uint64_t x, int64_t t) {
  const int32_t xh = (int32_t)(x >> 31), xl = (int32_t)(x & 0x7fffffff);
  const int32_t th = (int32_t)(t >> 10), tl = (int32_t)(t & 0x3ff);  // Q51 and the rest
  return ((int64_t)xh * th + (((int64_t)xh * tl) >> 10) + (((int64_t)xl * (th >> 12)) >> 19)) >> 20;
}

// 1 / sqrt(d) for d in Q58, 2^16 <= d <= 2^58, as Y 2^e: Y in (1/2, 1] (Q58),
// e >= 0
SV_FX int64_t fx_rsqrt_pivot(int64_t d, int& e) {
  const int h2 = fx_clz((uint64_t)d) & ~1;
  e = h2 / 2 - 2;
  uint32_t y0;
  uint64_t g0;
  const uint64_t m = (uint64_t)d << (h2 - 1);
  const int64_t t = fx_rsqrt_step(m, y0, g0);
  // Y = y0 (1 + t) / 2 in Q58
  const int32_t th = (int32_t)(t >> 16), tl = (int32_t)(t & 0xffff);
  const int64_t add = (int64_t)(int32_t)y0 * th + (((int64_t)(int32_t)y0 * tl) >> 16);  // Q74
  return ((int64_t)y0 << 28) + ((add + (1 << 16)) >> 17);
}

// e^-z (Q63) for z < 2^-8 ln 2 (Q70): the Taylor polynomial of degree 5
SV_FX uint64_t fx_exp_tail(uint64_t z) {
  const uint32_t zt = (uint32_t)(z >> 30);  // Q40
  // z^2 from the top 32 bits and their cross product with the rest: Q80
  const uint64_t z2 = (uint64_t)zt * zt + (((uint64_t)zt * (uint32_t)(((uint32_t)z & 0x3fffffffu) << 2)) >> 31);
  const uint32_t z2t = (uint32_t)(z2 >> 32);   // Q48
  const uint32_t z3 = 2 * fx_mulhi32(z2t, zt) + 1;  // Q57, with the mean of what is dropped
  // 1/6 - z/24 + z^2/120, Q34
  const uint32_t c3 = 2863311531u - fx_mulhi32(zt, 2796203u) + fx_mulhi32(z2t, 2185u);
  return (1ull << 63) - (z >> 7) + (z2 >> 18) - (((uint64_t)z3 * c3) >> 28);
}

// The squared distance of two points whose coordinates are split integers
// below 2^59: per input the square of the difference dh 2^30 + dl, exactly, as
// three sums at 2^60, 2^31 and 1. Differences first, so that a close pair keeps
// its relative accuracy however far both lie from the origin, and equal rows
// come out at 0 (|x|^2 + |y|^2 - 2 x.y is off by a unit of the whole extent's
// square: 31 ranges from the origin that reached 2^-46 of the variance, and
// had one sign for replicates). The limbs' differences are as many multiply-adds.
struct FxSq {
  uint64_t hh, ll;  // sums of 12 squares below 2^60
  int64_t hl;
};
SV_FX void fx_sqdiff(FxSq& a, Fx2 x, Fx2 y) {
  const int32_t dh = x.h - y.h, dl = x.l - y.l;  // |dh| <= 2^30, |dl| < 2^30
  a.hh += (uint64_t)((int64_t)dh * dh);
  a.hl += (int64_t)dh * dl;
  a.ll += (uint64_t)((int64_t)dl * dl);
}
// after 8 terms: room for 4 more in the middle sum, which is at most
// 2^30 sqrt(8 hh) (below 64 it needs none, and hh might go below 0)
SV_FX void fx_sqcarry(FxSq& a) {
  const int64_t t = a.hh >= 64 ? a.hl >> 29 : 0;
  a.hh += (uint64_t)t;
  a.hl -= (int64_t)((uint64_t)t << 29);
}
// The sum as s 2^(2 E) with s in [1/4, 1), Q64 (truncated), for coordinates in
// Q61 of 2^es; a sum of 0 reads as s = 1/4, E = es - 92 (es <= 7: it correlates
// by 1)
SV_FX uint64_t fx_sqnorm(const FxSq& a, int es, int& E) {
  const uint64_t l0 = a.hh << 60, l1 = (uint64_t)a.hl << 31;
  uint64_t lo = l0 + l1, hi = (a.hh >> 4) + (uint64_t)(a.hl >> 33) + (lo < l0 ? 1 : 0);
  lo += a.ll;
  hi += lo < a.ll ? 1 : 0;
  const bool low = hi == 0;
  hi = low ? lo : hi;
  lo = low ? 0 : lo;
  const bool none = hi == 0;
  hi |= none ? 1 : 0;
  const int z = fx_clz(hi) & ~1;
  E = es + 3 - z / 2 - (low ? 32 : 0) - (none ? 32 : 0);
  return hi << z | (lo >> 1) >> (63 - z);
}

// Matern 3/2 (code 1) and 5/2 (code 2) of a squared distance s 2^(2 E), s in
// [1/4, 1) (Q64): the correlation M, and the factor of its
// derivative, g = e^-c (3/2: M'(r)/r = -3 g) or (1 + c) e^-c (5/2:
// M'(r)/r = -5/3 g), c = sqrt(3) r or sqrt(5) r; both in Q61, absolute error
// a few 2^-59. SCALED: g 2^(2 E) instead (below 1.5, since 2^E < 2 r), to
// which squared differences in units of 2^E belong. exp(-c) = 2^-t,
// t = c log2 e: the integer part shifts, the
// next 8 bits index the table of 2^(-i/256) (Tang's table-driven method), the
// rest takes the Taylor polynomial of degree 5 of e^-z, z < 2^-8 ln 2. c and
// its powers keep their own exponent until they meet e^-c. The mean errors
// are below 2^-61: a common shift of all entries, 2^-58 say, would reach a
// small pivot of every block with the same sign, and add up over the blocks.
template <int CODE, bool SCALED>
SV_FX void fx_matern_norm(uint64_t s, int E, const uint64_t* T, uint64_t& M, uint64_t& g) {
  uint32_t y0;
  uint64_t q;
  const int64_t st = fx_rsqrt_step(s >> 1, y0, q);
  q = (q << 2) + (uint64_t)(fx_scale_step(q, st) * 4);  // sqrt(s), Q62
  const uint64_t t0 = fx_mulhi(q << 1, CODE == 1 ? kFxK3 : kFxK5) + 2;  // Q60; 2: the mean of what the products drop
  // t in Q57; beyond 79 (E > 5) the results are below 2^-70
  const int sh = 3 - E;
  const uint64_t t = sh >= 0 ? fx_shr(t0 + (fx_shl1(sh) >> 1), sh) : t0 << (E > 5 ? 0 : -sh);
  const uint32_t th = (uint32_t)(t >> 32);
  const int n = E > 5 ? 128 : (int)(th >> 25);
  const uint64_t rem = t & ((1ull << 49) - 1);
  const uint64_t e = fx_mulhi(fx_exp_tail(fx_mulhi(rem << 14, kFxLn2)), T[(th >> 17) & 255]);  // Q62
  const uint64_t c = fx_mulhi(q << 1, CODE == 1 ? kFxA3 : kFxA5);  // c = this 2^E, Q60
  const uint64_t F = fx_mulhi(c << 1, e << 1) + 1;                 // c e^-c, Q60 before the shift
  const uint64_t e0 = fx_shr(e, n + 1);
  const int kf = n - E - 1;  // -1 only at c < 1: the shift up by one
  const uint64_t eF = e0 + (kf < 0 ? F << 1 : fx_shr(F, kf));
  if (CODE == 1) {
    M = eF;
    g = SCALED ? fx_shr(e, n + 1 - 2 * E) : e0;
  } else {
    const uint64_t G = fx_mulhi(fx_mulhi(c << 1, F << 1) << 2, kFxThird) + 1;  // c^2 e^-c / 3, Q59
    const int kg = n - 2 * E - 2;
    M = eF + (kg < 0 ? G << -kg : fx_shr(G, kg)) + 1;
    const int ks = kf - 2 * E;
    g = SCALED ? fx_shr(e, n + 1 - 2 * E) + (ks < 0 ? F << -ks : fx_shr(F, ks)) : eF;
  }
}
// the same of s in Q62 of 2^(2 es); r = 0: M and g come out as 1 less the
// rounding
template <int CODE>
SV_FX void fx_matern(uint64_t s, int es, const uint64_t* T, uint64_t& M, uint64_t& g) {
  s = s > 0 ? s : 1;
  const int z = fx_clz(s) & ~1;
  fx_matern_norm<CODE, false>(s << z, es + 1 - z / 2, T, M, g);
}

// x 2^n, rounded to nearest (ties up) where bits are lost; the result fits
SV_FX int64_t fx_scale2(int64_t x, int n) {
  if (n >= 0) return (int64_t)((uint64_t)x << (n & 63));
  return n < -62 ? 0 : (x + (1ll << (-n - 1))) >> -n;
}
SV_FX int fx_bits(int64_t x) { return 64 - fx_clz((uint64_t)(x < 0 ? -x : x)); }

// v 2^ex as float64, rounded to nearest (ties up); no subnormal results
SV_FX double fx_to_double(uint64_t v, int ex) {
  if (v == 0) return 0.0;
  const int lz = fx_clz(v);
  v <<= lz;
  const uint64_t b = ((uint64_t)(ex + 63 - lz + 1022) << 52) + (v >> 11) + ((v >> 10) & 1);
#if defined(__CUDA_ARCH__)
  return __longlong_as_double((long long)b);
#else
  double r;
  memcpy(&r, &b, 8);
  return r;
#endif
}

// General Matern from tables in fixed point (a row: sv_matern.cuh's intervals
// as polynomials, see mtab_fix_interval).  The polynomial's 16 coefficients
// are Q58 of 2^ex (the top 16 bits of the last word; the sum of their
// magnitudes is below 2), by Horner's rule in t (Q58): value (Q58) of 2^ex.
constexpr uint64_t kFxTabS0 = 0x4d413cccfe779921ull;  // 2 (1 + sqrt 2), Q60
constexpr uint64_t kFxTabS1 = 0x36a09e667f3bcc90ull;  // 2 + sqrt 2, Q60
constexpr int64_t kFxTabO1 = 0x09a827999fcef324ll;    // 1 + sqrt 2, Q58
constexpr uint64_t kFxLog2e = 0x5c551d94ae0bf85eull;  // log2 e, Q62
// t in [-1, 1] (Q58) of the mantissa fraction f (52 bits) on the lower
// ([1, sqrt2)) or upper ([sqrt2, 2)) half of an octave
SV_FX int64_t fx_tab_t(uint64_t f, bool upper) {
  const uint64_t p = fx_mulhi(f << 11, upper ? kFxTabS1 : kFxTabS0);  // Q59
  return (int64_t)(p >> 1) - (upper ? kFxTabO1 : 1ll << 58);
}
// e^-c for c = (1 + f 2^-52) 2^e, -40 <= e < 9: the result (Q62) times 2^-n.
// t = c log2 e, its fraction in Q57: rounded to nearest below c = 8 (e^-c is
// within 2 units of 2^-58, and low or high by a third of one in the mean: an
// error common to all near pairs adds up), truncated above, where e^-c is
// small (the integer part must not take a carry)
SV_FX uint64_t fx_exp_neg(uint64_t f, int e, const uint64_t* T, int& n) {
  const uint64_t m = (1ull << 62) + (f << 10);
#if defined(__CUDA_ARCH__)
  const uint64_t p = __umul64hi(m, kFxLog2e), pl = m * kFxLog2e;  // Q124 before 2^e
#else
  const unsigned __int128 q = (unsigned __int128)m * kFxLog2e;
  const uint64_t p = (uint64_t)(q >> 64), pl = (uint64_t)q;
#endif
  const int sh = 3 - e;
  const uint64_t t = sh > 0 ? (p + (1ull << (sh - 1))) >> sh : p << -sh | (pl >> 1) >> (63 + sh);
  n = (int)(sh > 0 ? t >> 57 : p >> (57 + sh));
  const uint64_t rem = t & ((1ull << 49) - 1);
  return fx_mulhi(fx_exp_tail(fx_mulhi(rem << 14, kFxLn2)), T[(t >> 49) & 255]);
}

// mantissa and sign of a float64 (bits) as an integer in units of the power
// of two that puts the largest biased exponent exm of a group below 2^(53 + UP)
// (rounded to nearest; |x| < 2^(exm - 1022) becomes |X| < 2^(53 + UP))
template <int UP>
SV_FX int64_t fx_from_bits(int64_t bits, int exm) {
  const int ex = (int)((bits >> 52) & 0x7ff);
  if (ex == 0) return 0;
  const int64_t mant = (bits & 0xfffffffffffffll) | (1ll << 52);
  const int sh = ex - exm + UP;
  int64_t X;
  if (sh >= 0)
    X = mant << sh;
  else
    X = -sh > 54 ? 0 : (mant + (1ll << (-sh - 1))) >> -sh;
  return bits < 0 ? -X : X;
}

}  // namespace sv
