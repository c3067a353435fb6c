// 64-bit fixed-point arithmetic for the complex128 transforms.
//
// GB300 issues one FP64 instruction per 64 cycles and scheduler (measured: a
// warp's DFMA every 64 cycles against one FFMA per cycle, a 64-bit integer
// add in 1-2 and a 32 x 32 -> 64 bit multiply-add in 2), so FP64 butterflies
// leave the chip idle: the 1024^2 passes ran at 350-470 us with every other
// pipe under 5%.  A line of N FP64 points is therefore transformed as 64-bit
// integers with one exponent per line: value = int * 2^q.  Butterfly sums are
// exact integer adds, products keep the upper half of the 128-bit product.
//
// Headroom: a stage of radix R enlarges |z| at most R times, so a line enters
// its first stage with |z| < 2^(62.5 - bits(R)), bits(R) = max(2, ceil log2
// R), and the twiddles of every later stage carry the factor 2^-bits(R); no
// sum can leave 63 bits, whatever the data.  That scaling assumes values that
// all add up (a spectrum of unit modulus, domains of constant phase).  No
// partial sum of a transform exceeds the line's sum of |re| + |im| (its L1
// norm), which is much less for a spectrum of a few lines or a cloud in a
// large box, so the line is shifted up in front of its last stage by what its
// L1 norm leaves free (fx_room).  Behind a transform either every |z| is
// below 2^60.5 (its L1 norm had room), or their root sum square is below
// 2^62.5 (that of a line whose values all add up is its largest sum).
//
// Precision: a product is rounded within 0.6 units.  A line's values come in
// at 2^-(62 - bits(R)) of its largest, R the first radix: 2^-59 with 8 points
// per thread, 2^-60 with 4, 2^-58 with 12 (sides 3 * 2^k).  A line whose values
// meet in few of a stage's butterflies loses the stage's bits on the way and
// gets them back, rounded, in front of the last stage.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include <type_traits>

namespace sgpe {

typedef long long fx_t;

struct __align__(16) FxC {
  fx_t x, y;
};
template <class C> struct is_fx : std::false_type {};
template <> struct is_fx<FxC> : std::true_type {};

// v = h 2^32 + l with a signed low word (|l| <= 2^31), so that every partial
// product is one signed 32 x 32 -> 64 bit multiply-add.
struct FxSplit {
  int h, l;
};
__host__ __device__ __forceinline__ FxSplit fx_split(fx_t v) {
  FxSplit s;
  s.l = int(uint32_t(uint64_t(v)));
  s.h = int(v >> 32) + int(uint32_t(s.l) >> 31);
  return s;
}
// One IMAD.WIDE (written as C++, the compiler split 64-bit products of
// reassembled words into unsigned parts: 60 more instructions per point of
// the 1024^2 column pass).
__host__ __device__ __forceinline__ fx_t fx_mad(int a, int b, fx_t c) {
#ifdef __CUDA_ARCH__
  fx_t r;
  asm("mad.wide.s32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return fx_t(a) * fx_t(b) + c;
#endif
}

constexpr fx_t kFxHalf = fx_t(1) << 31;  // rounds the upper half

// a b / 2^64 + c.  |a| < 2^63, |b| <= 2^62: no partial sum leaves 64 bits.
// The product of the low words (under a quarter unit, zero mean) is dropped.
__host__ __device__ __forceinline__ fx_t fx_mul(FxSplit a, FxSplit b, fx_t c = 0) {
  const fx_t t = fx_mad(a.h, b.l, fx_mad(a.l, b.h, kFxHalf));
  return fx_mad(a.h, b.h, c + (t >> 32));
}

// a w / 2^64 (CONJ: a conj(w) / 2^64) + c for a split complex factor
// w = (re.h, re.l, im.h, im.l) of modulus at most 2^62 whose low words are
// not -2^31 (they are negated), |a| < 2^62.7.
template <bool CONJ> __host__ __device__ __forceinline__ FxC fx_cmul(FxSplit ax, FxSplit ay, int4 w, FxC c) {
  const int nh = -w.z, nl = -w.w;
  const int ih = CONJ ? nh : w.z, il = CONJ ? nl : w.w;  // im = ax * i + ay * re
  const int jh = CONJ ? w.z : nh, jl = CONJ ? w.w : nl;  // re = ax * re + ay * j
  const fx_t tr = fx_mad(ax.h, w.y, fx_mad(ax.l, w.x, fx_mad(ay.h, jl, fx_mad(ay.l, jh, kFxHalf))));
  const fx_t ti = fx_mad(ax.h, il, fx_mad(ax.l, ih, fx_mad(ay.h, w.y, fx_mad(ay.l, w.x, kFxHalf))));
  FxC r;
  r.x = fx_mad(ax.h, w.x, fx_mad(ay.h, jh, c.x + (tr >> 32)));
  r.y = fx_mad(ax.h, ih, fx_mad(ay.h, w.x, c.y + (ti >> 32)));
  return r;
}
template <bool CONJ> __host__ __device__ __forceinline__ FxC fx_cmul(FxC a, int4 w) {
  return fx_cmul<CONJ>(fx_split(a.x), fx_split(a.y), w, FxC{0, 0});
}
// split form of a complex factor |w| <= 2^62 computed at run time
__host__ __device__ __forceinline__ int4 fx_factor(fx_t re, fx_t im) {
  FxSplit a = fx_split(re), b = fx_split(im);
  b.l |= 1;  // never -2^31, which has no negative; one unit of 2^62
  int4 w;
  w.x = a.h;
  w.y = a.l;
  w.z = b.h;
  w.w = b.l;
  return w;
}

// a c for a constant c = K + W / 2^64, K = 0 or 1, |W| <= 2^63
template <int K, fx_t W> __host__ __device__ __forceinline__ fx_t fx_mulc(fx_t a) {
  constexpr int l = int(uint32_t(uint64_t(W)));
  constexpr int h = int(W >> 32) + int(uint32_t(l) >> 31);
  return fx_mul(fx_split(a), FxSplit{h, l}, K ? a : 0);
}
// ceil(log2 R), at least 2 (a factor of modulus one is held as 2^62)
__host__ __device__ constexpr int fx_bits(int radix) {
  int b = 2;
  while ((1 << b) < radix) ++b;
  return b;
}

// Bits free in front of the last stage of a line whose L1 norm is below
// l1 2^44, after stages that scaled it by 2^-scaled: the values there may be
// shifted up to 2^62.
__host__ __device__ __forceinline__ int fx_room(uint32_t l1, int scaled) {
#ifdef __CUDA_ARCH__
  const int b = 32 - __clz(int(l1));
#else
  const int b = l1 ? 32 - __builtin_clz(l1) : 0;
#endif
  const int up = 62 - 44 - b + scaled;
  return up > 0 ? up : 0;
}

// a 2^-B, rounded
template <int B> __host__ __device__ __forceinline__ FxC fx_scale_down(FxC a) {
  const fx_t half = fx_t(1) << (B - 1);
  return FxC{(a.x + half) >> B, (a.y + half) >> B};
}

// ------------------------------------------------ FP64 <-> fixed point
__host__ __device__ __forceinline__ uint64_t fx_shr(uint64_t m, int d) {  // d >= 0; 0 from 64 on
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(m), "r"(d));
  return r;
#else
  return d < 64 ? m >> d : 0;
#endif
}
// Biased exponent of a line from the largest (high word & 0x7fffffff) of its
// parts.  From 70 on, so that zeros and subnormals (biased exponent 0) shift
// out: parts below 2^-952 of a line that small read as zero.
__host__ __device__ __forceinline__ int fx_line_exp(uint32_t hi_max) {
  const int be = int(hi_max >> 20);
  return be < 70 ? 70 : be;
}
constexpr int kFxNonFinite = 0x7ff;
// exponent q of a line with biased exponent be held at |part| < 2^p
__host__ __device__ __forceinline__ int fx_line_q(int be, int p) { return be - 1022 - p; }
// part of an FP64 value (its two words) in a line of biased exponent be,
// |part| < 2^p, p <= 62
__host__ __device__ __forceinline__ fx_t fx_from_words(uint32_t hi, uint32_t lo, int be, int p) {
  const uint32_t mh = (hi << 11) | (lo >> 21) | 0x80000000u;
  const uint32_t ml = lo << 11;
  const int d = 64 - p + be - int((hi >> 20) & 0x7ff);
  const uint64_t m = fx_shr((uint64_t(mh) << 32) | ml, d);
  const fx_t s = fx_t(int(hi) >> 31);
  return (fx_t(m) ^ s) - s;
}
__host__ __device__ __forceinline__ int fx_clz(uint64_t a) {
#ifdef __CUDA_ARCH__
  return __clzll(fx_t(a));
#else
  return a ? __builtin_clzll(a) : 64;
#endif
}
// Words of v 2^q as FP64, rounded to 53 bits (ties away from zero); the
// result and its neighbours must be in the normal range (fx_q_safe) or zero.
__host__ __device__ __forceinline__ void fx_to_words(fx_t v, int q, uint32_t* hi, uint32_t* lo) {
  const uint32_t sign = uint32_t(v >> 32) & 0x80000000u;
  const uint64_t a = uint64_t(v < 0 ? -v : v);
  const int lz = fx_clz(a);
  const uint64_t n = a << (lz & 63);
  // n in [2^63, 2^64): value = n 2^(q - lz); the hidden bit adds one to the
  // exponent field, and so does a carry of the rounding
  const uint32_t e = uint32_t(q - lz + 63 + 1023 - 1) << 20;
  const uint64_t t = (n >> 11) + ((n >> 10) & 1);
  *lo = uint32_t(t);
  *hi = a == 0 ? sign : (uint32_t(t >> 32) + e) | sign;
  if (a == 0) *lo = 0;
}
__host__ __device__ __forceinline__ bool fx_q_safe(int q) { return q > -1020 && q < 950; }

// ------------------------------------- sin and cos of a small fixed phase
// X = x 2^64 with |x| < 1/8: sin x and cos x - 1 times 2^64.  Taylor series
// to x^9 and x^10 (the omitted terms are below 2^-58 and 2^-64); the terms
// small enough to need no more than 30 bits take 32-bit products.
__host__ __device__ constexpr fx_t fx_coef(int n) {  // 2^64 / n, n >= 5
  return fx_t(0xffffffffffffffffull / uint64_t(n));
}
__host__ __device__ constexpr int fx_coef32(int k, int n) {  // 2^k / n
  return int(((uint64_t(1) << k) + uint64_t(n) / 2) / uint64_t(n));
}
__host__ __device__ __forceinline__ void fx_sincos(fx_t X, fx_t* sn, fx_t* cm1) {
  const FxSplit xs = fx_split(X);
  const fx_t u = fx_mul(xs, xs);                    // x^2 2^64 < 2^58
  const FxSplit us = fx_split(u);
  const int uh = int(u >> 27);                      // x^2 2^37 < 2^31
  // sin x = x - x^3 (1/6 - x^2 (1/120 - x^2 (1/5040 - x^2 / 362880)))
  const int s7 = fx_coef32(42, 5040) - int(fx_mad(uh, fx_coef32(37, 362880), 0) >> 32);  // 2^42
  const fx_t s5 = fx_coef(120) - (fx_mad(uh, s7, 0) >> 15);
  const fx_t s3 = fx_coef(6) - fx_mul(us, fx_split(s5));
  const fx_t x3 = fx_mul(us, xs);                   // x^3 2^64
  *sn = X - fx_mul(fx_split(x3), fx_split(s3));
  // cos x - 1 = -x^2/2 + x^4 (1/24 - x^2 (1/720 - x^2 (1/40320 - x^2 / 3628800)))
  const int c8 = fx_coef32(34, 40320) - int(fx_mad(uh, fx_coef32(29, 3628800), 0) >> 32);  // 2^34
  const int c6 = fx_coef32(39, 720) - int(fx_mad(uh, c8, 0) >> 32);                        // 2^39
  const fx_t c4 = fx_coef(24) - (fx_mad(uh, c6, 0) >> 12);
  const fx_t g = fx_mul(us, fx_split(c4));
  *cm1 = fx_mul(us, fx_split(g)) - (u >> 1);
}
// exp(x) - 1 times 2^64, |x| < 1/8: Taylor series to x^11.
__host__ __device__ __forceinline__ fx_t fx_expm1(fx_t X) {
  const FxSplit xs = fx_split(X);
  const int xh = int(X >> 30);                      // x 2^34, |.| < 2^31
  // t = 1/5040 + x (1/40320 + x (1/362880 + x (1/3628800 + x / 39916800))), times 2^42
  int t = fx_coef32(42, 39916800);
  t = fx_coef32(42, 3628800) + int(fx_mad(xh, t, 0) >> 34);
  t = fx_coef32(42, 362880) + int(fx_mad(xh, t, 0) >> 34);
  t = fx_coef32(42, 40320) + int(fx_mad(xh, t, 0) >> 34);
  t = fx_coef32(42, 5040) + int(fx_mad(xh, t, 0) >> 34);
  fx_t p = fx_coef(720) + (fx_mad(xh, t, 0) >> 12);
  p = fx_coef(120) + fx_mul(xs, fx_split(p));
  p = fx_coef(24) + fx_mul(xs, fx_split(p));
  p = fx_coef(6) + fx_mul(xs, fx_split(p));
  // x + x^2 (1/2 + x p), the bracket times 2^62
  const fx_t u = fx_mul(xs, xs);
  const fx_t h = (fx_t(1) << 61) + (fx_mul(xs, fx_split(p)) >> 2);
  return X + 4 * fx_mul(fx_split(u), fx_split(h));
}

}  // namespace sgpe
