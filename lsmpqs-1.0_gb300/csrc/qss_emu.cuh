// qss_emu.cuh -- IEEE-754 binary64 arithmetic (round to nearest even) on the
// integer pipes.
//
// On GB300 the FP64 pipe takes one warp instruction per 77 cycles and
// scheduler (measured for DADD, DMUL and DFMA alike), a 32-bit ALU
// instruction 2 cycles of the ALU pipe and an integer product 2 cycles of
// the FMA pipe, all three side by side; and the WENO5 kernels of this library
// are bound by the FP64 pipe.  The functions below compute the correctly
// rounded IEEE results of x/y, sqrt(x), x*y, x+y, exact power-of-two
// scalings and comparisons from the operands' bit patterns with 32/64-bit integer
// instructions, so that part of the FP64 work moves to otherwise idle
// pipes.  Each function has a fast path for operands in a middle range of
// exponents (plus signed zeros where cheap) and falls back to the native FP64
// instruction for everything else (subnormals, infinities, NaNs, overflow,
// underflow), so every result is bit-identical to the native operation on
// all inputs.  Divisions and square roots start from the single-precision
// approximations (rcp / rsqrt.approx, whose error bounds the PTX manual
// states) and proceed by two digits with exact remainders, as in long
// division; the bounds that make the last digit right are stated with each.
//
// The header compiles for the host too (g++), where the same code is tested
// against the host's IEEE double arithmetic.
#pragma once
#include <math.h>
#include <stdint.h>
#ifndef __CUDACC__
#include <string.h>
#endif

#ifdef __CUDACC__
#define QSS_EMU_HD __host__ __device__ __forceinline__
#else
#define QSS_EMU_HD static inline
#endif

// hooks for the host check: count fallbacks, perturb the reciprocal seed
#ifndef QSS_EMU_FALLBACK
#define QSS_EMU_FALLBACK(op, expr) (expr)
#endif
#ifndef QSS_EMU_SEED_ADJUST
#define QSS_EMU_SEED_ADJUST(rb) (rb)
#endif

namespace qss_emu {

// The native instruction of a fallback.  Volatile, so that the compiler does
// not issue it ahead of the test that rarely selects it: one FP64
// instruction costs as much as a whole integer-pipe product.
#ifdef __CUDA_ARCH__
#define QSS_EMU_NATIVE(name, ptx)                                                       \
  __device__ __forceinline__ double name(double x, double y) {                          \
    double r;                                                                           \
    asm volatile(ptx " %0, %1, %2;" : "=d"(r) : "d"(x), "d"(y));                        \
    return r;                                                                           \
  }
QSS_EMU_NATIVE(native_mul, "mul.rn.f64")
QSS_EMU_NATIVE(native_add, "add.rn.f64")
#undef QSS_EMU_NATIVE
#else
QSS_EMU_HD double native_mul(double x, double y) { return x * y; }
QSS_EMU_HD double native_add(double x, double y) { return x + y; }
#endif

constexpr uint64_t kMant = (1ull << 52) - 1;
constexpr uint64_t kHidden = 1ull << 52;
constexpr uint64_t kSign = 1ull << 63;
constexpr uint64_t kAbs = ~kSign;

// Twice the magnitude bits, for comparisons of magnitudes: the sign is shifted
// out because the compiler takes (bits of a double) & kAbs for fabs and issues
// it on the FP64 pipe (77 cycles; two such tests were a fifth of the
// reinitialisation sweep).
QSS_EMU_HD uint64_t mag2(uint64_t b) { return b << 1; }
constexpr uint64_t kInf2 = 0x7ff0000000000000ull << 1;

// Opaque to the compiler on the device: it takes tests of the bits for what they
// say about the number ((bits << 1) == 0 for x == 0, bits & kAbs for fabs) and issues
// them on the FP64 pipe, where one costs as much as a whole integer-pipe product.
QSS_EMU_HD uint64_t bits(double x) {
#ifdef __CUDA_ARCH__
  uint64_t u;
  asm("mov.b64 %0, %1;" : "=l"(u) : "d"(x));
  return u;
#else
  uint64_t u;
  memcpy(&u, &x, 8);
  return u;
#endif
}

QSS_EMU_HD double from_bits(uint64_t u) {
#ifdef __CUDA_ARCH__
  return __longlong_as_double((long long)u);
#else
  double x;
  memcpy(&x, &u, 8);
  return x;
#endif
}

QSS_EMU_HD int clz64(uint64_t x) {
#ifdef __CUDA_ARCH__
  return __clzll((long long)x);
#else
  return x ? __builtin_clzll(x) : 64;
#endif
}

// ---------------------------------------------------------------------------
// 32-bit words.  A 32-bit logic, shift or compare instruction occupies the
// ALU pipe for 2 cycles of a scheduler, an integer product (32 x 32 -> 64
// included) the FMA pipe for 2, both at the same time, and one FP64
// instruction the FP64 pipe for 77 (GB300, measured); so the routines below
// work on 32-bit words, keep the count of ALU instructions low, and leave
// the exponent arithmetic packed in the high word.

QSS_EMU_HD uint32_t hi32(double x) { return (uint32_t)(bits(x) >> 32); }
QSS_EMU_HD uint32_t lo32(double x) { return (uint32_t)bits(x); }
QSS_EMU_HD uint64_t pack64(uint32_t hi, uint32_t lo) { return ((uint64_t)hi << 32) | lo; }

// low word of (hi:lo) >> s and high word of (hi:lo) << s, 0 <= s <= 31
QSS_EMU_HD uint32_t fsr(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_r(lo, hi, s);
#else
  return (uint32_t)((((uint64_t)hi << 32) | lo) >> s);
#endif
}
QSS_EMU_HD uint32_t fsl(uint32_t lo, uint32_t hi, uint32_t s) {
#ifdef __CUDA_ARCH__
  return __funnelshift_l(lo, hi, s);
#else
  return (uint32_t)(((((uint64_t)hi << 32) | lo) << s) >> 32);
#endif
}

// high word of the 53-bit significand
QSS_EMU_HD uint32_t mant_hi(uint32_t h) { return (h & 0xfffffu) | 0x100000u; }

// 32 x 32 -> 64-bit product plus a word
QSS_EMU_HD uint64_t madw(uint32_t a, uint32_t b, uint64_t c) {
#ifdef __CUDA_ARCH__
  uint64_t r;
  asm("mad.wide.u32 %0, %1, %2, %3;" : "=l"(r) : "r"(a), "r"(b), "l"(c));
  return r;
#else
  return (uint64_t)a * b + c;
#endif
}
QSS_EMU_HD uint32_t mulhi32(uint32_t a, uint32_t b) { return (uint32_t)(((uint64_t)a * b) >> 32); }

// Round to nearest even: (hi:lo) plus one where the discarded bits are at
// least half a unit (half holds them left-aligned: its top bit), then the
// lowest bit cleared where they were exactly half (rest is nonzero where
// anything lies below half).
QSS_EMU_HD double round_pack(uint32_t hi, uint32_t lo, uint32_t half, uint32_t rest) {
#ifdef __CUDA_ARCH__
  asm("{\n\t.reg .u32 t;\n\t"
      "add.cc.u32 t, %2, %2;\n\t"
      "addc.cc.u32 %1, %1, 0;\n\t"
      "addc.u32 %0, %0, 0;\n\t}"
      : "+r"(hi), "+r"(lo)
      : "r"(half));
  if (((half ^ 0x80000000u) | rest) == 0u) lo &= ~1u;
  return __hiloint2double((int)hi, (int)lo);
#else
  uint64_t r = (((uint64_t)hi << 32) | lo) + (half >> 31);
  if (((half ^ 0x80000000u) | rest) == 0u) r &= ~1ull;
  return from_bits(r);
#endif
}

// The fast paths take operands with exponents in [-255, 256]: products and
// quotients of two such are normal.  2 h - 0x60000000 (sign shifted out) is
// below 2^30 exactly there.
QSS_EMU_HD uint32_t win(uint32_t h) { return h * 2u - 0x60000000u; }
QSS_EMU_HD bool in_window(uint32_t xh) { return win(xh) < 0x40000000u; }
QSS_EMU_HD bool in_window(uint32_t xh, uint32_t yh) { return (win(xh) | win(yh)) < 0x40000000u; }

// ---------------------------------------------------------------------------
// x / y
//
// Significands N and D in [2^52, 2^53), N doubled where N < D (N'), so that
// N' / D is in [1, 2); d = D / 2^52.  The quotient N' 2^52 / D is built from
// two digits q1 2^26 + q2 with exact remainders, which need only their low
// 64 bits because their size is known:
//   S0   rcp.approx of the top 24 bits of d, 2^24 / d to 2^-22 relative
//        (truncation of d and 1 ulp of the approximation)
//   S1   one Newton step in fixed point: 2^30 / d, off by (-0.01, 1.5) units
//   q1   floor(x - 1/2) for x = (N' >> 22) S1 / 2^34, so that
//        R1 = N' 2^26 - q1 D has R1 / D in [0.125, 1.625)
//   q2   floor((R1 + 2^23 >> 24) S1 / 2^32), so that
//        R2 = R1 2^26 - q2 D has R2 / D in [-0.43, 1.13)
// and the correctly rounded quotient is q1 2^26 + q2 + (2 R2 > D) (no
// quotient lies half-way between two 53-bit numbers).  T = D - 2 R2.
// On the host, where the seed may be perturbed, a seed outside its bound
// falls back to the native division.

QSS_EMU_HD uint32_t recip_seed(uint32_t mh, uint32_t ml) {
  const uint32_t fb = fsl(ml, mh, 3) + 0x3f000000u;  // the float in [1, 2) of the top 24 bits
#ifdef __CUDA_ARCH__
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
  const uint32_t rb = __float_as_uint(r);
#else
  float f, r;
  memcpy(&f, &fb, 4);
  r = 1.0f / f;
  uint32_t rb;
  memcpy(&rb, &r, 4);
  rb = QSS_EMU_SEED_ADJUST(rb);
#endif
  return rb - 0x3e800000u;  // r 2^24, 2^24 itself for r = 1
}

// S1 of the significand (mh:ml)
QSS_EMU_HD uint32_t recip30(uint32_t mh, uint32_t ml, bool& ok) {
  const uint32_t S0 = recip_seed(mh, ml);
  const uint64_t P = (uint64_t)fsl(ml, mh, 11) * S0;  // 2^55 - e
#ifndef __CUDA_ARCH__
  ok = P - ((1ull << 55) - (1ull << 34)) < (1ull << 35);
#endif
  const int32_t E = (int32_t)fsr((uint32_t)P, (uint32_t)(P >> 32), 8);  // floor(-e / 2^8)
  const int32_t c = (int32_t)((uint64_t)((int64_t)E * (int32_t)S0) >> 32) >> 9;
  return S0 * 64u - (uint32_t)c;
}

// quotient of the normal numbers (xh:xl) / (yh:yl) where it is normal; S1 is
// recip30 of y's significand, which a loop over one divisor computes once
QSS_EMU_HD double div_recip(uint32_t xh, uint32_t xl, uint32_t yh, uint32_t yl, uint32_t S1) {
  const uint32_t mxh = mant_hi(xh), myh = mant_hi(yh);
  const uint64_t mx = pack64(mxh, xl), my = pack64(myh, yl);
  const uint32_t s = mx < my ? 1u : 0u;
  const uint32_t nh = fsr(xl, mxh, 22u - s);
  const uint32_t q1 = (mulhi32(nh, S1) - 2u) >> 2;
  const uint64_t R1c = pack64(fsl(xl, mxh, 26u + s), xl << (26u + s)) + (1ull << 23) - (uint64_t)q1 * my;  // R1 + 2^23
  const uint32_t q2 = mulhi32(fsr((uint32_t)R1c, (uint32_t)(R1c >> 32), 24), S1);
  const uint64_t T = (uint64_t)(2u * q2 + 1u) * my + (1ull << 50) - (R1c << 27);
  const uint64_t Q = madw(q1, 1u << 26, q2 + (uint32_t)(T >> 63));
  // (exponent - 1) << 52 plus the 53-bit significand; the signs add up mod 2
  const uint32_t e = (xh - mxh) - (yh - myh) + ((1022u - s) << 20);
  return from_bits(pack64((uint32_t)(Q >> 32) + e, (uint32_t)Q));
}
QSS_EMU_HD double div_win(uint32_t xh, uint32_t xl, uint32_t yh, uint32_t yl, bool& ok) {
  return div_recip(xh, xl, yh, yl, recip30(mant_hi(yh), yl, ok));
}

QSS_EMU_HD double div(double x, double y) {
  const uint32_t xh = hi32(x), yh = hi32(y);
  if (in_window(xh, yh)) {
    bool ok = true;
    const double q = div_win(xh, lo32(x), yh, lo32(y), ok);
    if (ok) return q;
  }
  return QSS_EMU_FALLBACK(0, x / y);
}

// ---------------------------------------------------------------------------
// sqrt(x)
//
// x = M 2^(2k-52) with M = mx or 2 mx, so that v = M / 2^52 is in [1, 4); the
// root's significand sqrt(M 2^52) = S 2^26 comes from two digits:
//   Y0   rsqrt.approx of the top 24 bits of v, 2^24 / sqrt(v) to 2^-22
//   Y1   one Newton step: 2^30 / sqrt(v), off by less than a unit
//   q1   (M >> 22) Y1 / 2^34 rounded, so that d1 = S - q1 is within +-0.88;
//        R1 = M - q1^2 = d1 (2 S - d1) fits 32 bits
//   q2   floor((2 R1 + 1) Y1 / 2^32): d1 2^26 less d1^2 / (2 sqrt(v)) <= 0.39
// so that S 2^26 - (q1 2^26 + q2) is in (-0.5, 1.5) and the rounded root is
// Q = q1 2^26 + q2, plus one where M 2^52 - Q^2 > Q (no root lies half-way).

// root of the positive normal number (xh:xl)
QSS_EMU_HD double sqrt_win(uint32_t xh, uint32_t xl, bool& ok) {
  const uint32_t ex = xh >> 20, odd = ~ex & 1u;
  const uint32_t mh = mant_hi(xh);
  const uint64_t M = pack64(mh, xl) << odd;
  const uint32_t fb = 0x3f800000u + (odd << 23) + fsl(xl, mh & 0xfffffu, 3);
#ifdef __CUDA_ARCH__
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(fb)));
  const uint32_t rb = __float_as_uint(r);
#else
  float f, r;
  memcpy(&f, &fb, 4);
  r = 1.0f / ::sqrtf(f);
  uint32_t rb;
  memcpy(&rb, &r, 4);
  rb = QSS_EMU_SEED_ADJUST(rb);
#endif
  // r = 1 would make Y0^2 >> 16 overflow 32 bits
  const uint32_t Y0 = rb < 0x3f800000u ? rb - 0x3e800000u : 0xffffffu;
  const uint32_t Mt = fsr(xl, mh, 22u - odd);  // v 2^30
  const uint64_t P = (uint64_t)Mt * (uint32_t)(((uint64_t)Y0 * Y0) >> 16);  // 2^62 - e
#ifndef __CUDA_ARCH__
  ok = P - ((1ull << 62) - (1ull << 42)) < (1ull << 43);
#endif
  const int32_t E = (int32_t)fsr((uint32_t)P, (uint32_t)(P >> 32), 16);  // floor(-e / 2^16)
  const int32_t c = (int32_t)((uint64_t)((int64_t)E * (int32_t)Y0) >> 32) >> 9;
  const uint32_t Y1 = Y0 * 64u - (uint32_t)c;
  const uint32_t q1 = ((uint32_t)(((uint64_t)Mt * Y1) >> 32) + 2u) >> 2;
  const int32_t R1 = (int32_t)((uint32_t)M - q1 * q1);
  const int32_t q2 = (int32_t)((uint64_t)((int64_t)(2 * R1 + 1) * (int32_t)Y1) >> 32);
  const uint64_t Q = ((uint64_t)q1 << 26) + (uint64_t)(int64_t)q2;
  const uint64_t T = Q + Q * Q - (M << 52);  // Q - (M 2^52 - Q^2)
  const uint32_t e = (((ex + 1023u - odd) >> 1) - 1u) << 20;
  return from_bits(Q + (T >> 63) + ((uint64_t)e << 32));
}
QSS_EMU_HD double sqrt_win(uint32_t xh, uint32_t xl) {
  bool ok = true;
  return sqrt_win(xh, xl, ok);
}

QSS_EMU_HD double sqrt(double x) {
  const uint32_t xh = hi32(x);
  if (xh - 0x30000000u < 0x20000000u) {  // positive, exponent in [-255, 256]
    bool ok = true;
    const double r = sqrt_win(xh, lo32(x), ok);
    if (ok) return r;
  } else if (mag2(bits(x)) == 0) {
    return x;  // sqrt(+-0) = +-0
  }
  return QSS_EMU_FALLBACK(3, ::sqrt(x));
}

// ---------------------------------------------------------------------------
// x * y: the 106-bit product in four words, the significand taken from it by
// one funnel shift per word (by 20 or 21 bits), then rounded.

// product of the normal numbers (xh:xl), (yh:yl), times 2^k, where it is normal
QSS_EMU_HD double mul_win(uint32_t xh, uint32_t xl, uint32_t yh, uint32_t yl, int k = 0) {
  const uint32_t mxh = mant_hi(xh), myh = mant_hi(yh);
  const uint64_t p00 = (uint64_t)xl * yl;
  const uint64_t t = madw(mxh, yl, madw(xl, myh, p00 >> 32));  // < 2^55
  const uint64_t p11 = madw(mxh, myh, t >> 32);
  const uint32_t w0 = (uint32_t)p00, w1 = (uint32_t)t, w2 = (uint32_t)p11, w3 = (uint32_t)(p11 >> 32);
  const uint32_t top = w3 >> 9;  // product >= 2^105
  const uint32_t sh = 20u + top;
  const uint32_t e = (xh - mxh) + (yh - myh) + ((uint32_t)(k - 1022) << 20) + top * 0x100000u;
  return round_pack(fsr(w2, w3, sh) + e, fsr(w1, w2, sh), fsr(0u, w1, sh), w0);
}

// square of the normal number (xh:xl), sign ignored, times 2^k, where normal
QSS_EMU_HD double sq_win(uint32_t xh, uint32_t xl, int k = 0) {
  const uint32_t mh = mant_hi(xh);
  const uint64_t p00 = (uint64_t)xl * xl;
  const uint64_t t = madw(2u * mh, xl, p00 >> 32);
  const uint64_t p11 = madw(mh, mh, t >> 32);
  const uint32_t w0 = (uint32_t)p00, w1 = (uint32_t)t, w2 = (uint32_t)p11, w3 = (uint32_t)(p11 >> 32);
  const uint32_t top = w3 >> 9;
  const uint32_t sh = 20u + top;
  const uint32_t e = 2u * (xh - mh) + ((uint32_t)(k - 1022) << 20) + top * 0x100000u;
  return round_pack(fsr(w2, w3, sh) + e, fsr(w1, w2, sh), fsr(0u, w1, sh), w0);
}

QSS_EMU_HD double mul(double x, double y) {
  const uint32_t xh = hi32(x), yh = hi32(y);
  if (in_window(xh, yh)) return mul_win(xh, lo32(x), yh, lo32(y));
  const uint64_t bx = bits(x), by = bits(y);
  const uint32_t ex = (xh >> 20) & 0x7ffu, ey = (yh >> 20) & 0x7ffu;
  if ((mag2(bx) == 0 && ey != 0x7ffu) || (mag2(by) == 0 && ex != 0x7ffu))
    return from_bits((bx ^ by) & kSign);  // zero times a finite number
  return QSS_EMU_FALLBACK(1, native_mul(x, y));
}

// ---------------------------------------------------------------------------
// x + y of non-negative operands (+0 included; no NaN): no cancellation, so
// the larger significand grows by at most one bit

// The larger operand is normal and the sum finite; the smaller may be +0 or
// subnormal.  No branch: the smaller significand is shifted as three words
// (a shift of 54 or more leaves less than half a unit of the larger, whatever
// stands in its place).
QSS_EMU_HD double add_pos(double x, double y) {
  const bool sw = hi32(x) < hi32(y);
  const uint32_t ah = sw ? hi32(y) : hi32(x), al = sw ? lo32(y) : lo32(x);
  const uint32_t bh = sw ? hi32(x) : hi32(y), bl = sw ? lo32(x) : lo32(y);
  const uint32_t mah = mant_hi(ah), mbh = mant_hi(bh);
  uint32_t d = ((ah - mah) - (bh - mbh)) >> 20;
  d = d < 63u ? d : 63u;
  const bool far = d >= 32u;
  const uint32_t b2 = far ? 0u : mbh, b1 = far ? mbh : bl, b0 = far ? bl : 0u, t = d & 31u;
  const uint64_t s = pack64(mah, al) + pack64(b2 >> t, fsr(b1, b2, t));
  const uint32_t f = fsr(b0, b1, t), rest = fsr(0u, b0, t);  // the bits of b below a's unit
  const uint32_t sl = (uint32_t)s, sh = (uint32_t)(s >> 32), top = sh >> 21;
  return round_pack((sh >> top) + (ah - mah) + top * 0x100000u, fsr(sl, sh, top), fsr(f, sl, top), rest | (f & top));
}

QSS_EMU_HD double add_nonneg(double x, double y) {
  if (in_window(hi32(x) < hi32(y) ? hi32(y) : hi32(x))) return add_pos(x, y);
  return QSS_EMU_FALLBACK(2, native_add(x, y));
}

// ---------------------------------------------------------------------------
// x + y

QSS_EMU_HD double add(double x, double y) {
  uint64_t ba = bits(x), bb = bits(y);
  // order by magnitude: |a| >= |b|
  if ((bb & kAbs) > (ba & kAbs)) {
    const uint64_t t = ba;
    ba = bb;
    bb = t;
  }
  const uint32_t ea = (uint32_t)(ba >> 52) & 0x7ffu, eb = (uint32_t)(bb >> 52) & 0x7ffu;
  if (ea - 1u < 2046u) {
    if ((bb & kAbs) == 0) return from_bits(ba);  // a + (+-0) = a for a nonzero normal
    if (eb != 0) {
      const uint64_t A = ((ba & kMant) | kHidden) << 10;  // 63 bits
      uint64_t B = ((bb & kMant) | kHidden) << 10;
      const uint32_t d = ea - eb;
      if (d > 0) {
        if (d >= 63) {
          B = 1;  // only the sticky bit survives
        } else {
          const uint64_t lost = B & ((1ull << d) - 1);
          B = (B >> d) | (lost ? 1u : 0u);
        }
      }
      uint64_t S;
      int e = (int)ea;
      if (((ba ^ bb) & kSign) == 0) {
        S = A + B;  // < 2^64
        if (S >> 63) {
          S = (S >> 1) | (S & 1);
          e += 1;
        }
      } else {
        S = A - B;
        if (S == 0) return 0.0;  // exact cancellation: +0 in round-to-nearest
        const int sh = clz64(S) - 1;  // bring the leading one to bit 62
        S <<= sh;
        e -= sh;
      }
      if (e >= 1 && e <= 2046) {
        const uint64_t sig = S >> 10, rb = S & 0x3ffu;
        const uint64_t up = (rb > 0x200u || (rb == 0x200u && (sig & 1))) ? 1u : 0u;
        return from_bits((ba & kSign) | ((((uint64_t)(e - 1)) << 52) + sig + up));
      }
    }
  } else if ((ba & kAbs) == 0) {  // both zero
    return from_bits(ba & bb & kSign);
  }
  return QSS_EMU_FALLBACK(2, native_add(x, y));
}

QSS_EMU_HD double neg(double x);
QSS_EMU_HD double sub(double x, double y) { return add(x, neg(y)); }

// x * 2^k for a small integer k (exact unless the result leaves the normal range)
QSS_EMU_HD double scale2(double x, int k) {
  const uint64_t b = bits(x);
  if (in_window((uint32_t)(b >> 32))) return from_bits(b + ((uint64_t)(int64_t)k << 52));
  const int e = (int)((b >> 52) & 0x7ffu);
  if (e >= 1 && e <= 2046 && e + k >= 1 && e + k <= 2046)
    return from_bits(b + ((uint64_t)(int64_t)k << 52));
  if (mag2(b) == 0) return x;
#ifdef __CUDA_ARCH__
  return x * __longlong_as_double((long long)((uint64_t)(1023 + k) << 52));
#else
  return x * from_bits((uint64_t)(1023 + k) << 52);
#endif
}

// ---------------------------------------------------------------------------
// sign flip and absolute value on the integer pipes.  Written as plain bit
// operations the compiler recognises them as FP64 negation / fabs and may
// issue them as FP64-pipe additions; the PTX logic op on the high word keeps
// them integer instructions.

QSS_EMU_HD double neg(double x) {
#ifdef __CUDA_ARCH__
  int hi = __double2hiint(x);
  asm("xor.b32 %0, %0, 0x80000000;" : "+r"(hi));
  return __hiloint2double(hi, __double2loint(x));
#else
  return from_bits(bits(x) ^ kSign);
#endif
}

QSS_EMU_HD double abs(double x) {
#ifdef __CUDA_ARCH__
  int hi = __double2hiint(x);
  asm("and.b32 %0, %0, 0x7fffffff;" : "+r"(hi));
  return __hiloint2double(hi, __double2loint(x));
#else
  return from_bits(bits(x) & kAbs);
#endif
}

// ---------------------------------------------------------------------------
// comparisons with IEEE semantics (false for NaN operands, -0 == +0)

QSS_EMU_HD bool isnan_bits(uint64_t b) { return mag2(b) > kInf2; }

// x > 0
QSS_EMU_HD bool gt0(double x) {
  const int64_t b = (int64_t)bits(x);
  return b > 0 && (uint64_t)b <= 0x7ff0000000000000ull;
}
// x >= 0
QSS_EMU_HD bool ge0(double x) {
  const uint64_t b = bits(x);
  return ((int64_t)b >= 0 && b <= 0x7ff0000000000000ull) || b == kSign;
}
// x < 0
QSS_EMU_HD bool lt0(double x) {
  const uint64_t b = bits(x);
  return (int64_t)b < 0 && b != kSign && b <= 0xfff0000000000000ull;
}

// x > y
QSS_EMU_HD bool gt(double x, double y) {
  const uint64_t a = bits(x), b = bits(y);
  if (isnan_bits(a) || isnan_bits(b)) return false;
  if (mag2(a | b) == 0) return false;  // both zero
  // negative numbers order as their magnitudes' complements
  const int64_t ka = (int64_t)a ^ (((int64_t)a >> 63) & (int64_t)kAbs);
  const int64_t kb = (int64_t)b ^ (((int64_t)b >> 63) & (int64_t)kAbs);
  return ka > kb;
}

// max of two non-negative, non-NaN values (e.g. squares): bit patterns order
// like the values
QSS_EMU_HD double max_nonneg(double a, double b) {
  const int64_t ia = (int64_t)bits(a), ib = (int64_t)bits(b);
  return from_bits((uint64_t)(ia > ib ? ia : ib));
}

}  // namespace qss_emu
