// FP64 multiplication, addition and division on the integer and FP32 pipes,
// correctly rounded to nearest-even, so they return the same bits as the
// IEEE-754 binary64 operations (and as the hardware DMUL / DADD / division).
//
// Why: GB300 executes 2 FP64 operations per clock per SM, against 64-128
// integer or FP32 operations.  The bit-exact FP64 kernels are bound by that
// pipe while most issue slots stay idle, so a kernel moves part of its FP64
// arithmetic here and keeps the rest on the FP64 pipe; both run at once.
//
// Method (the textbook software floating point of e.g. Muller et al.,
// "Handbook of Floating-Point Arithmetic", 2nd ed., ch. 7-8): unpack sign,
// exponent and significand; compute the exact result significand, or enough of
// it plus a sticky bit; round to nearest-even from the guard bit and the
// sticky bit; repack, letting a rounding carry propagate into the exponent.
// Operands of magnitude within 2^+-500 take this path (every result is then
// normal and finite), and so do zero operands with a finite partner (a product
// or sum with a zero is frequent: a uniform region has zero differences);
// subnormals, infinities, NaNs and extreme exponents go to the hardware
// instruction, so every input gives the IEEE result.
//
//   mul: the 106-bit product of the 53-bit significands from four 32x32-bit
//        integer multiplies; the rounding increment is the carry of one add.
//   add: the smaller operand aligned with 8 extra low bits and a jammed sticky
//        bit, integer add or subtract, renormalisation.
//   div: long division (Knuth, TAOCP vol. 2, 4.3.1) in digits of 18, 18 and 17
//        bits, each estimated from below from an FP32 reciprocal of the
//        divisor's top 24 bits; the exact integer remainder stays in
//        [0, 1.5 divisors) and is corrected once, after the last digit.
//
// The tests of the exponent and zero bits work on the two 32-bit halves taken
// through an opaque move, so the compiler cannot turn them into FP64
// comparisons (which would run on the FP64 pipe this code exists to relieve).
//
// Checked bitwise against the hardware operations on random and adversarial
// operands by fvh_debug_sf64 (tests/test_gpu_sf64.py).
#pragma once

#include <cstdint>

namespace fvh {
namespace sf64 {

constexpr unsigned long long kM52 = 0x000fffffffffffffull;
constexpr unsigned long long kH52 = 0x0010000000000000ull;

__device__ __forceinline__ unsigned long long bits(double x) {
  return (unsigned long long)__double_as_longlong(x);
}
__device__ __forceinline__ double dbl(unsigned long long u) {
  return __longlong_as_double((long long)u);
}

// The two 32-bit halves of a double and back, through an opaque move.
__device__ __forceinline__ void halves(double x, unsigned &lo, unsigned &hi) {
  asm("mov.b64 {%0, %1}, %2;" : "=r"(lo), "=r"(hi) : "d"(x));
}
__device__ __forceinline__ double join(unsigned lo, unsigned hi) {
  double x;
  asm("mov.b64 %0, {%1, %2};" : "=d"(x) : "r"(lo), "r"(hi));
  return x;
}

// Rare operands go to the hardware instruction in an out-of-line call, so it
// takes an FP64 issue slot only when a lane needs it (an inlined fallback is
// issued, predicated off, on every call).
__device__ __noinline__ double mul_rare(double a, double b) { return __dmul_rn(a, b); }
__device__ __noinline__ double add_rare(double a, double b) { return __dadd_rn(a, b); }
__device__ __noinline__ double div_rare(double a, double b) { return __ddiv_rn(a, b); }

// biased exponent field of the high half
__device__ __forceinline__ unsigned expo(unsigned hi) { return (hi >> 20) & 0x7ffu; }
// exponents in [523, 1523] (magnitudes within 2^+-500): sums, differences,
// products and quotients of two such values are normal and finite
__device__ __forceinline__ bool moderate(unsigned e) { return e - 523u < 1001u; }
__device__ __forceinline__ bool is_zero(unsigned lo, unsigned hi) {
  return ((hi & 0x7fffffffu) | lo) == 0u;
}
__device__ __forceinline__ bool is_finite(unsigned hi) {
  return (hi & 0x7ff00000u) != 0x7ff00000u;
}

// An operand taken apart: the significand (m : lo), 53 bits with the implied
// one, and the sign and exponent field as they stand in the high half.
struct parts {
  unsigned lo, m, se;
  bool zero;
};

// Takes a moderate value or a zero apart.
__device__ __forceinline__ parts take_plain(double x) {
  unsigned lo, hi;
  halves(x, lo, hi);
  parts p;
  p.lo = lo;
  p.m = (hi & 0xfffffu) | 0x100000u;
  p.se = hi & 0xfff00000u;
  p.zero = ((hi & 0x7fffffffu) | lo) == 0u;
  return p;
}
// Takes x apart; `rare` collects whether it is neither moderate nor a zero.
__device__ __forceinline__ parts take(double x, unsigned &rare) {
  const parts p = take_plain(x);
  unsigned lo, hi;
  halves(x, lo, hi);
  const unsigned h = hi & 0x7fffffffu;
  rare |= (unsigned)!((h - (523u << 20) < (1001u << 20)) | p.zero);
  return p;
}

// Rounded product of two moderate operands.  The sign and exponent fields are
// added as they stand: modulo 2^32 the sign bits add to their exclusive or.
__device__ __forceinline__ double mul_core(const parts &a, const parts &b) {
  // P = product of the significands in 32-bit words w3 w2 w1 w0, in [2^104, 2^106)
  const unsigned long long p0 = (unsigned long long)a.lo * b.lo;
  const unsigned long long t =
      (unsigned long long)a.m * b.lo + ((unsigned long long)a.lo * b.m + (p0 >> 32));
  const unsigned long long u = (unsigned long long)a.m * b.m + (t >> 32);
  const unsigned w0 = (unsigned)p0, w1 = (unsigned)t, w2 = (unsigned)u, w3 = (unsigned)(u >> 32);
  // shifted left by s the significand of the result is the words above w1
  const unsigned top = w3 >> 9, s = 12u - top;  // top = 1 when P >= 2^105
  const unsigned mhi = __funnelshift_l(w2, w3, s), mlo = __funnelshift_l(w1, w2, s);
  // what is below it, w0 jammed into the lowest bit (bit s after the shift),
  // and the result's lowest bit in bit 0: above 2^31 it rounds up, so adding
  // 2^31 - 1 carries exactly then
  const unsigned f = ((w1 | (w0 < 1u ? w0 : 1u)) << s) | (mlo & 1u);
  // exponent field of the result minus one (the significand's leading one,
  // bit 52, adds it back; a rounding carry to 2^53 moves on to the exponent)
  const unsigned e1 = a.se + b.se - (1024u << 20) + (top << 20);
  unsigned lo, hi;
  asm("{\n\t.reg .u32 t;\n\t"
      "add.cc.u32 t, %2, 0x7fffffff;\n\t"
      "addc.cc.u32 %0, %3, 0;\n\t"
      "addc.u32 %1, %4, %5;\n\t}"
      : "=r"(lo), "=r"(hi)
      : "r"(f), "r"(mlo), "r"(mhi), "r"(e1));
  return join(lo, hi);
}

// Product of two operands taken apart, zeros by a select (the sign of a
// product is that of the added sign bits).
__device__ __forceinline__ double mul_parts(const parts &a, const parts &b) {
  const double q = mul_core(a, b);
  return (a.zero | b.zero) ? join(0u, (a.se + b.se) & 0x80000000u) : q;
}

// a * b
__device__ __forceinline__ double mul(double a, double b) {
  unsigned al, ah, bl, bh;
  halves(a, al, ah);
  halves(b, bl, bh);
  const unsigned ea = expo(ah), eb = expo(bh);
  const unsigned sign = (ah ^ bh) & 0x80000000u;
  if (!(moderate(ea) & moderate(eb))) {
    // a zero times a finite value is the zero of the product's sign
    if ((is_zero(al, ah) & is_finite(bh)) | (is_zero(bl, bh) & is_finite(ah)))
      return join(0u, sign);
    return mul_rare(a, b);
  }
  unsigned rare = 0;
  return mul_core(take(a, rare), take(b, rare));
}

// a + b
__device__ __forceinline__ double add(double a, double b) {
  unsigned al, ah, bl, bh;
  halves(a, al, ah);
  halves(b, bl, bh);
  // x: the operand of larger magnitude
  const unsigned long long xa = ((unsigned long long)(ah & 0x7fffffffu) << 32) | al;
  const unsigned long long xb = ((unsigned long long)(bh & 0x7fffffffu) << 32) | bl;
  const bool swap = xa < xb;
  const unsigned long long mx = swap ? xb : xa, my = swap ? xa : xb;
  const unsigned sx = (swap ? bh : ah) & 0x80000000u;
  const unsigned ex = (unsigned)(mx >> 52), ey = (unsigned)(my >> 52);
  if (!(moderate(ex) & (ey != 0u))) {
    if ((my == 0) & (ex != 2047u)) {  // x + (+-0), x finite
      if (mx == 0) return join(0u, ah & bh & 0x80000000u);  // -0 only for (-0) + (-0)
      return swap ? b : a;
    }
    return add_rare(a, b);
  }
  // (ex moderate, y normal: the result exponent stays within [466, 1524])
  int d = (int)(ex - ey);
  d = d > 63 ? 63 : d;  // beyond 63 only the sticky bit remains either way
  const unsigned long long A = ((mx & kM52) | kH52) << 8;  // leading one at bit 60
  const unsigned long long B = ((my & kM52) | kH52) << 8;
  const unsigned long long Bs =
      d == 0 ? B : ((B >> d) | (unsigned long long)((B << (64 - d)) != 0));
  const bool sub = ((ah ^ bh) & 0x80000000u) != 0;
  const unsigned long long S = sub ? A - Bs : A + Bs;
  unsigned long long N;
  int e;
  if (S >> 61) {  // carry out of an addition
    N = (S >> 1) | (S & 1);
    e = (int)ex + 1;
  } else if (S >> 60) {
    N = S;
    e = (int)ex;
  } else {  // cancellation
    if (S == 0) return 0.0;  // x - x = +0 when rounding to nearest
    const int lz = __clzll((long long)S);  // >= 4
    N = S << (lz - 3);
    e = (int)ex - (lz - 3);
  }
  unsigned long long m = N >> 8;
  const unsigned guard = (unsigned)(N >> 7) & 1u;
  const unsigned sticky = (N & 0x7f) != 0;
  m += guard & (sticky | ((unsigned)m & 1u));
  return dbl((((unsigned long long)(e - 1) << 52) + m) | ((unsigned long long)sx << 32));
}

__device__ __forceinline__ double sub(double a, double b) {
  unsigned bl, bh;
  halves(b, bl, bh);
  return add(a, join(bl, bh ^ 0x80000000u));
}

// One quotient digit of K <= 18 bits: q <= r 2^K / d, r <- r 2^K - q d, for
// 0 <= r < 2 d, 2^52 <= d < 2^53 (nd = 2^64 - d).  ginv is 2^(K+2) times an
// FP32 reciprocal of dh = d >> 29 lowered by 2^-21.  With fr = r >> 31 < 2^23
// the estimate floor(fr ginv) never exceeds r 2^K / d: truncating d and the
// reciprocal's error raise it by less than 2^-22 of itself.  It falls short by
// less than 1.49 (1 for the floor, 2^(K-21) for truncating r, 0.36 for the
// lowered reciprocal at a digit below 2^19), so 0 <= r < 1.49 d again.  The
// remainder is exact modulo 2^64.
template <int K>
__device__ __forceinline__ unsigned div_digit(unsigned long long &r, unsigned long long nd,
                                              float ginv) {
  const float fr = __int_as_float(0x4b000000 | (int)(unsigned)(r >> 31)) - 8388608.0f;
  // floor(fr * ginv) for a value below 2^23: round toward zero onto 2^23
  const unsigned q = (unsigned)__float_as_int(__fmaf_rz(fr, ginv, 8388608.0f)) & 0x7fffffu;
  r = (r << K) + (unsigned long long)q * (unsigned)nd +
      ((unsigned long long)(q * (unsigned)(nd >> 32)) << 32);
  return q;
}

// Rounded quotient of two moderate operands.
__device__ __forceinline__ double div_core(const parts &a, const parts &b) {
  unsigned long long x = ((unsigned long long)a.m << 32) | a.lo;
  const unsigned long long d = ((unsigned long long)b.m << 32) | b.lo;
  const bool lt = x < d;
  x = lt ? x + x : x;  // d <= x < 2d: the quotient is in [1, 2)
  const unsigned long long nd = 0ull - d;
  // dh = d >> 29 in [2^23, 2^24), exactly a float
  const float fd = __int_as_float(0x4b000000 | ((unsigned)(d >> 29) & 0x7fffffu));
  float inv;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(inv) : "f"(fd));
  const float g18 = inv * (1048576.0f * (1.0f - 0x1p-21f));
  unsigned long long r = x;
  const unsigned q1 = div_digit<18>(r, nd, g18);
  const unsigned q2 = div_digit<18>(r, nd, g18);
  const unsigned q3 = div_digit<17>(r, nd, 0.5f * g18);
  // Q = floor(x 2^53 / d) in [2^53, 2^54): 53 bits and the guard bit.  A
  // quotient of two 53-bit significands is never halfway between two results
  // (d would have to be a multiple of 2^53), so the guard bit alone rounds.
  unsigned long long Q = (((unsigned long long)q1 << 18) + q2) * 131072ull + q3;
  Q += (unsigned long long)(r >= d) + 1ull;
  const unsigned long long m = Q >> 1;
  // exponent field minus one, and the sign (see mul_core)
  const unsigned e1 = a.se - b.se + ((lt ? 1021u : 1022u) << 20);
  return join((unsigned)m, (unsigned)(m >> 32) + e1);
}

// a / b
__device__ __forceinline__ double div(double a, double b) {
  unsigned al, ah, bl, bh;
  halves(a, al, ah);
  halves(b, bl, bh);
  const unsigned ea = expo(ah), eb = expo(bh);
  const unsigned sign = (ah ^ bh) & 0x80000000u;
  if (!(moderate(ea) & moderate(eb))) {
    // zero over a finite nonzero value: the zero of the quotient's sign
    if (is_zero(al, ah) & is_finite(bh) & !is_zero(bl, bh)) return join(0u, sign);
    return div_rare(a, b);
  }
  unsigned rare = 0;
  return div_core(take(a, rare), take(b, rare));
}

// ---------------------------------------------------------------------------
// Branch-free forms for optimistic evaluation: the integer path for every
// operand, with zeros handled by a select; `rare` collects whether any
// operand needs the hardware instruction, in which case the caller discards
// the results and evaluates the whole unit of work again with the FP64
// instructions.  A kernel then has no branch per operation.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double mul_opt(double a, double b, unsigned &rare) {
  const parts pa = take(a, rare), pb = take(b, rare);
  return mul_parts(pa, pb);
}

__device__ __forceinline__ double div_opt(double a, double b, unsigned &rare) {
  const parts pa = take(a, rare), pb = take(b, rare);
  rare |= (unsigned)pb.zero;
  const double q = div_core(pa, pb);
  return pa.zero ? join(0u, (pa.se + pb.se) & 0x80000000u) : q;
}

}  // namespace sf64
}  // namespace fvh
