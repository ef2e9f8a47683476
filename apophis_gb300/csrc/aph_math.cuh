// aph_math.cuh -- device arithmetic of the hydro flux path (sm_103a).
//
// On GB300 every FP64 instruction -- add, mul, fma, but also compare (DSETP), negation,
// absolute value and min/max -- holds a pipe that takes 17 cycles of an SM for a warp, where
// an integer or FP32 one takes a quarter of a cycle.  Quotients, roots, most products, predicates and
// min/max below therefore work on the IEEE bit patterns with integer instructions.
// They give the same answer as the IEEE comparison for every non-NaN input, -0.0 and
// +0.0 included, so using them changes no result bit.
//
// APH_EXACT selects the arithmetic:
//   1  the reference's operation order, one rounding per operation (the translation
//      unit is built with --fmad=false); bit-identical to the reference's FP64 CPU path.
//   0  the same algorithm with fused multiply-adds, shared reciprocals and
//      precomputed gamma-dependent constants; agrees to ~1e-15 relative per operation.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#ifndef APH_EXACT
#define APH_EXACT 0
#endif

namespace aph {

constexpr int IDN = 0, IM1 = 1, IM2 = 2, IM3 = 3, IEN = 4, NHYDRO = 5;
constexpr int IV1 = 1, IV2 = 2, IV3 = 3, IPR = 4;
constexpr int RECON_DC = 1, RECON_PLM = 2, RECON_PPM = 3;
constexpr int RS_NONE = 1, RS_HLLE = 2, RS_HLLC = 3, RS_LHLLC = 4;

constexpr double C_LIGHT = 2.99792458e10;        // hydro_hlle.hpp:26
constexpr double C_LIGHT2 = C_LIGHT * C_LIGHT;   // SQR(C_LIGHT)
constexpr double TINY_NUMBER = 1.0e-20;
constexpr double PPM_C2 = 1.25;                  // ppm_simple.hpp:36

// ---- integer-pipe predicates ------------------------------------------------
__device__ __forceinline__ bool is_neg(double x) {  // x < 0.0
  const int hi = __double2hiint(x), lo = __double2loint(x);
  return (hi < 0) & (((((unsigned)hi) << 1) | (unsigned)lo) != 0u);
}
__device__ __forceinline__ bool is_pos(double x) {  // x > 0.0
  const int hi = __double2hiint(x), lo = __double2loint(x);
  return (hi >= 0) & ((hi | lo) != 0);
}
// monotone integer key: a < b  <=>  okey(a) < okey(b)  (-0.0 and +0.0 share key 0)
__device__ __forceinline__ long long okey(double x) {
  const long long b = __double_as_longlong(x);
  return b >= 0 ? b : (long long)(0x8000000000000000ULL - (unsigned long long)b);
}
__device__ __forceinline__ bool lt(double a, double b) { return okey(a) < okey(b); }
__device__ __forceinline__ bool le(double a, double b) { return okey(a) <= okey(b); }
__device__ __forceinline__ bool gt(double a, double b) { return okey(a) > okey(b); }
// std::min / std::max tie rules (the first argument wins when neither is smaller)
__device__ __forceinline__ double smin(double a, double b) { return lt(b, a) ? b : a; }
__device__ __forceinline__ double smax(double a, double b) { return lt(a, b) ? b : a; }
// The sign bit is masked and flipped in PTX, out of the compiler's sight: it would make an FP64
// instruction (a DADD with an absolute or negated operand) of it.
__device__ __forceinline__ unsigned abs_hi(double x) {
  unsigned r;
  asm("and.b32 %0, %1, 0x7fffffff;" : "=r"(r) : "r"(__double2hiint(x)));
  return r;
}
__device__ __forceinline__ unsigned long long mag(double x) {
  return ((unsigned long long)abs_hi(x) << 32) | (unsigned)__double2loint(x);
}
__device__ __forceinline__ double dabs(double x) {
  return __hiloint2double((int)abs_hi(x), __double2loint(x));
}
// bits of 2*|x| (exact doubling: exponent +1, or a shift for subnormals; overflow -> inf)
__device__ __forceinline__ unsigned long long twice_mag(double x) {
  const unsigned long long m = mag(x);
  const unsigned long long e = m >> 52;
  if (e == 0) return m << 1;
  if (e >= 0x7feULL) return 0x7ff0000000000000ULL;
  return m + (1ULL << 52);
}
// v with its sign flipped when neg (SIGN(s) * v for SIGN in {-1, +1})
__device__ __forceinline__ double flip_if(double v, bool neg) {
  int hi;
  asm("xor.b32 %0, %1, %2;" : "=r"(hi) : "r"(__double2hiint(v)), "r"(neg ? 0x80000000u : 0u));
  return __hiloint2double(hi, __double2loint(v));
}
__device__ __forceinline__ double from_bits(unsigned long long b) { return __longlong_as_double((long long)b); }
// b strictly between a and c: the reference's sign test (b - a) * (c - b) > 0 without the FP64
// subtractions and product (a difference of finite doubles is zero only when they are
// equal; the two differ only where the product underflows to zero, for differences of
// order 1e-162).  Fast mode, and tame windows.
__device__ __forceinline__ bool strictly_between(double a, double b, double c) {
  const long long ka = okey(a), kb = okey(b), kc = okey(c);
  return ((ka < kb) & (kb < kc)) | ((ka > kb) & (kb > kc));
}
// x beyond both a and b on the same side: the sign test (x - a) * (b - x) < 0.  As above.
__device__ __forceinline__ bool strictly_outside(double x, double a, double b) {
  const long long kx = okey(x), ka = okey(a), kb = okey(b);
  return ((kx > ka) & (kx > kb)) | ((kx < ka) & (kx < kb));
}

// ---- exact operations on the integer pipe for tame operands -------------------------
// A value is tame when it is zero or a normal number with 2^-200 <= |x| < 2^201.  The
// reconstruction of a window of tame values only forms sums, differences and a few
// products and quotients of them, which stay zero or normal far from the underflow and
// overflow thresholds (a nonzero difference of tame values is at least 2^-252).  For those
// values the operations below give exactly the bits of the FP64 operation they replace:
//   half_x(x) == 0.5 * x and twice_x(x) == 2.0 * x (an exponent step; zero kept),
//   div6_x(x) == x / 6.0 (correctly rounded, see below),
// and the sign of a product of two differences is the product of their signs (no product
// underflows), which strictly_between / strictly_outside decide on the integer pipe.
__device__ __forceinline__ bool tame(double x) {
  const unsigned hi = (unsigned)__double2hiint(x) & 0x7fffffffu;
  const unsigned e = hi >> 20;  // biased exponent
  return (e - (1023u - 200u) <= 400u) | ((hi | (unsigned)__double2loint(x)) == 0u);
}
// Zero or 2^-110 <= |x| < 2^111.  From the face states of such cells the exact Riemann solvers form no
// product or quotient outside 2^+-1000 as long as their denominators and the few results they
// check stay within 2^+-400, so their other operations need no checks of their own.  The signs of
// a face's states do not follow from the cells': at a deep trough of positive cells PPM forms
// negative densities and pressures, whose roots are NaN, so the solvers look at those (positive).
__device__ __forceinline__ bool snug(double x) {
  const unsigned hi = abs_hi(x);
  return (hi - ((1023u - 110u) << 20) < (221u << 20)) | ((hi | (unsigned)__double2loint(x)) == 0u);
}
// (word by word: from a test of all 64 bits the compiler makes a DSETP, an FP64 instruction)
__device__ __forceinline__ bool is_zero(double x) {
  return ((((unsigned)__double2hiint(x)) << 1) | (unsigned)__double2loint(x)) == 0u;
}
__device__ __forceinline__ double half_x(double x) {
  const int hi = __double2hiint(x);
  return __hiloint2double(is_zero(x) ? hi : hi - 0x100000, __double2loint(x));
}
__device__ __forceinline__ double twice_x(double x) {
  const int hi = __double2hiint(x);
  return __hiloint2double(is_zero(x) ? hi : hi + 0x100000, __double2loint(x));
}
// x / 6.0 correctly rounded, on the integer pipe: x / 6 = (x / 3) / 2, and with the significand
// moved left by one or two bits to N, the quotient's significand is the integer nearest N / 3,
// which is floor((N + 1) / 3) (N / 3 is never halfway).  2^30 is 1 modulo 3, so for
// N + 1 = H 2^30 + L that is H (2^30 - 1) / 3 + floor((H + L) / 3).  Valid for x zero or normal with
// 2^-1000 < |x| < 2^1000.  9 SM-cycles per warp on GB300 (26 in an earlier form built on
// __umul64hi; a DADD takes 17).
__device__ __forceinline__ double div6_x(double x) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const unsigned hi = (unsigned)(u >> 32);
  const unsigned top = (hi >> 19) & 1u;  // the significand is 1.5 or more
  const unsigned long long M = (u & 0xfffffffffffffULL) | 0x10000000000000ULL;
  const unsigned long long N = (top ? M << 1 : M << 2) + 1;
  const unsigned L = (unsigned)N & 0x3fffffffu, H = (unsigned)(N >> 30);
  const unsigned long long m =
      (unsigned long long)H * 0x15555555u + (__umulhi(H + L, 0xAAAAAAABu) >> 1);
  // the exponent falls by 3 (2 if top), and m's leading bit adds one
  const unsigned e = (hi & 0xfff00000u) - (4u - top) * 0x100000u;
  const unsigned long long r = m + ((unsigned long long)e << 32);
  return is_zero(x) ? x : __longlong_as_double((long long)r);  // +-0 / 6 = +-0
}

// ---- IEEE double multiplications by constants on the integer pipe -------------------------
// RN(k * x) for k = C * 2^S2 with C = 3 (k = 3 or 6) or C = 5 (k = 1.25): the product of the
// significand and C is one or two (C = 5: two or three) bits longer than a significand.
template <int C, int S2>
__device__ __forceinline__ double mulk_x(double x) {
  const unsigned long long u = (unsigned long long)__double_as_longlong(x);
  const unsigned hi = (unsigned)(u >> 32);
  const unsigned long long P =
      ((u & 0xfffffffffffffULL) | 0x10000000000000ULL) * (unsigned long long)C;
  constexpr int s0 = C == 5 ? 2 : 1;
  const unsigned longer = (unsigned)(P >> (53 + s0));  // 0 or 1
  const unsigned sh = s0 + longer;
  const unsigned long long m = (P + ((1ULL << (sh - 1)) - 1 + ((P >> sh) & 1))) >> sh;  // to even
  const unsigned e = (hi & 0xfff00000u) + (unsigned)(s0 + S2 - 1 + (int)longer) * 0x100000u;
  const unsigned long long r = m + ((unsigned long long)e << 32);
  return is_zero(x) ? x : __longlong_as_double((long long)r);  // k * +-0 = +-0
}

// ---- correctly rounded quotients, reciprocals and square roots on the integer pipe ------
// GB300 spends 144 SM-cycles per warp on an IEEE double division and 151 on a square root (8-9
// instructions of a pipe that takes 17 cycles each).  The digit recurrences below take 20 cycles
// per warp in 32-bit integer instructions and give the same bits: a 32-bit reciprocal (or
// reciprocal square root) word from the hardware's FP32 approximation and one Newton step, the
// quotient's (root's) first ~30 bits by a multiplication with that word, the exact 64-bit
// remainder, the remaining bits the same way, and one correction by the exact final remainder.
// (Long division with an approximate reciprocal: D. E. Knuth, TAOCP 2, 4.3.1; Newton's iteration
// for 1/b and 1/sqrt(x).)  54 bits come out, the last one being the round bit: a quotient or
// root of doubles is never halfway between two doubles, so adding it rounds to nearest.
__device__ __forceinline__ unsigned long long mulw(unsigned a, unsigned b) {
  return (unsigned long long)a * (unsigned long long)b;
}
__device__ __forceinline__ unsigned long long significand(unsigned long long u) {
  return (u & 0xfffffffffffffULL) | 0x10000000000000ULL;
}

// R = Y - d, 1 <= d < 5, for Y = 2^84 / B and a significand B.  With y = 2^52 / B (1/2 < y <= 1)
// and f = B / 2^52 cut to 24 bits, the approximation (relative error 2^-23) lowered by 5 units of
// 2^-24, and kept at or above 1/2, is y0 in [y - 7 2^-24, y]; the Newton step y0 (2 - y0 / y)
// leaves (y - y0)^2 / y < 2^-41 plus at most two units of 2^-32 for B's dropped bits (upwards) and
// one for the cut products (downwards); 3 is subtracted so that R < Y, also modulo 2^32.
__device__ __forceinline__ unsigned rcp_word(unsigned long long B) {
  const unsigned b1 = (unsigned)(B >> 21);
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(0x3f800000u | ((b1 >> 8) & 0x7fffffu))));
  const unsigned rb = max(__float_as_uint(r) - 5u, 0x3f000000u);
  const unsigned R0 = (rb << 8) | 0x80000000u;
  const unsigned eh = (unsigned)((0x8000000000000000ULL - mulw(R0, b1)) >> 16);
  return R0 + (unsigned)(mulw(R0, eh) >> 47) - 3u;
}

// RN(a / b) from the bits of a and b, both normal with a normal quotient; R = rcp_word of b's
// significand.  With A the numerator's significand moved so that B <= A < 2B, q1 is at most 7
// below A 2^30 / B (cut operands 1 + 5, floor 1), so the remainder r1 < 7 B < 2^56, and q2 falls
// short of the integer part of r1 2^23 / B by at most one (cut operands 0.2, floors 1), which the
// remainder r2 shows.
__device__ __forceinline__ double quot_bits(unsigned long long ua, unsigned long long ub, unsigned R) {
  unsigned long long A = significand(ua);
  const unsigned long long B = significand(ub);
  const unsigned less = A < B ? 1u : 0u;
  A <<= less;
  const unsigned q1 = __umulhi((unsigned)(A >> 22), R);
  const unsigned long long r1 = (A << 30) - (unsigned long long)q1 * B;
  unsigned q2 = __umulhi((unsigned)(r1 >> 24), R) >> 5;
  const unsigned long long r2 = (r1 << 23) - (unsigned long long)q2 * B;
  q2 += r2 >= B ? 1u : 0u;
  const unsigned long long m = (((unsigned long long)q1 << 23) + q2 + 1) >> 1;  // 53 bits, rounded
  const unsigned ah = (unsigned)(ua >> 32), bh = (unsigned)(ub >> 32);
  const unsigned e = (ah & 0x7ff00000u) - (bh & 0x7ff00000u) + ((1022u - less) << 20);
  return __hiloint2double((int)(((unsigned)(m >> 32) + e) | ((ah ^ bh) & 0x80000000u)), (int)(unsigned)m);
}

// RN(sqrt(x)) for x normal and positive.  With x = X 4^k, 1 <= X < 4, M = X 2^52 and y = 1/sqrt(X):
// the approximation (relative error 2^-22.9) of X cut to 24 bits, lowered by 4 units of 2^-24, is
// y0 in [y - 6.2 2^-24, y]; the Newton step y0 (3 - X y0^2) / 2 leaves 1.5 (y - y0)^2 / y < 2^-41, up to
// 4 units of 2^-32 upwards for the cut products and one down, so R = Y - d, 1 <= d < 6.2, for
// Y = y 2^32.  s1 is at most 8.1 below sqrt(X) 2^30, the remainder r1 = M 2^8 - s1^2 < 2^35.1, and s2
// (ignoring s2^2: at most 0.3 low) at most 1.6 below the rest of the 54-bit root: r2, the remainder
// of M 2^54, shows whether one more fits.
__device__ __forceinline__ double sqrt_bits(unsigned long long u) {
  const unsigned e = (unsigned)(u >> 52);
  const unsigned odd = (e & 1u) ^ 1u;  // e - 1023 is odd
  const unsigned long long M = significand(u) << odd;
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;"
      : "=f"(r)
      : "f"(__uint_as_float((odd ? 0x40000000u : 0x3f800000u) | ((unsigned)(u >> 29) & 0x7fffffu))));
  const unsigned rb = max(__float_as_uint(r) - 4u, 0x3f000000u);
  const unsigned R0 = (rb << 8) | 0x80000000u;
  const unsigned x1 = (unsigned)(M >> 22);
  const unsigned eh = (unsigned)((0x4000000000000000ULL - mulw(x1, __umulhi(R0, R0))) >> 16);
  const unsigned R = R0 + (unsigned)(mulw(R0, eh) >> 47) - 5u;
  const unsigned s1 = __umulhi(x1, R);
  const unsigned long long r1 = (M << 8) - mulw(s1, s1);
  const unsigned s2 = (unsigned)(mulw((unsigned)(r1 >> 4), R) >> 36);
  const unsigned long long r2 = (((r1 << 22) - mulw(s1, s2)) << 24) - mulw(s2, s2);
  const unsigned long long S = ((unsigned long long)s1 << 23) + s2;
  const unsigned long long m = (S + 1 + (r2 > 2 * S ? 1u : 0u)) >> 1;
  return __longlong_as_double((long long)(m + ((unsigned long long)((e + 1022u - odd) >> 1) << 52)));
}

// How far the high word of |x| lies above that of 2^-400; kFar or more above: x is outside
// 2^-400 .. 2^401 (zero, infinite and NaN included; signed: also where x is negative).  Quotients,
// products of two and roots of values inside are normal.
constexpr unsigned kFar = 801u << 20;
__device__ __forceinline__ unsigned far_of(double x) { return abs_hi(x) - (623u << 20); }
__device__ __forceinline__ unsigned far_of_signed(double x) {
  return (unsigned)__double2hiint(x) - (623u << 20);
}

// A denominator and its reciprocal word, which several quotients may share.
struct Den {
  double b;
  unsigned R;
};

// Operations of a Riemann solve on the integer pipe, free of branches: far collects the largest
// distance over the denominators and what else the caller has it see; where that is out of range
// the solve is taken again with IeeeOps.  Other operands are not checked (snug states): the caller
// makes sure that numerators (div) are not zero and radicands are positive.  div0 allows a
// numerator of zero, mul any zeros.
struct IntOps {
  static constexpr bool kInt = true;
  unsigned far = 0;
  __device__ __forceinline__ Den den(double b) {
    far = max(far, far_of(b));
    return Den{b, rcp_word(significand((unsigned long long)__double_as_longlong(b)))};
  }
  __device__ __forceinline__ double div(double a, const Den &d) {
    return quot_bits((unsigned long long)__double_as_longlong(a),
                     (unsigned long long)__double_as_longlong(d.b), d.R);
  }
  __device__ __forceinline__ double div0(double a, const Den &d) {
    const double q = div(a, d);
    const int sg = (__double2hiint(a) ^ __double2hiint(d.b)) & (int)0x80000000;
    return is_zero(a) ? __hiloint2double(sg, 0) : q;
  }
  __device__ __forceinline__ double rcp(double b) { return div(1.0, den(b)); }
  // a value that has to be positive and inside the range, as such and as a denominator
  __device__ __forceinline__ void positive(double x) { far = max(far, far_of_signed(x)); }
  __device__ __forceinline__ Den den_positive(double b) {
    positive(b);
    return Den{b, rcp_word(significand((unsigned long long)__double_as_longlong(b)))};
  }
  __device__ __forceinline__ double rcp_positive(double b) { return div(1.0, den_positive(b)); }
  __device__ __forceinline__ double sqrt(double x) {
    return sqrt_bits((unsigned long long)__double_as_longlong(x));
  }
  // RN(a b), a and b zero or normal: the 106-bit product of the significands, rounded by a carry
  // chain.  13 SM-cycles per warp on pipes of its own, where a DMUL holds the FP64 pipe for 17.
  __device__ __forceinline__ double mul(double a, double b) {
    unsigned unused;
    return product(a, b, unused);
  }
  // far_e: far_of the product, before its exponent can wrap
  __device__ __forceinline__ double product(double a, double b, unsigned &far_e) {
    const unsigned ah = (unsigned)__double2hiint(a), bh = (unsigned)__double2hiint(b);
    const unsigned ea = ah & 0x7ff00000u, eb = bh & 0x7ff00000u;
    unsigned __int128 P = (unsigned __int128)significand((unsigned long long)__double_as_longlong(a)) *
                          (significand((unsigned long long)__double_as_longlong(b)) << 11);
    const unsigned low = ((unsigned)((unsigned long long)(P >> 64) >> 32) >> 20) ^ 1u;  // 1: below 2^116
    P <<= low;
    P += 0x7fffffffffffffffULL + ((unsigned)(unsigned long long)(P >> 64) & 1u);  // to even
    const unsigned long long m = (unsigned long long)(P >> 64);
    // (the leading bit of the significand adds one to the exponent)
    const unsigned e = ea + eb - ((1023u + low) << 20);
    const unsigned sg = (ah ^ bh) & 0x80000000u;
    const bool z = min(ea, eb) == 0u;
    far_e = z ? 0u : (unsigned)(m >> 32) + e - (623u << 20);
    return __hiloint2double((int)(z ? sg : (((unsigned)(m >> 32) + e) | sg)), (int)(z ? 0u : (unsigned)m));
  }
  __device__ __forceinline__ double half(double x) { return half_x(x); }
  __device__ __forceinline__ double twice(double x) { return twice_x(x); }
  // a value that has to be zero or inside the range
  __device__ __forceinline__ void see(double x) { far = max(far, is_zero(x) ? 0u : far_of(x)); }
  __device__ __forceinline__ void give_up() { far = ~0u; }
  __device__ __forceinline__ bool ok() const { return far < kFar; }
};
// The same with every operand and product checked, for arithmetic on any values.
struct CheckedOps : IntOps {
  __device__ __forceinline__ double div(double a, const Den &d) {
    far = max(far, far_of(a));
    return IntOps::div(a, d);
  }
  __device__ __forceinline__ double div0(double a, const Den &d) {
    see(a);
    return IntOps::div0(a, d);
  }
  __device__ __forceinline__ double rcp(double b) { return IntOps::div(1.0, den(b)); }
  __device__ __forceinline__ double sqrt(double x) {
    far = max(far, far_of_signed(x));
    return IntOps::sqrt(x);
  }
  __device__ __forceinline__ double mul(double a, double b) {
    const double r = IntOps::mul(a, b);
    see(r);
    return r;
  }
};
// The fast solvers': an operand of a product is a state value the solver has seen, a product, a
// quotient, a reciprocal root (seen: that of a zero is infinite, and a product with zero would hide
// it) or a sum of those, so it is finite and zero or normal, and the exponent of the product tells
// whether the result is.
struct FaceOps : CheckedOps {
  __device__ __forceinline__ double rsqrt(double x) {
    const double r = ::rsqrt(x);
    far = max(far, far_of(r));
    return r;
  }
  __device__ __forceinline__ double mul(double a, double b) {
    unsigned e;
    const double r = product(a, b, e);
    far = max(far, e);
    return r;
  }
};
struct IeeeOps {
  static constexpr bool kInt = false;
  __device__ __forceinline__ Den den(double b) { return Den{b, 0u}; }
  __device__ __forceinline__ double div(double a, const Den &d) { return __ddiv_rn(a, d.b); }
  __device__ __forceinline__ double div0(double a, const Den &d) { return __ddiv_rn(a, d.b); }
  __device__ __forceinline__ double rcp(double b) { return __drcp_rn(b); }
  __device__ __forceinline__ void positive(double) {}
  __device__ __forceinline__ Den den_positive(double b) { return Den{b, 0u}; }
  __device__ __forceinline__ double rcp_positive(double b) { return __drcp_rn(b); }
  __device__ __forceinline__ double sqrt(double x) { return __dsqrt_rn(x); }
  __device__ __forceinline__ double rsqrt(double x) { return ::rsqrt(x); }
  __device__ __forceinline__ double mul(double a, double b) { return __dmul_rn(a, b); }
  __device__ __forceinline__ double half(double x) { return __dmul_rn(0.5, x); }
  __device__ __forceinline__ double twice(double x) { return __dadd_rn(x, x); }
  __device__ __forceinline__ void see(double) {}
  __device__ __forceinline__ void give_up() {}
  __device__ __forceinline__ bool ok() const { return true; }
};

// A face's solve: the exact one takes snug states, the fast one any.
#if APH_EXACT
using SolveOps = IntOps;
#else
using SolveOps = FaceOps;
#endif

// Single operations for any operands: the digits, or the IEEE instruction where an operand is far
// (a branch: predicating the instruction instead leaves its whole FP64 sequence in the path, which
// cost the fast stage kernel 15 %).
__device__ __forceinline__ Den den(double b) {
  return Den{b, rcp_word(significand((unsigned long long)__double_as_longlong(b)))};
}
__device__ __forceinline__ double div_x(double a, const Den &d) {
  CheckedOps o;
  const double q = o.div0(a, d);
  if (max(o.far, far_of(d.b)) >= kFar) return __ddiv_rn(a, d.b);
  return q;
}
__device__ __forceinline__ double div_x(double a, double b) { return div_x(a, den(b)); }
__device__ __forceinline__ double rcp_x(double b) {
  if (far_of(b) >= kFar) return __drcp_rn(b);
  return quot_bits(0x3ff0000000000000ULL, (unsigned long long)__double_as_longlong(b), den(b).R);
}
__device__ __forceinline__ double sqrt_x(double x) {
  if (is_zero(x)) return x;
  if (far_of_signed(x) >= kFar) return __dsqrt_rn(x);
  return sqrt_bits((unsigned long long)__double_as_longlong(x));
}

// ---- gamma-dependent constants of a pack (fast mode) ---------------------------
struct GasConsts {
  double gm1, igm1, gamma;      // eos/gm1, 1/gm1, gm1+1
  double c2g;                   // C^2 * gamma
  double one_igm1;              // 1 + 1/gm1
  double hlle_k;                // (gamma+1)/sqrt(2 gamma)
  double hllc_k;                // (gamma+1)/(2 gamma)
};

// ---- ideal gas (singularity-eos IdealGas) ------------------------------------
// The reference's ConsToPrim arithmetic after the density floor (hydro.cpp:502-531), one
// rounded operation at a time in its order: the fast build contracts products and sums into
// FMAs, and these values must match the reference bit for bit where they feed the
// discontinuous PPM limiters (the adiabatic-index fields of blocks where a floor fired, which
// the fast mode otherwise replaces by the constants) or the non-idempotent pressure floor.
// u_d: the floored density.  Sets w, g_c, g_e and u[IEN]; returns whether the pressure floor
// fired (with IntOps, which gives up there, at a zero internal energy and on far operands: not
// valid then).
template <class OPS>
__device__ __forceinline__ bool cons_to_prim_tail(double *u, double *w, double &g_c, double &g_e,
                                                  double u_d, double gm1, double pfloor, OPS &o) {
  const Den rho = o.den(u_d);
  const double di = o.div(1.0, rho);
  const double m1 = u[IM1], m2 = u[IM2], m3 = u[IM3];
  double u_e = u[IEN];
  o.see(m1);
  o.see(m2);
  o.see(m3);
  o.see(u_e);
  w[IDN] = u_d;
  w[IV1] = o.mul(m1, di);
  w[IV2] = o.mul(m2, di);
  w[IV3] = o.mul(m3, di);
  const double e_k =
      o.mul(o.half(di), __dadd_rn(__dadd_rn(o.mul(m1, m1), o.mul(m2, m2)), o.mul(m3, m3)));
  double e_i = __dsub_rn(u_e, e_k);
  double sie = o.div0(e_i, rho);
  double w_p = o.mul(o.mul(gm1, u_d), sie);
  w_p = is_neg(w_p) ? 0.0 : w_p;  // eos_pressure
  const bool floored = !gt(w_p, pfloor);
  if (floored) {
    if (OPS::kInt) {
      o.give_up();
    } else {
      const double gm1q = __ddiv_rn(w_p, __dmul_rn(u_d, e_k));  // hydro.cpp:517
      u_e = __dadd_rn(__ddiv_rn(pfloor, gm1q), e_k);
      w_p = pfloor;
      e_i = __dsub_rn(u_e, e_k);
      sie = o.div0(e_i, rho);  // of the floored energy (unchanged otherwise)
    }
  }
  u[IEN] = u_e;
  w[IPR] = w_p;
  const double small = 10.0 * 2.2250738585072014e-308;
  double b = o.mul(o.mul(__dmul_rn(gm1, __dadd_rn(gm1, 1.0)), u_d), sie);  // eos_bulk_modulus
  b = lt(small, b) ? b : small;
  g_c = o.div(b, o.den(w_p));
  g_e = __dadd_rn(o.div(w_p, o.den(e_i)), 1.0);
  return floored;
}
// The same for any state: on the integer pipe, or again with the IEEE instructions.
__device__ __forceinline__ bool cons_to_prim_any(double *u, double *w, double &g_c, double &g_e,
                                                 double u_d, double gm1, double pfloor) {
  CheckedOps o;
  const double e = u[IEN];
  cons_to_prim_tail(u, w, g_c, g_e, u_d, gm1, pfloor, o);
  if (o.ok()) return false;
  IeeeOps ieee;
  u[IEN] = e;
  return cons_to_prim_tail(u, w, g_c, g_e, u_d, gm1, pfloor, ieee);
}

#if !APH_EXACT
// Velocities into w and the returned pressure of the fast ConsToPrim.
template <class OPS>
__device__ __forceinline__ double fast_prim(const double *u, double u_d, double gm1, double *w, OPS &o) {
  const double di = o.rcp(u_d);
  w[IV1] = o.mul(u[IM1], di);
  w[IV2] = o.mul(u[IM2], di);
  w[IV3] = o.mul(u[IM3], di);
  return o.mul(gm1, fma(-o.half(di), fma(u[IM3], u[IM3], fma(u[IM1], u[IM1], o.mul(u[IM2], u[IM2]))), u[IEN]));
}
#endif

// ConsToPrim for one cell (hydro.cpp:459-531, ideal gas).  u[] is updated in place
// by the floors (density, energy); w[] gets rho, v1, v2, v3, p; g_c, g_e the two
// adiabatic indices.  Returns true when the pressure floor was applied.
__device__ __forceinline__ bool cons_to_prim_cell(double *u, double *w, double &g_c, double &g_e,
                                                  double gm1, double dfloor, double pfloor) {
  double u_d = u[IDN];
  const bool dens_ok = gt(u_d, dfloor);
  u_d = dens_ok ? u_d : dfloor;
  u[IDN] = u_d;
#if !APH_EXACT
  // fast: p = gm1 rho ((E - e_k) / rho) = gm1 (E - e_k), and with the floors inactive both
  // adiabatic indices are gamma (B / p = gm1 + 1 = p / (rho e) + 1), so one division per cell
  // (a floored density takes the reference's arithmetic below, whose indices are kept)
  if (dens_ok) {
    w[IDN] = u_d;
    FaceOps o;
    o.see(u[IM1]);
    o.see(u[IM2]);
    o.see(u[IM3]);
    o.see(u[IEN]);
    double pe = fast_prim(u, u_d, gm1, w, o);
    if (!o.ok()) {
      IeeeOps ieee;
      pe = fast_prim(u, u_d, gm1, w, ieee);
    }
    const double wp = is_neg(pe) ? 0.0 : pe;
    if (gt(wp, pfloor)) {
      w[IPR] = wp;
      g_c = gm1 + 1.0;
      g_e = g_c;
      return false;
    }
  }
#endif
  return cons_to_prim_any(u, w, g_c, g_e, u_d, gm1, pfloor);
}

// The reference's adiabatic indices (gamma_c, gamma_e) of a cell whose floors did not fire,
// from its conserved state after ConsToPrim (u: the cell's five values).
__device__ __forceinline__ void gamma_ref(const double *u, double gm1, double &g_c, double &g_e) {
  double uu[NHYDRO] = {u[0], u[1], u[2], u[3], u[4]}, w[NHYDRO];
  cons_to_prim_any(uu, w, g_c, g_e, u[IDN], gm1, -1.0);
}

// ---- reconstruction (src/recon) --------------------------------------------------
__device__ __forceinline__ void plm(double q_im1, double q_i, double q_ip1, double &ql_ip1,
                                    double &qr_i) {
  const double dql = q_i - q_im1;
  const double dqr = q_ip1 - q_i;
  double dqm = 0.0;
#if APH_EXACT
  const double dq2 = dql * dqr;
  if (is_pos(dq2)) dqm = div_x(dq2, dql + dqr);
#else
  FaceOps o;  // (the fast kernel's FP64 pipe is the busier one)
  o.see(dql);
  o.see(dqr);
  double dq2 = o.mul(dql, dqr);
  if (is_pos(dq2)) dqm = o.div(dq2, o.den(dql + dqr));
  if (!o.ok()) {
    dq2 = dql * dqr;
    dqm = is_pos(dq2) ? __ddiv_rn(dq2, dql + dqr) : 0.0;
  }
#endif
  ql_ip1 = q_i + dqm;
  qr_i = q_i - dqm;
}

// PPM split in two.  The limited interface value at a face is a function of the four
// cells around it only, and the reference computes it identically from both adjacent
// cells (its symmetric grouping of the stencil sums makes the two evaluations the same
// operations on the same operands).  ppm_face() evaluates it once per face;
// ppm_cell() then applies the cell's parabola limiter.  Together they give exactly
// PPM(q_im2..q_ip2) of ppm_simple.hpp:32-161.
//
// dd(c) = 0.5*(q[c+1]-q[c]) + 0.5*(q[c]-q[c-1]);  d2(c) = (q[c-1]+q[c+1]) - 2*q[c]
//
// TAME (every window value tame): the same bits with the scalings by constants, the quotient and
// (exact mode) the sign tests of products of differences on the integer pipe, and the limited value
// formed only at the faces that take it.
// (An RK2 step in fast mode, PPM + HLLC, of a 128^3 pack with its host copies: 8.90 -> 6.22 ms.)
template <bool TAME = false>
__device__ __forceinline__ double ppm_dd(double qm1, double q0, double qp1) {
#if APH_EXACT
  if (TAME) return half_x(qp1 - q0) + half_x(q0 - qm1);
  return 0.5 * (qp1 - q0) + 0.5 * (q0 - qm1);
#else
  // the same quantity with one rounding
  return TAME ? half_x(qp1 - qm1) : 0.5 * (qp1 - qm1);
#endif
}
template <bool TAME = false>
__device__ __forceinline__ double ppm_d2(double qm1, double q0, double qp1) {
  if (APH_EXACT && TAME) return (qm1 + qp1) - twice_x(q0);
  return (qm1 + qp1) - 2.0 * q0;
}
// Face between cells c-1 (value qm1) and c (value q0): ddm1 = dd(c-1), dd0 = dd(c),
// d2m1 = d2(c-1), d20 = d2(c).
template <bool TAME = false>
__device__ __forceinline__ double ppm_face(double qm1, double q0, double ddm1, double dd0,
                                           double d2m1, double d20) {
#if APH_EXACT
  if (TAME) {
    const double s = qm1 + q0;
    const double avg = half_x(s);
    double dph = avg + div6_x(ddm1 - dd0);
    // (dph - qm1) * (q0 - dph) < 0, the differences being nonzero and their product normal; the
    // limited value, which only such a face takes, is formed there
    // (selects inside: lanes that part in a nested branch would take the last addition one
    // group after the other)
    if (strictly_outside(dph, qm1, q0)) {
      const double qa = mulk_x<3, 0>(s - twice_x(dph));
      const bool sa = is_neg(qa);
      const unsigned long long mb = mag(d2m1), mc = mag(d20), ma = mag(qa);
      const unsigned long long mm = mag(mulk_x<5, -2>(from_bits(mc < mb ? mc : mb)));  // PPM_C2 = 5/4
      const bool same = (sa == is_neg(d2m1)) & (sa == is_neg(d20));
      const double qd = flip_if(from_bits(ma < mm ? ma : mm), sa);
      dph = avg - div6_x(same ? qd : 0.0);
    }
    return dph;
  }
#else
  if (TAME) {
    const double s = qm1 + q0;
    const double avg = half_x(s);
    double dph = fma(ddm1 - dd0, 1.0 / 6.0, avg);
    if (strictly_outside(dph, qm1, q0)) {
      const double qa = mulk_x<3, 0>(fma(-2.0, dph, s));
      const bool sa = is_neg(qa);
      const unsigned long long mb = mag(d2m1), mc = mag(d20), ma = mag(qa);
      const unsigned long long mm = mag(mulk_x<5, -2>(from_bits(mc < mb ? mc : mb)));  // PPM_C2 = 5/4
      const bool same = (sa == is_neg(d2m1)) & (sa == is_neg(d20));
      const double qd = flip_if(from_bits(ma < mm ? ma : mm), sa);
      dph = fma(same ? qd : 0.0, -1.0 / 6.0, avg);
    }
    return dph;
  }
#endif
  const double avg = 0.5 * (qm1 + q0);
#if APH_EXACT
  double dph = avg + (ddm1 - dd0) / 6.0;
#else
  double dph = fma(ddm1 - dd0, 1.0 / 6.0, avg);
#endif
#if APH_EXACT
  const double qa_tmp = dph - qm1;
  const double qb_tmp = q0 - dph;
#endif
  const double qa = 3.0 * (qm1 + q0 - 2.0 * dph);
  double qd = 0.0;
  const bool sa = is_neg(qa);
  if (sa == is_neg(d2m1) && sa == is_neg(d20)) {
    // min(C2|qb|, min(C2|qc|, |qa|)) with the two scalings merged (scaling by a positive
    // constant is monotone, so min(C2 x, C2 y) == C2 min(x, y) bit for bit)
    const unsigned long long mb = mag(d2m1), mc = mag(d20);
    const double m = PPM_C2 * from_bits(mc < mb ? mc : mb);
    const unsigned long long mm = mag(m), ma = mag(qa);
    qd = flip_if(from_bits(ma < mm ? ma : mm), sa);
  }
#if APH_EXACT
  if (is_neg(qa_tmp * qb_tmp)) dph = avg - qd / 6.0;
#else
  if (strictly_outside(dph, qm1, q0)) dph = fma(qd, -1.0 / 6.0, avg);
#endif
  return dph;
}

// The limited curvature of an extremum with d2qf, tame operands; guard: whether d2qf counts; src:
// where it comes from (0 nowhere, 1..3 the cell i-1, i, i+1, 4 d2qf itself).
__device__ __forceinline__ double extremum_qe(double d2qf, double d2m1, double d20, double d2p1, double q_im2,
                                              double q_im1, double q_i, double q_ip1, double q_ip2, bool &guard,
                                              int &src) {
  const bool sd = is_neg(d2qf);
  unsigned long long m = mag(d2m1);
  const unsigned long long m0 = mag(d20), m1 = mag(d2p1), md = mag(d2qf);
  src = m0 < m ? 2 : 1;
  m = m0 < m ? m0 : m;
  src = m1 < m ? 3 : src;
  m = m1 < m ? m1 : m;
  const unsigned long long ms = mag(mulk_x<5, -2>(from_bits(m)));
  const bool same = (sd == is_neg(d2m1)) & (sd == is_neg(d20)) & (sd == is_neg(d2p1));
  const double qe = same ? flip_if(from_bits(md < ms ? md : ms), sd) : 0.0;
  src = same ? (md < ms ? 4 : src) : 0;
  unsigned long long mx = mag(q_im2);
  const unsigned long long a1 = mag(q_im1), a2 = mag(q_i), a3 = mag(q_ip1), a4 = mag(q_ip2);
  mx = a1 > mx ? a1 : mx;
  mx = a2 > mx ? a2 : mx;
  mx = a3 > mx ? a3 : mx;
  mx = a4 > mx ? a4 : mx;
  // the roundoff guard |d2qf| > 1e-12 * max|q| (ppm_simple.hpp:132); RN(1e-12 * mx) lies in
  // [2^-40, 2^-38) times mx's binade, so the exponents decide it except within two binades
  // (0 > anything is false, a nonzero value over 0 true)
  IntOps o;
  const int ed = (int)(md >> 52), em = (int)(mx >> 52);
  guard = ed >= em - 38;
  if ((ed < em - 38) & (ed > em - 41)) guard = md > mag(o.mul(1.0e-12, from_bits(mx)));
  guard = guard & (md != 0ULL);
  return qe;
}

// Cell limiter: dph_lo, dph_hi are the limited values at faces i-1/2, i+1/2.
// Outputs ql_ip1 (left state of face i+1/2) and qr_i (right state of face i-1/2).
template <bool TAME = false>
__device__ __forceinline__ void ppm_cell(double q_im2, double q_im1, double q_i, double q_ip1,
                                         double q_ip2, double d2m1, double d20, double d2p1,
                                         double dph_lo, double dph_hi, double &ql_ip1,
                                         double &qr_i) {
  double qr = dph_lo, ql = dph_hi;
  const double dqf_minus = q_i - qr;
  const double dqf_plus = ql - q_i;
#if APH_EXACT
  if (TAME) {
    // the states are qr = q_i - xm where sub_m, ql = q_i + xp where add_p: one addition each
    // for all lanes whatever branch formed the steps
    double xm = 0.0, xp = 0.0;
    bool sub_m, add_p;
    // the signs of the two products of differences, as in ppm_face
    if (!strictly_between(qr, q_i, ql) | !strictly_between(q_im1, q_i, q_ip1)) {
      const double d2qf = mulk_x<3, 1>((dph_lo + dph_hi) - twice_x(q_i));
      bool guard;
      int src;
      const double qe = extremum_qe(d2qf, d2m1, d20, d2p1, q_im2, q_im1, q_i, q_ip1, q_ip2, guard, src);
      IntOps o;  // (tame operands: all in range)
      // rho = qe / d2qf with the guard, else +0.  Where it is a zero (of qe's and d2qf's signs with
      // the guard) the steps are signed zeros; where qe is d2qf it is 1 > 1 - 1e-12: the face
      // values stay
      const bool none = is_zero(qe) | !guard;
      const double rho = o.div(qe, o.den(d2qf));
      const unsigned rs = guard ? (unsigned)(__double2hiint(qe) ^ __double2hiint(d2qf)) & 0x80000000u : 0u;
      auto step = [&](double dqf) {
        const double z = __hiloint2double((int)(rs ^ ((unsigned)__double2hiint(dqf) & 0x80000000u)), 0);
        const double r = o.mul(rho, dqf);
        return none ? z : r;
      };
      xm = step(dqf_minus);
      xp = step(dqf_plus);
      sub_m = add_p = none | le(rho, 1.0 - 1.0e-12);
    } else {
      sub_m = mag(dqf_minus) >= twice_mag(dqf_plus);
      add_p = mag(dqf_plus) >= twice_mag(dqf_minus);
      xm = twice_x(dqf_plus);
      xp = twice_x(dqf_minus);
    }
    const double rm = q_i - xm, lp = q_i + xp;
    qr_i = sub_m ? rm : qr;
    ql_ip1 = add_p ? lp : ql;
    return;
  }
  const double qa_tmp = dqf_minus * dqf_plus;
  const double qb_tmp = (q_ip1 - q_i) * (q_i - q_im1);
  if (!is_pos(qa_tmp) || !is_pos(qb_tmp)) {
#else
  if (TAME) {
    // the states are q_i -+ f times a difference: one fused operation each for all lanes
    double f = 2.0, xm = dqf_plus, xp = dqf_minus;
    bool sub_m = mag(dqf_minus) >= twice_mag(dqf_plus), add_p = mag(dqf_plus) >= twice_mag(dqf_minus);
    if (!strictly_between(qr, q_i, ql) | !strictly_between(q_im1, q_i, q_ip1)) {
      const double d2qf = mulk_x<3, 1>(fma(-2.0, q_i, dph_lo + dph_hi));
      bool guard;
      int src;
      const double qe = extremum_qe(d2qf, d2m1, d20, d2p1, q_im2, q_im1, q_i, q_ip1, q_ip2, guard, src);
      IntOps o;
      const double rho = o.div0(qe, o.den(d2qf));
      f = guard ? rho : 0.0;
      xm = dqf_minus;
      xp = dqf_plus;
      sub_m = add_p = le(f, 1.0 - 1.0e-12);
    }
    const double rm = fma(-f, xm, q_i), lp = fma(f, xp, q_i);
    qr_i = sub_m ? rm : qr;
    ql_ip1 = add_p ? lp : ql;
    return;
  }
  if (!strictly_between(qr, q_i, ql) || !strictly_between(q_im1, q_i, q_ip1)) {
#endif
    // local extremum: limit with rho = qe/qd (CS eq 22-23, MC eq 27)
    const double d2qf = 6.0 * (dph_lo + dph_hi - 2.0 * q_i);
    double qe = 0.0;
    const bool sd = is_neg(d2qf);
    if (sd == is_neg(d2m1) && sd == is_neg(d20) && sd == is_neg(d2p1)) {
      unsigned long long m = mag(d2m1);
      const unsigned long long m0 = mag(d20), m1 = mag(d2p1);
      m = m0 < m ? m0 : m;
      m = m1 < m ? m1 : m;
      const unsigned long long ms = mag(PPM_C2 * from_bits(m));
      const unsigned long long md = mag(d2qf);
      qe = flip_if(from_bits(md < ms ? md : ms), sd);
    }
    unsigned long long mx = mag(q_im2);
    const unsigned long long a1 = mag(q_im1), a2 = mag(q_i), a3 = mag(q_ip1), a4 = mag(q_ip2);
    mx = a1 > mx ? a1 : mx;
    mx = a2 > mx ? a2 : mx;
    mx = a3 > mx ? a3 : mx;
    mx = a4 > mx ? a4 : mx;
    double rho = 0.0;
    if (mag(d2qf) > mag(1.0e-12 * from_bits(mx))) rho = div_x(qe, d2qf);
    if (le(rho, 1.0 - 1.0e-12)) {
#if APH_EXACT
      qr = q_i - rho * dqf_minus;
      ql = q_i + rho * dqf_plus;
#else
      qr = fma(-rho, dqf_minus, q_i);
      ql = fma(rho, dqf_plus, q_i);
#endif
    }
  } else {
    if (mag(dqf_minus) >= twice_mag(dqf_plus)) qr = q_i - 2.0 * dqf_plus;
    if (mag(dqf_plus) >= twice_mag(dqf_minus)) ql = q_i + 2.0 * dqf_minus;
  }
  ql_ip1 = ql;
  qr_i = qr;
}

#if APH_EXACT
// ---- reconstruction of the adiabatic indices as small integers --------------------------
// Where no floor fired, gamma_c = B / p and gamma_e = p / (rho e) + 1 are gamma up to a few
// rounding errors.  A window whose indices all lie within kGamMax units u of the last place of
// gamma = gm1 + 1 (M u, in one binade) is reconstructed on the offsets k = g / u - M: every sum,
// difference and rounding of PPM and PLM on such values is a small integer operation with the
// same result (a sum of two values of the binade is rounded to a multiple of 2 u, half to even;
// a value added to such a mean is rounded to a multiple of u).  In PPM's extremum branch
// |d2qf| <= 6 (2 (kGamMax + 41) + 2 kGamMax + 1) u stays below the roundoff guard's 1e-12 |q| (at least
// 4503 u), so rho is 0 and both face values are the cell's.
constexpr int kGamMax = 100;
__device__ __forceinline__ int gam_round_half(int K, int odd) {  // RN((2 M + K) / 2) - M; odd: of M
  const int h = K >> 1;
  return h + (K & (h + odd) & 1);
}
__device__ __forceinline__ int gam_round_12(int j, int odd) {  // RN(M + j / 12) - M, |j| < 2000
  const int t = j + 6 + 12 * 256;
  const int q = (t * 5462) >> 16;  // floor(t / 12) for 0 <= t < 8160
  return q - 256 - ((t - 12 * q == 0) & (q + odd) & 1);
}
// The limited value at the face between cells of offsets b and c (a, d: the next ones), as
// ppm_face.  avg = M + h; the interpolation adds j / 12 with j the difference of the slopes;
// qa = -6 m u, the second differences 2 e u, and the limited qd / 6 is (qd / u * 2) / 12 u.
__device__ __forceinline__ int gam_face(int a, int b, int c, int d, int odd) {
  const int h = gam_round_half(b + c, odd);
  const int m = gam_round_12((c - a) - (d - b), odd + h);
  int f = h + m;
  if ((f > b && f > c) || (f < b && f < c)) {
    const int eb = gam_round_half(a + c, odd) - b, ec = gam_round_half(b + d, odd) - c;
    int q = 0;
    if ((m > 0) == (eb < 0) && (m > 0) == (ec < 0)) {
      const int lim = 5 * min(abs(eb), abs(ec));
      q = min(12 * abs(m), lim);
      if (m > 0) q = -q;
    }
    f = h + gam_round_12(-q, odd + h);
  }
  return f;
}
// ppm_cell: lo, hi the face values of cell q0 (qm, qp: its neighbours)
__device__ __forceinline__ void gam_cell(int qm, int q0, int qp, int lo, int hi, int &ql, int &qr) {
  const int dm = q0 - lo, dp = hi - q0;
  const bool between = (dm > 0 && dp > 0) || (dm < 0 && dp < 0);
  const bool monotone = (qm < q0 && q0 < qp) || (qm > q0 && q0 > qp);
  if (!between || !monotone) {
    ql = qr = q0;
  } else {
    qr = abs(dm) >= 2 * abs(dp) ? q0 - 2 * dp : lo;
    ql = abs(dp) >= 2 * abs(dm) ? q0 + 2 * dm : hi;
  }
}
// plm: q0 +- dl dr / (dl + dr), rounded half to even
__device__ __forceinline__ void gam_plm(int qm, int q0, int qp, int odd, int &ql, int &qr) {
  const int dl = q0 - qm, dr = qp - q0;
  ql = qr = q0;
  if (dl * dr <= 0) return;
  const unsigned num = dl * dr, sum = abs(dl + dr);
  const int x = (int)(num / sum);
  const unsigned rest = 2 * (num - x * sum);
  const int up = rest > sum || (rest == sum && ((q0 + x + odd) & 1));  // x or x + 1, either way
  const int s = dl > 0 ? x + up : -(x + up);
  ql = q0 + s;
  qr = q0 - s;
}
#endif

// ---- Riemann solvers (src/hydro/rsolvers) -------------------------------------------
// wl, wr: (rho, v_normal, v_t1, v_t2, p).  gl*, gr*: reconstructed (gamma_c, gamma_e).
// With CONSTG the adiabatic indices are the pack's constants (gc) instead.
// flx: (mass, normal momentum, t1 momentum, t2 momentum, energy).

// c-limited sound speed C*sqrt(gamma / (1 + (1/gm1 + rho C^2 / p))) (hydro_hlle.hpp:63-66)

#if APH_EXACT
// A side's density, pressure and adiabatic indices, all positive with gamma_e above 1: then every
// radicand of the exact solvers is positive (rho C^2 / p, 1 / (gamma_e - 1) and gamma are; a shock
// factor is taken where the middle pressure is above p), and no numerator is zero.  Returns
// 1 / (gamma_e - 1).
template <class OPS>
__device__ __forceinline__ double see_side(double rho, double gc, double ge, OPS &o) {
  o.positive(rho);
  o.positive(gc);
  return o.rcp_positive(ge - 1);
}
template <class OPS>
__device__ __forceinline__ double sound_speed(double rho, const Den &p, double gamma, double igm1, OPS &o) {
  return o.mul(C_LIGHT, o.sqrt(o.div(gamma, o.den(1 + (igm1 + o.div(o.mul(rho, C_LIGHT2), p))))));
}

template <class OPS>
__device__ __forceinline__ void solve_hlle_exact(const double *wli, const double *wri, double glc,
                                                 double gle, double grc, double gre, double *flxi,
                                                 OPS &o) {
  const double igm1l = see_side(wli[IDN], glc, gle, o), igm1r = see_side(wri[IDN], grc, gre, o);
  const Den pl = o.den_positive(wli[IPR]), pr = o.den_positive(wri[IPR]);
  const double cl = sound_speed(wli[IDN], pl, glc, igm1l, o);
  const double cr = sound_speed(wri[IDN], pr, grc, igm1r, o);
  auto energy = [&](const double *w, double igm1) {
    return o.mul(w[IPR], igm1) +
           o.mul(o.half(w[IDN]), o.mul(w[IV1], w[IV1]) + o.mul(w[IV2], w[IV2]) + o.mul(w[IV3], w[IV3]));
  };
  const double el = energy(wli, igm1l), er = energy(wri, igm1r);
  const double rhoa = o.half(wli[IDN] + wri[IDN]);
  const double ca = o.half(cl + cr);
  const double pmid = o.half(wli[IPR] + wri[IPR] + o.mul(o.mul(wli[IV1] - wri[IV1], rhoa), ca));
  double ql = 1.0, qr = 1.0;
  if (gt(pmid, wli[IPR]))
    ql = 1.0 + o.mul(o.div(glc + 1, o.den(o.sqrt(o.twice(glc)))), o.div(pmid, pl) - 1.0);
  if (gt(pmid, wri[IPR]))
    qr = 1.0 + o.mul(o.div(grc + 1, o.den(o.sqrt(o.twice(grc)))), o.div(pmid, pr) - 1.0);
  const double al = wli[IV1] - o.mul(cl, ql);
  const double ar = wri[IV1] + o.mul(cr, qr);
  const double bp = is_pos(ar) ? ar : 0.0;
  const double bm = is_neg(al) ? al : 0.0;
  double tmp = 0.0;
  if (__double_as_longlong(bp) != __double_as_longlong(bm) && (mag(bp) | mag(bm)) != 0ULL)
    tmp = o.div0(o.half(bp + bm), o.den(bp - bm));
  double fl[NHYDRO], fr[NHYDRO];
  auto fluxes = [&](const double *w, double b, double e, double *f) {
    const double vx = w[IV1] - b;
    f[IDN] = o.mul(w[IDN], vx);
    f[IV1] = o.mul(o.mul(w[IDN], w[IV1]), vx) + w[IPR];
    f[IV2] = o.mul(o.mul(w[IDN], w[IV2]), vx);
    f[IV3] = o.mul(o.mul(w[IDN], w[IV3]), vx);
    f[IEN] = o.mul(e, vx) + o.mul(w[IPR], w[IV1]);
  };
  fluxes(wli, bm, el, fl);
  fluxes(wri, bp, er, fr);
#pragma unroll
  for (int n = 0; n < NHYDRO; ++n) flxi[n] = o.half(fl[n] + fr[n]) + o.mul(fl[n] - fr[n], tmp);
}

#else
// The fast solvers name every fused multiply-add themselves: left to the compiler, which products
// are fused depends on how it splits the code into blocks, and PPM's discontinuous limiters turn
// a difference of one rounding into a different flux, so that builds and launches would no
// longer agree with one another.
// Their plain products take the integer pipe (FaceOps), the same bits: with PLM + HLLE the stage
// kernel held the FP64 pipe for 67 % of its cycles (PPM + HLLC: 77 %) and the ALU for 6 (12) %.  A
// step of the 512^2 Kelvin-Helmholtz pack (PLM + HLLE) went from 547 to 479 us with it, of the
// 512^2 rollout the forward and backward from 8.41 to 7.94 ms (415 us and 6.55 ms with the products
// of PLM and ConsToPrim there too).
__device__ __forceinline__ double add(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sub(double a, double b) { return __dsub_rn(a, b); }
template <class OPS>
__device__ __forceinline__ double square3(double a, double b, double c, OPS &o) {  // a^2 + b^2 + c^2
  return fma(c, c, fma(a, a, o.mul(b, b)));
}

// the square of the sound speed as num / den
template <bool CONSTG, class OPS>
__device__ __forceinline__ void sound_parts(double rho, double p, double gamma, double igm1,
                                            const GasConsts &gc, double &num, double &root, OPS &o) {
  num = CONSTG ? o.mul(gc.c2g, p) : o.mul(o.mul(C_LIGHT2, gamma), p);
  const double den = fma(p, CONSTG ? gc.one_igm1 : add(1.0, igm1), o.mul(rho, C_LIGHT2));
  root = o.rsqrt(o.mul(num, den));  // the speed is num * root
}
template <bool CONSTG, class OPS>
__device__ __forceinline__ double sound_speed(double rho, double p, double gamma, double igm1,
                                              const GasConsts &gc, OPS &o) {
  double num, root;
  sound_parts<CONSTG>(rho, p, gamma, igm1, gc, num, root, o);
  return o.mul(num, root);
}
// the values a face's products start from
template <bool CONSTG, class OPS>
__device__ __forceinline__ void see_face(const double *wl, const double *wr, double glc, double gle,
                                         double grc, double gre, OPS &o) {
#pragma unroll
  for (int n = 0; n < NHYDRO; ++n) {
    o.see(wl[n]);
    o.see(wr[n]);
  }
  if (!CONSTG) {
    o.see(glc);
    o.see(gle);
    o.see(grc);
    o.see(gre);
  }
}

template <bool CONSTG, class OPS>
__device__ __forceinline__ void solve_hlle(const double *wl, const double *wr, double glc, double gle,
                                           double grc, double gre, const GasConsts &gc, double *flx,
                                           OPS &o) {
  see_face<CONSTG>(wl, wr, glc, gle, grc, gre, o);
  const double gl = CONSTG ? gc.gamma : glc, gr = CONSTG ? gc.gamma : grc;
  const double il = CONSTG ? gc.igm1 : o.rcp(sub(gle, 1)), ir = CONSTG ? gc.igm1 : o.rcp(sub(gre, 1));
  const double cl = sound_speed<CONSTG>(wl[IDN], wl[IPR], gl, il, gc, o);
  const double cr = sound_speed<CONSTG>(wr[IDN], wr[IPR], gr, ir, gc, o);
  const double el = fma(wl[IPR], il, o.mul(o.half(wl[IDN]), square3(wl[IV1], wl[IV2], wl[IV3], o)));
  const double er = fma(wr[IPR], ir, o.mul(o.half(wr[IDN]), square3(wr[IV1], wr[IV2], wr[IV3], o)));
  const double rhoa = o.half(add(wl[IDN], wr[IDN])), ca = o.half(add(cl, cr));
  const double pmid = o.half(fma(o.mul(sub(wl[IV1], wr[IV1]), rhoa), ca, add(wl[IPR], wr[IPR])));
  double ql = 1.0, qr = 1.0;
  const bool bl = gt(pmid, wl[IPR]), br = gt(pmid, wr[IPR]);
  if (bl || br) {
    const double ipp = o.rcp(o.mul(wl[IPR], wr[IPR]));  // shared reciprocal
    const double kl = CONSTG ? gc.hlle_k : o.mul(add(gl, 1), o.rsqrt(o.twice(gl)));
    const double kr = CONSTG ? gc.hlle_k : o.mul(add(gr, 1), o.rsqrt(o.twice(gr)));
    if (bl) ql = fma(kl, fma(o.mul(pmid, wr[IPR]), ipp, -1.0), 1.0);
    if (br) qr = fma(kr, fma(o.mul(pmid, wl[IPR]), ipp, -1.0), 1.0);
  }
  const double al = fma(-cl, ql, wl[IV1]), ar = fma(cr, qr, wr[IV1]);
  const double bp = is_pos(ar) ? ar : 0.0, bm = is_neg(al) ? al : 0.0;
  const double vl = sub(wl[IV1], bm), vr = sub(wr[IV1], bp);
  double fl[NHYDRO], fr[NHYDRO];
  fl[IDN] = o.mul(wl[IDN], vl);
  fr[IDN] = o.mul(wr[IDN], vr);
  fl[IV1] = fma(o.mul(wl[IDN], wl[IV1]), vl, wl[IPR]);
  fr[IV1] = fma(o.mul(wr[IDN], wr[IV1]), vr, wr[IPR]);
  fl[IV2] = o.mul(o.mul(wl[IDN], wl[IV2]), vl);
  fr[IV2] = o.mul(o.mul(wr[IDN], wr[IV2]), vr);
  fl[IV3] = o.mul(o.mul(wl[IDN], wl[IV3]), vl);
  fr[IV3] = o.mul(o.mul(wr[IDN], wr[IV3]), vr);
  fl[IEN] = fma(el, vl, o.mul(wl[IPR], wl[IV1]));
  fr[IEN] = fma(er, vr, o.mul(wr[IPR], wr[IV1]));
  double t = 0.0;
  if (__double_as_longlong(bp) != __double_as_longlong(bm) && (mag(bp) | mag(bm)) != 0ULL)
    t = o.div0(o.half(add(bp, bm)), o.den(sub(bp, bm)));
#pragma unroll
  for (int n = 0; n < NHYDRO; ++n) flx[n] = fma(0.5, add(fl[n], fr[n]), o.mul(sub(fl[n], fr[n]), t));
}

// HLLC; LOWMACH: the pstar of hydro_lhllc.hpp:71-79, whose "Mach" is the speed |v| itself
template <bool CONSTG, bool LOWMACH, class OPS>
__device__ __forceinline__ void solve_hllc(const double *wl, const double *wr, double glc, double gle,
                                           double grc, double gre, const GasConsts &gc, double *flx,
                                           OPS &o) {
  see_face<CONSTG>(wl, wr, glc, gle, grc, gre, o);
  const double gl = CONSTG ? gc.gamma : glc, gr = CONSTG ? gc.gamma : grc;
  const double il = CONSTG ? gc.igm1 : o.rcp(sub(gle, 1)), ir = CONSTG ? gc.igm1 : o.rcp(sub(gre, 1));
  const double cl = sound_speed<CONSTG>(wl[IDN], wl[IPR], gl, il, gc, o);
  const double cr = sound_speed<CONSTG>(wr[IDN], wr[IPR], gr, ir, gc, o);
  const double rhoa = o.half(add(wl[IDN], wr[IDN])), ca = o.half(add(cl, cr));
  double x = o.mul(o.mul(o.half(sub(wr[IV1], wl[IV1])), rhoa), ca);
  if (LOWMACH) {
    auto root = [&](double q) { return is_zero(q) ? q : o.sqrt(is_zero(q) ? 1.0 : q); };
    const double chi = smax(root(square3(wl[IV1], wl[IV2], wl[IV3], o)), root(square3(wr[IV1], wr[IV2], wr[IV3], o)));
    x = o.mul(x, o.mul(chi, sub(2.0, chi)));
  }
  const double pstar = fma(.5, add(wl[IPR], wr[IPR]), -x);
  double ql = 1.0, qr = 1.0;
  const bool bl = gt(pstar, wl[IPR]), br = gt(pstar, wr[IPR]);
  if (bl || br) {
    const double ipp = o.rcp(o.mul(wl[IPR], wr[IPR]));
    const double k = CONSTG ? gc.hllc_k : o.div(add(gl, 1), o.den(o.twice(gr)));
    if (bl) ql = o.sqrt(fma(k, fma(o.mul(pstar, wr[IPR]), ipp, -1.0), 1.0));
    if (br) qr = o.sqrt(fma(k, fma(o.mul(pstar, wl[IPR]), ipp, -1.0), 1.0));
  }
  const double sl = fma(-cl, ql, wl[IV1]), sr = fma(cr, qr, wr[IV1]);
  const double bp = is_pos(sr) ? sr : TINY_NUMBER;
  const double bm = is_neg(sl) ? sl : -TINY_NUMBER;
  const double vl = sub(wl[IV1], sl), vr = sub(wr[IV1], sr);
  const double tl = fma(o.mul(vl, wl[IDN]), wl[IV1], wl[IPR]);
  const double tr = fma(o.mul(vr, wr[IDN]), wr[IV1], wr[IPR]);
  const double ml = o.mul(wl[IDN], vl), mr = -o.mul(wr[IDN], vr);
  const double imm = o.rcp(add(ml, mr));
  const double sstar = o.mul(sub(tl, tr), imm);
  double cp = o.mul(fma(ml, tr, o.mul(mr, tl)), imm);
  cp = is_pos(cp) ? cp : 0.0;
  // one-sided: the flux is sstar/(sstar - b) times the physical flux of the upwind side of
  // the contact (left with b = bm when sstar >= 0, else right with b = bp) plus the pressure
  // terms; the other side's weight is exactly 0, so this is the two-sided sum of the reference
  // with its zero term dropped
  const bool L = !is_neg(sstar);
  const double rho = L ? wl[IDN] : wr[IDN], u = L ? wl[IV1] : wr[IV1];
  const double v = L ? wl[IV2] : wr[IV2], z = L ? wl[IV3] : wr[IV3];
  const double p = L ? wl[IPR] : wr[IPR];
  const double b = L ? bm : bp;
  const double e = fma(p, L ? il : ir, o.mul(o.half(rho), square3(u, v, z, o)));
  const double id = o.rcp(sub(sstar, b));
  const double coef = o.mul(sstar, id);
  const double ustar = o.mul(-b, id);
  const double vx = sub(u, b);
  flx[IDN] = o.mul(coef, o.mul(rho, vx));
  flx[IV1] = fma(coef, fma(o.mul(rho, u), vx, p), o.mul(ustar, cp));
  flx[IV2] = o.mul(coef, o.mul(o.mul(rho, v), vx));
  flx[IV3] = o.mul(coef, o.mul(o.mul(rho, z), vx));
  flx[IEN] = fma(o.mul(ustar, cp), sstar, o.mul(coef, fma(p, u, o.mul(e, vx))));
}
#endif

// x = 2^k with x and 1/x both normal: then y / x == y * (1/x) exactly for every y (both are
// the correctly rounded y * 2^-k), so a division by x is a multiplication.
__device__ __forceinline__ bool pow2_normal(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  const unsigned long long e = b >> 52;  // the sign bit must be 0
  return (b & 0xfffffffffffffULL) == 0 && e >= 1 && e <= 2045;
}
// x times 2^k, k within +-400: an exponent step for x in range or zero, else the product with c = 2^k
__device__ __forceinline__ double scale_x(double x, double c, int k) {
  if (far_of(x) < kFar)
    return __longlong_as_double(__double_as_longlong(x) + ((long long)k << 52));
  return is_zero(x) ? x : x * c;
}
// k where x = 2^k within +-400, else kNoStep
constexpr int kNoStep = 1 << 20;
__device__ __forceinline__ int pow2_step(double x) {
  const int k = (__double2hiint(x) >> 20) - 1023;
  return pow2_normal(x) && k >= -400 && k <= 400 ? k : kNoStep;
}
// y / vol, correctly rounded; ivol = 1 / vol, p2 = pow2_normal(vol) (uniform over a block)
__device__ __forceinline__ double div_vol(double y, double vol, double ivol, bool p2) {
  if (!p2) return div_x(y, vol);
  const int k = (__double2hiint(ivol) >> 20) - 1023;
  return k >= -400 && k <= 400 ? scale_x(y, ivol, k) : y * ivol;
}
// RN(RN(gam0 u0) + RN(gam1 u1)) of an RK stage, with the products by 0, 1 and powers of two (every
// stage of RK1, RK2 and VL2) taken off the FP64 pipe.
struct RkForm {
  double gam0, gam1;
  int form;    // 1: gam0 = 0 and gam1 = 1; 2: both powers of two, exponents k0 and k1; 0: any
  int k0, k1;
};
__device__ __forceinline__ RkForm rk_form(double gam0, double gam1) {
  RkForm r{gam0, gam1, 0, (__double2hiint(gam0) >> 20) - 1023, (__double2hiint(gam1) >> 20) - 1023};
  if (gam0 == 0.0 && gam1 == 1.0) r.form = 1;
  else if (pow2_normal(gam0) && pow2_normal(gam1) && abs(r.k0) <= 400 && abs(r.k1) <= 400) r.form = 2;
  return r;
}
__device__ __forceinline__ double rk_sum(const RkForm &r, double u0, double u1) {
  // 0 u0 + u1 is u1 unless u1 is a zero (whose sign the sum decides) or u0 not finite
  if (r.form == 1 && !is_zero(u1) && ((__double2hiint(u0) >> 20) & 0x7ff) != 0x7ff) return u1;
  if (r.form == 2) return scale_x(u0, r.gam0, r.k0) + scale_x(u1, r.gam1, r.k1);
  return r.gam0 * u0 + r.gam1 * u1;
}

#if APH_EXACT
// The reference's c-limited sound speed C sqrt(gamma / (1 + (igm1 + rho C^2 / p)))
// (hydro_hllc.hpp:57-60) with its roundings.  Where X = rho C^2 / p is at least 2^55 times
// both igm1 and 1 (always for non-relativistic gas: X ~ (c_light / c_sound)^2), each addition
// adds less than a quarter ulp of X and returns X, so both are skipped.
template <class OPS>
__device__ __forceinline__ double csound_exact(double rho, const Den &p, double gamma, double igm1, OPS &o) {
  const double X = o.div(o.mul(rho, C_LIGHT2), p);
  const long long ex = (long long)(mag(X) >> 52), ei = (long long)(mag(igm1) >> 52);
  const double d = (ex >= 1023 + 55 && ex >= ei + 55 && ex < 2047) ? X : 1 + (igm1 + X);
  return o.mul(C_LIGHT, o.sqrt(o.div(gamma, o.den(d))));
}

// HLLC in the exact mode with the reference's roundings (hydro_hllc.hpp:45-145, and the
// low-Mach pstar of hydro_lhllc.hpp:71-79), arranged for the GPU without changing a bit:
//  * the shock factor (gamma_l + 1) / (2 gamma_r), which the reference writes identically
//    for both sides, is formed once, and a face shocked on one side only takes one
//    division and square root whichever side it is;
//  * the contact branch picks its operands instead of its code, so both branches are the
//    same two divisions: ul = sstar / (sstar - bm), ustar = -bm / (sstar - bm) when
//    sstar >= 0, else ur = -sstar / (bp - sstar), ustar = bp / (bp - sstar);
//  * with IntOps (snug states) the flux is formed from the upwind
//    side only.  The reference's ul*fl + ur*fr has one weight exactly 0, and RN(a + (+-0)) == a
//    for every a but -0: there the other side's term 0 * f is +0 or -0 by the sign of f, which
//    for the mass and transverse fluxes is that of its factors (the normal momentum's and the
//    energy's -0 give up).  With IeeeOps both sides' terms are formed.
template <bool LOWMACH, class OPS>
__device__ __forceinline__ void solve_hllc_exact(const double *wli, const double *wri, double glc,
                                                 double gle, double grc, double gre, double *flxi,
                                                 OPS &o) {
  const double gammal = glc, gammar = grc;
  const double igm1l = see_side(wli[IDN], glc, gle, o), igm1r = see_side(wri[IDN], grc, gre, o);
  // the sound speed and the shock factor divide by the pressures
  const Den pl = o.den_positive(wli[IPR]), pr = o.den_positive(wri[IPR]);
  const double cl = csound_exact(wli[IDN], pl, gammal, igm1l, o);
  const double cr = csound_exact(wri[IDN], pr, gammar, igm1r, o);
  const double rhoa = o.half(wli[IDN] + wri[IDN]);
  const double ca = o.half(cl + cr);
  auto square3 = [&](const double *w) {
    return o.mul(w[IV1], w[IV1]) + o.mul(w[IV2], w[IV2]) + o.mul(w[IV3], w[IV3]);
  };
  double dp = o.mul(o.mul(o.half(wri[IV1] - wli[IV1]), rhoa), ca);
  if (LOWMACH) {
    auto root = [&](double x) { return is_zero(x) ? x : o.sqrt(is_zero(x) ? 1.0 : x); };
    const double chi = smax(root(square3(wli)), root(square3(wri)));
    dp = o.mul(dp, o.mul(chi, 2.0 - chi));
  }
  const double pstar = o.half(wli[IPR] + wri[IPR]) - dp;
  double cql = cl, cqr = cr;  // the sound speeds times the shock factors
  const bool bl = gt(pstar, wli[IPR]), br = gt(pstar, wri[IPR]);
  if (bl || br) {
    const double k = o.div(gammal + 1, o.den(o.twice(gammar)));
    const double q1 = o.mul(bl ? cl : cr, o.sqrt(1.0 + o.mul(k, o.div(pstar, bl ? pl : pr) - 1.0)));
    if (bl) cql = q1;
    else cqr = q1;
    if (bl && br) cqr = o.mul(cr, o.sqrt(1.0 + o.mul(k, o.div(pstar, pr) - 1.0)));
  }
  const double sl = wli[IV1] - cql;
  const double sr = wri[IV1] + cqr;
  const double bp = is_pos(sr) ? sr : TINY_NUMBER;
  const double bm = is_neg(sl) ? sl : -TINY_NUMBER;
  const double ml = o.mul(wli[IDN], wli[IV1] - sl);
  const double xr = o.mul(wri[IDN], wri[IV1] - sr), mr = -xr;
  const double tl = wli[IPR] + o.mul(ml, wli[IV1]);
  const double tr = wri[IPR] + o.mul(xr, wri[IV1]);
  const Den m = o.den(ml + mr);
  const double sstar = o.div0(tl - tr, m);
  double cp = o.div0(o.mul(ml, tr) + o.mul(mr, tl), m);
  cp = is_pos(cp) ? cp : 0.0;
  const bool L = !is_neg(sstar);  // sstar >= 0.0
  const Den d = o.den(L ? sstar - bm : bp - sstar);
  const double coef = o.div0(L ? sstar : -sstar, d);  // ul (or ur)
  const double ustar = o.div(L ? -bm : bp, d);
  // the upwind side (u) and the other one (v)
  double wu[NHYDRO], wv[NHYDRO];
#pragma unroll
  for (int n = 0; n < NHYDRO; ++n) {
    wu[n] = L ? wli[n] : wri[n];
    wv[n] = L ? wri[n] : wli[n];
  }
  const double bu = L ? bm : bp, bv = L ? bp : bm;
  auto side = [&](const double *w, double b, double igm1, double *f) {
    const double vx = w[IV1] - b;
    f[IDN] = o.mul(w[IDN], vx);
    f[IV1] = o.mul(o.mul(w[IDN], w[IV1]), vx) + w[IPR];
    f[IV2] = o.mul(o.mul(w[IDN], w[IV2]), vx);
    f[IV3] = o.mul(o.mul(w[IDN], w[IV3]), vx);
    const double e = o.mul(w[IPR], igm1) + o.mul(o.half(w[IDN]), square3(w));
    f[IEN] = o.mul(e, vx) + o.mul(w[IPR], w[IV1]);
  };
  double t[NHYDRO];
  side(wu, bu, L ? igm1l : igm1r, t);
#pragma unroll
  for (int n = 0; n < NHYDRO; ++n) t[n] = o.mul(coef, t[n]);
  if (OPS::kInt) {
    const bool back = lt(wv[IV1], bv);  // the sign of the other side's v - b
    auto add_zero = [](double x, bool negative) {
      return __double_as_longlong(x) == (long long)0x8000000000000000ULL && !negative ? 0.0 : x;
    };
    t[IDN] = add_zero(t[IDN], back);
    t[IV2] = add_zero(t[IV2], back != (__double2hiint(wv[IV2]) < 0));
    t[IV3] = add_zero(t[IV3], back != (__double2hiint(wv[IV3]) < 0));
    if (__double_as_longlong(t[IV1]) == (long long)0x8000000000000000ULL ||
        __double_as_longlong(t[IEN]) == (long long)0x8000000000000000ULL)
      o.give_up();
  } else {
    double f[NHYDRO];
    side(wv, bv, L ? igm1r : igm1l, f);
#pragma unroll
    for (int n = 0; n < NHYDRO; ++n) {
      const double z = o.mul(0.0, f[n]);
      t[n] = L ? t[n] + z : z + t[n];  // the reference's order: ul*fl + ur*fr
    }
  }
  o.see(sstar);
  o.see(cp);
  o.see(coef);
  const double pu = o.mul(ustar, cp);
  flxi[IDN] = t[IDN];
  flxi[IV1] = t[IV1] + pu;
  flxi[IV2] = t[IV2];
  flxi[IV3] = t[IV3];
  flxi[IEN] = t[IEN] + o.mul(pu, sstar);
}

#endif

// Fluxes of one face.  The caller checks o.ok() (IntOps), and takes the face again with IeeeOps
// where it is false.
template <int RS, bool CONSTG, class OPS>
__device__ __forceinline__ void riemann(const double *wl, const double *wr, double glc, double gle,
                                        double grc, double gre, const GasConsts &gc, double *flx,
                                        OPS &o) {
#if APH_EXACT
  if (RS == RS_HLLE) solve_hlle_exact(wl, wr, glc, gle, grc, gre, flx, o);
  else if (RS == RS_HLLC || RS == RS_LHLLC)
    solve_hllc_exact<RS == RS_LHLLC>(wl, wr, glc, gle, grc, gre, flx, o);
#else
  if (RS == RS_HLLE) solve_hlle<CONSTG>(wl, wr, glc, gle, grc, gre, gc, flx, o);
  else if (RS == RS_HLLC || RS == RS_LHLLC)
    solve_hllc<CONSTG, RS == RS_LHLLC>(wl, wr, glc, gle, grc, gre, gc, flx, o);
#endif
  else {
#pragma unroll
    for (int n = 0; n < NHYDRO; ++n) flx[n] = 0.0;
  }
}

// EstimateTimestep per-cell candidate (hydro.cpp:384-415): min over active directions
// of dx_d / (|v_d| + lambda).  dt_cell below is the form the stage kernel uses.
template <class OPS>
__device__ __forceinline__ double dt_candidate_ops(const double *w, double e_cons, const double *dx,
                                                   int ndim, double gm1, OPS &o) {
#pragma unroll
  for (int n = 0; n < NHYDRO; ++n) o.see(w[n]);
  o.see(e_cons);
#if APH_EXACT
  const double v2 = o.mul(w[IV1], w[IV1]) + o.mul(w[IV2], w[IV2]) + o.mul(w[IV3], w[IV3]);
  const double e_k = o.mul(o.half(w[IDN]), v2);
  const double e_i = e_cons - e_k;
#else
  const double e_i = fma(-o.half(w[IDN]), square3(w[IV1], w[IV2], w[IV3], o), e_cons);
#endif
  const double e_internal = o.div0(e_i, o.den(w[IDN]));
  const double small = 10.0 * 2.2250738585072014e-308;
  double bulkmod = o.mul(o.mul(__dmul_rn(gm1, __dadd_rn(gm1, 1.0)), w[IDN]), e_internal);  // eos_bulk_modulus
  bulkmod = lt(small, bulkmod) ? bulkmod : small;
  const Den p = o.den(w[IPR]);
  const double gamma_c = o.div(bulkmod, p);
  const double rat = o.div(o.mul(__dadd_rn(e_internal, C_LIGHT2), w[IDN]), p);
  const double root = o.sqrt(o.div(gamma_c, o.den(__dadd_rn(1, rat))));  // lambda is C times this
#if APH_EXACT
  const double lam = o.mul(C_LIGHT, root);
  auto rate = [&](int d) { return dabs(w[IV1 + d]) + lam; };
#else
  auto rate = [&](int d) { return fma(C_LIGHT, root, dabs(w[IV1 + d])); };
#endif
  double m = o.div(dx[0], o.den(rate(0)));
  if (ndim > 1) {
    const double c2 = o.div(dx[1], o.den(rate(1)));
    m = lt(c2, m) ? c2 : m;
  }
  if (ndim > 2) {
    const double c3 = o.div(dx[2], o.den(rate(2)));
    m = lt(c3, m) ? c3 : m;
  }
  return m;
}
__device__ __forceinline__ double dt_candidate(const double *w, double e_cons, const double *dx,
                                               int ndim, double gm1) {
  CheckedOps o;
  const double m = dt_candidate_ops(w, e_cons, dx, ndim, gm1, o);
  if (o.ok()) return m;
  IeeeOps ieee;
  return dt_candidate_ops(w, e_cons, dx, ndim, gm1, ieee);
}

// dt candidate of a cell just converted by cons_to_prim_cell (floored: its return value).
// Fast mode with the floors inactive: lambda is the c-limited sound speed of the constant
// gamma (the same quantity: rho e = p / gm1), and one reciprocal of the largest rate
// (|v_d| + lambda) / dx_d replaces a division per direction.
__device__ __forceinline__ double dt_cell(const double *w, double e_cons, const double *dx, int ndim,
                                          const GasConsts &gc, bool floored) {
#if APH_EXACT
  return dt_candidate(w, e_cons, dx, ndim, gc.gm1);
#else
  if (floored) return dt_candidate(w, e_cons, dx, ndim, gc.gm1);
  double num, root;
  IeeeOps o;
  sound_parts<true>(w[IDN], w[IPR], 0.0, 0.0, gc, num, root, o);
  double r = div_x(fma(num, root, dabs(w[IV1])), dx[0]);
  if (ndim > 1) {
    const double r2 = div_x(fma(num, root, dabs(w[IV2])), dx[1]);
    r = lt(r, r2) ? r2 : r;
  }
  if (ndim > 2) {
    const double r3 = div_x(fma(num, root, dabs(w[IV3])), dx[2]);
    r = lt(r, r3) ? r3 : r;
  }
  return rcp_x(r);
#endif
}

}  // namespace aph
