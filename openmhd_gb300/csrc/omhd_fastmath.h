// omhd_fastmath.h -- FP64 reciprocal and square roots, and binary32 <-> binary64
// conversions, on the integer pipes (device code).
#pragma once

namespace omhd {

// ---------------------------------------------------------------------------
// FP64 reciprocal and square roots without the FP64 pipe.  That pipe takes one
// warp instruction in 19 cycles (an SM issues 76 other ones in that time) and
// bounds the FP64 kernels, so the performance variants (FAST = true) compute
// 1/x, 1/sqrt(x) and sqrt(x) on the integer pipes: the argument's significand
// as a 64-bit fixed-point number, a binary32 seed of the special-function unit
// as a 32-bit one, and one third-order step of Newton's iteration (the series
// of (1-e)^-1 and (1-e)^(-1/2) up to e^2) in 64-bit products:
//   rcp_nr   : y0 <= 1/m from the seed, lowered by kSeedBias so that
//              e = 1 - m*y0 is in [0, 2^-20); 1/m = y0*(1 + e + e^2 + O(e^3)),
//              truncation below 2^-60;
//   rsqrt_nr : e = 1 - m*y0^2 in [0, 2^-19), 1/sqrt(m) =
//              y0*(1 + e/2 + 3e^2/8 + O(e^3)), truncation below 2^-58, with
//              m in [1,4) and the exponent even;
//   sqrt_nr  : m * 1/sqrt(m), the same series before it is rounded.
// The 64-bit result is rounded once, to nearest: within 0.51 ulp (measured on
// 6e7 arguments against extended precision; the FP64-pipe refinements these
// replaced were within 1 ulp).  Measured on GB300 with 12 warps per SM, SM
// cycles per warp operation: rcp 12.8, rsqrt 23, sqrt 27 (FP64-pipe forms: 52,
// ~92, 92; a DFMA: 19), and beside a stream of DFMAs they cost no time at all
// (16 DFMAs: 306 cycles; 16 DFMAs and 8 reciprocals: 305).
// tests/test_gpu_fastmath.py enforces 1 ulp over 2^-60..2^59 and over each
// function's whole domain: |x| in [2^-1022, 2^1022] for rcp_nr (x and 1/x
// normal; zero, subnormal and larger arguments, infinities and NaN give NaN),
// positive normal x for the square roots, which take the IEEE operation outside
// it (a branch that the solver's arguments never take).  The parity variant
// (FAST = false) keeps the reference's IEEE operations.
//
// rcp_nr_fp, rsqrt_nr_fp and sqrt_nr_fp are the refinements on the FP64 pipe (3,
// 5 and 5 operations from a binary64 seed, within 1 ulp).  The FP32-mixed kernels keep them for the
// CFL speed: another rounding of dt moves every cell of a mixed run by an ulp,
// and a state that differs in its last bit now and then rounds to the
// neighbouring binary32 number.
// ---------------------------------------------------------------------------
#ifdef __CUDACC__
constexpr unsigned kSeedBias = 1100u;  // in units of 2^-32; seed error <= 2^-23 + 2^-23 relative (1024 units)

// a seed r in [1/2, 1] (its binary32 bits) as a 0.32 fixed-point number, lowered by kSeedBias
__device__ __forceinline__ unsigned seed_fixed(float r) {
  return __float_as_uint(r) * 256u + (0x80000000u - kSeedBias);
}

// 1/m for the significand m of a number with high and low words hi, lo: m = mh:ml *
// 2^-63 in [1,2), returns 2^63/m to a few units
__device__ __forceinline__ unsigned long long rcp_fixed(unsigned hi, unsigned lo, unsigned& mh, unsigned& ml) {
  mh = __funnelshift_l(lo, hi, 11) | 0x80000000u;
  ml = lo << 11;
  float r;
  asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float((mh >> 8) + 0x3f000000u)));
  const unsigned y0 = seed_fixed(r);
  const unsigned long long e = 0x8000000000000000ull - ((unsigned long long)mh * y0 + __umulhi(ml, y0));  // e * 2^63
  const unsigned e32 = __funnelshift_r((unsigned)e, (unsigned)(e >> 32), 11);                             // e * 2^52
  const unsigned long long s = e + 0x8000000000000000ull + (__umulhi(e32, e32) >> 9);  // (1 + e + e^2) * 2^63
  return (unsigned long long)y0 * (unsigned)(s >> 32) + __umulhi(y0, (unsigned)s);
}

__device__ __forceinline__ double rcp_nr(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  unsigned mh, ml;
  const unsigned long long q = (rcp_fixed(hi, lo, mh, ml) + 512u) >> 10;  // 53 bits (2^53 where 1/m rounds to 1)
  const unsigned f = hi & 0xfff00000u;                                    // sign and exponent
  const unsigned rh = (f & 0x7ff00000u) - 0x00100000u < 0x7fd00000u ? 0x7fc00000u - f + (unsigned)(q >> 32) : 0x7ff80000u;
  return __hiloint2double((int)rh, (int)(unsigned)q);
}

// x positive, normal and finite (one integer compare on the bit pattern)
__device__ __forceinline__ bool pos_normal(double x) {
  const unsigned long long b = (unsigned long long)__double_as_longlong(x);
  return b - 0x0010000000000000ULL < 0x7fe0000000000000ULL;
}

// x = m 4^q with m = mh:ml * 2^-62 in [1,4); t = 2^63 / sqrt(m); the exponent
// field of 2^q, less that of 1/2, as ex (positive normal x)
__device__ __forceinline__ void rsqrt_fixed(double x, unsigned& mh, unsigned& ml, unsigned long long& t, unsigned& ex) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned sh = 11u - ((hi >> 20) & 1u);
  mh = __funnelshift_l(lo, (hi & 0xfffffu) | 0x100000u, sh);
  ml = lo << sh;
  const unsigned g = (__funnelshift_l(lo, hi, 3) & 0xffffffu) ^ 0x800000u;  // significand and exponent parity
  float r;
  asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(__uint_as_float(g + 0x3f800000u)));
  const unsigned y0 = seed_fixed(r);
  const unsigned long long y2 = (unsigned long long)y0 * y0;
  const unsigned y2h = (unsigned)(y2 >> 32);
  const unsigned long long e =
      0x4000000000000000ull - ((unsigned long long)mh * y2h + __umulhi(mh, (unsigned)y2) + __umulhi(ml, y2h));  // e * 2^62
  const unsigned e32 = __funnelshift_r((unsigned)e, (unsigned)(e >> 32), 11);                                   // e * 2^51
  const unsigned long long s = e + 0x8000000000000000ull + __umulhi(__umulhi(e32, e32), 3u << 22);  // (1 + e/2 + 3e^2/8) * 2^63
  t = (unsigned long long)y0 * (unsigned)(s >> 32) + __umulhi(y0, (unsigned)s);
  ex = ((hi + 0x100000u) >> 1) & 0xfff00000u;
}

__device__ __forceinline__ double rsqrt_nr(double x) {
  if (!pos_normal(x)) return 1.0 / sqrt(x);
  unsigned mh, ml, ex;
  unsigned long long t;
  rsqrt_fixed(x, mh, ml, t, ex);
  const unsigned long long q = (t + 512u) >> 10;
  return __hiloint2double((int)((1533u << 20) - ex + (unsigned)(q >> 32)), (int)(unsigned)q);
}

__device__ __forceinline__ double sqrt_nr(double x) {
  if (!pos_normal(x)) return sqrt(x);
  unsigned mh, ml, ex;
  unsigned long long t;
  rsqrt_fixed(x, mh, ml, t, ex);
  const unsigned th = (unsigned)(t >> 32);
  const unsigned long long p = (unsigned long long)mh * th + __umulhi(mh, (unsigned)t) + __umulhi(ml, th);  // sqrt(m) * 2^61
  const unsigned long long q = (p + 256u) >> 9;
  return __hiloint2double((int)((510u << 20) + ex + (unsigned)(q >> 32)), (int)(unsigned)q);
}

// a / b and sqrt(x), correctly rounded, on the integer pipes: the IEEE results bit
// for bit, for the kernels that reproduce the reference's operations.  A quotient or
// root cut to 53 bits from the approximations above, made to lie below the true
// value by less than a unit, then corrected and rounded by its exact remainder, of
// which 64 bits are enough.  Zero dividends are taken; everything else outside the
// normal range, or whose quotient may leave it, goes through the IEEE operation (a
// branch: its expansion is too long to be predicated).  ~65 and ~55 instructions,
// at 39 and 35 SM cycles a warp operation, beside FP64 work for less; the IEEE
// expansions take 4.4 and 7.2 operations of the FP64 pipe, 135 and 140 cycles.
struct Divisor {  // b prepared once for several quotients
  double b;
  unsigned long long t;  // 2^63 / m
  unsigned hi, mh, ml;
};
__device__ __forceinline__ Divisor divisor(double b) {
  Divisor d;
  d.b = b;
  d.hi = (unsigned)__double2hiint(b);
  d.t = rcp_fixed(d.hi, (unsigned)__double2loint(b), d.mh, d.ml);
  return d;
}
__device__ __forceinline__ double div_rn(double a, const Divisor& d) {
  const unsigned ah = (unsigned)__double2hiint(a), al = (unsigned)__double2loint(a);
  const unsigned ea = (ah >> 20) & 0x7ffu, eb = (d.hi >> 20) & 0x7ffu;
  const bool zero = (ah * 2u | al) == 0u;
  // both normal, and the quotient's exponent well inside the normal range
  if (!(eb - 1u < 2046u && (zero || (ea - 1u < 2046u && ea - eb + 1020u < 2040u)))) return a / d.b;
  const unsigned long long ma = ((unsigned long long)(__funnelshift_l(al, ah, 11) | 0x80000000u) << 32) | (al << 11);
  const unsigned long long mb = ((unsigned long long)d.mh << 32) | d.ml;
  const unsigned mah = (unsigned)(ma >> 32), mal = (unsigned)ma, th = (unsigned)(d.t >> 32), tl = (unsigned)d.t;
  // (ma/mb) 2^62, less 4: the reciprocal may be a unit high
  const unsigned long long p = (unsigned long long)mah * th + __umulhi(mah, tl) + __umulhi(mal, th) - 4u;
  const unsigned ge = ma >= mb ? 1u : 0u;  // ma/mb in [1,2), else in (1/2,1)
  unsigned long long q = p >> (9u + ge);
  const unsigned long long b53 = mb >> 11;
  // remainder ma53 * 2^(53 - ge) - q * b53, exact modulo 2^64
  unsigned long long r = ((unsigned long long)(al << (21u - ge)) << 32) - q * b53;
  if (r >= b53) {
    r -= b53;
    ++q;
  }
  if (2 * r > b53) ++q;
  const unsigned rh = ((ea - eb + 1021u + ge) << 20) + (unsigned)(q >> 32);
  const unsigned sg = (ah ^ d.hi) & 0x80000000u;
  return __hiloint2double((int)((zero ? 0u : rh) | sg), (int)(zero ? 0u : (unsigned)q));
}
__device__ __forceinline__ double div_rn(double a, double b) { return div_rn(a, divisor(b)); }

__device__ __forceinline__ double sqrt_rn(double x) {
  if (!pos_normal(x)) return sqrt(x);
  unsigned mh, ml, ex;
  unsigned long long t;
  rsqrt_fixed(x, mh, ml, t, ex);
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x), th = (unsigned)(t >> 32);
  // sqrt(m) 2^61, less 8: the reciprocal root may be a few units high
  const unsigned long long p = (unsigned long long)mh * th + __umulhi(mh, (unsigned)t) + __umulhi(ml, th) - 8u;
  unsigned long long q = p >> 9;
  // remainder m53 * 2^(52 or 53) - q^2, exact modulo 2^64
  unsigned long long r = ((unsigned long long)(lo << (21u - ((hi >> 20) & 1u))) << 32) - q * q;
  if (r > 2 * q) {
    r -= 2 * q + 1;
    ++q;
  }
  if (r > q) ++q;
  return __hiloint2double((int)((510u << 20) + ex + (unsigned)(q >> 32)), (int)(unsigned)q);
}

// a * b, rounded to nearest, on the integer pipes: the exact 106-bit product of
// the significands in four 32-bit multiplies, cut to 53 bits and rounded on the
// next bit (the IEEE product but for exact ties, which round up instead of to
// even, and for products below 2^-1022, which become signed zeros; subnormal
// operands are taken as zeros).  An operand of magnitude 2^511 or more, infinity
// or NaN sets bad, and the caller redoes its work with FP64-pipe operations (a
// predicated DMUL in its place would hold the pipe even where no lane takes it:
// measured, 19 SM cycles a warp operation with all lanes predicated off).  ~35
// instructions; 13 SM cycles a warp operation with 12 warps per SM (DMUL: 19),
// and next to nothing beside FP64 work: 16 DFMAs 306 cycles, 16 DFMAs and 16 of
// these 270-310, 16 DFMAs and 16 DMULs 617.
__device__ __forceinline__ double mul_int(double a, double b, bool& bad) {
  const unsigned ah = (unsigned)__double2hiint(a), al = (unsigned)__double2loint(a);
  const unsigned bh = (unsigned)__double2hiint(b), bl = (unsigned)__double2loint(b);
  // sign and exponent (less one: the significand's leading bit adds it)
  const unsigned f = (ah & 0xfff00000u) + (bh & 0xfff00000u) - 0x40000000u;
  const bool zero = min(ah * 2u, bh * 2u) < 0x00200000u || (int)(f ^ ah ^ bh) < 0;  // a zero operand, or underflow
  bad |= max(ah * 2u, bh * 2u) >= 0xbfc00000u;
  const unsigned mah = (ah & 0xfffffu) | 0x100000u, mbh = (bh & 0xfffffu) | 0x100000u;
  const unsigned long long c =
      (unsigned long long)mah * bl + ((unsigned long long)al * mbh + __umulhi(al, bl));  // product >> 32, without mah*mbh
  const unsigned long long p = (unsigned long long)mah * mbh + (c >> 32);                // product >> 64, in [2^40, 2^42)
  const unsigned ph = (unsigned)(p >> 32), pl = (unsigned)p, cl = (unsigned)c;
  const unsigned two = ph >> 9, sh = 12u - two;  // product of the significands >= 2
  const unsigned qh = __funnelshift_l(pl, ph, sh), ql = __funnelshift_l(cl, pl, sh), half = (cl << sh) >> 31;
  const unsigned long long r = (((unsigned long long)(f + (two << 20) + qh) << 32) | ql) + half;
  const unsigned rh = zero ? (ah ^ bh) & 0x80000000u : (unsigned)(r >> 32), rl = zero ? 0u : (unsigned)r;
  return __hiloint2double((int)rh, (int)rl);
}

// x / 2, rounded to nearest: the IEEE result for all arguments, by the exponent or,
// below 2^-1021, where the bits of |x| are its value in units of 2^-1074 (exponent field
// included), as an integer, to even.  Written out with one select a word: as half_exact
// with a second select the mixed 3D kernel took 0.5 to 1.3 % longer (Harris 256x128x256,
// 14.02-14.13 ms for 2 steps, against 13.94; without the integer halves 13.93).
__device__ __forceinline__ double half_rn(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), mh = hi & 0x7fffffffu, lo = (unsigned)__double2loint(x);
  const unsigned long long m =
      (((unsigned long long)(mh >> 1) << 32) | __funnelshift_r(lo, mh, 1)) + (lo & (lo >> 1) & 1u);
  const bool tiny = mh < 0x00200000u;
  const unsigned h = mh >= 0x7ff00000u ? hi : hi - 0x00100000u;  // infinity and NaN stay
  return __hiloint2double((int)(tiny ? (unsigned)(m >> 32) | (hi & 0x80000000u) : h), (int)(tiny ? (unsigned)m : lo));
}

// its exponent part alone (probed; exact; results below 2^-1022 become signed zeros)
__device__ __forceinline__ double half_exact(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x), e = hi & 0x7ff00000u;
  const bool tiny = e < 0x00200000u;
  const unsigned h = e == 0x7ff00000u ? hi : hi - 0x00100000u;  // infinity and NaN stay
  return __hiloint2double((int)(tiny ? hi & 0x80000000u : h), (int)(tiny ? 0u : lo));
}

__device__ __forceinline__ double rcp_nr_fp(double x) {
  double y;
  asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
  const double e = fma(-x, y, 1.0);
  return fma(fma(e, e, e), y, y);
}

__device__ __forceinline__ double rsqrt_nr_fp(double x) {
  if (!pos_normal(x)) return 1.0 / sqrt(x);
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double e = fma(-(x * r), r, 1.0);
  return fma(r * e, fma(0.375, e, 0.5), r);
}

__device__ __forceinline__ double sqrt_nr_fp(double x) {
  if (!pos_normal(x)) return sqrt(x);
  double r;
  asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
  const double s = x * r;
  const double e = fma(-s, r, 1.0);
  return fma(s * e, fma(0.375, e, 0.5), s);
}

// ---------------------------------------------------------------------------
// binary32 <-> binary64 conversions on the integer pipe.  GB300 executes the
// F2F conversions on its FP64 pipe, one slot each like an FMA; the FP32-mixed
// kernels convert every loaded primitive to binary32 and every face flux back,
// which took a quarter of their FP64-pipe time.  These forms move the bits with
// 8-15 integer instructions instead (IEEE 754 formats: binary32 = 1/8/23 bits,
// bias 127; binary64 = 1/11/52 bits, bias 1023):
//   widen_f32  : exact for normal floats, +-0, +-inf and NaN (payload kept);
//                a subnormal float (|f| < 2^-126) becomes a signed zero.
//   narrow_f64 : round to nearest, ties to even, as cvt.rn.f32.f64, for every
//                argument of magnitude 2^-126 or more, with overflow to
//                +-inf; a smaller argument gives a signed zero (no subnormal
//                results); NaN stays NaN (quiet).
// tests/test_gpu_convert.py checks both against IEEE conversions on the host,
// bit for bit, over random bit patterns and every boundary of the formats;
// tests/test_convert_algorithm.py restates the bit manipulation in numpy and
// checks it the same way without a GPU.
// ---------------------------------------------------------------------------
__device__ __forceinline__ double widen_f32(float f) {
  const unsigned u = __float_as_uint(f);
  const unsigned mag = u & 0x7fffffffu;
  // rebias the exponent: + (1023 - 127) in the high word's exponent field, and
  // twice that for inf/NaN so that exponent 255 lands on 2047
  unsigned hi = (mag >> 3) + (mag >= 0x7f800000u ? 0x70000000u : 0x38000000u);
  unsigned lo = u << 29;  // the three low mantissa bits
  if (mag < 0x00800000u) hi = lo = 0u;
  return __hiloint2double((int)(hi | (u & 0x80000000u)), (int)lo);
}

// widen_f32(a) - widen_f32(b), rounded to binary64, without the FP64 pipe (the same
// bits for all arguments; a NaN stays one).  s = a - b in
// binary32 and its exact error e (Knuth's two-sum) add up to a - b; s's binary64
// bits and e in units of s's last binary64 place are then added as integers, which
// cannot carry out of s's binade but where s is a power of two and e points to the
// binade below, whose places are half as wide.  e in those units has to be rounded
// to an integer only if it reaches below 53 bits, and to even as the sum's own parity
// is e's (s ends in 29 zeros).  Two operands below 2^-30 are scaled by 2^96 so that s
// and e stay normal, others by 2^-2 so that s stays finite.  ~33 instructions; the FP64 subtraction holds the SM's FP64 pipe
// for 19 cycles, in which its four schedulers issue 76.
__device__ __forceinline__ float mul_ftz(float x, float y) {  // subnormals are zeros
  float r;
  asm("mul.rn.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"(x), "f"(y));
  return r;
}
__device__ __forceinline__ double sub_f32(float a, float b) {
  const bool small = fmaxf(fabsf(a), fabsf(b)) < 0x1p-30f;
  const float scale = small ? 0x1p96f : 0x1p-2f;
  a = mul_ftz(a, scale);
  b = mul_ftz(b, scale);
  const float s = __fsub_rn(a, b), t = __fsub_rn(s, a);
  const float e = __fsub_rn(__fsub_rn(a, __fsub_rn(s, t)), __fadd_rn(b, t));
  const unsigned u = __float_as_uint(s), mag = u & 0x7fffffffu;
  // +-2^(1-Es), the sign that of s; 0 for infinity and NaN
  const float x = __fmul_rn(e, __uint_as_float((0x7f800000u - (u & 0x7f800000u)) | (u & 0x80000000u)));
  const bool below = (u << 9) == 0u && x < 0.0f;
  const int j = __float2int_rn(__fmul_rn(x, below ? 0x1p52f : 0x1p51f));  // 0 for NaN
  const unsigned hi = (mag >> 3) + (mag >= 0x7f800000u ? 0x70000000u : small ? 0x32000000u : 0x38200000u);
  unsigned long long r = (((unsigned long long)hi << 32) | (u << 29)) + (unsigned long long)(long long)j;
  r = mag == 0u ? 0ull : r;
  return __hiloint2double((int)((unsigned)(r >> 32) | (u & 0x80000000u)), (int)(unsigned)r);
}

__device__ __forceinline__ float narrow_f64(double x) {
  const unsigned hi = (unsigned)__double2hiint(x), lo = (unsigned)__double2loint(x);
  const unsigned ahi = hi & 0x7fffffffu;
  // round the 64-bit magnitude at bit 29: add half an ulp of the result minus
  // one, plus the kept lowest bit (ties go to even), then drop 29 bits
  const unsigned long long a = ((unsigned long long)ahi << 32) | lo;
  const unsigned long long r = a + (0x0fffffffull + ((lo >> 29) & 1u));
  unsigned f = (unsigned)(r >> 29) - (896u << 23);  // rebias 1023 -> 127
  f = ahi >= 0x47f00000u ? 0x7f800000u : f;         // |x| >= 2^128: inf (also inf/NaN inputs)
  f = ahi < 0x38100000u ? 0u : f;                   // |x| < 2^-126: zero
  f = a > 0x7ff0000000000000ull ? 0x7fc00000u : f;  // NaN
  return __uint_as_float(f | (hi & 0x80000000u));
}
#endif

}  // namespace omhd
