// fp64ops.cuh -- exact replacements for FP64 operations, off the FP64 pipe.
//
// GB300 issues FP64 at 2 operations per SM per cycle (1/64 of FP32) and a double
// division or square root costs about 8.5 of those slots, while the integer and
// FP32 pipes sit idle in these kernels.  Each helper here returns exactly the IEEE
// result of the operation it replaces (round to nearest even), using integer
// instructions, or a shorter FP64 sequence, wherever that is exact, and the plain
// operation otherwise.  The float overloads are the plain operations.
#pragma once
#include <cstring>
#include <cuda_runtime.h>

namespace hgpu {

__device__ __forceinline__ long long bitsOf(double x) { return __double_as_longlong(x); }
__device__ __forceinline__ double fromBits(long long b) { return __longlong_as_double(b); }

// Class tests on the two 32-bit words: a test of the whole 64-bit pattern is
// recognised by the compiler as a floating-point class test or compare and issued to
// the FP64 unit; on the words it stays on the integer pipes.
__device__ __forceinline__ bool isNaNBits(double x) {
    const int hi = __double2hiint(x) & 0x7FFFFFFF, lo = __double2loint(x);
    return hi > 0x7FF00000 || (hi == 0x7FF00000 && lo != 0);
}

__device__ __forceinline__ bool isNaNBits(float x) { return x != x; }

// x >= 0.  (-0 >= 0 is true, NaN >= 0 is false)
__device__ __forceinline__ bool geZero(double x) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    return hi >= 0 ? (hi < 0x7FF00000 || (hi == 0x7FF00000 && lo == 0)) : (hi == (int)0x80000000 && lo == 0);
}
// x is +0 or -0
__device__ __forceinline__ bool isZeroBits(double x) {
    return ((__double2hiint(x) & 0x7FFFFFFF) | __double2loint(x)) == 0;
}
__device__ __forceinline__ bool geZero(float x) { return x >= 0.f; }
__device__ __forceinline__ bool isZeroBits(float x) { return (__float_as_int(x) & 0x7FFFFFFF) == 0; }

// .5 * x exactly: decrement the exponent of a normal x whose half is normal; a zero, an
// infinity or a NaN is its own half.  The rare other operands (subnormal, or with a
// subnormal half) take the FP64 unit out of line, so the compiler cannot issue that
// product for every operand and select.
static __device__ __noinline__ double halfNative(double x) { return x * .5; }
__device__ __forceinline__ double halfOf(double x) {
    const int hi = __double2hiint(x), lo = __double2loint(x), e = hi & 0x7FF00000;
    if ((unsigned)e - 0x00200000u < 0x7FD00000u) return __hiloint2double(hi - 0x00100000, lo);
    if (isZeroBits(x) || e == 0x7FF00000) return x;
    return halfNative(x);
}
__device__ __forceinline__ float halfOf(float x) { return x * .5f; }

// total-order key of a non-NaN double (-0 < +0 here; callers treat zeros as equal)
__device__ __forceinline__ long long orderKey(long long b) { return b ^ ((b >> 63) & 0x7FFFFFFFFFFFFFFFLL); }

// C library fmin/fmax semantics (the oracle's): a NaN operand yields the other
// operand; equal operands (including -0 and +0) yield the second one.  The choice is
// made on the bit patterns and the result selected as an integer: a select between
// two doubles issues FP64-unit instructions on this part.
__device__ __forceinline__ bool fminTakesFirst(double x, double y) {
    const long long bx = bitsOf(x), by = bitsOf(y);
    const bool bothZero = ((bx | by) & 0x7FFFFFFFFFFFFFFFLL) == 0;
    return isNaNBits(y) || (!isNaNBits(x) && !bothZero && orderKey(bx) < orderKey(by));
}
__device__ __forceinline__ bool fmaxTakesFirst(double x, double y) {
    const long long bx = bitsOf(x), by = bitsOf(y);
    const bool bothZero = ((bx | by) & 0x7FFFFFFFFFFFFFFFLL) == 0;
    return isNaNBits(y) || (!isNaNBits(x) && !bothZero && orderKey(bx) > orderKey(by));
}
// c ? a : b, selected as an integer
__device__ __forceinline__ double selectD(bool c, double a, double b) {
    return fromBits(c ? bitsOf(a) : bitsOf(b));
}
__device__ __forceinline__ float selectD(bool c, float a, float b) { return c ? a : b; }
__device__ __forceinline__ double fminLibm(double x, double y) { return selectD(fminTakesFirst(x, y), x, y); }
__device__ __forceinline__ double fmaxLibm(double x, double y) { return selectD(fmaxTakesFirst(x, y), x, y); }
// c ? 1. : -1., selected as an integer
__device__ __forceinline__ double plusMinusOne(bool c) {
    return fromBits(c ? 0x3FF0000000000000LL : (long long)0xBFF0000000000000ULL);
}
// fmax(0, x) and fmin(0, x), the sign of a zero result aside (NaN gives 0), on the words:
// through fmaxLibm / fminLibm with a constant 0 the compiler issues FP64 compares
__device__ __forceinline__ double positivePart(double x) {
    return selectD(__double2hiint(x) < 0 || isNaNBits(x), 0., x);
}
__device__ __forceinline__ double negativePart(double x) {
    return selectD(__double2hiint(x) >= 0 || isNaNBits(x), 0., x);
}
__device__ __forceinline__ float positivePart(float x) { return x > 0.f ? x : 0.f; }
__device__ __forceinline__ float negativePart(float x) { return x < 0.f ? x : 0.f; }
// x <= 0 (-0 and +0 included, NaN false) and a <= b, on the words / bit patterns
__device__ __forceinline__ bool leZero(double x) { return isZeroBits(x) || (__double2hiint(x) < 0 && !isNaNBits(x)); }
__device__ __forceinline__ bool leZero(float x) { return x <= 0.f; }
__device__ __forceinline__ bool leD(double a, double b) {
    if (isNaNBits(a) || isNaNBits(b)) return false;
    return (isZeroBits(a) && isZeroBits(b)) || orderKey(bitsOf(a)) <= orderKey(bitsOf(b));
}
__device__ __forceinline__ bool leD(float a, float b) { return a <= b; }
// x is finite / x is finite and nonzero, on the words
__device__ __forceinline__ bool finiteD(double x) { return (__double2hiint(x) & 0x7FF00000) != 0x7FF00000; }
__device__ __forceinline__ bool finiteNonzeroD(double x) { return finiteD(x) && !isZeroBits(x); }
__device__ __forceinline__ float fminLibm(float x, float y) { return (x < y || y != y) ? x : y; }
__device__ __forceinline__ float fmaxLibm(float x, float y) { return (x > y || y != y) ? x : y; }



// x * y computed on the integer pipes, bit-identical to the FP64 unit's product.
// The FP64 unit issues 2 operations per SM per clock on this part while the integer
// and FP32 pipes stand idle in the FP64-bound kernels; products routed here run on
// those pipes, concurrently with the native adds.  Fast path: both operands normal
// and the biased exponent sum in [1, 2045].  The significands' exact product is formed
// from 32-bit limbs (four 32x32+64-bit multiply-adds), the second one scaled by 2^11 so
// that the rounded significand falls on the upper two words; it is rounded to nearest,
// ties to even, by a carry out of the next word (the lowest word as a sticky bit); the
// carry of a round-up into bit 53 increments the exponent field (to +-Inf only from the
// largest binade, as IEEE 754 requires).  Zeros, subnormals, Inf, NaN and products that
// could leave the normal range take the FP64 unit.  hgpu_fp64_selftest compares it with
// the FP64 unit (all exponent ranges, short significands, extremes).  Throughput: 613
// G/s with one operand shared by four products, 489 G/s for the form on 64-bit words
// before it and for the FP64 unit.
// the rare native product, kept out of line: inlined, it would be if-converted and
// issued to the FP64 unit for every operand pair
static __device__ __noinline__ double mulNative(double x, double y) { return x * y; }

__device__ __forceinline__ double productBits(unsigned xh, unsigned xl, unsigned yh, unsigned yl) {
    const unsigned a1 = (xh & 0xFFFFFu) | 0x100000u;                                     // 53 bits: a1, xl
    const unsigned b1 = __funnelshift_l(yl, yh, 11) | 0x80000000u, b0 = yl << 11;        // 64 bits
    const unsigned long long t0 = (unsigned long long)xl * b0, t1 = (unsigned long long)xl * b1 + (t0 >> 32);
    const unsigned long long t2 = (unsigned long long)a1 * b0 + (unsigned)t1;
    const unsigned long long h = (unsigned long long)a1 * b1 + (t1 >> 32) + (t2 >> 32);  // [2^51, 2^53)
    unsigned h1 = (unsigned)(h >> 32), h0 = (unsigned)h, w = (unsigned)t2 | ((unsigned)t0 ? 1u : 0u);
    unsigned bias = 1023u << 20;                     // the leading bit of h1 adds one to the field
    if (h1 < 0x100000u) {
        h1 = __funnelshift_l(h0, h1, 1);
        h0 = __funnelshift_l(w, h0, 1);
        w <<= 1;
        bias = 1024u << 20;
    }
    const unsigned up = (unsigned)(((unsigned long long)w + 0x7FFFFFFFu + (h0 & 1u)) >> 32);
    const unsigned long long r = (((unsigned long long)((xh & 0x7FF00000u) + (yh & 0x7FF00000u) - bias + h1) << 32) | h0) + up;
    return __hiloint2double((int)((unsigned)(r >> 32) | ((xh ^ yh) & 0x80000000u)), (int)(unsigned)r);
}
__device__ __forceinline__ double mulI(double x, double y) {
    const unsigned xh = (unsigned)__double2hiint(x), yh = (unsigned)__double2hiint(y);
    const unsigned ex = xh & 0x7FF00000u, ey = yh & 0x7FF00000u;
    if (ex - 0x00100000u >= 0x7FE00000u || ey - 0x00100000u >= 0x7FE00000u || ex + ey - (1024u << 20) >= (2045u << 20))
        return mulNative(x, y);
    return productBits(xh, (unsigned)__double2loint(x), yh, (unsigned)__double2loint(y));
}
__device__ __forceinline__ float mulI(float x, float y) { return x * y; }

static __device__ __noinline__ double divNative(double x, double y) { return x / y; }

// 2^64 / d for the significand d in [1, 2) of y (its words given; y normal), from below
// and by less than 11.  The FP32 reciprocal of d's top 24 bits (rounded up), lowered past
// its error, is a 32-bit v0 <= 2^32 / d within 2^-21; two fixed-point Newton steps
// v += v (1 - d v), the residual formed from the whole of d and every truncation
// downwards, keep it from below: 2^-31, then second order 2^-62 plus truncations.
__device__ __forceinline__ unsigned long long recipBits(unsigned yh, unsigned yl) {
    const unsigned dh = __funnelshift_l(yl, yh, 11) | 0x80000000u, dl = yl << 11;
    float rf;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(rf) : "f"(__uint_as_float((0x3F800000u | (dh >> 8 & 0x7FFFFFu)) + 1u)));
    const unsigned v0 = (__float_as_uint(rf) << 8) + (0x80000000u - 0x200u);
    const unsigned long long e0 = 0x7FFFFFFFFFFFFFFFull - ((unsigned long long)dh * v0 + __umulhi(dl, v0));
    const unsigned v1 = v0 + (__umulhi(v0, (unsigned)(e0 >> 11)) >> 20);
    const unsigned long long e1 = 0x7FFFFFFFFFFFFFFFull - ((unsigned long long)dh * v1 + __umulhi(dl, v1));   // < 2^32.01
    return ((unsigned long long)v1 << 32) + (((unsigned long long)v1 * (unsigned)(e1 >> 1)) >> 30);
}

// x / y given v = recipBits(y) (or any value from below by less than 11), x and y normal
// and the quotient safely normal.  q = significand(x) v / 2^64 from 32-bit limbs, on the
// same two words as mulI's product, is the truncated quotient or one less (then its
// remainder is barely above y's significand); the remainder, exact modulo 2^64, against
// half of y's significand rounds it to nearest (a quotient is never a tie).
__device__ __forceinline__ double quotientBits(unsigned xh, unsigned xl, unsigned yh, unsigned yl,
                                               unsigned long long v) {
    const unsigned b1 = (unsigned)(v >> 32), b0 = (unsigned)v, a1 = (xh & 0xFFFFFu) | 0x100000u;
    const unsigned long long t1 = (unsigned long long)xl * b1 + __umulhi(xl, b0);
    const unsigned long long t2 = (unsigned long long)a1 * b0 + (unsigned)t1;
    const unsigned long long h = (unsigned long long)a1 * b1 + (t1 >> 32) + (t2 >> 32);
    unsigned h1 = (unsigned)(h >> 32), h0 = (unsigned)h, n = xl << 20, bias = 1022u << 20;
    if (h1 < 0x100000u) {
        h1 = __funnelshift_l(h0, h1, 1);
        h0 = __funnelshift_l((unsigned)t2, h0, 1);
        n <<= 1;
        bias = 1021u << 20;
    }
    const unsigned m1 = (yh & 0xFFFFFu) | 0x100000u;
    const unsigned long long lo = (unsigned long long)h0 * yl;
    const unsigned long long rem = ((unsigned long long)(n - ((unsigned)(lo >> 32) + h0 * m1 + h1 * yl)) << 32) -
                                   (unsigned)lo;
    const unsigned long long half = (((unsigned long long)m1 << 32) | yl) >> 1;
    const unsigned long long r =
        (((unsigned long long)((xh & 0x7FF00000u) - (yh & 0x7FF00000u) + bias + h1) << 32) | h0) + (rem > half ? 1u : 0u);
    return __hiloint2double((int)((unsigned)(r >> 32) | ((xh ^ yh) & 0x80000000u)), (int)(unsigned)r);
}

// x / y on the integer pipes, bit-identical to the IEEE quotient (round to nearest
// even).  Fast path: both operands normal and the quotient's biased exponent safely
// inside [1, 2046].  A zero operand beside a finite one is resolved with integer
// operations; everything else takes the FP64 unit.  hgpu_fp64_selftest compares it with
// the FP64 unit's quotient.  Four quotients by one divisor 567 G/s, against 126 for the
// form before it (two Newton steps on 64-bit words, the remainder corrected twice each
// way) and 70 for the FP64 unit's division.
__device__ __forceinline__ double divI(double x, double y) {
    const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
    const unsigned yh = (unsigned)__double2hiint(y), yl = (unsigned)__double2loint(y);
    const unsigned ex = xh & 0x7FF00000u, ey = yh & 0x7FF00000u;
    if (ex - 0x00100000u >= 0x7FE00000u || ey - 0x00100000u >= 0x7FE00000u ||
        ex - ey + (1021u << 20) >= (2044u << 20)) {
        // a zero operand beside a finite one: 0/0 = NaN, x/0 = +-Inf, 0/y = +-0 (the
        // limiter ratios of flat states are mostly these); the rest on the FP64 unit
        const bool xz = ((xh << 1) | xl) == 0, yz = ((yh << 1) | yl) == 0;
        if ((xz || yz) && ex != 0x7FF00000u && ey != 0x7FF00000u) {
            const unsigned sgn = (xh ^ yh) & 0x80000000u;
            const bool nan = xz && yz;
            return __hiloint2double((int)(nan ? 0x7FFFFFFFu : xz ? sgn : (sgn | 0x7FF00000u)), nan ? -1 : 0);
        }
        return divNative(x, y);
    }
    return quotientBits(xh, xl, yh, yl, recipBits(yh, yl));
}
__device__ __forceinline__ float divI(float x, float y) { return x / y; }

// sqrt(x) on the integer pipes, bit-identical to the FP64 unit's: x normal and positive (its
// words given).  With M in [1, 4) the significand, doubled where the exponent is odd, and
// a = M / 4: y ~ 1 / sqrt(a) is seeded by the FP32 reciprocal square root of a's top bits
// (rounded up, the result lowered by 4 units), refined by two fixed-point Newton steps
// y += y (1 - a y^2) / 2 that keep it from below (2^-28, then 2^-57); q = floor(2^53 a y) is
// the truncated root or one less, and the remainder, exact modulo 2^64, against q rounds it
// to nearest (a root is never a tie).  Some 60 instructions against about ten FP64
// operations of 64 issue slots each: KH 2048^2 eigenbasis 867 -> 525 us a launch (with roe.cuh's
// left rows off the FP64 unit too), HLLC wave speeds at 1021x1030 154 -> 105 us, at 160x144x136
// 889 -> 713 us.
__device__ __forceinline__ double rootBits(unsigned xh, unsigned xl) {
    const unsigned odd = (~xh >> 20) & 1u, mh = (xh & 0xFFFFFu) | 0x100000u;
    const unsigned ah = __funnelshift_l(xl, mh, 10 + odd), al = xl << (10 + odd);          // a 2^64
    float rf;
    asm("rsqrt.approx.ftz.f32 %0, %1;"
        : "=f"(rf)
        : "f"(__uint_as_float(((0x3E800000u + (odd << 23)) | (__funnelshift_l(xl, mh, 3) & 0x7FFFFFu)) + 1u)));
    const unsigned y0 = (__float_as_uint(rf) - 4u) << 8;                                   // y 2^31
    const unsigned e0 = (unsigned)((0x4000000000000000ull - (unsigned long long)ah * __umulhi(y0, y0)) >> 12);
    const unsigned y1 = y0 + (__umulhi(y0, e0) >> 19) - 4u;
    const unsigned long long a = ((unsigned long long)ah << 32) | al;
    const unsigned long long e1 = 0x3FFFFFFFFFFFFFFFull - __umul64hi(a, (unsigned long long)y1 * y1);   // < 2^35
    const unsigned long long y2 = ((unsigned long long)y1 << 32) + (((unsigned long long)y1 * (unsigned)(e1 >> 4)) >> 27);
    const unsigned long long q = __umul64hi(a, y2) >> 10;
    const unsigned q0 = (unsigned)q, q1 = (unsigned)(q >> 32);
    const unsigned long long lo = (unsigned long long)q0 * q0;
    const unsigned long long rem = ((unsigned long long)((xl << (20 + odd)) - ((unsigned)(lo >> 32) + 2u * q0 * q1)) << 32) -
                                   (unsigned)lo;
    const unsigned top = ((((xh >> 20) + 1023u) >> 1) - 1u) << 20;
    return __longlong_as_double((long long)(((unsigned long long)top << 32) + q + (rem > q ? 1u : 0u)));
}
static __device__ __noinline__ double sqrtNative(double x) { return sqrt(x); }
__device__ __forceinline__ double sqrtI(double x) {
    const unsigned h = (unsigned)__double2hiint(x);
    if (h - 0x00100000u >= 0x7FE00000u) return sqrtNative(x);     // negative, zero, subnormal, Inf, NaN
    return rootBits(h, (unsigned)__double2loint(x));
}
__device__ __forceinline__ float sqrtI(float x) { return sqrt(x); }

// Arithmetic on a group of operands that were tested once, without a branch of its own, so
// that the compiler can interleave the independent products and quotients (each a dependent
// chain of some 30 integer instructions, which a warp otherwise waits out one by one).
// Magnitudes in [2^-480, 2^481) have safely normal products and quotients:
//   GroupPlain  every operand's magnitude in that window;
//   GroupZeros  zeros too (flat states, gas at rest), resolved by selects.
// Both give the IEEE results (GroupZeros the signed zeros, infinities and NaN of mulI and
// divI).  warpAll() takes the class for all active lanes of the warp together: lanes of
// different classes would run every class's code one after the other.  KH 2048^2 step 6.41
// -> 6.05 ms with the Roe transforms and corrections in groups, 1D shock tube step 32.8 ->
// 27.7 us (with the plain group for some lanes and the tested products for the others 36.4).
__device__ __forceinline__ bool inWindow(double x) {
    const unsigned h = (unsigned)__double2hiint(x);
    return h + h - (543u << 21) < (961u << 21);
}
template <int N>
__device__ __forceinline__ bool allInWindow(const double* v) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < N; ++i) ok &= inWindow(v[i]);
    return ok;
}
template <int N>
__device__ __forceinline__ bool allInWindowOrZero(const double* v) {
    bool ok = true;
#pragma unroll
    for (int i = 0; i < N; ++i) ok &= inWindow(v[i]) | isZeroBits(v[i]);
    return ok;
}
__device__ __forceinline__ bool warpAll(bool p) { return __all_sync(__activemask(), p); }

struct GroupPlain {
    static __device__ __forceinline__ double mul(double x, double y) {
        return productBits((unsigned)__double2hiint(x), (unsigned)__double2loint(x), (unsigned)__double2hiint(y),
                           (unsigned)__double2loint(y));
    }
    static __device__ __forceinline__ double div(double x, double y) {
        const unsigned yh = (unsigned)__double2hiint(y), yl = (unsigned)__double2loint(y);
        return quotientBits((unsigned)__double2hiint(x), (unsigned)__double2loint(x), yh, yl, recipBits(yh, yl));
    }
    // half of a product
    static __device__ __forceinline__ double half(double p) {
        return __hiloint2double(__double2hiint(p) - 0x00100000, __double2loint(p));
    }
};
struct GroupZeros {
    static __device__ __forceinline__ double mul(double x, double y) {
        const double p = GroupPlain::mul(x, y);
        const bool z = (((unsigned)__double2hiint(x) & 0x7FF00000u) == 0) | (((unsigned)__double2hiint(y) & 0x7FF00000u) == 0);
        const int sgn = (__double2hiint(x) ^ __double2hiint(y)) & (int)0x80000000u;
        return __hiloint2double(z ? sgn : __double2hiint(p), z ? 0 : __double2loint(p));
    }
    static __device__ __forceinline__ double div(double x, double y) {
        const double q = GroupPlain::div(x, y);
        const bool xz = ((unsigned)__double2hiint(x) & 0x7FF00000u) == 0, yz = ((unsigned)__double2hiint(y) & 0x7FF00000u) == 0;
        const int sgn = (__double2hiint(x) ^ __double2hiint(y)) & (int)0x80000000u;
        const int hi = yz ? (xz ? 0x7FFFFFFF : sgn | 0x7FF00000) : sgn, lo = xz & yz ? -1 : 0;
        return __hiloint2double(xz | yz ? hi : __double2hiint(q), xz | yz ? lo : __double2loint(q));
    }
    static __device__ __forceinline__ double half(double p) { return isZeroBits(p) ? p : GroupPlain::half(p); }
};

// A divisor used by several quotients (a density, the cell size, an HLLC denominator):
// its reciprocal bits are formed once, on the host for a constant, and a quotient then
// costs about a product.  v is 0 where b is not normal.
template <typename real> struct Divisor { real b; };
template <> struct Divisor<double> { double b; unsigned long long v; };

__device__ __forceinline__ Divisor<float> divisorOf(float b) { return {b}; }
__device__ __forceinline__ Divisor<double> divisorOf(double b) {
    const unsigned h = (unsigned)__double2hiint(b);
    return {b, (h & 0x7FF00000u) - 0x00100000u < 0x7FE00000u ? recipBits(h, (unsigned)__double2loint(b)) : 0ull};
}
inline void hostDivisor(float b, Divisor<float>& d) { d.b = b; }
inline void hostDivisor(double b, Divisor<double>& d) {
    unsigned long long u;
    memcpy(&u, &b, 8);
    const unsigned long long m = (u & 0xFFFFFFFFFFFFFull) | (1ull << 52), e = (u >> 52) & 0x7FF;
    d.b = b;
    d.v = e - 1 >= 2046 ? 0ull : m == (1ull << 52) ? ~0ull : (unsigned long long)(((unsigned __int128)1 << 116) / m);
}

// x / d.b, the IEEE quotient (as divI)
__device__ __forceinline__ float quotBy(float x, const Divisor<float>& d) { return x / d.b; }
__device__ __forceinline__ double quotBy(double x, const Divisor<double>& d) {
    const unsigned xh = (unsigned)__double2hiint(x), xl = (unsigned)__double2loint(x);
    const unsigned yh = (unsigned)__double2hiint(d.b), yl = (unsigned)__double2loint(d.b);
    const unsigned ex = xh & 0x7FF00000u, ey = yh & 0x7FF00000u;
    if (ex - 0x00100000u >= 0x7FE00000u || d.v == 0 || ex - ey + (1021u << 20) >= (2044u << 20)) {
        if (((xh << 1) | xl) == 0 && d.v != 0) return __hiloint2double((int)((xh ^ yh) & 0x80000000u), 0);
        return divNative(x, d.b);
    }
    return quotientBits(xh, xl, yh, yl, d.v);
}

// x / d for x and d.b in the window (GroupPlain's quotient by a shared divisor)
__device__ __forceinline__ double quotPlain(double x, const Divisor<double>& d) {
    return quotientBits((unsigned)__double2hiint(x), (unsigned)__double2loint(x), (unsigned)__double2hiint(d.b),
                        (unsigned)__double2loint(d.b), d.v);
}

// The operations of a longer computation: AnyOps tests each operand pair (mulI, divI);
// CheckedOps assumes ordinary magnitudes and keeps in `ok` whether every operand had one, for
// the caller to do the whole computation again with AnyOps if not.
template <typename real>
struct AnyOps {
    bool ok = true;
    __device__ __forceinline__ real mul(real x, real y) { return mulI(x, y); }
    __device__ __forceinline__ real div(real x, real y) { return divI(x, y); }
    __device__ __forceinline__ real half(real x) { return halfOf(x); }
    __device__ __forceinline__ real root(real x) { return sqrtI(x); }
    __device__ __forceinline__ Divisor<real> divisor(real b) { return divisorOf(b); }
    __device__ __forceinline__ real quot(real x, const Divisor<real>& d) { return quotBy(x, d); }
};
struct CheckedOps {
    bool ok = true;
    __device__ __forceinline__ double mul(double x, double y) {
        ok &= inWindow(x) & inWindow(y);
        return GroupPlain::mul(x, y);
    }
    __device__ __forceinline__ double div(double x, double y) {
        ok &= inWindow(x) & inWindow(y);
        return GroupPlain::div(x, y);
    }
    __device__ __forceinline__ double half(double x) {
        ok &= inWindow(x);
        return GroupPlain::half(x);
    }
    __device__ __forceinline__ double root(double x) {
        ok &= inWindow(x) & (__double2hiint(x) >= 0);
        return rootBits((unsigned)__double2hiint(x), (unsigned)__double2loint(x));
    }
    // 2 x of a product (exact)
    __device__ __forceinline__ double twice(double x) {
        ok &= inWindow(x);
        return __hiloint2double(__double2hiint(x) + 0x00100000, __double2loint(x));
    }
    __device__ __forceinline__ Divisor<double> divisor(double b) {
        ok &= inWindow(b);
        return {b, recipBits((unsigned)__double2hiint(b), (unsigned)__double2loint(b))};
    }
    __device__ __forceinline__ double quot(double x, const Divisor<double>& d) {
        ok &= inWindow(x);
        return quotPlain(x, d);
    }
};

// (float)((double)c - (double)a * (double)b) for floats, on the FP32 pipes.  The product
// is exact in double (48 bits), so the value is c - a*b rounded to 53 bits and then to 24;
// one fma rounds it to 24 directly, the same unless the 53-bit value is the midpoint of
// two floats.  The distance x - r of the exact value from the fma's result r is formed
// from the product's and the sum's error terms (fma residual, Knuth's two-sum) to well
// below 2^-18 of half an ulp; results within that of a midpoint, or with error terms that
// are not numbers (a product past the floats beside a c that brings the result back: the
// comparison is false for NaN), and r a power of two, whose lower neighbour is closer, and
// tiny r, take the double expression out of line.
// The three conversions to double, the product, the difference and the conversion back
// ran on the FP64 unit and were most of the FP32 flux kernel: KH 2048^2 550 us a launch,
// 163 us with this form (the rest of it: loads at the HBM rate).
static __device__ __noinline__ float subProductNative(float c, float a, float b) {
    return (float)((double)c - (double)a * (double)b);
}
__device__ __forceinline__ float subProduct(float c, float a, float b) {
    const float r = fmaf(-a, b, c);
    const float p = __fmul_rn(a, b), pe = fmaf(a, b, -p);                    // a*b = p + pe
    const float s = __fsub_rn(c, p), v = __fsub_rn(s, c);
    const float t = __fsub_rn(__fsub_rn(c, __fsub_rn(s, v)), __fadd_rn(p, v));   // c - p = s + t
    const float e = __fsub_rn(__fadd_rn(__fsub_rn(s, r), t), pe);
    const unsigned rb = __float_as_uint(r);
    const float half = __uint_as_float(rb & 0x7F800000u) * 0x1p-24f;         // half an ulp of r
    const bool near = !(fabsf(fabsf(e) - half) >= 0x1p-18f * (half + fabsf(pe) + fabsf(t)));
    const bool edge = (rb << 1) != 0 && ((rb << 9) == 0 || (rb & 0x7FFFFFFFu) < 0x12800000u);   // |r| < 2^-90
    return near || edge ? subProductNative(c, a, b) : r;
}


}  // namespace hgpu
