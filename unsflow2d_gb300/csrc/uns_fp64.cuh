// uns_fp64.cuh -- IEEE double arithmetic arranged for GB300, whose FP64 unit
// is the scarcest resource of the FP64 kernels: it accepts one warp
// instruction per SM sub-partition every 64-76 cycles, while the integer and
// FP32 pipes beside it take one every 1-4.  F64 is a double whose operators
// give the bits of the IEEE operations (round to nearest even) by cheaper
// routes, each measured on the GB300 (cycles a warp instruction holds its
// sub-partition, 8 warps each):
//
//   a + b, a * b   as an FMA whose three operands are vector registers, with
//                  an opaque 1.0 or -0.0 as the third: 64.1, against 76.1 for
//                  the add and multiply instructions and for an FMA with one
//                  constant operand;
//   a / b, sqrt a  on the integer pipe by digit recurrence: 90 and 96,
//                  against 550 and 573 for the FP64 sequences, and beside the
//                  FP64 unit rather than on it (four additions and a division
//                  take what the four additions take);
//   comparisons, min, max, halving, conversion from and to float: integer
//                  operations (4-18 cycles).
//
// Operands outside the middle of the exponent range (2^-255 .. 2^256; a zero
// numerator stays on the fast route) take the native operation, so every
// input gives the IEEE result; tests/test_gpu_fp64_ops.py compares them
// bit by bit.
//
// In the contracted build (UNS_FP64_CONTRACT) + - * are the language's own,
// which the compiler may fuse.
#pragma once
#include <cuda_runtime.h>

namespace uns {

// -0.0 and 1.0 in vector registers whose value the compiler does not know:
// bit 31 of %lanemask_ge is set in every lane.  (A constant or uniform
// operand would put the FMA back to 76 cycles.)
__device__ __forceinline__ double opaque_mzero() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_ge;" : "=r"(m));
    return __hiloint2double((int)(m & 0x80000000u), 0);
}
__device__ __forceinline__ double opaque_one() {
    unsigned m;
    asm("mov.u32 %0, %%lanemask_ge;" : "=r"(m));
    return __hiloint2double((int)((m & 0x80000000u) ^ 0xbff00000u), 0);
}

__device__ __forceinline__ double add64(double a, double b) {
#ifdef UNS_FP64_CONTRACT
    return a + b;
#else
    return __fma_rn(a, opaque_one(), b);
#endif
}
__device__ __forceinline__ double sub64(double a, double b) {
#ifdef UNS_FP64_CONTRACT
    return a - b;
#else
    return __fma_rn(a, opaque_one(), -b);
#endif
}
__device__ __forceinline__ double mul64(double a, double b) {
#ifdef UNS_FP64_CONTRACT
    return a * b;
#else
    return __fma_rn(a, b, opaque_mzero());
#endif
}

__device__ __forceinline__ unsigned dhi(double x) { return (unsigned)__double2hiint(x); }
__device__ __forceinline__ unsigned dlo(double x) { return (unsigned)__double2loint(x); }
__device__ __forceinline__ double dmake(unsigned hi, unsigned lo) { return __hiloint2double((int)hi, (int)lo); }
__device__ __forceinline__ unsigned long long u64(unsigned hi, unsigned lo) {
    return ((unsigned long long)hi << 32) | lo;
}

// -a on the sign bit, and a with its sign flipped where minus (a negation that
// no FMA operand absorbs is an addition on the FP64 unit).
__device__ __forceinline__ double neg64(double a) { return dmake(dhi(a) ^ 0x80000000u, dlo(a)); }
__device__ __forceinline__ double flip64(double a, bool minus) { return dmake(dhi(a) ^ (minus ? 0x80000000u : 0u), dlo(a)); }

// The native operations where they are rarely needed, as calls: branched
// around (predicated off, they would hold the FP64 unit all the same), and
// once in a kernel's code.
static __device__ __noinline__ double native_mul(double a, double b) { return a * b; }
static __device__ __noinline__ double add_rare(double a, double b) { return a + b; }
static __device__ __noinline__ double mul_rare(double a, double b) {
    // zeros (uniform flow, the first steps of a solve) without the unit
    const unsigned ha = dhi(a), hb = dhi(b);
    const bool za = ((ha << 1) | dlo(a)) == 0, zb = ((hb << 1) | dlo(b)) == 0;
    const bool fa = (ha & 0x7ff00000u) != 0x7ff00000u, fb = (hb & 0x7ff00000u) != 0x7ff00000u;
    if ((za && fb) || (zb && fa)) return dmake((ha ^ hb) & 0x80000000u, 0u);
    return native_mul(a, b);
}
static __device__ __noinline__ double div_rare(double a, double b) { return a / b; }
static __device__ __noinline__ double sqrt_rare(double a) { return sqrt(a); }
static __device__ __noinline__ double widen_rare(float a) {  // a NaN as FP32 arithmetic gives it, whatever sign a flip left on it
    return a != a ? dmake(0x7fffffffu, 0xe0000000u) : (double)a;
}
static __device__ __noinline__ float narrow_rare(double a) { return (float)a; }

// (double)a and (float)a on the integer pipe (the conversions hold the FP64
// unit 76-99 cycles).
__device__ __forceinline__ double widen(float a) {
    const unsigned b = __float_as_uint(a);
    const bool zero = (b << 1) == 0;
    if ((b & 0x7f800000u) - 0x00800000u >= 0x7f000000u && !zero) return widen_rare(a);  // subnormal, infinite, NaN
    const unsigned hi = ((b >> 3) & 0x0fffffffu) + 0x38000000u;
    return dmake((b & 0x80000000u) | (zero ? 0u : hi), b << 29);
}
__device__ __forceinline__ float narrow(double a) {
    const unsigned h = dhi(a), l = dlo(a), m = h & 0x7fffffffu;
    const bool zero = (m | l) == 0;
    if (m - 0x38100000u >= 0x0fd00000u && !zero) return narrow_rare(a);  // outside [2^-126, 2^127)
    const unsigned r = __funnelshift_l(l, m - 0x38000000u, 3), rem = l << 3;  // 24-bit significand and what it drops
    const unsigned up = (rem >= 0x80000000u && (rem > 0x80000000u || (r & 1u))) ? 1u : 0u;
    return __uint_as_float((h & 0x80000000u) | (zero ? 0u : r + up));
}

// Division and square root by digit recurrence with accurate quotient digits
// (D. Wong, M. Flynn, "Fast division using accurate quotient
// approximations", IEEE Trans. Computers 41(8), 1992): every digit is the
// leading 32 bits of the remainder times a 32-bit reciprocal Y that is never
// too large and short by at most 2^-19.9 of itself, so a digit is never too
// large either and the remainders, kept exactly modulo 2^64, stay
// non-negative.  Three digits give floor(q 2^54) or one less; the last
// remainder tells which.  A quotient or root of 53-bit significands is never
// halfway between two of them, so rounding needs no further sticky bit.

// Y = 2^32 y (1 - 2^-21 ...) for y in (1/2, 1] given to 2^-23 of itself.
__device__ __forceinline__ unsigned recip_digits(float y) {
    return __float_as_uint(__fmaf_rd(y, 1.0f - 0x1p-21f, 1.0f)) << 9;
}

// The reciprocal of b's significand for div_digits: from its leading 24 bits.
__device__ __forceinline__ unsigned div_recip(double b) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(__uint_as_float(0x3f800000u | (__funnelshift_l(dlo(b), dhi(b), 3) & 0x7fffffu))));
    return recip_digits(y);
}

// a / b with Y = div_recip(b), which a caller that has b early forms early.
__device__ __forceinline__ double div_digits(double a, double b, unsigned Y) {
    const unsigned ha = dhi(a), la = dlo(a), hb = dhi(b), lb = dlo(b);
    const unsigned ea = ha & 0x7ff00000u, eb = hb & 0x7ff00000u, sign = (ha ^ hb) & 0x80000000u;
    const bool zero = ((ha << 1) | la) == 0;
    // exponent fields of both within [768, 1279]
    if ((((zero ? 0u : ea - 0x30000000u) | (eb - 0x30000000u)) & 0xe0000000u) != 0) return div_rare(a, b);
    const unsigned long long ma = u64((ha & 0xfffffu) | 0x100000u, la), mb = u64((hb & 0xfffffu) | 0x100000u, lb);
    const unsigned d1 = __umulhi((unsigned)(ma >> 21), Y) >> 2;                   // q to 2^-29
    const unsigned long long r1 = (ma << 29) - (unsigned long long)d1 * mb;      // < 2^63.2
    const unsigned d2 = __umulhi((unsigned)(r1 >> 32), Y);                        // to 2^-49
    const unsigned long long r2 = (r1 << 20) - (unsigned long long)d2 * mb;      // < 2^63.4
    const unsigned d3 = __umulhi((unsigned)(r2 >> 32), Y) >> 15;                  // to 2^-54
    const unsigned long long r3 = (r2 << 5) - (unsigned long long)d3 * mb;       // < 2 mb
    unsigned long long f = ((unsigned long long)d1 << 25) + ((unsigned long long)d2 << 5) + d3 + (r3 >= mb ? 1 : 0);
    const unsigned t = (unsigned)(f >> 54);  // q >= 1
    f = (f + (1u << t)) >> (1 + t);
    const unsigned hi = (unsigned)(f >> 32) + (ea - eb) + ((1021u + t) << 20);
    return dmake(zero ? sign : (hi | sign), zero ? 0u : (unsigned)f);
}
__device__ __forceinline__ double div_digits(double a, double b) { return div_digits(a, b, div_recip(b)); }

__device__ __forceinline__ double sqrt_digits(double a) {
    const unsigned ha = dhi(a), la = dlo(a);
    if (ha - 0x30000000u >= 0x20000000u) return sqrt_rare(a);  // exponent field within [768, 1279], positive
    const unsigned odd = ((ha >> 20) & 1u) ^ 1u;          // of the unbiased exponent
    const unsigned long long m = u64((ha & 0xfffffu) | 0x100000u, la) << odd;  // 2^52 times a value in [1, 4)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;"
        : "=f"(y) : "f"(__uint_as_float((0x3f800000u + (odd << 23)) | (((ha & 0xfffffu) << 3) | (la >> 29)))));
    const unsigned Y = recip_digits(y);
    const unsigned s1 = __umulhi((unsigned)(m >> 22), Y);                           // root to 2^-30
    const unsigned long long r1 = (m << 8) - (unsigned long long)s1 * s1;
    const unsigned s2 = __umulhi((unsigned)(r1 >> 12), Y);                          // to 2^-49
    const unsigned long long r2 = (r1 << 38) - (((unsigned long long)s1 * s2) << 20) - (unsigned long long)s2 * s2;
    const unsigned s3 = __umulhi((unsigned)(r2 >> 32), Y) >> 13;                    // to 2^-54
    const unsigned long long s = (((unsigned long long)s1 << 19) + s2) << 5;
    unsigned long long f = s + s3;
    const unsigned long long r3 = (r2 << 10) - (s + f) * s3;
    f += (r3 > 2 * f) ? 1 : 0;
    f = (f + 2) >> 2;
    return __longlong_as_double((long long)(f + ((unsigned long long)(((ha >> 20) - odd + 1) / 2 + 510) << 52)));
}

// a * b on the integer pipe: the 106-bit product of the significands, its top
// 53 bits rounded to nearest even.  About 40 cycles of its own pipe, beside
// the FP64 unit: kernels bound by that unit put products here and keep sums
// there.
__device__ __forceinline__ double mul_digits(double a, double b) {
    const unsigned ha = dhi(a), la = dlo(a), hb = dhi(b), lb = dlo(b);
    const unsigned ea = ha & 0x7ff00000u, eb = hb & 0x7ff00000u, sign = (ha ^ hb) & 0x80000000u;
    if ((((ea - 0x30000000u) | (eb - 0x30000000u)) & 0xe0000000u) != 0) return mul_rare(a, b);  // fields within [768, 1279]
    const unsigned mah = (ha & 0xfffffu) | 0x100000u, mbh = (hb & 0xfffffu) | 0x100000u;
    const unsigned long long t0 = (unsigned long long)la * lb;
    const unsigned long long t1 = (unsigned long long)mah * lb + (t0 >> 32);
    const unsigned long long t2 = (unsigned long long)la * mbh + t1;                    // < 2^54
    const unsigned long long p = (unsigned long long)mah * mbh + (t2 >> 32);            // product >> 64, < 2^42
    const unsigned low = (unsigned)t2 | min((unsigned)t0, 1u);                          // bit 0 sticky
    const unsigned top = (unsigned)(p >> 41), sh = 20 + top;                            // significands' product >= 2
    const unsigned mlo = __funnelshift_r(low, (unsigned)p, sh), mhi = __funnelshift_r((unsigned)p, (unsigned)(p >> 32), sh);
    const unsigned rem = low << (12 - top);                                             // discarded bits
    const unsigned long long m = u64(mhi + (ea + eb - 0x40000000u) + (top << 20) + sign, mlo);
    return __longlong_as_double((long long)(m + (rem + (mlo & 1u) > 0x80000000u ? 1 : 0)));
}

// a < b on the integer pipe: false where either is a NaN, and for two zeros.
__device__ __forceinline__ bool dlt(double a, double b) {
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    const long long kx = x ^ (long long)((unsigned long long)(x >> 63) >> 1), ky = y ^ (long long)((unsigned long long)(y >> 63) >> 1);
    const unsigned long long ax = (unsigned long long)x << 1, ay = (unsigned long long)y << 1;
    return kx < ky && (ax | ay) != 0 && ax <= 0xffe0000000000000ULL && ay <= 0xffe0000000000000ULL;
}
// a <= b likewise.
__device__ __forceinline__ bool dle(double a, double b) {
    const long long x = __double_as_longlong(a), y = __double_as_longlong(b);
    const long long kx = x ^ (long long)((unsigned long long)(x >> 63) >> 1), ky = y ^ (long long)((unsigned long long)(y >> 63) >> 1);
    const unsigned long long ax = (unsigned long long)x << 1, ay = (unsigned long long)y << 1;
    return (kx <= ky || (ax | ay) == 0) && ax <= 0xffe0000000000000ULL && ay <= 0xffe0000000000000ULL;
}
// Running extremes as order-preserving signed keys (11 integer operations for
// both, where a maximum and a minimum instruction hold the FP64 unit 76 cycles
// each): a NaN changes neither.
__device__ __forceinline__ long long order_key(double a) {
    const long long x = __double_as_longlong(a);
    return x ^ (long long)((unsigned long long)(x >> 63) >> 1);
}
__device__ __forceinline__ double from_key(long long k) {
    return __longlong_as_double(k ^ (long long)((unsigned long long)(k >> 63) >> 1));
}
__device__ __forceinline__ void extend(double a, long long& lo, long long& hi) {
    const long long k = order_key(a);
    if (((unsigned long long)__double_as_longlong(a) << 1) > 0xffe0000000000000ULL) return;
    hi = k > hi ? k : hi;
    lo = k < lo ? k : lo;
}

// 0 < a and a < 0 (false for NaN).
__device__ __forceinline__ bool dpos(double a) {
    return (unsigned long long)__double_as_longlong(a) - 1ULL < 0x7ff0000000000000ULL;
}
__device__ __forceinline__ bool dneg(double a) { return dpos(neg64(a)); }

// 0.5 * a: the exponent field less one; zero stays, the ends of the range take the multiplication.
__device__ __forceinline__ double dhalf(double a) {
    const unsigned h = dhi(a), l = dlo(a);
    const bool in = (h & 0x7ff00000u) - 0x00200000u < 0x7fd00000u, zero = ((h << 1) | l) == 0;
    if (!in && !zero) return mul_rare(0.5, a);
    return dmake(in ? h - 0x00100000u : h, l);
}
// 2 * a likewise.
__device__ __forceinline__ double dtwice(double a) {
    const unsigned h = dhi(a), l = dlo(a);
    const bool in = (h & 0x7ff00000u) - 0x00100000u < 0x7fd00000u, zero = ((h << 1) | l) == 0;
    if (!in && !zero) return mul_rare(2.0, a);
    return dmake(in ? h + 0x00100000u : h, l);
}

// A value (a constant, a kernel parameter) in vector registers: as an operand
// of the FMAs above it does not cost the 12 cycles of a constant one.
__device__ __forceinline__ double in_register(double x) {
#ifdef UNS_FP64_CONTRACT
    return x;
#else
    unsigned m;
    asm("mov.u32 %0, %%lanemask_ge;" : "=r"(m));
    return dmake(dhi(x) ^ (m & 0x80000000u) ^ 0x80000000u, dlo(x));
#endif
}

// A double with these operators (in a namespace of its own, so that its sqrt,
// fabs and pow are found by argument-dependent lookup alone).
namespace f64 {

struct F64 {
    double v;
    __device__ __forceinline__ F64() {}
    __device__ __forceinline__ F64(double x) : v(x) {}
    __device__ __forceinline__ explicit operator double() const { return v; }
    __device__ __forceinline__ explicit operator float() const { return (float)v; }
};
__device__ __forceinline__ F64 operator+(F64 a, F64 b) { return add64(a.v, b.v); }
__device__ __forceinline__ F64 operator-(F64 a, F64 b) { return sub64(a.v, b.v); }
__device__ __forceinline__ F64 operator-(F64 a) { return neg64(a.v); }
__device__ __forceinline__ F64 operator*(F64 a, F64 b) { return mul64(a.v, b.v); }
__device__ __forceinline__ F64 operator/(F64 a, F64 b) { return div_digits(a.v, b.v); }
__device__ __forceinline__ bool operator<(F64 a, F64 b) { return dlt(a.v, b.v); }
__device__ __forceinline__ bool operator>(F64 a, F64 b) { return dlt(b.v, a.v); }
__device__ __forceinline__ bool operator<=(F64 a, F64 b) { return dle(a.v, b.v); }
__device__ __forceinline__ bool operator>=(F64 a, F64 b) { return dle(b.v, a.v); }
__device__ __forceinline__ F64 half(F64 a) { return dhalf(a.v); }
__device__ __forceinline__ F64 twice(F64 a) { return dtwice(a.v); }
__device__ __forceinline__ F64 quarter(F64 a) { return dhalf(dhalf(a.v)); }
__device__ __forceinline__ F64 sqrt(F64 a) { return sqrt_digits(a.v); }
__device__ __forceinline__ F64 fabs(F64 a) { return __longlong_as_double(__double_as_longlong(a.v) & 0x7fffffffffffffffLL); }
__device__ __forceinline__ F64 pow(F64 a, F64 b) { return ::pow(a.v, b.v); }

}  // namespace f64
using f64::F64;
// F64 whose products run on the integer pipe (mul_digits), for kernels whose
// sums alone keep the FP64 unit busy.
namespace f64 {
struct F64I {
    double v;
    __device__ __forceinline__ F64I() {}
    __device__ __forceinline__ F64I(double x) : v(x) {}
    __device__ __forceinline__ F64I(F64 x) : v(x.v) {}
    __device__ __forceinline__ explicit operator double() const { return v; }
    __device__ __forceinline__ explicit operator float() const { return (float)v; }
};
__device__ __forceinline__ F64I operator+(F64I a, F64I b) { return add64(a.v, b.v); }
__device__ __forceinline__ F64I operator-(F64I a, F64I b) { return sub64(a.v, b.v); }
__device__ __forceinline__ F64I operator-(F64I a) { return neg64(a.v); }
#ifdef UNS_FP64_CONTRACT
__device__ __forceinline__ F64I operator*(F64I a, F64I b) { return a.v * b.v; }
#else
__device__ __forceinline__ F64I operator*(F64I a, F64I b) { return mul_digits(a.v, b.v); }
#endif
__device__ __forceinline__ F64I operator/(F64I a, F64I b) { return div_digits(a.v, b.v); }
__device__ __forceinline__ bool operator<(F64I a, F64I b) { return dlt(a.v, b.v); }
__device__ __forceinline__ bool operator>(F64I a, F64I b) { return dlt(b.v, a.v); }
__device__ __forceinline__ bool operator<=(F64I a, F64I b) { return dle(a.v, b.v); }
__device__ __forceinline__ bool operator>=(F64I a, F64I b) { return dle(b.v, a.v); }
__device__ __forceinline__ F64I half(F64I a) { return dhalf(a.v); }
__device__ __forceinline__ F64I twice(F64I a) { return dtwice(a.v); }
__device__ __forceinline__ F64I quarter(F64I a) { return dhalf(dhalf(a.v)); }
__device__ __forceinline__ F64I sqrt(F64I a) { return sqrt_digits(a.v); }
__device__ __forceinline__ F64I fabs(F64I a) { return fabs(F64(a.v)).v; }
__device__ __forceinline__ F64I pow(F64I a, F64I b) { return ::pow(a.v, b.v); }
}  // namespace f64
using f64::F64I;

// The type that a kernel template instantiated on double or float computes in.
template <class R> struct Arith { typedef R type; };
template <> struct Arith<double> { typedef F64 type; };

// 0.5 a, 2 a and a / 4 of any other arithmetic type.
template <class R> __device__ __forceinline__ R half(R a) { return R(0.5) * a; }
template <class R> __device__ __forceinline__ R twice(R a) { return R(2) * a; }
template <class R> __device__ __forceinline__ R quarter(R a) { return R(0.25) * a; }

}  // namespace uns
