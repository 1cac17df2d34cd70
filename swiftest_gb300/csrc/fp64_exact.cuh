// fp64_exact.cuh -- correctly rounded FP64 square root, quotient and product that leave
// the FP64 pipe alone.
//
// GB300 issues one FP64 warp instruction per SM every 16 cycles (DFMA, DMUL; 19 for DADD
// and DSETP), against one FP32 or integer instruction every 0.25 to 1.5 cycles, so an FP64
// divide (137 cycles per warp and SM, measured) or square root (143) costs as much as
// hundreds of cheap ones.  The functions here form the same correctly rounded results from
// an FP32 approximation and integer arithmetic:
//
//  1. an FP32 estimate of 24 bits (PTX rsqrt.approx / rcp.approx, whose documented maximum
//     relative errors are 2^-22.9 and 2^-23), refined once in FP32 pairs to about 45 bits
//     (Newton's iteration on the residual);
//  2. as an integer mantissa with an error of at most a few hundred units in the last
//     place, whose exact remainder (x - s^2, g - q p) fits 64 bits, so its low 64 bits,
//     computed modulo 2^64, are the remainder;
//  3. remainder / divisor in FP32 gives the distance to the exact result to better than
//     2^-11 units; it is rounded to the nearest integer, and where it lies within 2^-10 of a
//     midpoint the exact remainder decides (Markstein's remainder test; neither a square
//     root nor a quotient of 53-bit numbers is ever a midpoint).
//
// Valid for positive normal operands with a normal result.  The callers pass operands with exponents within
// +-XR_EXP of one (x_ok), or results of such operands whose exponents stay normal, and send
// everything else (zeros, subnormals, infinities, NaN, extreme exponents) to the native
// operations.  Each function reports in `bad` the lanes it could not decide, which take the native
// form too: an estimate that falls into the neighbouring binade, about one random operand in 2^22, and
// in x_div every divisor that is a power of two (its reciprocal's estimate is one).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

namespace swg {

constexpr int XR_EXP = 100;

// positive (sign bit clear), normal, exponent within +-XR_EXP; hi: the high word
__device__ __forceinline__ bool x_ok(int hi) {
    return (unsigned)((hi >> 20) - (1023 - XR_EXP)) <= (unsigned)(2 * XR_EXP);
}
__device__ __forceinline__ float x_rsqrt_approx(float x) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}
__device__ __forceinline__ float x_rcp_approx(float x) {
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
}

// the leading 24 mantissa bits of a double as a float in [1, 2)
__device__ __forceinline__ float x_mant_hi(int hi, int lo) {
    return __int_as_float((__funnelshift_l(lo, hi, 3) & 0x7fffff) | 0x3f800000);
}
// the remaining 29 bits, at the same scale (odd: twice that)
__device__ __forceinline__ float x_mant_lo(int lo, int odd) {
    return __int2float_rn(lo & 0x1fffffff) * __int_as_float((75 + odd) << 23);
}

constexpr float X_MAGIC = 12582912.0f;  // 1.5 * 2^23: adding it rounds a small float to an integer

// sqrt(x), x_ok(x).  Error budget in units of the result's last place (2^-52 of [1, 2)):
// the FP32 pair is off by at most 640 (each rounding counted at its worst), the remainder
// wraps at 512 to 1024, so |delta| <= 380 is the remainder itself.
__device__ __forceinline__ double x_sqrt(double x, bool &bad) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    // x = m 4^k, m in [1, 4); the exponent's bias is odd
    const int odd = (~hi >> 20) & 1;
    const float mh = __int_as_float(((__funnelshift_l(lo, hi, 3) & 0xffffff) ^ 0x800000) + 0x3f800000);
    const float ml = x_mant_lo(lo, odd);
    const float y = x_rsqrt_approx(mh);
    const float th = y * y, tl = fmaf(y, y, -th);
    const float e = fmaf(-mh, th, 1.0f) - fmaf(mh, tl, ml * th);     // 1 - m y^2
    const float c = y * fmaf(0.375f * e, e, 0.5f * e);               // y + c = m^-1/2
    const float sh = mh * y;
    const float sl = fmaf(mh, c, fmaf(ml, y, fmaf(mh, y, -sh)));     // sh + sl = m^1/2
    const int sb = __float_as_int(sh);
    const uint64_t s1 = ((uint64_t)(uint32_t)((sb & 0x7fffff) | 0x800000) << 29) +
                        (int64_t)__float2int_rn(sl * 4503599627370496.0f);
    const uint64_t r = ((uint64_t)((uint32_t)lo << (20 + odd)) << 32) - s1 * s1;  // m 2^104 - s1^2
    const float d = __int2float_rn((int)(r >> 32)) * (y * 4.76837158203125e-7f);  // / (2 s1)
    const float t = d + X_MAGIC;
    const int n = __float_as_int(t) - __float_as_int(X_MAGIC);
    uint64_t s = s1 + (int64_t)n;
    if (fabsf(d - (t - X_MAGIC)) > 0.5f - 1.0f / 1024) {  // near a midpoint: the remainder of s decides
        const int64_t rem = (int64_t)(r - (uint64_t)(int64_t)n * (s1 + s));
        if (rem > (int64_t)s) s++;
        else if (rem <= -(int64_t)s) s--;
    }
    bad |= (sb >> 23) != 127 || (s >> 52) != 1 || fabsf(d) > 380.0f;
    return __hiloint2double((((hi - 0x3ff00000) >> 1) & 0xfff00000) + 0x3fe00000 + (int)(s >> 32), (int)s);
}

// a * b for normal operands whose product is normal; a > 0.  The 106-bit product of the
// mantissas from four 32-bit products (the cross terms fit one 64-bit sum), half a unit of
// the result's last place added at its position (product below or above 2^105), the
// rest cut; an exact tie clears the last bit (round to even).
__device__ __forceinline__ double x_mul(double a, double b) {
    const int ah = __double2hiint(a), al = __double2loint(a), bh = __double2hiint(b), bl = __double2loint(b);
    const uint32_t Ah = (ah & 0xfffff) | 0x100000, Al = (uint32_t)al;
    const uint32_t Bh = (bh & 0xfffff) | 0x100000, Bl = (uint32_t)bl;
    const uint64_t t0 = (uint64_t)Al * Bl;
    const uint64_t x = (uint64_t)Al * Bh + ((uint64_t)Ah * Bl + (t0 >> 32));
    const uint64_t top = (uint64_t)Ah * Bh + (x >> 32);
    const int c = (int)(top >> 41), s = 12 - c;  // c: the product is 2^105 or more
    uint32_t r, m0, m1;
    asm("{add.cc.u32 %0, %3, %4; addc.cc.u32 %1, %5, 0; addc.u32 %2, %6, 0;}"
        : "=r"(r), "=r"(m0), "=r"(m1)
        : "r"((uint32_t)x), "r"(0x80000u << c), "r"((uint32_t)top), "r"((uint32_t)(top >> 32)));
    uint32_t o0 = __funnelshift_l(r, m0, s);
    if (((r << s) | (uint32_t)t0) == 0) o0 &= ~1u;
    const int e = (ah & 0x7ff00000) + (bh & 0xfff00000) - 0x40000000 + (c << 20);
    return __hiloint2double((int)__funnelshift_l(m0, m1, s) + e, (int)o0);
}

// a * a for a normal operand whose square is normal
__device__ __forceinline__ double x_sqr(double a) {
    const double p = __hiloint2double(__double2hiint(a) & 0x7fffffff, __double2loint(a));  // no FP64 instruction
    return x_mul(p, p);
}

// Numerator of x_div, formed once where it serves several quotients: mantissa as an FP32 pair.
struct XNum {
    float h, l;
    int hi, lo;
};
__device__ __forceinline__ XNum x_num(double g) {
    XNum a;
    a.hi = __double2hiint(g);
    a.lo = __double2loint(g);
    a.h = x_mant_hi(a.hi, a.lo);
    a.l = x_mant_lo(a.lo, 0);
    return a;
}

// g / p, normal with a normal quotient.  The FP32 pair is off by at most 450 units in the last place; the
// remainder wraps at 1024.
__device__ __forceinline__ double x_div(const XNum &g, double p, bool &bad) {
    const int hi = __double2hiint(p), lo = __double2loint(p);
    const float z = x_rcp_approx(x_mant_hi(hi, lo));  // in (1/2, 1]
    const int zb = __float_as_int(z);
    const uint64_t P = ((uint64_t)(uint32_t)((hi & 0xfffff) | 0x100000) << 32) | (uint32_t)lo;
    const uint32_t Z = (zb & 0x7fffff) | 0x800000;       // z 2^24
    const int64_t rho = -(int64_t)(P * Z);               // 2^76 (1 - p z), modulo 2^64
    const float rf = __int2float_rn((int)(rho >> 24)) * 2.220446049250313e-16f;
    const float zl = z * fmaf(rf, rf, rf);               // z + zl = 1 / p
    const float qh = g.h * z;
    const float ql = fmaf(g.h, zl, fmaf(g.l, z, fmaf(g.h, z, -qh)));
    const int qb = __float_as_int(qh);
    const int low = 127 - (qb >> 23);                    // 0: quotient in [1, 2), 1: in [1/2, 1)
    const uint64_t q1 = ((uint64_t)(uint32_t)((qb & 0x7fffff) | 0x800000) << 29) +
                        (int64_t)__float2int_rn(ql * __int_as_float((127 + 52 + low) << 23));
    const uint64_t r = ((uint64_t)((uint32_t)g.lo << (20 + low)) << 32) - q1 * P;  // g 2^(52+low) - q1 p
    const float d = __int2float_rn((int)(r >> 32)) * (z * 9.5367431640625e-7f);    // / p
    const float t = d + X_MAGIC;
    const int n = __float_as_int(t) - __float_as_int(X_MAGIC);
    uint64_t q = q1 + (int64_t)n;
    if (fabsf(d - (t - X_MAGIC)) > 0.5f - 1.0f / 1024) {
        const int64_t rem2 = 2 * (int64_t)(r - (uint64_t)(int64_t)n * P);
        if (rem2 > (int64_t)P) q++;
        else if (rem2 < -(int64_t)P) q--;
    }
    bad |= (zb >> 23) != 126 || (q >> 52) != 1;
    return __hiloint2double((g.hi & 0x7ff00000) - (hi & 0x7ff00000) - (low << 20) + 0x3fe00000 + (int)(q >> 32), (int)q);
}

// Conversions by integer instructions (the conversion instructions take the FP64 pipe): a
// double cut to its leading 24 bits, a float as a double, and the rounded float of a double.
__device__ __forceinline__ float x_to_float(double x) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    if (!x_ok(hi & 0x7fffffff)) return ((hi & 0x7fffffff) | lo) == 0 ? 0.0f : (float)x;
    return __int_as_float((__funnelshift_l(lo, hi - ((1023 - 127) << 20), 3) & 0x7fffffff) | (hi & 0x80000000));
}
__device__ __forceinline__ double x_to_double(float f) {
    const int b = __float_as_int(f), m = b & 0x7fffffff;
    if (m < 0x800000 && m != 0) return (double)f;  // subnormal
    return __hiloint2double((b & 0x80000000) | (m == 0 ? 0 : (m >> 3) + ((1023 - 127) << 20)), b << 29);
}
// (float)x, rounded to nearest even
__device__ __forceinline__ float x_to_float_rn(double x) {
    const int hi = __double2hiint(x), lo = __double2loint(x);
    if (!x_ok(hi & 0x7fffffff)) return (float)x;
    const unsigned f = __funnelshift_l(lo, (hi & 0x7fffffff) - ((1023 - 127) << 20), 3);
    const unsigned up = ((lo & 0x1fffffffu) + 0x0fffffffu + (f & 1u)) >> 29;
    return __int_as_float((int)((f + up) | (hi & 0x80000000)));
}

// hi = (float)x, lo = (float)(x - hi), both rounded to nearest even: with x = +-(1.m) 2^e the
// remainder is an integer of at most 29 bits times 2^(e - 52), so one integer conversion rounds it.
static __device__ __noinline__ float2 x_native_split(double x) {
    const float hi = (float)x;
    return make_float2(hi, (float)(x - (double)hi));
}
__device__ __forceinline__ void x_split(double x, float &hi, float &lo) {
    const int h = __double2hiint(x), l = __double2loint(x), m = h & 0x7fffffff;
    const int e = (m >> 20) - 1023;
    if ((unsigned)(e + 70) > 170u) {  // out of range (zeros too): lo may be subnormal, hi infinite
        const float2 s = x_native_split(x);
        hi = s.x;
        lo = s.y;
        return;
    }
    const unsigned f = __funnelshift_l(l, m - ((1023 - 127) << 20), 3);
    const int rest = l & 0x1fffffff, up = (int)(((unsigned)rest + 0x0fffffffu + (f & 1u)) >> 29);
    const int k = rest - (up << 29);
    hi = __int_as_float((int)((f + up) | (h & 0x80000000)));
    lo = (float)(h < 0 ? -k : k) * __int_as_float((e - 52 + 127) << 23);
}

__device__ __forceinline__ double x_half(double a) {
    const int h = __double2hiint(a);
    if (!x_ok(h & 0x7fffffff)) return 0.5 * a;
    return __hiloint2double(h - 0x100000, __double2loint(a));
}

// ---- any operands: the exact forms above where they apply, else the native operation (out of
// line).  xdiv and xsqrt give the bits of a / b and sqrt(x).
static __device__ __noinline__ double x_native_div(double a, double b) { return a / b; }
static __device__ __noinline__ double x_native_sqrt(double x) { return sqrt(x); }

__device__ __forceinline__ double xdiv(double a, double b) {
    const int ah = __double2hiint(a), bh = __double2hiint(b);
    const int am = ah & 0x7fffffff, bm = bh & 0x7fffffff;
    bool bad = !x_ok(am) || !x_ok(bm);
    const double q = x_div(x_num(__hiloint2double(am, __double2loint(a))), __hiloint2double(bm, __double2loint(b)), bad);
    if (bad) return x_native_div(a, b);
    return __hiloint2double(__double2hiint(q) | ((ah ^ bh) & 0x80000000), __double2loint(q));
}
__device__ __forceinline__ double xsqrt(double x) {
    bool bad = !x_ok(__double2hiint(x));
    const double s = x_sqrt(x, bad);
    return bad ? x_native_sqrt(x) : s;
}

// The same out of line, for code with many of them that few warps run once per pass (the
// recursion's kicks and checks, the universal-variable drift): its instructions come late, and
// one copy stays in the instruction cache (recursion kick 5.2k -> 4.7k cycles; the drift's main
// branch, one long chain per body, is faster inline).
static __device__ __noinline__ double xdiv_call(double a, double b) { return xdiv(a, b); }
static __device__ __noinline__ double xsqrt_call(double x) { return xsqrt(x); }
static __device__ __noinline__ double rsqrt_call(double x) { return rsqrt(x); }
static __device__ __noinline__ double x_native_mul(double a, double b) { return a * b; }
__device__ __forceinline__ double xmul(double a, double b) {
    const int ah = __double2hiint(a), bh = __double2hiint(b);
    const int am = ah & 0x7fffffff, bm = bh & 0x7fffffff;
    if (!x_ok(am) || !x_ok(bm)) return x_native_mul(a, b);
    const double p = x_mul(__hiloint2double(am, __double2loint(a)), __hiloint2double(bm, __double2loint(b)));
    return __hiloint2double(__double2hiint(p) | ((ah ^ bh) & 0x80000000), __double2loint(p));
}

// Additions as fma(a, 1, b), the same rounding: DFMA takes the FP64 pipe for 16 cycles, DADD
// for 19 (the factor sits in constant memory so that the compiler does not fold it).
static __constant__ double x_one = 1.0;
static __constant__ double x_minus_one = -1.0;
__device__ __forceinline__ double xadd(double a, double b) { return fma(a, x_one, b); }
__device__ __forceinline__ double xsub(double a, double b) { return fma(b, x_minus_one, a); }

// a < b, a > b for a, b >= 0 (b finite), without an FP64 compare; false for NaN
__device__ __forceinline__ bool x_less(double a, double b) {
    return (unsigned long long)__double_as_longlong(a) < (unsigned long long)__double_as_longlong(b);
}
__device__ __forceinline__ bool x_greater(double a, double b) {
    const unsigned long long u = __double_as_longlong(a);
    return u > (unsigned long long)__double_as_longlong(b) && u <= 0x7ff0000000000000ull;
}
__device__ __forceinline__ double x_abs(double a) {
    return __hiloint2double(__double2hiint(a) & 0x7fffffff, __double2loint(a));
}
// A double whose operators are the functions above: an expression in xd has the bits of the
// same expression in double (compiled without contraction).  INTMUL: products by x_mul too (9
// cycles of the integer pipes against 16 of the FP64 pipe, but 26 instructions more to fetch
// and a longer chain: for kernels that fill the GPU).
template <bool INTMUL>
struct xd {
    double v;
    __device__ __forceinline__ xd() {}
    __device__ __forceinline__ xd(double x) : v(x) {}
    friend __device__ __forceinline__ xd operator+(xd a, xd b) { return xadd(a.v, b.v); }
    friend __device__ __forceinline__ xd operator-(xd a, xd b) { return xsub(a.v, b.v); }
    friend __device__ __forceinline__ xd operator*(xd a, xd b) { return INTMUL ? xmul(a.v, b.v) : a.v * b.v; }
    friend __device__ __forceinline__ xd operator/(xd a, xd b) { return xdiv(a.v, b.v); }
    friend __device__ __forceinline__ xd root(xd a) { return xsqrt(a.v); }
    __device__ __forceinline__ xd operator-() const {
        return __hiloint2double(__double2hiint(v) ^ 0x80000000, __double2loint(v));
    }
};

}  // namespace swg
