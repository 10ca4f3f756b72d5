// tm_f64.cuh -- correctly rounded binary64 multiply, divide and square root in
// 32-bit integer arithmetic.
//
// GB300's FP64 pipe takes one warp instruction per 64-76 cycles and scheduler
// (measured; one lane or 32, multiply, add or fused alike), a divide or a square
// root several of them (344 and 572 cycles), while integer and FP32 instructions
// issue every cycle or two.  The FP64 kernels are bound by that pipe alone (83 %
// busy at 7 % of the issue slots), so the operations below compute the same IEEE
// results -- round to nearest even, bit for bit -- on the integer pipe: mantissa
// products and exact remainders, with the FP32 reciprocal units for first
// estimates that the remainders correct.  Operands or results outside the normal
// range (zeros, subnormals, infinities, NaN) take the hardware instruction.
//
// The header also compiles for the host (the tests compare it there with the
// host's own arithmetic).
#pragma once
#include <stdint.h>
#include <string.h>

#ifdef __CUDACC__
#define TM_HD __host__ __device__ __forceinline__
#else
#define TM_HD static inline
#endif

namespace tmf {

constexpr uint64_t kFrac = 0x000fffffffffffffULL, kOne = 0x0010000000000000ULL, kSign = 0x8000000000000000ULL;

TM_HD uint64_t f64_bits(double x)
{
#ifdef __CUDA_ARCH__
    return (uint64_t)__double_as_longlong(x);
#else
    uint64_t u;
    memcpy(&u, &x, 8);
    return u;
#endif
}
TM_HD double bits_f64(uint64_t u)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((long long)u);
#else
    double x;
    memcpy(&x, &u, 8);
    return x;
#endif
}
TM_HD uint32_t umulhi32(uint32_t a, uint32_t b)
{
#ifdef __CUDA_ARCH__
    return __umulhi(a, b);
#else
    return (uint32_t)(((uint64_t)a * b) >> 32);
#endif
}
TM_HD int f64_exp_field(uint64_t u) { return (int)((uint32_t)(u >> 52) & 0x7ffu); }
// exponent field of a normal number
TM_HD bool field_normal(int e) { return (uint32_t)(e - 1) < 2046u; }

TM_HD uint32_t f32_bits(float x)
{
#ifdef __CUDA_ARCH__
    return __float_as_uint(x);
#else
    uint32_t u;
    memcpy(&u, &x, 4);
    return u;
#endif
}
TM_HD float bits_f32(uint32_t u)
{
#ifdef __CUDA_ARCH__
    return __uint_as_float(u);
#else
    float x;
    memcpy(&x, &u, 4);
    return x;
#endif
}

// FP32 estimates of 1/x and 1/sqrt(x), within 2^-21 relative
TM_HD float est_rcp(float x)
{
#ifdef __CUDA_ARCH__
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / x;
#endif
}
TM_HD float est_rsqrt(float x)
{
#ifdef __CUDA_ARCH__
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
#else
    return 1.0f / __builtin_sqrtf(x);
#endif
}
// The hardware operations, for operands or results outside the normal range.  As
// volatile assembly they stay behind their branch.
TM_HD double hw_mul(double a, double b)
{
#ifdef __CUDA_ARCH__
    double r;
    asm volatile("mul.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
    return r;
#else
    return a * b;
#endif
}
TM_HD double hw_div(double a, double b)
{
#ifdef __CUDA_ARCH__
    double r;
    asm volatile("div.rn.f64 %0, %1, %2;" : "=d"(r) : "d"(a), "d"(b));
    return r;
#else
    return a / b;
#endif
}
TM_HD double hw_sqrt(double a)
{
#ifdef __CUDA_ARCH__
    double r;
    asm volatile("sqrt.rn.f64 %0, %1;" : "=d"(r) : "d"(a));
    return r;
#else
    return __builtin_sqrt(a);
#endif
}

// ---------------------------------------------------------------- multiply
// Product of two normal numbers, by their bits; e is the exponent field of the
// result (which the caller checks lies in 1..2046 after rounding).
TM_HD uint64_t mul_core(uint64_t ua, uint64_t ub, int& e)
{
    const uint64_t A = ((ua & kFrac) | kOne) << 11, B = ((ub & kFrac) | kOne) << 1;
    // 128-bit product in [2^116, 2^118): the high word holds the 53 or 54 leading bits
    const uint32_t a0 = (uint32_t)A, a1 = (uint32_t)(A >> 32), b0 = (uint32_t)B, b1 = (uint32_t)(B >> 32);
    const uint64_t p00 = (uint64_t)a0 * b0;
    const uint64_t p01 = (uint64_t)a0 * b1 + (p00 >> 32);
    const uint64_t p10 = (uint64_t)a1 * b0 + (uint32_t)p01;
    uint64_t hi = (uint64_t)a1 * b1 + (p01 >> 32) + (p10 >> 32);
    uint64_t lo = (p10 << 32) | (uint32_t)p00;
    const uint32_t up = (uint32_t)(hi >> 53);       // one bit too many: drop it (the product's low 12 bits are 0)
    lo = up ? (lo >> 1) | (hi << 63) : lo;
    hi >>= up;
    e += (int)up;
    // nearest, ties to even: carry out of lo + (2^63 - 1) + (hi & 1)
    const uint64_t t = lo + (0x7fffffffffffffffULL + (hi & 1u));
    hi += (t < lo) ? 1u : 0u;
    return ((uint64_t)(uint32_t)(e - 1) << 52) + hi;     // the leading 1 (or a carry) adds to the exponent
}

// a b for operands and a result known to be normal
TM_HD double mul_normal(double a, double b)
{
    const uint64_t ua = f64_bits(a), ub = f64_bits(b);
    int e = f64_exp_field(ua) + f64_exp_field(ub) - 1023;
    const uint64_t r = mul_core(ua, ub, e);
    return bits_f64(r | ((ua ^ ub) & kSign));
}

// a b for any operands (a zero with a finite operand, common on empty lattices, stays
// on the integer pipe)
TM_HD double mul(double a, double b)
{
    const uint64_t ua = f64_bits(a), ub = f64_bits(b);
    const int ea = f64_exp_field(ua), eb = f64_exp_field(ub);
    int e = ea + eb - 1023;
    if (!(field_normal(ea) && field_normal(eb) && (uint32_t)(e - 2) < 2042u)) {
        if (((ua << 1) == 0 || (ub << 1) == 0) && ea < 2047 && eb < 2047) return bits_f64((ua ^ ub) & kSign);
        return hw_mul(a, b);
    }
    const uint64_t r = mul_core(ua, ub, e);
    return bits_f64(r | ((ua ^ ub) & kSign));
}

// ---------------------------------------------------------------- divide
// Reciprocal of a mantissa mb in [2^52, 2^53): R ~ 2^31 / (mb 2^-53), below it by
// at most 16.  An FP32 estimate and one Newton step in 32-bit fixed point.
TM_HD uint32_t recip31(uint64_t mb)
{
    const uint32_t dh = (uint32_t)(mb >> 21);                       // [2^31, 2^32)
    // the estimate's argument lies 2^-22 above the truncated divisor, so the
    // estimate stays below 1; both are kept inside the binade
    uint32_t fb = 0x3f800002u + ((dh >> 8) & 0x7fffffu);
    fb = fb < 0x3fffffffu ? fb : 0x3fffffffu;
    uint32_t rb = f32_bits(est_rcp(bits_f32(fb)));
    rb = rb > 0x3f000000u ? rb : 0x3f000000u;
    const uint32_t r0 = ((rb & 0x7fffffu) | 0x800000u) << 8;
    const int32_t delta = (int32_t)(0x80000000u - umulhi32(r0, dh));   // |delta| < 2^11
    const int32_t corr = (int32_t)(((int64_t)(int32_t)(r0 >> 1) * delta) >> 30);
    return r0 + (uint32_t)(corr - 8);
}

// a / b from their bits and b's reciprocal (recip31): 54 quotient bits in two
// digits with exact 64-bit remainders.  An exact tie cannot occur (a 54-bit odd
// quotient times mb exceeds any shifted ma), so one guard bit rounds.
TM_HD uint64_t div_core(uint64_t ua, uint64_t ub, uint32_t R, int& e)
{
    const uint64_t ma = (ua & kFrac) | kOne, mb = (ub & kFrac) | kOne;
    const bool ge = ma >= mb;
    const uint64_t D = mb << 6;                                     // [2^58, 2^59)
    const uint64_t N = ge ? ma << 5 : ma << 6;                       // N < D, N / D in [1/2, 1)
    if (!ge) e -= 1;
    const uint32_t t = umulhi32((uint32_t)(N >> 27), R);             // N / D 2^31, low by < 16
    const uint64_t r1 = (N << 31) - (uint64_t)t * D;                 // < 16 D < 2^63
    uint32_t q2 = umulhi32((uint32_t)(r1 >> 31), R) >> 4;            // r1 / D 2^23, low by at most 1
    const uint64_t r2 = (r1 << 23) - (uint64_t)q2 * D;
    q2 += (r2 >= D) ? 1u : 0u;
    const uint64_t Q = ((uint64_t)t << 23) + q2;                     // [2^53, 2^54)
    return ((uint64_t)(uint32_t)(e - 1) << 52) + ((Q + 1) >> 1);
}

TM_HD bool div_fields_ok(int ea, int eb)
{
    return field_normal(ea) && field_normal(eb) && (uint32_t)(ea - eb + 1023 - 2) < 2043u;
}

// a / b with b's reciprocal R where b is normal
TM_HD double div_by(double a, double b, uint32_t R)
{
    const uint64_t ua = f64_bits(a), ub = f64_bits(b);
    const int ea = f64_exp_field(ua), eb = f64_exp_field(ub);
    if (!div_fields_ok(ea, eb)) {
        if ((ua << 1) == 0 && field_normal(eb)) return bits_f64((ua ^ ub) & kSign);
        return hw_div(a, b);
    }
    int e = ea - eb + 1023;
    const uint64_t r = div_core(ua, ub, R, e);
    return bits_f64(r | ((ua ^ ub) & kSign));
}
TM_HD uint32_t recip_of(double b) { return recip31((f64_bits(b) & kFrac) | kOne); }

// a / b for any operands
TM_HD double div(double a, double b) { return div_by(a, b, recip_of(b)); }

// ---------------------------------------------------------------- square root
// sqrt of a positive normal number: a 32-bit root from the FP32 estimate and one
// Newton step, its exact remainder, 22 more bits from it, and a correction by the
// sign of the final remainder.  No tie can occur (an odd 54-bit root squares to
// an odd 107-bit number).
TM_HD uint64_t sqrt_core(uint64_t u)
{
    const int e = f64_exp_field(u) - 1023;
    const int odd = e & 1;
    const uint64_t X = ((u & kFrac) | kOne) << (10 + odd);           // M 2^62, M in [1, 4)
    const uint32_t mh = (uint32_t)(X >> 32);                         // M 2^30
    const float est = est_rsqrt(bits_f32(((uint32_t)(127 + odd) << 23) | ((uint32_t)(u >> 29) & 0x7fffffu)));
    const uint32_t fb = f32_bits(est);
    uint32_t y0 = ((fb & 0x7fffffu) | 0x800000u) << ((fb >> 23) - 119);   // y 2^31, y = 1/sqrt(M)
    y0 -= y0 >> 20;                                                  // below 1/sqrt(M): Newton stays below
    const uint32_t s0 = (uint32_t)(((uint64_t)mh * y0) >> 30);       // M y 2^31 < 2^32
    const int32_t d = (int32_t)(0x40000000u - umulhi32(s0, y0));     // (1 - M y^2) 2^30
    const uint32_t y = y0 + (uint32_t)(int32_t)(((int64_t)(int32_t)(y0 >> 1) * d) >> 30) - 4u;
    const uint32_t s1 = (uint32_t)(((uint64_t)mh * y) >> 30);        // sqrt(M) 2^31, low by < 32
    const uint64_t r1 = X - (uint64_t)s1 * s1;                       // < 2^38
    // r1 2^22 / (2 s1) = r1 y 2^-41, at most 1 off
    const uint32_t q = umulhi32((uint32_t)(r1 >> 6), y) >> 3;
    uint64_t S = ((uint64_t)s1 << 22) + q;
    const int64_t r2 = (int64_t)((r1 << 44) - (uint64_t)q * (((uint64_t)s1 << 23) + q));   // X 2^44 - S^2
    if (r2 < 0) S -= 1;
    else if ((uint64_t)r2 > 2 * S) S += 1;
    return ((uint64_t)(uint32_t)(((e - odd) >> 1) + 1022) << 52) + ((S + 1) >> 1);
}

TM_HD double sqrt(double a)
{
    const uint64_t u = f64_bits(a);
    if ((u >> 63) || !field_normal(f64_exp_field(u))) return hw_sqrt(a);
    return bits_f64(sqrt_core(u));
}

// ---------------------------------------------------------------- conversions and tests by bits
// (x + 0.5) 2^-53 of a 53-bit integer, rounded to nearest even as the FP64 sum is
TM_HD double open_unit(uint64_t x)
{
    // the sum has 54 bits from 2^52 on: round half to even there
    uint64_t v = (x >> 52) ? (x + (x & 1u)) << 1 : (x << 1) | 1u;    // 2 (x + 0.5), exact after the rounding
#ifdef __CUDA_ARCH__
    const int lz = __clzll((long long)v);
#else
    const int lz = __builtin_clzll(v);
#endif
    // v = 1.f 2^(63 - lz); the value is v 2^-54
    v <<= lz;
    return bits_f64(((uint64_t)(uint32_t)(1023 + 63 - lz - 54 - 1) << 52) + (v >> 11));
}

// a non-negative integer below 2^31 as binary64
TM_HD double from_u31(uint32_t n)
{
    if (n == 0) return 0.0;
#ifdef __CUDA_ARCH__
    const int lz = __clz((int)n);
#else
    const int lz = __builtin_clz(n);
#endif
    const uint32_t f = n << lz;                                       // leading 1 at bit 31
    return bits_f64(((uint64_t)(((uint32_t)(1023 + 31 - lz - 1) << 20) + (f >> 11)) << 32) | (uint32_t)(f << 21));
}

// nearest-below FP32 of a positive binary64 in FP32's normal range (0 below it)
TM_HD float trunc_f32(double x)
{
    const uint64_t u = f64_bits(x);
    const uint32_t hi = (uint32_t)(u >> 32);
    if (hi < ((uint32_t)897 << 20)) return 0.0f;
    return bits_f32(((hi - ((uint32_t)896 << 20)) << 3) | ((uint32_t)u >> 29));
}

TM_HD bool is_zero(double x) { return (f64_bits(x) << 1) == 0; }
// The sign by its bit (the compiler's own negation and absolute value are FP64 additions).
TM_HD double abs_bits(double x) { return bits_f64(f64_bits(x) & ~kSign); }
TM_HD double with_sign(double x, bool negative) { return bits_f64((f64_bits(x) & ~kSign) | (negative ? kSign : 0)); }
// a < b by the hardware's comparison, kept behind the caller's branch.
TM_HD bool hw_less(double a, double b)
{
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\tsetp.lt.f64 p, %1, %2;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r) : "d"(a), "d"(b));
    return r != 0;
#else
    return a < b;
#endif
}
// x in [lo, hi) by the hardware's comparisons, kept behind the caller's branch.
TM_HD bool hw_in_range(double x, double lo, double hi)
{
#ifdef __CUDA_ARCH__
    uint32_t r;
    asm volatile("{\n\t.reg .pred p, q;\n\tsetp.lt.f64 p, %1, %3;\n\tsetp.ge.and.f64 q, %1, %2, p;\n\t"
                 "selp.u32 %0, 1, 0, q;\n\t}"
                 : "=r"(r) : "d"(x), "d"(lo), "d"(hi));
    return r != 0;
#else
    return x < hi && x >= lo;
#endif
}

}  // namespace tmf
