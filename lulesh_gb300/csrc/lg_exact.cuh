// lg_exact.cuh -- IEEE division and square root on the integer pipes.
//
// The strict build's quotients and roots are the IEEE ones (round to nearest
// even), and GB300's FP64 pipe pays 5 instructions for a reciprocal, 8 for a
// quotient and about 10 for a root, at 2 lanes per SM and clock.  Here a 60-bit
// approximation on the integer pipes (lg_fixed_eos.cuh's reciprocal and root, off by
// at most 2^-57) gives a 53-bit candidate that is off by at most one unit, and
// the exact remainder, which fits 64 bits, decides: 50 to 90 integer instructions
// at 128 lanes.  Neither a quotient nor a root of 53-bit numbers can lie halfway
// between two of them, so no tie has to be broken.  Operands or results outside
// the normal range take the hardware's operation, out of line.
#pragma once

#include "lg_fixed_eos.cuh"

namespace lg {
namespace fx {

#ifdef __CUDACC__
#define LG_FX_SLOW static __device__ __noinline__
LG_FX_SLOW double slow_div(double a, double b) { return a / b; }
LG_FX_SLOW double slow_sqrt(double a) { return sqrt(a); }
#endif
LG_FX double general_div(double a, double b)
{
#ifdef __CUDA_ARCH__
    return slow_div(a, b);
#else
    return a / b;
#endif
}
LG_FX double general_sqrt(double a)
{
#ifdef __CUDA_ARCH__
    return slow_sqrt(a);
#else
    return std::sqrt(a);
#endif
}

#ifdef __CUDACC__
LG_FX_SLOW double slow_mul(double a, double b) { return a * b; }
#endif
// a 2^K by the exponent field; zeros as they are
template <int K>
LG_FX double times_pow2(double a)
{
    const double f = K < 0 ? 1.0 / (1 << (K < 0 ? -K : 0)) : (double)(1 << (K < 0 ? 0 : K));
    const int e = expo(a);
    if (e == 0 && (bits(a) << 1) == 0) return a;
    if (e < 1 + (K < 0 ? -K : 0) || e > 2046 - (K > 0 ? K : 0)) {
#ifdef __CUDA_ARCH__
        return slow_mul(a, f);
#else
        return a * f;
#endif
    }
    return from_bits(bits(a) + ((u64)(i64)K << 52));
}

// q + (-1, 0 or 1) so that |2 r| <= d for the remainder r of q
LG_FX u64 adjust(u64 q, i64 r, i64 d)
{
    if (2 * r > d) ++q;
    if (2 * r < -d) --q;
    return q;
}

// 1 / b
LG_FX double exact_rcp(double b)
{
    const u64 m = significand(b);
    const int e = expo(b);
    if (e < 1 || e > 2044) return general_div(1.0, b);
    // 1 / m in (1/2, 1]: 53 bits in units of 2^-105
    u64 q = (u64)(reciprocal((i64)(m << 7)) + 64) >> 7;
    q = adjust(q, -(i64)(q * m), (i64)m);
    // q = 2^53 for a power of two carries into the exponent; the hidden bit
    // of q adds 1
    return from_bits((bits(b) & 0x8000000000000000ull) + ((u64)(unsigned)(2044 - e) << 52) + q);
}

// a / b
LG_FX double exact_div(double a, double b)
{
    const u64 sign = (bits(a) ^ bits(b)) & 0x8000000000000000ull;
    const int ea = expo(a), eb = expo(b);
    const bool zero = (bits(a) << 1) == 0;
    const int e = ea - eb;
    if (eb < 1 || eb > 2046 || ea > 2046 || (!zero && (ea < 1 || e < -1020 || e > 1020)))
        return general_div(a, b);
    const u64 ma = significand(a), mb = significand(b);
    const int lt = ma < mb;
    // ma / mb in units of 2^-60, then 53 bits of it
    Acc p = acc0<4>();
    mac(p, split((i64)(ma << 7)), split(reciprocal((i64)(mb << 7))));
    // ma 2^7 (y 2^-60 2^-59 2^7...): units of 2^-59
    const u64 w = (u64)value<4>(p);
    u64 q = lt ? (w + 32) >> 6 : (w + 64) >> 7;
    const i64 r = (i64)((ma << (52 + lt)) - q * mb);
    q = adjust(q, r, (i64)mb);
    return from_bits(sign | (zero ? 0 : ((u64)(unsigned)(e - lt + 1022) << 52) + q));
}

// sqrt(a) for a >= 0
LG_FX double exact_sqrt(double a)
{
    const int e = expo(a);
    if (e < 1 || e > 2046 || (i64)bits(a) < 0) return general_sqrt(a);
    const u64 m = significand(a);
    const int odd = (e - 1075) & 1;  // a = m 2^(e - 1075)
    // sqrt(m 2^(52 + odd)) is in [2^52, 2^53)
    const Num s = root(num((i64)m, 52 + odd));  // 60 bits, unit 2^s.e (about -7)
    u64 q = (u64)((s.m + ((i64)1 << (-s.e - 1))) >> -s.e);
    const i64 r = (i64)((m << (52 + odd)) - q * q);
    // (q + 1/2)^2 = q^2 + q + 1/4
    if (r > (i64)q) ++q;
    if (r <= -(i64)q) --q;
    return from_bits(((u64)(unsigned)((e - 1075 - odd - 52) / 2 + 1074) << 52) + q);
}

// A factor of rounded products: h:l the 53-bit significand (0 for a zero), e the
// sign and the exponent field in their places.
struct Factor {
    unsigned h, l, e;
};
// bad gets bits of a value that is neither zero nor within 2^-510 .. 2^511
// (products of two values within stay normal)
LG_FX Factor factor(double a, unsigned &bad)
{
    const unsigned ah = (unsigned)(bits(a) >> 32), al = (unsigned)bits(a);
    const unsigned t = ah & 0x7fffffffu;
    const bool in = t - 0x20100000u < 0x3fe00000u;
    bad |= in ? 0u : t | al;
    Factor f;
    f.h = in ? (ah & 0xfffffu) | 0x100000u : 0u;
    f.l = al;
    f.e = ah & 0xfff00000u;
    return f;
}
LG_FX u64 umad(unsigned a, unsigned b, u64 c)
{
#ifdef __CUDA_ARCH__
    u64 d;
    asm("{ .reg .u64 t; mul.wide.u32 t, %1, %2; add.u64 %0, t, %3; }"
        : "=l"(d)
        : "r"(a), "r"(b), "l"(c));
    return d;
#else
    return (u64)a * b + c;
#endif
}
// a b rounded to nearest even: 22 integer instructions, where the FP64 pipe is
// occupied for 64 clocks by each warp's multiplication
LG_FX double product(Factor a, Factor b)
{
    // the product of 105 or 106 bits in words w3 : w2 : w1 : w0
    const u64 low = (u64)a.l * b.l, high = (u64)a.h * b.h;
    const u64 mid = umad(a.l, b.h, (u64)a.h * b.l);
    const unsigned w0 = (unsigned)low;
    unsigned w1, w2, w3;
#ifdef __CUDA_ARCH__
    asm("add.cc.u32 %0, %3, %4; addc.cc.u32 %1, %5, %6; addc.u32 %2, %7, 0;"
        : "=r"(w1), "=r"(w2), "=r"(w3)
        : "r"((unsigned)(low >> 32)), "r"((unsigned)mid), "r"((unsigned)(mid >> 32)),
          "r"((unsigned)high), "r"((unsigned)(high >> 32)));
#else
    const u64 m1 = mid + (low >> 32), top = high + (m1 >> 32);
    w1 = (unsigned)m1;
    w2 = (unsigned)top;
    w3 = (unsigned)(top >> 32);
#endif
    // moved up by 11 or 12 it is q : r : rest with q of 53 bits
    const bool up = (w3 & 0x200u) != 0;
    const int sh = up ? 11 : 12;
    const unsigned qh = funnel(w3, w2, sh), ql = funnel(w2, w1, sh), r = funnel(w1, w0, sh);
    // r = 2^31 rounds up if a bit below is set (of w0: those of its bits that went
    // into r are zero then) or q is odd
    const unsigned half = (w0 | (ql & 1)) != 0 ? 0x80000000u : 0x7fffffffu;
    // modulo 2^32: the signs' sum is their exclusive or, the fields' less 1,024 or 1,023
    // is below 2,048
    const unsigned e = a.e + b.e - (up ? 0x3ff00000u : 0x40000000u);
    unsigned lo, hi;
#ifdef __CUDA_ARCH__
    asm("{ .reg .u32 t; add.cc.u32 t, %2, %3; addc.cc.u32 %0, %4, 0; addc.u32 %1, %5, %6; }"
        : "=r"(lo), "=r"(hi)
        : "r"(r), "r"(half), "r"(ql), "r"(qh), "r"(e));
#else
    const u64 q = ((u64)qh << 32 | ql) + (((u64)r + half) >> 32);
    lo = (unsigned)q;
    hi = (unsigned)(q >> 32) + e;
#endif
    return from_bits((u64)(qh ? hi : (a.e ^ b.e) & 0x80000000u) << 32 | lo);
}

// a b of any two doubles
LG_FX double exact_mul(double a, double b)
{
    unsigned bad = 0;
    const double r = product(factor(a, bad), factor(b, bad));
#ifdef __CUDA_ARCH__
    return bad ? slow_mul(a, b) : r;
#else
    return bad ? a * b : r;
#endif
}

}  // namespace fx
}  // namespace lg
