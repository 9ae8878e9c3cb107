// lg_fixed.cuh -- 64-bit fixed-point arithmetic on the integer pipes.
//
// GB300 issues 2 FP64 lanes per SM and clock (1.9 measured) against 64 lanes of
// 32 x 32 + 64 -> 64 multiply-adds (58.6 measured) and 128 of 32-bit adds, and
// the pipes run side by side.  A product of two 64-bit fixed-point numbers is
// three such multiply-adds, a sum two 32-bit adds, so work whose operands share a
// known scale costs an order of magnitude less here than on the FP64 pipe, at
// 59 or 60 bits of the largest operand instead of 53 of each.
//
//   Op    a number v = h 2^32 + l with both halves signed (|l| <= 2^31), so that
//         every partial product is a signed 32 x 32 multiply;
//   Acc   a sum of products: hh collects h h', hl the two cross terms; the l l'
//         terms lie 2^-64 below h h' 2^64 and are left out (at most 1/4 of the
//         unit of hh for each product, mean 0).
//
// Bounds are stated at each use: |h| < 2^(n - 32) for |v| < 2^n.  Everything is
// host code too (the tests evaluate it beside extended precision).
#pragma once

#include <cmath>
#include <cstdint>
#include <cstring>

#include "lg_geometry.cuh"

#ifdef __CUDACC__
#define LG_FX __host__ __device__ __forceinline__
#else
#define LG_FX inline
#endif

namespace lg {
namespace fx {

typedef long long i64;
typedef unsigned long long u64;

struct alignas(8) Op {
    int h, l;
};
struct Acc {
    i64 hh, hl;
};

LG_FX i64 shl(i64 v, int n) { return (i64)((u64)v << n); }

LG_FX Op split(i64 v)
{
    Op o;
    o.l = (int)(unsigned)(u64)v;
    o.h = (int)(v >> 32) + (int)((unsigned)o.l >> 31);
    return o;
}

LG_FX i64 join(Op o) { return shl(o.h, 32) + o.l; }

// a sum of products whose result is taken by value<K>
template <int K>
LG_FX Acc acc0()
{
    Acc a;
    a.hh = 0;
    a.hl = (i64)1 << (31 - K);  // rounds the cross terms' share to nearest
    return a;
}
// a b + c in one instruction (written out: the compiler splits the sums of
// several products into products and additions)
LG_FX i64 mad(int a, int b, i64 c)
{
#ifdef __CUDA_ARCH__
    i64 d;
    asm("{ .reg .s64 t; mul.wide.s32 t, %1, %2; add.s64 %0, t, %3; }"
        : "=l"(d)
        : "r"(a), "r"(b), "l"(c));
    return d;
#else
    return (i64)a * b + c;
#endif
}
LG_FX void mac(Acc &a, Op x, Op y)
{
    a.hh = mad(x.h, y.h, a.hh);
    a.hl = mad(x.h, y.l, a.hl);
    a.hl = mad(x.l, y.h, a.hl);
}
// the sum / 2^(64 - K)
template <int K>
LG_FX i64 value(const Acc &a)
{
    return shl(a.hh, K) + (a.hl >> (32 - K));
}

// (a b - c d) / 2^(64 - K)
template <int K = 0>
LG_FX i64 det2(Op a, Op b, Op c, Op d)
{
    Acc p = acc0<K>(), q;
    q.hh = q.hl = 0;
    mac(p, a, b);
    mac(q, c, d);
    p.hh -= q.hh;
    p.hl -= q.hl;
    return value<K>(p);
}

LG_FX u64 bits(double v)
{
#ifdef __CUDA_ARCH__
    return (u64)__double_as_longlong(v);
#else
    u64 b;
    std::memcpy(&b, &v, sizeof b);
    return b;
#endif
}
LG_FX double from_bits(u64 b)
{
#ifdef __CUDA_ARCH__
    return __longlong_as_double((i64)b);
#else
    double v;
    std::memcpy(&v, &b, sizeof v);
    return v;
#endif
}
LG_FX int clz64(u64 v)  // 64 for 0
{
#ifdef __CUDA_ARCH__
    return __clzll((i64)v);
#else
    return v ? __builtin_clzll(v) : 64;
#endif
}
LG_FX int clz32(unsigned v)  // 32 for 0
{
#ifdef __CUDA_ARCH__
    return __clz((int)v);
#else
    return v ? __builtin_clz(v) : 32;
#endif
}
// the upper word of (h : l) 2^sh, 0 < sh < 32
LG_FX unsigned funnel(unsigned h, unsigned l, int sh)
{
#ifdef __CUDA_ARCH__
    return __funnelshift_l(l, h, sh);
#else
    return h << sh | l >> (32 - sh);
#endif
}
// float -> double on the integer pipe, for normal numbers
LG_FX double widen(float f)
{
    unsigned u;
#ifdef __CUDA_ARCH__
    u = __float_as_uint(f);
#else
    std::memcpy(&u, &f, sizeof u);
#endif
    const unsigned hi = (u & 0x80000000u) | (((u & 0x7fffffffu) >> 3) + (896u << 20));
    return from_bits(((u64)hi << 32) | (u << 29));
}
LG_FX int imin(int a, int b) { return a < b ? a : b; }
LG_FX int imax(int a, int b) { return a > b ? a : b; }

// biased exponent of a double
LG_FX int expo(double v) { return (int)(bits(v) >> 52) & 0x7ff; }
// largest of |v|'s upper word and m (an order of the exponents)
LG_FX int top_word(int m, double v) { return imax(m, (int)(bits(v) >> 32) & 0x7fffffff); }
// signed 53-bit significand (a normal number's; 0 and subnormals get the hidden bit too)
LG_FX u64 significand(double v)
{
    return (bits(v) & 0xfffffffffffffull) | 0x10000000000000ull;
}
// v in units of 2^(emax - 1022 - T), |result| < 2^T, truncated, all on the
// integer pipe (14 instructions; the FP64 pipe's conversion is one instruction
// that occupies it as long as an addition does, and k_forces with 48 of them
// took 928 us at s=150 against 878 with integer conversions).  emax >= 64 is at least v's biased exponent
// (0 and subnormals give 0)
template <int T>
LG_FX i64 fixed_int(double v, int emax)
{
    const u64 m = (significand(v) << (T - 53)) >> imin(emax - expo(v), 63);
    const i64 s = (i64)bits(v) >> 63;
    return ((i64)m ^ s) - s;
}
// r 2^e as a double, rounded to nearest, for |e| <= 900
LG_FX double real_of(i64 r, int e)
{
    const u64 b = bits((double)r);
    return from_bits(r == 0 ? 0 : b + ((u64)(i64)e << 52));
}
// 1 / d, d^(-1/3) and (below) d^(-1/2) and a / b for positive d and b in FP32's normal
// range, which the caller checks (seedable): an FP32 seed of about 21 bits and one
// third-order Householder step, 3 to 6 FP64 instructions.  The step's residual is exact
// but for its own last bit (the seed's square has 48 bits), so the results are off
// by one rounding, the cube root's by 1.4.
LG_FX bool seedable(double d)
{
    const int h = (int)(bits(d) >> 52);  // 2^-123 to 2^123
    return h >= 900 && h <= 1146;
}
LG_FX double recip(double d)
{
    const float f = geom::f32_trunc(d);
#ifdef __CUDA_ARCH__
    float y32;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y32) : "f"(f));
#else
    const float y32 = 1.0f / f;
#endif
    const double y = widen(y32);
    const double r = fma(-d, y, 1.0);
    return fma(y, fma(r, r, r), y);
}
// the product's quotient corrected by its residual
LG_FX double quotient(double a, double b)
{
    const double r = recip(b), q = a * r;
    return fma(fma(-b, q, a), r, q);
}
LG_FX double recip_cbrt(double d)
{
    const float f = geom::f32_trunc(d);
#ifdef __CUDA_ARCH__
    float l, y32;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(l) : "f"(f));
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(y32) : "f"(l * (-1.0f / 3.0f)));
#else
    const float y32 = powf(f, -1.0f / 3.0f);
#endif
    const double y = widen(y32);
    const double r = fma(-d, y * y * y, 1.0);
    return fma(y * r, fma(2.0 / 9.0, r, 1.0 / 3.0), y);
}

// a^(-1/2), as recip
LG_FX double recip_sqrt(double a)
{
    const float f = geom::f32_trunc(a);
#ifdef __CUDA_ARCH__
    float y32;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y32) : "f"(f));
#else
    const float y32 = 1.0f / sqrtf(f);
#endif
    const double y = widen(y32);
    const double r = fma(-a, y * y, 1.0);
    return fma(y * r, fma(0.375, r, 0.5), y);
}

// whether b holds in a lane that runs along
LG_FX bool any_lane(bool b)
{
#ifdef __CUDA_ARCH__
    return __any_sync(__activemask(), b);
#else
    return b;
#endif
}

// collects the bits of |v|'s upper half (one's complement of a negative v)
LG_FX void magnitude(int &mag, i64 v)
{
    const int h = (int)(v >> 32);
    mag |= h ^ (h >> 31);
}

// The sum of eight doubles, each in units of 2^-59 of the largest; false where
// an exponent is out of range (the caller sums in FP64)
LG_FX bool sum_of(const double v[8], double &sum)
{
    int top = 200 << 20;
#pragma unroll
    for (int i = 0; i < 8; ++i) top = top_word(top, v[i]);
    const int emax = top >> 20;
    i64 s = 0;
#pragma unroll
    for (int i = 0; i < 8; ++i) s += fixed_int<59>(v[i], emax);
    sum = real_of(s, emax - 1081);
    return emax <= 1900;
}

}  // namespace fx
}  // namespace lg
