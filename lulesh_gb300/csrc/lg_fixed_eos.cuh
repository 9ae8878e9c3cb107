// lg_fixed_eos.cuh -- the EOS repetitions of one element on the integer pipes.
//
// EvalEOSForElems' predictor-corrector (lulesh.cc:2048-2324) mixes volumes,
// energies and pressures of any ratio, so its numbers carry an exponent each:
// Num is m 2^e with |m| < 2^60.  Sums align the smaller operand, products keep
// the upper half, and nothing is renormalised: a cancelled sum is off by its
// last bits as it is in FP64, only 2^-58 of its operands instead of 2^-53.
// One repetition is about 620 integer instructions (128 lanes per SM and clock)
// for an element at rest and 830 for a moving one, against 63 and 110 FP64 ones (2
// lanes), which bound the phase: the FMA build's k_material at s=150 (11
// regions, cost 1) 2,137 -> 958 us (716 with the steps noted below and at the kernels),
// the mixed one's at s=192 (16 regions, cost 4) 7,084 -> 2,542 us (2,063).
#pragma once

#include "lg_fixed_geometry.cuh"

namespace lg {
namespace fx {

typedef Scale Num;

LG_FX Num num(i64 m, int e)
{
    Num r;
    r.m = m;
    r.e = e;
    return r;
}
LG_FX Num neg(Num a) { return num(-a.m, a.e); }
LG_FX Num twice(Num a, int n) { return num(a.m, a.e + n); }  // a 2^n
LG_FX Num mul(Num a, Num b)
{
    Acc p = acc0<4>();
    mac(p, split(a.m), split(b.m));
    return num(value<4>(p), a.e + b.e + 60);
}
LG_FX Num add(Num a, Num b)
{
    const int e = imax(a.e, b.e) + 1;
    return num((a.m >> imin(e - a.e, 63)) + (b.m >> imin(e - b.e, 63)), e);
}
// the same number with |m| in [2^59, 2^60)
LG_FX Num norm(Num a)
{
    const int n = clz64((u64)(a.m ^ (a.m >> 63))) - 4;
    return num(shl(a.m, n), a.e - n);
}
// |a| < |b|
LG_FX bool below(Num a, Num b)
{
    const int e = imax(a.e, b.e);
    const i64 s = a.m >> 63;
    return (((a.m ^ s) - s) >> imin(e - a.e, 63)) < (b.m >> imin(e - b.e, 63));
}

// 24 bits of 1 / v and 1 / sqrt(v) for the 24-bit significand v of [1, 2) and [1, 4)
LG_FX unsigned seed(unsigned f, bool root)
{
    float x, y;
    unsigned r;
#ifdef __CUDA_ARCH__
    x = __uint_as_float(f);
    if (root)
        asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    else
        asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    r = __float_as_uint(y);
#else
    std::memcpy(&x, &f, sizeof x);
    y = root ? 1.0f / sqrtf(x) : 1.0f / x;
    std::memcpy(&r, &y, sizeof r);
#endif
    // y in [1/2, 1], which the approximation may leave by its last bit: the
    // significand, in units of 2^-24
    if (r < 0x3f000000u) r = 0x3f000000u;
    return r >= 0x3f800000u ? 0xffffffu : ((r & 0x7fffffu) | 0x800000u);
}

// 1 / (v 2^-59) in units of 2^-60 for v in [2^59, 2^60): the seed's residual is
// exact, and one third-order step leaves 2^-60
LG_FX i64 reciprocal(i64 v)
{
    const unsigned y = seed(0x3f800000u | ((unsigned)(v >> 36) & 0x7fffffu), false);
    const Op o = split(v);
    // 1 - v y, units of 2^-83, |.| < 2^62
    const i64 r = -(shl(mad(o.h, (int)y, 0), 32) + mad(o.l, (int)y, 0));
    const Op q = split(r >> 23);  // 2^-60
    const int t = (int)(r >> 38);  // 2^-45
    const i64 p = shl(mad(q.h, (int)y, 0), 32) + mad(q.l, (int)y, 0);  // 2^-84
    const i64 c = mad((int)(mad(t, t, 0) >> 30), (int)(y >> 8), 0) >> 16;
    return shl((i64)y, 36) + (p >> 24) + c;
}

// sqrt(a) for a > 0 (relative error about 2^-58)
LG_FX Num root(Num a)
{
    const int n = clz64((u64)a.m);          // >= 4
    const int odd = (a.e - n + 1) & 1;
    // x = a 2^-2k in [1, 4), units of 2^-60: top bit 60 or 61 (a split's upper
    // half has to stay below 2^31 when its lower half rounds up)
    const u64 top = (u64)shl(a.m, n & 63);
    const i64 x = (i64)(top >> (3 - odd));
    const unsigned y = seed((0x3f800000u + ((unsigned)odd << 23)) |
                                ((unsigned)(top >> 40) & 0x7fffffu), true);
    const Op o = split(x);
    // s = x y, 2^-60, and its residual x - s^2
    const i64 s = shl(mad(o.h, (int)y, 0), 8) + (mad(o.l, (int)y, 0) >> 24);
    const Op so = split(s);
    Acc sq = acc0<4>();
    mac(sq, so, so);
    const Op r = split(x - value<4>(sq));
    // first order: r y / 2; second: 3/2 y of its square
    const i64 c = shl(mad(r.h, (int)y, 0), 7) + (mad(r.l, (int)y, 0) >> 25);
    const int t = (int)(c >> 16);  // 2^-44
    const int t2 = (int)(mad(t, t, 0) >> 28);  // 2^-60
    const i64 c2 = mad(t2, (int)((y >> 9) + (y >> 10)), 0) >> 15;
    // a = x 2^-60 2^(a.e - n - odd + 63), an even power
    return num((s + c + c2) >> 1, ((a.e - n - odd + 63) >> 1) - 59);
}

// Thresholds of the EOS (positive), as Nums.
struct EosCuts {
    Num e, p, q;
};

// One element's inputs; ok of eos_inputs says whether the repetitions may run
// here.
struct EosIn {
    Num e, p, q, qq, ql, delv, v;
};
LG_FX bool eos_inputs(double e, double delv, double p, double q, double qq, double ql, double v,
                      EosIn &in)
{
    bool ok = true;
    in.e = scale_of(e, ok);
    in.delv = scale_of(delv, ok);
    in.p = scale_of(p, ok);
    in.q = scale_of(q, ok);
    in.qq = scale_of(qq, ok);
    in.ql = scale_of(ql, ok);
    in.v = scale_of(v, ok);
    // v in [2^-28, 2^29), |delv| < v, and magnitudes far from overflow (delv (p + q)
    // can still reach the energy floor: eos_repetition looks)
    const int ev = expo(v);
    ok = ok && in.v.m > 0 && ev >= 995 && ev <= 1051 && expo(delv) < ev;
    return ok && expo(e) <= 1069 && expo(p) <= 1069 && expo(q) <= 1069 && expo(qq) <= 1069 &&
           expo(ql) <= 1069;
}

LG_FX Num cut(Num a, Num eps) { return num(below(a, eps) ? 0 : a.m, a.e); }
// a pressure: below the cut-off or negative (pmin = 0) is 0
LG_FX Num cut_positive(Num a, Num eps)
{
    const int e = imax(a.e, eps.e);
    const bool less = (a.m >> imin(e - a.e, 63)) < (eps.m >> imin(e - eps.e, 63));
    return num(less ? 0 : a.m, a.e);
}
// The sound speed term sqrt(2/3 e + v^2 bvc p) with its floor (lulesh.cc:2083-2090
// and its repetitions, for refdens = 1), bvc = 2/3 / v.  p is bvc e, or 0 where the
// cut-off or pmin took it, so the argument is (2/3 + 4/9) e or 2/3 e: no product
// with v and no sum.  A warp without an element above the floor skips the root.
LG_FX Num sound_speed(Num en, Num p, bool wanted)
{
    // c + c^2 and c for c = 2.0 / 3.0, in units of 2^-59
    const i64 both = 0x8e38e38e38e38b2ll, one = 0x15555555555555ll << 6;
    const Num s = mul(num(p.m > 0 ? both : one, -59), en);
    // above .1111111e-36: by the exponent, then by the significand with its top bit at 63
    // (both of which the root starts from)
    const int n = clz64((u64)s.m), e = s.e - n;
    const bool above =
        s.m > 0 && (e > -186 || (e == -186 && (u64)shl(s.m, n & 63) > 0x973c9151be8d0000ull));
    Num r = num(0xc4c3e773fa1ce80ll, -121);  // .3333333e-18
    if (any_lane(above && wanted)) {
        const Num t = root(s);
        if (above) r = t;
    }
    return r;
}
LG_FX Num viscosity(Num e, Num p, const EosIn &in, bool wanted)
{
    return add(mul(sound_speed(e, p, wanted), in.ql), in.qq);
}

// One repetition of CalcEnergyForElems with CalcPressureForElems, for refdens
// = 1, pmin = 0 and volumes inside the EOS' limits.  False: an energy of 2^49 or
// more (the floor emin, -1e15 or below, is not applied here), or a half-step volume far
// from v.
LG_FX bool eos_repetition(const EosIn &in, const EosCuts &cuts, Num &p3, Num &e3, Num &q3)
{
    const Num c1s = num(0x15555555555555ll << 7, -60);      // 2.0 / 3.0
    const Num sixth = num(-(0x15555555555555ll << 7), -62);  // -1.0 / 6.0
    const bool shrink = in.delv.m <= 0;
    // no viscosity while expanding: a zero at qq's exponent would take the digits of
    // what it is added to
    const Num none = num(0, -5000);
    const Num dh = num(-in.delv.m, in.delv.e - 1), pq = add(in.p, in.q);  // -delv / 2
    // half-step volume, normalised, and both reciprocals
    const i64 w = in.v.m + (dh.m >> imin(in.v.e - dh.e, 63));
    const int n = clz64((u64)w) - 4;  // -1, 0, 1
    const bool half = w > ((i64)1 << 57);
    const i64 vh = shl(w, (n + 1) & 3) >> 1;
    const Num b = mul(c1s, num(reciprocal(in.v.m), -119 - in.v.e));
    const Num bh = mul(c1s, num(reciprocal(vh), n - 119 - in.v.e));

    const Num e1 = add(in.e, mul(dh, pq));
    const Num ph = cut_positive(mul(bh, e1), cuts.p);
    Num q1 = viscosity(e1, ph, in, shrink);
    if (!shrink) q1 = none;
    const Num pq1 = add(ph, q1);
    // -(3 (p + q) - 4 (ph + q1))
    const Num t = add(twice(pq1, 2), num(-((pq.m + shl(pq.m, 1)) >> 2), pq.e + 2));
    const Num e2 = cut(norm(add(e1, mul(dh, norm(t)))), cuts.e);
    const Num p2 = cut_positive(mul(b, e2), cuts.p);
    Num qt = viscosity(e2, p2, in, shrink);
    if (!shrink) qt = none;
    const Num u = add(pq, neg(twice(t, 1)));  // 7 (p + q) - 8 (ph + q1)
    const Num d6 = mul(in.delv, sixth);
    e3 = cut(add(e2, mul(norm(add(u, add(p2, qt))), d6)), cuts.e);
    p3 = cut_positive(mul(b, e3), cuts.p);
    q3 = cut(viscosity(e3, p3, in, shrink), cuts.q);
    if (!shrink) q3.m = 0;
    // |m| < 2^60 in each: none is below -2^49 = -5.6e14
    return half && imax(e1.e, imax(e2.e, e3.e)) <= -11;
}

}  // namespace fx
}  // namespace lg
