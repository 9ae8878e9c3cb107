// lg_exact_geometry.cuh -- the strict build's corner forces with their products and
// coordinate sums on the integer pipes, every one rounded as in IEEE arithmetic.
//
// GB300's FP64 pipe issues 2 lanes per SM and clock and bounds the strict kernels;
// the integer pipes issue 128.  Three kinds of operations move there bit for bit:
// products (product() of lg_exact.cuh), sums of an element's coordinates, and the
// powers of two.  An element's eight x (y, z) are nearly of one size: as 64-bit
// integers in one unit, with up to six bits between the largest and the smallest, a
// sum is an integer addition and a rounding to 53 bits, 14 instructions without
// the alignment and normalisation of two floating-point numbers.  The sums of
// products, whose terms differ in size, stay on the FP64 pipe.  Elements that do not
// fit (zeros do) are flagged, and the caller takes the FP64 form.
#pragma once

#include "lg_exact.cuh"

namespace lg {
namespace fx {

// The eight values of one coordinate as multiples of 2^(emax - 1082): even integers
// below 2^60, in every BS-th word of n.
template <int BS>
LG_FX int align8(const double (&a)[8], i64 *n, unsigned &bad)
{
    int top = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) top = top_word(top, a[j]);
    const int emax = top >> 20;
    bad |= emax < 600 || emax > 1500;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const bool zero = (bits(a[j]) << 1) == 0;
        const int d = emax - expo(a[j]);
        bad |= !zero && d > 6;
        const i64 m = zero ? 0 : (i64)(significand(a[j]) << ((7 - d) & 63));
        const i64 s = (i64)bits(a[j]) >> 63;
        n[j * BS] = (m ^ s) - s;
    }
    return emax;
}
// an even |s| < 2^63 rounded to 53 bits, ties to even (in two's complement the rule
// is the same on both sides of zero)
LG_FX i64 rounded(i64 s)
{
    const int hi = (int)(s >> 32);
    const int k = imax(1, 11 - clz32((unsigned)(hi ^ (hi >> 31))));
    const unsigned mask = (1u << k) - 1;
    const unsigned odd = ((unsigned)s >> k) & 1;
    return (s + (mask >> 1) + odd) & ~(i64)mask;
}
// a rounded sum in units of 2^(emax - 1082) as a factor
LG_FX void normal_form(i64 s, int emax, u64 &m, unsigned &e)
{
    const i64 sign = s >> 63;
    const u64 a = (u64)((s ^ sign) - sign);
    const int c = clz64(a);
    m = a << (c & 63);
    e = ((unsigned)(emax + 4 - c) << 20) | ((unsigned)sign & 0x80000000u);
}
LG_FX Factor factor_of(i64 s, int emax)
{
    u64 m;
    Factor f;
    normal_form(s, emax, m, f.e);
    m >>= 11;
    f.h = (unsigned)(m >> 32);
    f.l = (unsigned)m;
    return f;
}
LG_FX double double_of(i64 s, int emax)
{
    u64 m;
    unsigned e;
    normal_form(s, emax, m, e);
    // the hidden bit adds one to the exponent field
    return from_bits(m == 0 ? 0 : (m >> 11) + ((u64)(e - (1u << 20)) << 32));
}

// corners a, b, c, d of face f, three bits each, in SumElemFaceNormal's order
LG_FX unsigned face_corners(int f)
{
    constexpr u64 faces = 03210ull | 01540ull << 12 | 02651ull << 24 | 03762ull << 36 |
                          00473ull << 48;
    return f == 5 ? 05674u : (unsigned)(faces >> 12 * f) & 07777u;
}
// the three faces of corner j in the order their areas are added, three bits each
LG_FX unsigned corner_faces(int j)
{
    constexpr u64 low = 0410ull | 0210ull << 9 | 0320ull << 18 | 0430ull << 27;
    constexpr u64 high = 0541ull | 0521ull << 9 | 0532ull << 18 | 0543ull << 27;
    return (unsigned)((j < 4 ? low : high) >> 9 * (j & 3)) & 0777u;
}

// 16 x the areas of count faces from first (face_area_x16), component c of face f at
// area[(3 f + c) BS]
template <int BS>
LG_FX void face_areas(const i64 *n, const int (&emax)[3], int first, int count,
                      double *area)
{
#pragma unroll 1
    for (int f = first; f < first + count; ++f) {
        const unsigned code = face_corners(f);
        const i64 *const pa = n + (code & 7) * BS, *const pb = n + (code >> 3 & 7) * BS,
                        *const pc = n + (code >> 6 & 7) * BS, *const pd = n + (code >> 9) * BS;
        Factor b0[3];
        Factor b1[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const i64 na = pa[8 * c * BS], nb = pb[8 * c * BS], nc = pc[8 * c * BS],
                      nd = pd[8 * c * BS];
            b0[c] = factor_of(rounded(rounded(rounded(nd + nc) - nb) - na), emax[c]);
            b1[c] = factor_of(rounded(rounded(rounded(nc + nb) - nd) - na), emax[c]);
        }
        area[(3 * f + 0) * BS] = product(b0[1], b1[2]) - product(b0[2], b1[1]);
        area[(3 * f + 1) * BS] = product(b0[2], b1[0]) - product(b0[0], b1[2]);
        area[(3 * f + 2) * BS] = product(b0[0], b1[1]) - product(b0[1], b1[0]);
    }
}

// Component c of the volume derivatives (CalcElemVolumeDerivative, lulesh.cc:591-663),
// corner j at out[(8 c + j) BS].  dx is F(y, z), dy -F(x, z) and dz -F(y, x) of
//   F(p, q) = (p1 + p2)(q0 + q1) - (p0 + p1)(q1 + q2) + (p0 + p4)(q3 + q4)
//           - (p3 + p4)(q0 + q4) - (p2 + p5)(q3 + q5) + (p3 + p5)(q2 + q5),
// term for term with the same roundings; the pair sums are the element's 12 edges.
template <int BS>
LG_FX void volume_derivatives(const i64 *n, const int (&emax)[3], int c, double *out,
                              unsigned &bad)
{
    constexpr int V[8][6] = {{1, 2, 3, 4, 5, 7}, {2, 3, 0, 5, 6, 4}, {3, 0, 1, 6, 7, 5},
                             {0, 1, 2, 7, 4, 6}, {7, 6, 5, 0, 3, 1}, {4, 7, 6, 1, 0, 2},
                             {5, 4, 7, 2, 1, 3}, {6, 5, 4, 3, 2, 0}};
    // edge of two corners: 0..3 bottom, 4..7 top, 8..11 upright
    constexpr int A[12] = {0, 1, 2, 3, 4, 5, 6, 7, 0, 1, 2, 3};
    constexpr int B[12] = {1, 2, 3, 0, 5, 6, 7, 4, 4, 5, 6, 7};
    constexpr int G[8][8] = {{0, 0, 0, 3, 8, 0, 0, 0}, {0, 0, 1, 0, 0, 9, 0, 0},
                             {0, 1, 0, 2, 0, 0, 10, 0}, {3, 0, 2, 0, 0, 0, 0, 11},
                             {8, 0, 0, 0, 0, 4, 0, 7}, {0, 9, 0, 0, 4, 0, 5, 0},
                             {0, 0, 10, 0, 0, 5, 0, 6}, {0, 0, 0, 11, 7, 0, 6, 0}};
    const Factor twelfth = factor(1.0 / 12.0, bad);
    const i64 *const np = n + (c == 1 ? 0 : 8 * BS), *const nq = n + (c == 2 ? 0 : 16 * BS);
    const int ep = c == 1 ? emax[0] : emax[1], eq = c == 2 ? emax[0] : emax[2];
    Factor p[12];
    Factor q[12];
#pragma unroll
    for (int i = 0; i < 12; ++i) {
        p[i] = factor_of(rounded(np[A[i] * BS] + np[B[i] * BS]), ep);
        q[i] = factor_of(rounded(nq[A[i] * BS] + nq[B[i] * BS]), eq);
    }
    const u64 flip = c == 0 ? 0 : 0x8000000000000000ull;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
#define LG_EDGE(a, b) G[V[j][a]][V[j][b]]
        const double F = product(p[LG_EDGE(1, 2)], q[LG_EDGE(0, 1)]) -
                         product(p[LG_EDGE(0, 1)], q[LG_EDGE(1, 2)]) +
                         product(p[LG_EDGE(0, 4)], q[LG_EDGE(3, 4)]) -
                         product(p[LG_EDGE(3, 4)], q[LG_EDGE(0, 4)]) -
                         product(p[LG_EDGE(2, 5)], q[LG_EDGE(3, 5)]) +
                         product(p[LG_EDGE(3, 5)], q[LG_EDGE(2, 5)]);
#undef LG_EDGE
        const double d = product(factor(F, bad), twelfth);
        out[(8 * c + j) * BS] = from_bits(bits(d) ^ flip);
    }
}

// gam(m, j) < 0 at bit j
LG_FX unsigned mode_signs(int m) { return (0xa5aa963cu >> 8 * m) & 0xffu; }
// sum_j gam(m, j) x_j from left to right (lulesh.cc:894-912)
template <int BS>
LG_FX i64 hourglass_mode(const i64 *n, unsigned signs)
{
    i64 s = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const i64 f = -(i64)(signs >> j & 1);
        s += (n[j * BS] ^ f) - f;
        if (j) s = rounded(s);
    }
    return s;
}

// 12 x the volume (CalcElemVolume, lulesh.cc:1273-1356): the triple product t
// = a . (b x c) of its three, of a = (r0 - r1) + (r2 - r3), b = r4 - r5, c = r6 - r7
template <int BS>
LG_FX double volume_triple(const i64 *n, const int (&emax)[3], int t, unsigned &bad)
{
    // corners r0 .. r7, three bits each
    const unsigned code = t == 0 ? 002362713u : t == 1 ? 007467534u : 005165241u;
    const i64 *r[8];
#pragma unroll
    for (int i = 0; i < 8; ++i) r[i] = n + (code >> 3 * i & 7) * BS;
    Factor a[3], b[3];
    Factor c[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int o = 8 * d * BS;
        a[d] = factor_of(rounded(rounded(r[0][o] - r[1][o]) + rounded(r[2][o] - r[3][o])), emax[d]);
        b[d] = factor_of(rounded(r[4][o] - r[5][o]), emax[d]);
        c[d] = factor_of(rounded(r[6][o] - r[7][o]), emax[d]);
    }
    const double x = product(b[1], c[2]) - product(b[2], c[1]);
    const double y = product(b[2], c[0]) - product(b[0], c[2]);
    const double z = product(b[0], c[1]) - product(b[1], c[0]);
    return product(a[0], factor(x, bad)) + product(a[1], factor(y, bad)) +
           product(a[2], factor(z, bad));
}

// The largest of 0 and count of CalcElemCharacteristicLength's AreaFace values from first
// (lulesh.cc:1370-1435)
template <int BS>
LG_FX double largest_area_face(const i64 *n, const int (&emax)[3], int first, int count,
                               unsigned &bad)
{
    double largest = 0.0;
#pragma unroll 1
    for (int t = first; t < first + count; ++t) {
        constexpr u64 faces = 03210ull | 07654ull << 12 | 04510ull << 24 | 05621ull << 36 |
                              06732ull << 48;
        const unsigned code = t == 5 ? 07403u : (unsigned)(faces >> 12 * t) & 07777u;
        const i64 *const pa = n + (code & 7) * BS, *const pb = n + (code >> 3 & 7) * BS,
                        *const pc = n + (code >> 6 & 7) * BS, *const pd = n + (code >> 9) * BS;
        double ff = 0., gg = 0., fg = 0.;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int o = 8 * c * BS;
            const i64 p = rounded(pc[o] - pa[o]), q = rounded(pd[o] - pb[o]);
            const i64 f = rounded(p - q), g = rounded(p + q);
            const Factor f1 = factor_of(f, emax[c]), g1 = factor_of(g, emax[c]);
            const double a = product(f1, f1), b = product(g1, g1), d = product(f1, g1);
            ff = c ? ff + a : a;
            gg = c ? gg + b : b;
            fg = c ? fg + d : d;
        }
        const Factor fg1 = factor(fg, bad);
        const double area =
            product(factor(ff, bad), factor(gg, bad)) - product(fg1, fg1);
        largest = geom::lt(area, largest) ? largest : area;
    }
    return largest;
}

// CalcMonotonicQGradientsForElems' differences of one coordinate (lulesh.cc:1613-1757,
// without the factors 0.25): directions xi, eta, zeta at out[0], out[BS], out[2 BS]
template <int BS>
LG_FX void gradient_sums(const i64 *n, int emax, double *out)
{
    constexpr int S[3][8] = {{1, 2, 6, 5, 0, 3, 7, 4}, {0, 1, 5, 4, 3, 2, 6, 7},
                             {4, 5, 6, 7, 0, 1, 2, 3}};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        i64 s[2];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            s[i] = rounded(n[S[d][4 * i] * BS] + n[S[d][4 * i + 1] * BS]);
            s[i] = rounded(s[i] + n[S[d][4 * i + 2] * BS]);
            s[i] = rounded(s[i] + n[S[d][4 * i + 3] * BS]);
        }
        const double v = double_of(rounded(s[0] - s[1]), emax);
        // eta is the difference negated, a zero's sign too
        out[d * BS] = d == 1 ? from_bits(bits(v) ^ 0x8000000000000000ull) : v;
    }
}

}  // namespace fx
}  // namespace lg
