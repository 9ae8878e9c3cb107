// lg_fixed_geometry.cuh -- the FMA build's element geometry in fixed point.
//
// An element's coordinates enter as differences from its corner 0, each
// component scaled by its own power of two to |R| < 2^60 ("1").  Coordinates
// of one binade are exact multiples of that unit, so every difference and sum
// of them is exact; products round at 2^-56 of 1 and better where it matters.
// Where a bound below fails (an element flattened to a few percent, folded or
// inverted; extreme scales; infinities; NaN) the functions return false and
// the caller evaluates the element in FP64.
#pragma once

#include "lg_fixed.cuh"

namespace lg {
namespace fx {

// Per-element scratch of the corner forces: i64 (or Op) values, `stride` apart
// (a thread's column of shared memory).
enum ForceSlots { FS_D = 0, FS_MODES = 36, FS_COUNT = 48 };
LG_FX void put(i64 *s, Op o) { *reinterpret_cast<Op *>(s) = o; }
LG_FX Op get(const i64 *s) { return *reinterpret_cast<const Op *>(s); }

// Component c of the corners: its twelve node differences (elem_differences'
// order, |d| < 2^61) and hourglass mode sums (hourglass_modes', < 7 x 2^60) into
// the scratch, and the exponent u of its unit.
LG_FX bool force_component(const double a[8], int c, i64 *s, int stride, int &u)
{
    int top = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) top = top_word(top, a[j]);
    const int emax = top >> 20;
    const bool ok = emax >= 700 && emax <= 1081;
    const int k = imax(imin(1081 - emax, 381), 0);  // |a| 2^k < 2^59
    i64 R[8];
    const i64 a0 = fixed_of(a[0], k);
    int mag = 0;
    R[0] = 0;
#pragma unroll
    for (int j = 1; j < 8; ++j) {
        R[j] = fixed_of(a[j], k) - a0;  // |.| < 2^60
        magnitude(mag, R[j]);
    }
    const int n = (clz32((unsigned)mag) - 4) & 31;  // top bit of the largest to bit 59
#pragma unroll
    for (int j = 1; j < 8; ++j) R[j] = shl(R[j], n);
    u = -k - n;
    i64 *d = s + (FS_D + 12 * c) * stride, *m = s + (FS_MODES + 4 * c) * stride;
    put(d + 0 * stride, split(R[2]));
    put(d + 1 * stride, split(R[3] - R[1]));
    put(d + 2 * stride, split(R[5]));
    put(d + 3 * stride, split(R[1] - R[4]));
    put(d + 4 * stride, split(R[6] - R[1]));
    put(d + 5 * stride, split(R[2] - R[5]));
    put(d + 6 * stride, split(R[7] - R[2]));
    put(d + 7 * stride, split(R[6] - R[3]));
    put(d + 8 * stride, split(R[4] - R[3]));
    put(d + 9 * stride, split(R[7]));
    put(d + 10 * stride, split(R[6] - R[4]));
    put(d + 11 * stride, split(R[5] - R[7]));
    const i64 d23 = R[2] - R[3], s23 = R[2] + R[3], d45 = R[4] - R[5], s45 = R[4] + R[5];
    const i64 d67 = R[6] - R[7], s67 = R[6] + R[7];
    const i64 p = d67 - R[1], q = d23 + d45;
    m[0 * stride] = (R[1] + s67) - (s23 + s45);
    m[1 * stride] = p - q;
    m[2 * stride] = p + q;
    m[3 * stride] = (d45 + d67) - (d23 - R[1]);
    return ok && mag > 0;
}

// k's sign in hourglass mode m (lulesh.cc:743-776)
LG_FX constexpr bool gam_plus(int m, int k)
{
    constexpr unsigned char P[4] = {0xc3, 0x69, 0x55, 0x5a};  // bit k: +1
    return (P[m] >> k) & 1;
}

// The face areas (8 x, six faces in node_normals_x8_diff's order, units of
// 2^-56) into the scratch (slots area_slot(c) + f), and the hourglass shape
// vectors hourgam in units of 2^-59.  vi12 = 1 / (12 det); u the components'
// units.
LG_FX int area_slot(int c) { return c == 2 ? FS_D : FS_D + 24 + 6 * c; }

LG_FX bool force_shape(i64 *s, int stride, const int u[3], double vi12, Op hg[8][4])
{
    Op G[3][8];
    i64 A[3][6];
    int J[3][3];  // 8 x the Jacobian's columns, 2^-28
    int magG = 0, magH = 0, magh = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int ci = (c + 1) % 3, cj = (c + 2) % 3;
        Op U[12], V[12];
#pragma unroll
        for (int i = 0; i < 12; ++i) {
            U[i] = get(s + (FS_D + 12 * ci + i) * stride);
            V[i] = get(s + (FS_D + 12 * cj + i) * stride);
        }
        J[0][ci] = (U[7].h + U[11].h) + (U[3].h + U[0].h);
        J[1][ci] = (U[10].h + U[1].h) - (U[11].h - U[0].h);
        J[2][ci] = (U[4].h + U[2].h) + (U[6].h + U[8].h);
#define LG_FX_CR(q, p) det2(U[q], V[p], V[q], U[p])
        A[c][0] = LG_FX_CR(1, 0);
        A[c][1] = LG_FX_CR(3, 2);
        A[c][2] = LG_FX_CR(5, 4);
        A[c][3] = LG_FX_CR(6, 7);
        A[c][4] = LG_FX_CR(8, 9);
        A[c][5] = LG_FX_CR(11, 10);
        // volume_gradient_x12_diff, component c, units of 2^-56 (< 48)
        const Op u1 = split(join(U[1]) + join(U[6])), v1 = split(join(V[1]) + join(V[6]));
        const Op u2 = split(join(U[8]) + join(U[11])), v2 = split(join(V[8]) + join(V[11]));
        const Op u3 = split(join(U[3]) + join(U[5])), v3 = split(join(V[3]) + join(V[5]));
        const i64 X1 = LG_FX_CR(7, 0), X2 = LG_FX_CR(10, 9), X3 = LG_FX_CR(4, 2);
        const i64 Y1 = det2(U[0], v1, V[0], u1), Z1 = det2(u1, V[7], v1, U[7]);
        const i64 Y2 = det2(U[9], v2, V[9], u2), Z2 = det2(u2, V[10], v2, U[10]);
        const i64 Y3 = det2(U[2], v3, V[2], u3), Z3 = det2(u3, V[4], v3, U[4]);
        i64 v[8];
        v[0] = -(Z1 + Z2 + Z3);
        v[1] = (X3 - X1) - Y3;
        v[2] = (X3 - X1) + Z1;
        v[3] = (X1 - X2) - Y1;
        v[4] = (X2 - X3) - Y2;
        v[5] = (X2 - X3) + Z3;
        v[6] = Y1 + Y2 + Y3;
        v[7] = (X1 - X2) + Z2;
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            magnitude(magG, v[k]);
            G[c][k] = split(v[k]);
        }
#undef LG_FX_CR
        // component 2's differences are done with after c = 1, component 0's
        // after c = 2
        if (c > 0) {
#pragma unroll
            for (int f = 0; f < 6; ++f) {
                s[(area_slot(c) + f) * stride] = A[c][f];
                if (c == 1) s[(area_slot(0) + f) * stride] = A[0][f];
            }
        }
    }
    // The Jacobian's sign (lulesh.cc:1082-1091): the triple product is 64 det J in
    // units of 2^-51, off by less than 2^38 of them
    bool ok;
    {
        const i64 cx = ((i64)J[0][1] * J[1][2] - (i64)J[0][2] * J[1][1]) >> 33;
        const i64 cy = ((i64)J[0][2] * J[1][0] - (i64)J[0][0] * J[1][2]) >> 33;
        const i64 cz = ((i64)J[0][0] * J[1][1] - (i64)J[0][1] * J[1][0]) >> 33;
        const i64 j = (i64)(int)cx * J[2][0] + (i64)(int)cy * J[2][1] + (i64)(int)cz * J[2][2];
        ok = j > ((i64)1 << 39);
    }
    // -1 / (12 det) in units of 2^-59, |.| in (2^-7, 8)
    Op vi;
    {
        const int sh = expo(vi12) + (u[0] + u[1] + u[2] + 180) - 1016;
        ok = ok && sh >= 0 && sh <= 9 && (i64)bits(vi12) > 0;
        vi = split(-(i64)(significand(vi12) << (sh & 15)));
    }
    Op H[3][4];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            const i64 v = s[(FS_MODES + 4 * c + m) * stride];
            magnitude(magH, v);
            Acc a = acc0<7>();
            mac(a, split(v), vi);
            magnitude(magh, a.hh);
            H[c][m] = split(value<7>(a));  // 2^-62
        }
    ok = ok && (magG >> 27) == 0 && (magH >> 29) == 0;  // |G| < 8, |modes| < 2
#pragma unroll
    for (int k = 0; k < 8; ++k)
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            Acc a = acc0<5>();
            a.hh = gam_plus(m, k) ? (i64)1 << 54 : -((i64)1 << 54);
            mac(a, G[0][k], H[0][m]);
            mac(a, G[1][k], H[1][m]);
            mac(a, G[2][k], H[2][m]);
            magnitude(magh, a.hh);
            hg[k][m] = split(value<5>(a));
        }
    return ok && (magh >> 23) == 0;  // |H| < 1, |hourgam| < 2
}

// A double as a 60-bit significand and its unit's exponent; an infinity or
// NaN clears ok.
struct Scale {
    i64 m;
    int e;
};
LG_FX Scale scale_of(double v, bool &ok)
{
    const int be = expo(v);
    const i64 s = (i64)bits(v) >> 63;
    const i64 m = (i64)(significand(v) << 7);
    ok = ok && be != 0x7ff;
    Scale r;
    r.e = be ? be - 1082 : -5000;
    r.m = be ? (m ^ s) - s : 0;
    return r;
}

// Corner forces of component c: k1 (sums of three areas) + k2 hourgam
// (hourgam^T v).  k1 = (p + q) / 8, k2 the hourglass coefficient; u12 the sum
// of the other two components' units.
LG_FX bool force_corners(const i64 *s, int stride, const Op hg[8][4], int c, Scale k1, int u12,
                         Scale k2, const double v[8], double F[8])
{
    const int E1 = k1.e + 125 + u12;
    int top = 200 << 20;
#pragma unroll
    for (int j = 0; j < 8; ++j) top = top_word(top, v[j]);
    const int emax = top >> 20;
    bool ok = emax <= 1081;
    const int k = imax(1081 - emax, 0);  // |v| 2^k < 2^59
    i64 hx[4];
    i64 mag = 0;
    {
        Op U[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) U[j] = split(fixed_of(v[j], k));
#pragma unroll
        for (int m = 0; m < 4; ++m) {
            Acc a = acc0<2>();
#pragma unroll
            for (int j = 0; j < 8; ++j) mac(a, hg[j][m], U[j]);
            hx[m] = value<2>(a);  // units of 2^(3 - k), < 2^60
            mag |= hx[m] ^ (hx[m] >> 63);
        }
    }
    const int n = imax(clz64((u64)mag) - 4, 0);
    Op h[4];
#pragma unroll
    for (int m = 0; m < 4; ++m) h[m] = split(shl(hx[m], n));
    const int E2 = k2.e + 66 - k - n;
    // both terms in units of 2^E: the smaller one's factor is shifted
    const int E = imax(E1, E2);
    ok = ok && E < 800;
    const Op q1 = split(k1.m >> imin(E - E1, 63)), q2 = split(k2.m >> imin(E - E2, 63));
    const i64 *a = s + area_slot(c) * stride;
    const i64 A0 = a[0], A1 = a[stride], A2 = a[2 * stride], A3 = a[3 * stride],
              A4 = a[4 * stride], A5 = a[5 * stride];
    i64 N[8];
    N[0] = (A0 + A1) + A4;
    N[1] = (A0 + A1) + A2;
    N[2] = (A0 + A2) + A3;
    N[3] = (A0 + A3) + A4;
    N[4] = (A1 + A4) + A5;
    N[5] = (A1 + A2) + A5;
    N[6] = (A2 + A3) + A5;
    N[7] = (A3 + A4) + A5;
    const bool some = E > -900;
    const int e = some ? E : 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        Acc a = acc0<3>(), r = acc0<3>();
#pragma unroll
        for (int m = 0; m < 4; ++m) mac(a, hg[j][m], h[m]);
        mac(r, split(N[j]), q1);
        mac(r, split(value<3>(a)), q2);  // value: units of 2^(5 - k - n), < 2^61
        F[j] = real_of(some ? value<3>(r) : 0, e);
    }
    return ok;
}

}  // namespace fx
}  // namespace lg
