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
    i64 R[8];
    const i64 a0 = fixed_int<59>(a[0], emax);
    int mag = 0;
    R[0] = 0;
#pragma unroll
    for (int j = 1; j < 8; ++j) {
        R[j] = fixed_int<59>(a[j], emax) - a0;  // |.| < 2^60
        magnitude(mag, R[j]);
    }
    const int n = (clz32((unsigned)mag) - 4) & 31;  // top bit of the largest to bit 59
#pragma unroll
    for (int j = 1; j < 8; ++j) R[j] = shl(R[j], n);
    u = emax - 1081 - n;
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
    const int k = 1081 - emax;  // |v| 2^k < 2^59
    i64 hx[4];
    i64 mag = 0;
    {
        Op U[8];
#pragma unroll
        for (int j = 0; j < 8; ++j) U[j] = split(fixed_int<59>(v[j], emax));
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

// ---------------------------------------------------------------------------
// CalcKinematicsForElems and CalcMonotonicQGradientsForElems
// ---------------------------------------------------------------------------
// scratch of kinematics(): the three components' twelve differences
enum KinSlots { KS_D = 0, KS_COUNT = 36 };

// the xi, eta, zeta differences (diag_directions) of eight values below 2^60:
// |.| < 2^63
LG_FX void directions(const i64 v[8], i64 d[3])
{
    const i64 D0 = v[6] - v[0], D1 = v[5] - v[3], D2 = v[7] - v[1], D3 = v[4] - v[2];
    const i64 s = D0 + D1, t = D2 + D3, p = D0 - D1, q = D2 - D3;
    d[0] = s - t;
    d[1] = p + q;
    d[2] = s + t;
}

// Component c of the coordinates: differences to the scratch, quarter
// directions P, unit exponent u.
LG_FX bool kin_component(const double a[8], int c, i64 *s, int stride, Op P[3], int &u)
{
    int top = 0;
#pragma unroll
    for (int j = 0; j < 8; ++j) top = top_word(top, a[j]);
    const int emax = top >> 20;
    i64 R[8];
    const i64 a0 = fixed_int<59>(a[0], emax);
    int mag = 0;
    R[0] = 0;
#pragma unroll
    for (int j = 1; j < 8; ++j) {
        R[j] = fixed_int<59>(a[j], emax) - a0;  // |.| < 2^60
        magnitude(mag, R[j]);
    }
    const int n = (clz32((unsigned)mag) - 4) & 31;
#pragma unroll
    for (int j = 1; j < 8; ++j) R[j] = shl(R[j], n);
    u = emax - 1081 - n;
    i64 *d = s + (KS_D + 12 * c) * stride;
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
    i64 p[3];
    directions(R, p);
#pragma unroll
    for (int i = 0; i < 3; ++i) P[i] = split(p[i] >> 2);  // < 2^61
    // extents between 2^-24 and 2^24: areas and volumes stay seedable
    return emax >= 700 && mag > 0 && u >= -84 && u <= -36;
}

// The velocities' directions: direction d of component c in units of
// 2^(lambda[c] + u[c]), |.| < 2^62.  Each component has the unit of its own largest
// velocity, so that a small one beside a stream keeps its digits; a difference is exact
// to 2^-59 of that velocity.
LG_FX bool kin_velocities(const double v[3][8], const int u[3], Op V[3][3], int lambda[3])
{
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        int top = 300 << 20;
#pragma unroll
        for (int j = 0; j < 8; ++j) top = top_word(top, v[c][j]);
        const int e = top >> 20;
        i64 w[8], dir[3];
#pragma unroll
        for (int j = 0; j < 8; ++j) w[j] = fixed_int<59>(v[c][j], e);
        directions(w, dir);
#pragma unroll
        for (int d = 0; d < 3; ++d) V[c][d] = split(dir[d]);
        lambda[c] = e - 1083 - u[c];  // a quarter of the sums
        ok = ok && e <= 1200;
    }
    return ok;
}

// A factor of the rates, m 2^e with |m| in [2^59, 2^60), or a zero with e = kNoRate.
// sure: m has its digits (see cofactor).
constexpr int kNoRate = -100000;
struct Rate {
    i64 m;
    int e;
    bool sure;
};
LG_FX Rate rate_of(Op V, int lambda)
{
    const i64 v = join(V);
    const int n = clz64((u64)(v ^ (v >> 63))) - 4;  // >= -2
    Rate r;
    r.m = shl(v, (n + 2) & 63) >> 2;
    r.e = v == 0 ? kNoRate : lambda - n;
    r.sure = true;
    return r;
}
// (a b - c d) 2^-64 from all of the products' bits but the last 32, so that a small one
// (an edge nearly along an axis) keeps its digits as a product in FP64 does.
// |a|, ... < 2^61.  Not sure: below 2^-24 of 1, where m is short of its 60 bits.
LG_FX Rate cofactor(Op a, Op b, Op c, Op d)
{
    Acc p, q;
    p.hh = p.hl = q.hh = q.hl = 0;
    mac(p, a, b);
    mac(q, c, d);
    const i64 low = mad(a.l, b.l, 0) - mad(c.l, d.l, 0);
    const i64 hl = (p.hl - q.hl) + (low >> 32);
    const i64 hh = (p.hh - q.hh) + (hl >> 32);
    const int top = (int)(hh >> 32);
    const int n = clz32((unsigned)(top ^ (top >> 31))) - 4;  // 1 to 28
    Rate r;
    r.m = (i64)((u64)funnel((unsigned)top, (unsigned)hh, n) << 32 |
                funnel((unsigned)hh, (unsigned)hl, n));
    r.e = r.m == 0 ? kNoRate : -n;
    r.sure = n < 28;
    return r;
}
// sum_c a[c] V[c] = t 2^(60 + e), |t| < 2^62, with the products aligned at the largest; not
// ok where that one is not sure
struct RateSum {
    i64 t;
    int e;
    bool ok;
};
LG_FX RateSum rate_sum(const Rate a[3], const Rate V[3])
{
    RateSum s;
    int e[3], sure = 3 * kNoRate;
    s.e = 3 * kNoRate;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        e[c] = a[c].e + V[c].e;
        s.e = imax(s.e, e[c]);
        sure = imax(sure, a[c].sure ? e[c] : 3 * kNoRate);
    }
    s.ok = s.e - sure <= 2 || s.e < kNoRate / 2;
    Acc t = acc0<4>();
    i64 low = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const Op x = split(a[c].m), y = split(V[c].m >> imin(s.e - e[c], 63));
        mac(t, x, y);
        low = mad(x.l, y.l, low);
    }
    t.hl += low >> 32;
    s.t = value<4>(t);
    return s;
}

// CalcElemVolume from the corners' coordinates relative to corner 0 (r[c][0] is
// not read).  Each triple product is off by at most 2^-53 of the product of the
// three extents, 12 of which are a box's volume.
LG_FX bool relative_volume(const double r[3][8], double &volume)
{
    Op D[3][12];
    Op a[3][3];
    int S = 0;
    bool ok = true;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        int top = 0;
#pragma unroll
        for (int j = 1; j < 8; ++j) top = top_word(top, r[c][j]);
        const int emax = top >> 20;
        i64 R[8];
#pragma unroll
        for (int j = 1; j < 8; ++j) R[j] = fixed_int<60>(r[c][j], emax);
        D[c][7] = split(R[6] - R[3]);
        D[c][0] = split(R[2]);
        D[c][10] = split(R[6] - R[4]);
        D[c][9] = split(R[7]);
        D[c][4] = split(R[6] - R[1]);
        D[c][2] = split(R[5]);
        a[c][0] = split((R[3] - R[1]) + (R[7] - R[2]));
        a[c][1] = split((R[4] - R[3]) + (R[5] - R[7]));
        a[c][2] = split((R[1] - R[4]) + (R[2] - R[5]));
        ok = ok && emax >= 998 && emax <= 1046;  // extents between 2^-25 and 2^24
        S += emax - 1082;
    }
    i64 V12 = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const int i = (c + 1) % 3, j = (c + 2) % 3;
        Acc t = acc0<2>();
        mac(t, a[c][0], split(det2(D[i][7], D[j][0], D[j][7], D[i][0])));
        mac(t, a[c][1], split(det2(D[i][10], D[j][9], D[j][10], D[i][9])));
        mac(t, a[c][2], split(det2(D[i][4], D[j][2], D[j][4], D[i][2])));
        V12 += value<2>(t);  // units of 2^-54
    }
    volume = real_of(V12, 126 + S) * (1.0 / 12.0);
    return ok && V12 > ((i64)1 << 40);
}

struct Kinematics {
    double volume;   // CalcElemVolume
    double arealg;   // CalcElemCharacteristicLength
    double vdov;     // trace of the velocity gradient at the half step
    double delx[3], delv[3];  // xi, eta, zeta
};

// P, u and the scratch from kin_component; V, lambda from kin_velocities; dt2
// half the time step.  The volume is that of the differences; delx and delv
// are CalcMonotonicQGradientsForElems' for that volume.
LG_FX bool kinematics(const i64 *s, int stride, const Op P[3][3], const int u[3],
                      const Op V[3][3], const int lambda[3], double dt2, Kinematics &k)
{
    const int S = u[0] + u[1] + u[2];
    const int umin = imin(u[0], imin(u[1], u[2]));
    bool ok = true;
    // faces' areas (units of 2^-58 of their components' scales) and volume
    double m2;
    {
        i64 A[6][3];
        i64 V12 = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int ci = (c + 1) % 3, cj = (c + 2) % 3;
            Op U[12], W[12];
#pragma unroll
            for (int i = 0; i < 12; ++i) {
                U[i] = get(s + (KS_D + 12 * ci + i) * stride);
                W[i] = get(s + (KS_D + 12 * cj + i) * stride);
            }
            const i64 *dc = s + (KS_D + 12 * c) * stride;
            const int sh = imin(u[c] - umin, 63);
#define LG_FX_CR(q, p) det2<2>(U[q], W[p], W[q], U[p])
            A[0][c] = LG_FX_CR(1, 0) >> sh;
            A[1][c] = LG_FX_CR(3, 2) >> sh;
            A[2][c] = LG_FX_CR(5, 4) >> sh;
            A[3][c] = LG_FX_CR(6, 7) >> sh;
            A[4][c] = LG_FX_CR(8, 9) >> sh;
            A[5][c] = LG_FX_CR(11, 10) >> sh;
#undef LG_FX_CR
            Acc a = acc0<2>();
            mac(a, split(join(get(dc + 1 * stride)) + join(get(dc + 6 * stride))),
                split(det2(U[7], W[0], W[7], U[0])));
            mac(a, split(join(get(dc + 8 * stride)) + join(get(dc + 11 * stride))),
                split(det2(U[10], W[9], W[10], U[9])));
            mac(a, split(join(get(dc + 3 * stride)) + join(get(dc + 5 * stride))),
                split(det2(U[4], W[2], W[4], U[2])));
            V12 += value<2>(a);  // units of 2^-54
        }
        ok = V12 > ((i64)1 << 40);
        k.volume = real_of(V12, 126 + S) * (1.0 / 12.0);
        i64 best = 0;
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            Acc a = acc0<4>();
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                const Op o = split(A[f][c]);
                mac(a, o, o);
            }
            const i64 w = value<4>(a);  // units of 2^-56
            best = w > best ? w : best;
        }
        ok = ok && best > ((i64)1 << 40);
        m2 = real_of(best, 2 * (S - umin + 120) - 56);
    }
    k.arealg = 2.0 * k.volume * recip_sqrt(m2);
    // A warp of elements at rest skips the rates.
    int some = 0;
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int d = 0; d < 3; ++d) some |= V[c][d].h | V[c][d].l;
    const bool moving = any_lane(some != 0);
    ok = ok && expo(dt2) != 0x7ff && (i64)bits(dt2) >= 0;
    // monotonic-Q gradients
    const double norm = recip(k.volume + 1.e-36);
    double T1 = 0.0;
    Acc e = acc0<2>();
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const int p = (d + 1) % 3, q = (d + 2) % 3;
        Rate a[3];
        int top = 3 * kNoRate;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int i = (c + 1) % 3, j = (c + 2) % 3;
            a[c] = cofactor(P[i][p], P[j][q], P[i][q], P[j][p]);
            top = imax(top, a[c].e - u[c]);
        }
        ok = ok && top + umin >= -18;
        Acc w = acc0<4>();
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const Op o = split(a[c].m >> imin(top - (a[c].e - u[c]), 63));
            mac(w, o, o);
        }
        const double a2 = real_of(value<4>(w), 60 + 2 * (S + 64 + top)) + 1.e-36;
        k.delx[d] = k.volume * recip_sqrt(a2);
        k.delv[d] = 0.0;
        if (moving) {
            Rate r[3];
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                r[c] = rate_of(V[c][d], lambda[c]);
                // the determinant, a in units of 2^-58
                if (d == 1) mac(e, split(shl(a[c].m, 2) >> imin(-a[c].e, 63)), P[c][d]);
            }
            const RateSum t = rate_sum(a, r);
            ok = ok && t.ok;
            const double t1 = real_of(t.t, 124 + S + t.e);
            k.delv[d] = norm * t1;
            T1 = d ? T1 + t1 : t1;
        }
    }
    // Trace of the velocity gradient at the half step, where the Jacobian is P - h V: its
    // determinant det P - h T1 + h^2 T2 - h^3 T3 (T1 = sum cof(P) V, T2 = sum cof(V) P,
    // T3 = det V) and minus that one's derivative in h are the quotient.  An error of T2
    // or T3 counts by the share of the element that moves in half a step, so a component's
    // three differences share one unit here.
    k.vdov = 0.0;
    if (moving) {
        Op U[3][3];
        int g[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            i64 v[3], mag = 0;
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                v[d] = join(V[c][d]);
                mag |= v[d] ^ (v[d] >> 63);
            }
            const int n = clz64((u64)mag) - 4;  // >= -2
#pragma unroll
            for (int d = 0; d < 3; ++d) U[c][d] = split(shl(v[d], (n + 2) & 63) >> 2);
            g[c] = mag == 0 ? kNoRate : lambda[c] - n;
            // half a step moves it by less than its extent
            ok = ok && expo(dt2) + g[c] <= 1022;
        }
        i64 r[3];
        int E[3];
        Acc z = acc0<2>();
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const int i = (c + 1) % 3, j = (c + 2) % 3;
            Acc y = acc0<2>();
#pragma unroll
            for (int d = 0; d < 3; ++d) {
                const int p = (d + 1) % 3, q = (d + 2) % 3;
                const Op cof = split(det2<2>(U[i][p], U[j][q], U[i][q], U[j][p]));
                mac(y, cof, P[c][d]);
                if (c == 0) mac(z, cof, U[c][d]);
            }
            r[c] = value<2>(y);
            E[c] = g[i] + g[j];
        }
        const int top = imax(E[0], imax(E[1], E[2])), E3 = E[0] + g[0];
        i64 t2 = 0;
#pragma unroll
        for (int c = 0; c < 3; ++c) t2 += r[c] >> imin(top - E[c], 63);
        const i64 t3 = value<2>(z), det = value<2>(e);
        ok = ok && det > ((i64)1 << 36) && (t2 == 0 || top > -600) && (t3 == 0 || E3 > -600);
        const double T0 = real_of(det, 124 + S), T2 = real_of(t2, 124 + S + top),
                     T3 = real_of(t3, 124 + S + E3);
        const double h3 = dt2 * T3;
        const double D = fma(-dt2, fma(-dt2, T2 - h3, T1), T0);
        ok = ok && D > 0.0625 * T0;
        k.vdov = fma(-dt2, fma(-3.0, h3, 2.0 * T2), T1) * recip(D);
    }
    return ok;
}

}  // namespace fx
}  // namespace lg
