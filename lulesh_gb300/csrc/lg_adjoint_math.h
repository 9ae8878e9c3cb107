// lg_adjoint_math.h -- element-local vector-Jacobian products of the
// leap-frog cycle (reverse mode, FP64), usable on the device and the host.
//
// Each function recomputes the forward values it needs from the same inputs
// the forward kernel read and accumulates the adjoints (suffix "b") of those
// inputs from the adjoints of its outputs.  Non-smooth operations: the
// physical clamps and switches (emin, pmin, eosvmin/eosvmax, the monotonic
// limiter's min/max and its vdov > 0 switch, the sound-speed floor) take the
// derivative of the branch the forward took (zero when they fire); the
// numerical noise cut-offs (|e| < e_cut, |p| < p_cut, |q| < q_cut, and in
// the node and volume updates u_cut and v_cut), which zero values within
// ~1e-7 of zero, pass the derivative through -- the derivative of the map
// without its noise suppressor, which is what finite differences of any
// resolvable step see.  The time step is an input (frozen), so the
// Courant/hydro constraints and everything only they read (arealg, vdov's
// value) have no
// adjoint.  Forward formulas: lulesh.cc lines cited at each function.
#pragma once

#include "lg_geometry.cuh"

namespace lg {
namespace adj {

using geom::gam;

struct V3 {
    double x, y, z;
};
LG_HD V3 cross(const V3 &a, const V3 &b)
{
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
LG_HD double dot(const V3 &a, const V3 &b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

// ---------------------------------------------------------------------------
// The element's twelve node differences d[c][i] (geom::elem_differences) carry
// both the face areas of CalcElemNodeNormals (lulesh.cc:381-474) and the volume
// gradient of CalcElemVolumeDerivative (591-663), so their adjoints collect in
// db[c][i] and go to the nodes once.
// ---------------------------------------------------------------------------
LG_HD V3 diff(const double (*d)[12], int i) { return {d[0][i], d[1][i], d[2][i]}; }
LG_HD void add_to(double (*db)[12], int i, const V3 &g)
{
    db[0][i] += g.x;
    db[1][i] += g.y;
    db[2][i] += g.z;
}

// d[i] = u[P] - u[M] for one coordinate: ub from db
LG_HD void differences_vjp(const double db[12], double ub[8])
{
    ub[0] -= (db[0] + db[2]) + db[9];
    ub[1] += db[3] - (db[1] + db[4]);
    ub[2] += (db[0] + db[5]) - db[6];
    ub[3] += db[1] - (db[7] + db[8]);
    ub[4] += db[8] - (db[3] + db[10]);
    ub[5] += (db[2] - db[5]) + db[11];
    ub[6] += (db[4] + db[7]) + db[10];
    ub[7] += (db[6] + db[9]) - db[11];
}

// face f's four corners and its two diagonals (q, p): area = (q x p) / 8
LG_HD void face_corners(int f, int n[4])
{
    const int F[6][4] = {{0, 1, 2, 3}, {0, 4, 5, 1}, {1, 5, 6, 2},
                         {2, 6, 7, 3}, {3, 7, 4, 0}, {4, 7, 6, 5}};
    for (int i = 0; i < 4; ++i) n[i] = F[f][i];
}
LG_HD int face_q(int f)
{
    const int Q[6] = {1, 3, 5, 6, 8, 11};
    return Q[f];
}
LG_HD int face_p(int f)
{
    const int P[6] = {0, 2, 4, 7, 9, 10};
    return P[f];
}

// sum of the adjoints g[c][node] over face f's corners
LG_HD V3 face_sum(const double *gx, const double *gy, const double *gz, int f)
{
    int n[4];
    face_corners(f, n);
    return {(gx[n[0]] + gx[n[1]]) + (gx[n[2]] + gx[n[3]]),
            (gy[n[0]] + gy[n[1]]) + (gy[n[2]] + gy[n[3]]),
            (gz[n[0]] + gz[n[1]]) + (gz[n[2]] + gz[n[3]])};
}
// face f's q x p, and the adjoints of q and p from that of q x p
LG_HD V3 face_cross(const double (*d)[12], int f) { return cross(diff(d, face_q(f)), diff(d, face_p(f))); }
LG_HD void face_cross_vjp(const double (*d)[12], int f, const V3 &A, double (*db)[12])
{
    add_to(db, face_q(f), cross(diff(d, face_p(f)), A));
    add_to(db, face_p(f), cross(A, diff(d, face_q(f))));
}

// CalcElemNodeNormals' adjoint alone: each node's normal sums its faces' areas.  Only
// tests/adjoint_selftest.cc calls it (and volume_derivative_vjp and pat below); the sweep
// has the same terms inside forces_vjp.
LG_HD void node_normals_vjp(const double *x, const double *y, const double *z, const double *pbx,
                            const double *pby, const double *pbz, double *xb, double *yb,
                            double *zb)
{
    double d[3][12], db[3][12];
    geom::elem_differences(x, d[0]);
    geom::elem_differences(y, d[1]);
    geom::elem_differences(z, d[2]);
    for (int c = 0; c < 3; ++c)
        for (int i = 0; i < 12; ++i) db[c][i] = 0.;
    for (int f = 0; f < 6; ++f) {
        const V3 S = face_sum(pbx, pby, pbz, f);
        face_cross_vjp(d, f, {0.125 * S.x, 0.125 * S.y, 0.125 * S.z}, db);
    }
    differences_vjp(db[0], xb);
    differences_vjp(db[1], yb);
    differences_vjp(db[2], zb);
}

// The adjoints db of the differences from those of 12 x the volume gradient
// (gb[c][node]): node by node the gradient is a signed sum of the nine cross
// products X_k = b_k x c_k, Y_k = c_k x a_k, Z_k = a_k x b_k
// (geom::volume_gradient_x12_diff).
LG_HD void volume_gradient_vjp(const double (*d)[12], const double (*gb)[8], double (*db)[12])
{
    const int bi[3] = {7, 10, 4}, ci[3] = {0, 9, 2}, a0[3] = {1, 8, 3}, a1[3] = {6, 11, 5};
    V3 g[8];
#pragma unroll
    for (int k = 0; k < 8; ++k) g[k] = {gb[0][k], gb[1][k], gb[2][k]};
    auto sub = [](const V3 &u, const V3 &v) { return V3{u.x - v.x, u.y - v.y, u.z - v.z}; };
    const V3 g12 = {g[1].x + g[2].x, g[1].y + g[2].y, g[1].z + g[2].z};
    const V3 g37 = {g[3].x + g[7].x, g[3].y + g[7].y, g[3].z + g[7].z};
    const V3 g45 = {g[4].x + g[5].x, g[4].y + g[5].y, g[4].z + g[5].z};
    const V3 X[3] = {sub(g37, g12), sub(g45, g37), sub(g12, g45)};
    const V3 Y[3] = {sub(g[6], g[3]), sub(g[6], g[4]), sub(g[6], g[1])};
    const V3 Z[3] = {sub(g[2], g[0]), sub(g[7], g[0]), sub(g[5], g[0])};
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const V3 b = diff(d, bi[k]), c = diff(d, ci[k]);
        const V3 p = diff(d, a0[k]), q = diff(d, a1[k]);
        const V3 a = {p.x + q.x, p.y + q.y, p.z + q.z};
        // z = u x v: ub = v x zb, vb = zb x u
        const V3 ab0 = cross(Y[k], c), ab1 = cross(b, Z[k]);
        const V3 ab = {ab0.x + ab1.x, ab0.y + ab1.y, ab0.z + ab1.z};
        add_to(db, bi[k], cross(c, X[k]));
        add_to(db, bi[k], cross(Z[k], a));
        add_to(db, ci[k], cross(X[k], b));
        add_to(db, ci[k], cross(a, Y[k]));
        add_to(db, a0[k], ab);
        add_to(db, a1[k], ab);
    }
}

// CalcElemVolumeDerivative's adjoint alone (its factor 1/12 applied): xb, yb, zb
// from the adjoints of dV/dx, dV/dy, dV/dz
LG_HD void volume_derivative_vjp(const double *x, const double *y, const double *z,
                                 const double *dxb, const double *dyb, const double *dzb,
                                 double *xb, double *yb, double *zb)
{
    double d[3][12], db[3][12], gb[3][8];
    geom::elem_differences(x, d[0]);
    geom::elem_differences(y, d[1]);
    geom::elem_differences(z, d[2]);
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        gb[0][k] = dxb[k] * (1.0 / 12.0);
        gb[1][k] = dyb[k] * (1.0 / 12.0);
        gb[2][k] = dzb[k] * (1.0 / 12.0);
    }
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int i = 0; i < 12; ++i) db[c][i] = 0.;
    volume_gradient_vjp(d, gb, db);
    differences_vjp(db[0], xb);
    differences_vjp(db[1], yb);
    differences_vjp(db[2], zb);
}

// ---------------------------------------------------------------------------
// Element forces (lulesh.cc:273-286, 494-587, 710-1057): stress forces
// -sig * normals, sig = -p - q, plus the FB hourglass forces
//   f_c[i] = coef * sum_m hourgam[i][m] * hxx_c[m],
//   hxx_c[m] = sum_j hourgam[j][m] u_c[j],
//   hourgam[i][m] = gamma[m][i] - sum_c g_c[i] h_c[m],
//   g = 12 dV/dx, h = volinv / 12 * hourmod, coef = -hg 0.01 ss mass / cbrt(volo v).
// fb[c][i]: adjoint of the corner force component c at corner i (stress and
// hourglass parts are summed into the same node force, so they share it).
// With s_c[m] = sum_i hourgam[i][m] fb_c[i], coef's adjoint is sum hxx s and
// u's is coef hourgam s, so no product with hourgam is formed twice.  About
// 1,500 FP64 operations for each element in place of 3,200 for the
// corner-by-corner forms, which bound the kernel that runs this: 200 -> 135 us a
// cycle at s=32, 113 -> 77 us at s=20.
// ---------------------------------------------------------------------------
struct ForceAdj {
    double pb, qb, vb, ssb, hgb;
};

LG_HD void forces_vjp(const double *x, const double *y, const double *z, const double *xd,
                      const double *yd, const double *zd, double p, double q, double v, double volo,
                      double ss, double mass, double hg, const double (*fb)[8], double *xb,
                      double *yb, double *zb, double *xdb, double *ydb, double *zdb, ForceAdj &o)
{
    double d[3][12], db[3][12];
    geom::elem_differences(x, d[0]);
    geom::elem_differences(y, d[1]);
    geom::elem_differences(z, d[2]);
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int i = 0; i < 12; ++i) db[c][i] = 0.;
    // stress part: f = -sig / 8 sum of three faces' q x p
    {
        const double sig8 = (-p - q) * 0.125;
        double sigb = 0.0;
#pragma unroll
        for (int f = 0; f < 6; ++f) {
            const V3 S = face_sum(fb[0], fb[1], fb[2], f);
            sigb += dot(face_cross(d, f), S);
            face_cross_vjp(d, f, {-sig8 * S.x, -sig8 * S.y, -sig8 * S.z}, db);
        }
        o.pb += sigb * 0.125;
        o.qb += sigb * 0.125;
    }
    if (hg > 0.) {
        double g[3][8], h[3][4];
        geom::volume_gradient_x12_diff(d[0], d[1], d[2], g[0], g[1], g[2]);
        geom::hourglass_modes(x, h[0]);
        geom::hourglass_modes(y, h[1]);
        geom::hourglass_modes(z, h[2]);
        const double vol = volo * v;
        const double volinv = geom::rcp_op(vol), vi12 = volinv * (1.0 / 12.0);
#pragma unroll
        for (int c = 0; c < 3; ++c)
#pragma unroll
            for (int m = 0; m < 4; ++m) h[c][m] *= vi12;
        double hg_[8][4], G[8][4];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                hg_[i][m] = gam(m, i) - (g[0][i] * h[0][m] + g[1][i] * h[1][m] + g[2][i] * h[2][m]);
                G[i][m] = 0.0;
            }
        const double cr = cbrt(vol);
        const double coef = geom::div_op(-hg * 0.01 * ss * mass, cr);
        const double *vel[3] = {xd, yd, zd};
        double *velb[3] = {xdb, ydb, zdb};
        double coefb = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double *u = vel[c];
            double hx[4], s[4];
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                double a = 0., b = 0.;
#pragma unroll
                for (int j = 0; j < 8; ++j) {
                    a += hg_[j][m] * u[j];
                    b += hg_[j][m] * fb[c][j];
                }
                coefb += a * b;
                hx[m] = coef * a;
                s[m] = coef * b;
            }
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                double ub = 0.;
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    G[i][m] += fb[c][i] * hx[m] + s[m] * u[i];
                    ub += s[m] * hg_[i][m];
                }
                velb[c][i] += ub;
            }
        }
        // hourgam = gamma - g . h
        double gb[3][8], vib = 0.0;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            double hb[4] = {0., 0., 0., 0.};
#pragma unroll
            for (int i = 0; i < 8; ++i) {
                double a = 0.;
#pragma unroll
                for (int m = 0; m < 4; ++m) {
                    a -= G[i][m] * h[c][m];
                    hb[m] -= G[i][m] * g[c][i];
                }
                gb[c][i] = a;
            }
            // h = vi12 hourmod: vib collects hb . h = vi12 x its adjoint
#pragma unroll
            for (int m = 0; m < 4; ++m) {
                vib += hb[m] * h[c][m];
                hb[m] *= vi12;
            }
            // the modes' signs, transposed
            double *ub = c == 0 ? xb : c == 1 ? yb : zb;
            const double s12 = hb[1] + hb[2], d12 = hb[1] - hb[2];
            const double s03 = hb[0] + hb[3], d03 = hb[0] - hb[3];
            ub[0] += d03 + s12;
            ub[1] += s03 - s12;
            ub[2] -= s03 + d12;
            ub[3] += d12 - d03;
            ub[4] -= d03 + d12;
            ub[5] += d12 - s03;
            ub[6] += s03 + s12;
            ub[7] += d03 - s12;
        }
        volume_gradient_vjp(d, gb, db);
        // coef = -hg 0.01 ss mass vol^(-1/3); vi12 = 1 / (12 vol); vol = volo v
        o.hgb += coefb * geom::div_op(-0.01 * ss * mass, cr);
        o.ssb += coefb * geom::div_op(-hg * 0.01 * mass, cr);
        // the divisions take forward values: an adjoint dividend is 0 for most
        // elements, and a zero dividend takes division's special-operand path
        double volb = coefb * geom::div_op(coef * (-1.0 / 3.0), vol);
        volb -= vib * volinv;
        o.vb += volb * volo;
    }
    differences_vjp(db[0], xb);
    differences_vjp(db[1], yb);
    differences_vjp(db[2], zb);
}

// ---------------------------------------------------------------------------
// CalcMonotonicQGradientsForElems (lulesh.cc:1613-1757).  Per direction
// (zeta: a = Di x Dj, xi: a = Dj x Dk, eta: a = Dk x Di):
//   delx = vol / sqrt(|a|^2 + ptiny),  delv = norm * (a . V),
//   vol = volo vnew, norm = 1 / (vol + ptiny).
// In: node positions/velocities, volo, vnew and the adjoints of
// delx[3], delv[3] (order xi, eta, zeta).  Accumulates node adjoints and
// returns the adjoint of vnew.
// ---------------------------------------------------------------------------
LG_HD void pattern_i(const double *u, double &s) { s = 0.25 * ((u[1] + u[2] + u[6] + u[5]) - (u[0] + u[3] + u[7] + u[4])); }
LG_HD void pattern_j(const double *u, double &s) { s = -0.25 * ((u[0] + u[1] + u[5] + u[4]) - (u[3] + u[2] + u[6] + u[7])); }
LG_HD void pattern_k(const double *u, double &s) { s = 0.25 * ((u[4] + u[5] + u[6] + u[7]) - (u[0] + u[1] + u[2] + u[3])); }
LG_HD V3 pat(void (*f)(const double *, double &), const double *x, const double *y,
             const double *z)
{
    V3 r;
    f(x, r.x);
    f(y, r.y);
    f(z, r.z);
    return r;
}
// the same quarters of the xi, eta, zeta differences of one coordinate
// (geom::diag_directions of its body diagonals), and their adjoints' way back
LG_HD void directions(const double *u, double &i, double &j, double &k)
{
    double D[4];
    geom::body_diagonals(u, D);
    geom::diag_directions(D, i, j, k);
    i *= 0.25;
    j *= 0.25;
    k *= 0.25;
}
LG_HD void directions_vjp(double i, double j, double k, double *ub)
{
    i *= 0.25;
    j *= 0.25;
    k *= 0.25;
    // D0..D3 = r6 - r0, r5 - r3, r7 - r1, r4 - r2; i = D0 + D1 - D2 - D3,
    // j = D0 - D1 + D2 - D3, k = D0 + D1 + D2 + D3
    const double s = i + k, e = k - i;
    const double g0 = s + j, g1 = s - j, g2 = e + j, g3 = e - j;
    ub[6] += g0; ub[0] -= g0;
    ub[5] += g1; ub[3] -= g1;
    ub[7] += g2; ub[1] -= g2;
    ub[4] += g3; ub[2] -= g3;
}

LG_HD double qgrad_vjp(const double *x, const double *y, const double *z, const double *xd,
                       const double *yd, const double *zd, double volo, double vnew,
                       const double delxb[3], const double delvb[3], double *xb, double *yb,
                       double *zb, double *xdb, double *ydb, double *zdb)
{
    const double ptiny = 1.e-36;
    const double vol = volo * vnew;
    const double norm = geom::rcp_op(vol + ptiny);
    V3 Di, Dj, Dk, Vi, Vj, Vk;
    directions(x, Di.x, Dj.x, Dk.x);
    directions(y, Di.y, Dj.y, Dk.y);
    directions(z, Di.z, Dj.z, Dk.z);
    directions(xd, Vi.x, Vj.x, Vk.x);
    directions(yd, Vi.y, Vj.y, Vk.y);
    directions(zd, Vi.z, Vj.z, Vk.z);
    V3 Dib = {0, 0, 0}, Djb = {0, 0, 0}, Dkb = {0, 0, 0}, Vib = {0, 0, 0}, Vjb = {0, 0, 0},
       Vkb = {0, 0, 0};
    double volb = 0.0, normb = 0.0;
    // (P, Q, V, adjoint index) for xi, eta, zeta
    const V3 *Ps[3] = {&Dj, &Dk, &Di}, *Qs[3] = {&Dk, &Di, &Dj}, *Vs[3] = {&Vi, &Vj, &Vk};
    V3 *Pb[3] = {&Djb, &Dkb, &Dib}, *Qb[3] = {&Dkb, &Dib, &Djb}, *Vb[3] = {&Vib, &Vjb, &Vkb};
#pragma unroll
    for (int d = 0; d < 3; ++d) {
        const V3 a = cross(*Ps[d], *Qs[d]);
        const double s = geom::sqrt_op(dot(a, a) + ptiny);
        const double gx = delxb[d], gv = delvb[d];
        const double rs = geom::rcp_op(s);  // gx, an adjoint, is 0 for most elements
        volb += gx * rs;
        const double ka = -gx * (vol * (rs * rs * rs));
        V3 ab = {ka * a.x + gv * norm * Vs[d]->x, ka * a.y + gv * norm * Vs[d]->y,
                 ka * a.z + gv * norm * Vs[d]->z};
        normb += gv * dot(a, *Vs[d]);
        Vb[d]->x += gv * norm * a.x;
        Vb[d]->y += gv * norm * a.y;
        Vb[d]->z += gv * norm * a.z;
        const V3 pb = cross(*Qs[d], ab), qb = cross(ab, *Ps[d]);
        Pb[d]->x += pb.x; Pb[d]->y += pb.y; Pb[d]->z += pb.z;
        Qb[d]->x += qb.x; Qb[d]->y += qb.y; Qb[d]->z += qb.z;
    }
    directions_vjp(Dib.x, Djb.x, Dkb.x, xb);
    directions_vjp(Dib.y, Djb.y, Dkb.y, yb);
    directions_vjp(Dib.z, Djb.z, Dkb.z, zb);
    directions_vjp(Vib.x, Vjb.x, Vkb.x, xdb);
    directions_vjp(Vib.y, Vjb.y, Vkb.y, ydb);
    directions_vjp(Vib.z, Vjb.z, Vkb.z, zdb);
    volb -= normb * norm * norm;
    return volb * volo;  // adjoint of vnew
}

// ---------------------------------------------------------------------------
// One direction of the monotonic limiter (lulesh.cc:1778-1813).  kind_m /
// kind_p: 0 neighbour value, 1 own value (symmetry), 2 zero (free).
// Forward phi; reverse from phib: adjoint of the own value (selfb) and of the
// neighbour values (nbmb, nbpb).
// ---------------------------------------------------------------------------
struct PhiFwd {
    double phi, norm, m, p;
    int branch;  // 0 average, 1 2m, 2 2p, 3 zero, 4 max slope
};

LG_HD PhiFwd phi_forward(double self, double src_m, double src_p, double lim, double maxs)
{
    const double ptiny = 1.e-36;
    PhiFwd f;
    f.norm = geom::rcp_op(self + ptiny);
    f.m = src_m * f.norm;
    f.p = src_p * f.norm;
    double phi = .5 * (f.m + f.p);
    int br = 0;
    const double m2 = f.m * lim, p2 = f.p * lim;
    if (m2 < phi) { phi = m2; br = 1; }
    if (p2 < phi) { phi = p2; br = 2; }
    if (phi < 0.) { phi = 0.; br = 3; }
    if (phi > maxs) { phi = maxs; br = 4; }
    f.phi = phi;
    f.branch = br;
    return f;
}

LG_HD void phi_vjp(const PhiFwd &f, double src_m, double src_p, double lim, double phib,
                   double &selfb, double &srcmb, double &srcpb)
{
    double mb = 0., pb = 0.;
    if (f.branch == 0) { mb = .5 * phib; pb = .5 * phib; }
    else if (f.branch == 1) mb = lim * phib;
    else if (f.branch == 2) pb = lim * phib;
    srcmb = mb * f.norm;
    srcpb = pb * f.norm;
    const double normb = mb * src_m + pb * src_p;
    selfb -= normb * f.norm * f.norm;
}

// qlin / qquad of CalcMonotonicQRegionForElems (lulesh.cc:1892-1916) for an
// element with vdov <= 0.  In: delv[3], delx[3], phi[3], rho; adjoints of
// qlin, qquad.  Out: adjoints of delv, delx, phi, rho.
LG_HD void qlq_vjp(const double delv[3], const double delx[3], const double phi[3], double rho,
                   double qlc, double qqc, double qlb, double qqb, double delvb[3],
                   double delxb[3], double phib[3], double &rhob)
{
    double dx[3];
    bool clip[3];
    double S1 = 0., S2 = 0.;
    for (int d = 0; d < 3; ++d) {
        dx[d] = delv[d] * delx[d];
        clip[d] = dx[d] > 0.;
        if (clip[d]) dx[d] = 0.;
        S1 += dx[d] * (1. - phi[d]);
        S2 += dx[d] * dx[d] * (1. - phi[d] * phi[d]);
    }
    rhob = qlb * (-qlc) * S1 + qqb * qqc * S2;
    for (int d = 0; d < 3; ++d) {
        const double dxb = qlb * (-qlc * rho) * (1. - phi[d]) +
                           qqb * (qqc * rho) * 2. * dx[d] * (1. - phi[d] * phi[d]);
        phib[d] = qlb * (-qlc * rho) * (-dx[d]) + qqb * (qqc * rho) * dx[d] * dx[d] * (-2. * phi[d]);
        delvb[d] = clip[d] ? 0. : dxb * delx[d];
        delxb[d] = clip[d] ? 0. : dxb * delv[d];
    }
}

// ---------------------------------------------------------------------------
// EOS of one element, one repetition (EvalEOSForElems / CalcEnergyForElems /
// CalcPressureForElems / CalcSoundSpeedForElems, lulesh.cc:2014-2324; the
// repetitions recompute identical values, so one pass is the function).
// ---------------------------------------------------------------------------
struct EosConst {
    double e_cut, p_cut, q_cut, eosvmin, eosvmax, pmin, emin, rho0;
};

struct EosFwd {
    double comp, chs, vhalf, bvcH, e1, pH, sscH, qn1, e2, e3, bvc, pn1, sscT, qt, e4, pn2, sscF,
        qn2, ss;
    bool vmin, vmax, e1clamp, pHkeep, sscHsqrt, e3keep, pn1keep, sscTsqrt, e4keep, pn2keep,
        sscFsqrt, qn2keep, sssqrt, comp_gt;
};

// Keeps the compiler from moving the computation of v out of the branch it
// sits in (on the device; nothing on the host).  A hoisted square root or
// division runs for every element, and an element at rest gives it the
// operands of the special-operand path (a zero numerator).
LG_HD void adj_fence(double &v)
{
#ifdef __CUDA_ARCH__
    asm volatile("" : "+d"(v));
#else
    (void)v;
#endif
}

// The sound-speed term; kUnitRho (refdens == 1, decided once by the caller)
// skips x / 1.0, which is x.
template <bool kUnitRho>
LG_HD double ssc_val(double num, double rho0, bool &took_sqrt)
{
    double ssc = kUnitRho ? num : geom::div_op(num, rho0);
    took_sqrt = !(ssc <= .1111111e-36);
    if (!took_sqrt) return .3333333e-18;
    adj_fence(ssc);
    return geom::sqrt_op(ssc);
}

// pressure with its cut-off and clamps; keep = the derivative passes (the
// p_cut noise cut-off keeps it, the eosvmax and pmin clamps do not)
LG_HD double p_eval(const EosConst &K, double bvc, double e, double vc, bool &keep)
{
    double p = bvc * e;
    keep = true;
    if (fabs(p) < K.p_cut) p = 0.0;
    if (vc >= K.eosvmax) { p = 0.0; keep = false; }
    if (p < K.pmin) { p = K.pmin; keep = false; }
    return p;
}

template <bool kUnitRho>
LG_HD EosFwd eos_forward_rho(const EosConst &K, double e_old, double delvc, double p_old,
                             double q_old, double qq, double ql, double vc)
{
    EosFwd f;
    const double c1s = 2.0 / 3.0, sixth = 1.0 / 6.0;
    f.comp = geom::rcp_op(vc) - 1.;
    const double vchalf = vc - delvc * .5;
    f.chs = geom::rcp_op(vchalf) - 1.;
    f.vmin = (K.eosvmin != 0. && vc <= K.eosvmin);
    if (f.vmin) f.chs = f.comp;
    f.vmax = (K.eosvmax != 0. && vc >= K.eosvmax);
    if (f.vmax) { p_old = 0.; f.comp = 0.; f.chs = 0.; }
    f.e1 = e_old - .5 * delvc * (p_old + q_old);
    f.e1clamp = f.e1 < K.emin;
    if (f.e1clamp) f.e1 = K.emin;
    f.bvcH = c1s * (f.chs + 1.);
    f.pH = p_eval(K, f.bvcH, f.e1, vc, f.pHkeep);
    f.vhalf = geom::rcp_op(1. + f.chs);
    f.comp_gt = delvc > 0.;
    if (f.comp_gt) {
        f.qn1 = 0.;
        f.sscH = 0.;
        f.sscHsqrt = false;
    } else {
        f.sscH = ssc_val<kUnitRho>(c1s * f.e1 + f.vhalf * f.vhalf * f.bvcH * f.pH, K.rho0, f.sscHsqrt);
        f.qn1 = f.sscH * ql + qq;
    }
    f.e2 = f.e1 + .5 * delvc * (3.0 * (p_old + q_old) - 4.0 * (f.pH + f.qn1));
    f.e3 = f.e2;
    f.e3keep = true;
    if (fabs(f.e3) < K.e_cut) f.e3 = 0.;
    if (f.e3 < K.emin) { f.e3 = K.emin; f.e3keep = false; }
    f.bvc = c1s * (f.comp + 1.);
    f.pn1 = p_eval(K, f.bvc, f.e3, vc, f.pn1keep);
    if (f.comp_gt) {
        f.qt = 0.;
        f.sscT = 0.;
        f.sscTsqrt = false;
    } else {
        f.sscT = ssc_val<kUnitRho>(c1s * f.e3 + vc * vc * f.bvc * f.pn1, K.rho0, f.sscTsqrt);
        f.qt = f.sscT * ql + qq;
    }
    f.e4 = f.e3 - (7.0 * (p_old + q_old) - 8.0 * (f.pH + f.qn1) + (f.pn1 + f.qt)) * delvc * sixth;
    f.e4keep = true;
    if (fabs(f.e4) < K.e_cut) f.e4 = 0.;
    if (f.e4 < K.emin) { f.e4 = K.emin; f.e4keep = false; }
    f.pn2 = p_eval(K, f.bvc, f.e4, vc, f.pn2keep);
    f.qn2 = f.qn1;
    f.qn2keep = false;
    f.sscF = 0.;
    f.sscFsqrt = false;
    if (!f.comp_gt) {
        f.sscF = ssc_val<kUnitRho>(c1s * f.e4 + vc * vc * f.bvc * f.pn2, K.rho0, f.sscFsqrt);
        f.qn2 = f.sscF * ql + qq;
        f.qn2keep = true;
        if (fabs(f.qn2) < K.q_cut) f.qn2 = 0.;
    }
    f.ss = ssc_val<kUnitRho>(c1s * f.e4 + vc * vc * f.bvc * f.pn2, K.rho0, f.sssqrt);
    return f;
}

LG_HD EosFwd eos_forward(const EosConst &K, double e_old, double delvc, double p_old,
                         double q_old, double qq, double ql, double vc)
{
    if (K.rho0 == 1.0) return eos_forward_rho<true>(K, e_old, delvc, p_old, q_old, qq, ql, vc);
    return eos_forward_rho<false>(K, e_old, delvc, p_old, q_old, qq, ql, vc);
}

struct EosAdj {
    double e_oldb, delvcb, p_oldb, q_oldb, qqb, qlb, vcb;
};

// From the adjoints of (p_new = pn2, e_new = e4, q_new, ss).
LG_HD EosAdj eos_vjp(const EosConst &K, const EosFwd &f, double e_old, double delvc,
                     double p_old_in, double q_old, double qq, double ql, double vc, double pb,
                     double eb, double qb, double ssb)
{
    (void)e_old;
    (void)qq;
    const double c1s = 2.0 / 3.0, sixth = 1.0 / 6.0, r0 = K.rho0;
    const double p_old = f.vmax ? 0. : p_old_in;
    EosAdj a = {0, 0, 0, 0, 0, 0, 0};
    double e4b = eb, pn2b = pb, bvcb = 0.;
    // ss = sqrt((c1s e4 + vc^2 bvc pn2) / rho0)
    if (f.sssqrt) {
        const double nb = ssb * geom::rcp_op(2. * f.ss * r0);
        e4b += nb * c1s;
        a.vcb += nb * 2. * vc * f.bvc * f.pn2;
        bvcb += nb * vc * vc * f.pn2;
        pn2b += nb * vc * vc * f.bvc;
    }
    // q_new
    if (!f.comp_gt && f.qn2keep) {
        const double sb = qb * ql;
        a.qlb += qb * f.sscF;
        a.qqb += qb;
        if (f.sscFsqrt) {
            const double nb = sb * geom::rcp_op(2. * f.sscF * r0);
            e4b += nb * c1s;
            a.vcb += nb * 2. * vc * f.bvc * f.pn2;
            bvcb += nb * vc * vc * f.pn2;
            pn2b += nb * vc * vc * f.bvc;
        }
    }
    double qn1b = 0.;  // q_new = qn1 when delvc > 0 (then qn1 = 0: no flow)
    // pn2 = bvc e4
    if (f.pn2keep) {
        bvcb += pn2b * f.e4;
        e4b += pn2b * f.bvc;
    }
    // e4 = e3 - W delvc / 6
    double e3b = 0., pHb = 0., pn1b = 0., qtb = 0.;
    if (f.e4keep) {
        const double W = 7.0 * (p_old + q_old) - 8.0 * (f.pH + f.qn1) + (f.pn1 + f.qt);
        e3b += e4b;
        const double Wb = -e4b * delvc * sixth;
        a.delvcb += -e4b * W * sixth;
        a.p_oldb += 7. * Wb;
        a.q_oldb += 7. * Wb;
        pHb += -8. * Wb;
        qn1b += -8. * Wb;
        pn1b += Wb;
        qtb += Wb;
    }
    // qt = sscT ql + qq
    if (!f.comp_gt) {
        a.qlb += qtb * f.sscT;
        a.qqb += qtb;
        if (f.sscTsqrt) {
            const double nb = qtb * ql * geom::rcp_op(2. * f.sscT * r0);
            e3b += nb * c1s;
            a.vcb += nb * 2. * vc * f.bvc * f.pn1;
            bvcb += nb * vc * vc * f.pn1;
            pn1b += nb * vc * vc * f.bvc;
        }
    }
    if (f.pn1keep) {
        bvcb += pn1b * f.e3;
        e3b += pn1b * f.bvc;
    }
    // e3 = e2 (cut-offs)
    const double e2b = f.e3keep ? e3b : 0.;
    // e2 = e1 + 0.5 delvc (3 (p_old + q_old) - 4 (pH + qn1))
    double e1b = e2b, bvcHb = 0., vhalfb = 0.;
    {
        const double G = .5 * delvc * e2b;
        a.delvcb += e2b * .5 * (3.0 * (p_old + q_old) - 4.0 * (f.pH + f.qn1));
        a.p_oldb += 3. * G;
        a.q_oldb += 3. * G;
        pHb += -4. * G;
        qn1b += -4. * G;
    }
    // qn1 = sscH ql + qq
    if (!f.comp_gt) {
        a.qlb += qn1b * f.sscH;
        a.qqb += qn1b;
        if (f.sscHsqrt) {
            const double nb = qn1b * ql * geom::rcp_op(2. * f.sscH * r0);
            e1b += nb * c1s;
            vhalfb += nb * 2. * f.vhalf * f.bvcH * f.pH;
            bvcHb += nb * f.vhalf * f.vhalf * f.pH;
            pHb += nb * f.vhalf * f.vhalf * f.bvcH;
        }
    }
    double chsb = -vhalfb * f.vhalf * f.vhalf;
    if (f.pHkeep) {
        bvcHb += pHb * f.e1;
        e1b += pHb * f.bvcH;
    }
    chsb += bvcHb * c1s;
    // e1 = e_old - 0.5 delvc (p_old + q_old)
    if (!f.e1clamp) {
        a.e_oldb += e1b;
        a.delvcb += -.5 * e1b * (p_old + q_old);
        a.p_oldb += -.5 * delvc * e1b;
        a.q_oldb += -.5 * delvc * e1b;
    }
    double compb = bvcb * c1s;
    if (f.vmax) {
        a.p_oldb = 0.;  // p_old, compression, compHalfStep were set to zero
        compb = 0.;
        chsb = 0.;
    }
    if (f.vmin) {
        compb += chsb;  // compHalfStep = compression
        chsb = 0.;
    }
    // chs = 1 / (vc - 0.5 delvc) - 1; comp = 1 / vc - 1.  By reciprocals:
    // at rest chsb and compb are 0, and a zero dividend would send a division
    // down its special-operand path.
    const double vchalf = vc - delvc * .5;
    const double vchb = -chsb * geom::rcp_op(vchalf * vchalf);
    a.vcb += vchb;
    a.delvcb += -.5 * vchb;
    a.vcb += -compb * geom::rcp_op(vc * vc);
    return a;
}

}  // namespace adj
}  // namespace lg
