// fixed_selftest.cc -- the fixed-point element geometry and EOS of the FMA and
// mixed builds (lg_fixed_geometry.cuh, lg_fixed_eos.cuh), evaluated on the host
// beside the same formulas in long double.
//
//   fixed_selftest forces|kinematics|eos|sums|exact|elements|refused
//
// Prints one line for each case and exits 1 when an error exceeds its bound.
// The bounds follow from the formats: see each check.
#include <cmath>
#include <cstdio>
#include <cstring>
#include <limits>
#include <random>
#include <string>

// extended-precision overload for the reference formulas
namespace lg {
namespace geom {
inline long double rsqrt_fast(long double a) { return 1.0L / std::sqrt(a); }
}  // namespace geom
}  // namespace lg
#include "lg_exact_geometry.cuh"
#include "lg_fixed_eos.cuh"
#include "lg_fixed_geometry.cuh"

using namespace lg;
typedef long double R;

static std::mt19937_64 rng(11);
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }
static int fails = 0;
static void report(const char *what, const char *name, double worst, double bound)
{
    const bool ok = worst <= bound;
    std::printf("%s %s: worst %.3e bound %.3e%s\n", what, name, worst, bound, ok ? "" : "  FAIL");
    if (!ok) fails = 1;
}

struct Shape {
    const char *name;
    double jitter, ax, ay, az;  // node jitter in units of the edge; edges
    int at;                     // elements from the origin
    double size;
};
static const Shape kShapes[] = {
    {"cube", 0, 1, 1, 1, 70, 1.125 / 150},     {"origin", 0.05, 1, 1, 1, 0, 1.125 / 30},
    {"moved", 1e-7, 1, 1, 1, 100, 1.125 / 150}, {"bent", 0.1, 1, 1, 1, 40, 1.125 / 96},
    {"worn", 0.25, 1, 1, 1, 5, 1.125 / 8},      {"flat", 0.1, 1, 1, 0.01, 3, 0.1},
    {"large", 0.1, 1, 1, 1, 9, 4096.0},         {"small", 0.1, 1, 1, 1, 9, 1e-6},
    {"behind", 0.1, 1, 1, 1, -9, 0.01}};

static void element(const Shape &s, double x[3][8], double u[3][8], double speed, double spread)
{
    static const int C[3][8] = {{0, 1, 1, 0, 0, 1, 1, 0}, {0, 0, 1, 1, 0, 0, 1, 1},
                                {0, 0, 0, 0, 1, 1, 1, 1}};
    const double e[3] = {s.ax * s.size, s.ay * s.size, s.az * s.size};
    for (int c = 0; c < 3; ++c)
        for (int j = 0; j < 8; ++j) {
            x[c][j] = e[c] * (s.at + C[c][j] + s.jitter * uni(-1, 1));
            u[c][j] = speed * ((c == 1 ? 0.01 : 1.0) + spread * uni(-1, 1));
        }
}

// Corner forces.  hourgam is off by at most 2^-54, hourgam^T u by 8 (2^-54 + 2^-58) u,
// so the hourglass force by 4 (2 x 2^-51 + 16 x 2^-54) k2 u < 2^-47 k2 u; the sum
// of three areas by 3 x 2^-55 of the product of two extents.
static void forces()
{
    for (const Shape &s : kShapes) {
        double worst = 0;
        int taken = 0;
        for (int t = 0; t < 4000; ++t) {
            double x[3][8], u[3][8];
            element(s, x, u, std::exp(uni(-8, 8)), std::exp(uni(-12, 0)));
            const double det = geom::elem_volume(x[0], x[1], x[2]) * (1 + 1e-3 * uni(-1, 1));
            if (!(det > 0)) continue;
            const double pq = t % 5 ? std::exp(uni(-8, 8)) : 0.0, k2 = -std::exp(uni(-8, 8));
            fx::i64 sm[fx::FS_COUNT];
            int unit[3];
            fx::Op hg[8][4];
            bool ok = fx::seedable(det);
            for (int c = 0; c < 3; ++c) ok = fx::force_component(x[c], c, sm, 1, unit[c]) && ok;
            ok = fx::force_shape(sm, 1, unit, fx::recip(det) * (1.0 / 12.0), hg) && ok;
            const fx::Scale s1 = fx::scale_of(pq * 0.125, ok), s2 = fx::scale_of(k2, ok);
            double F[3][8];
            for (int c = 0; c < 3; ++c)
                ok = fx::force_corners(sm, 1, hg, c, s1, unit[0] + unit[1] + unit[2] - unit[c], s2,
                                       u[c], F[c]) && ok;
            if (!ok) continue;
            ++taken;
            R X[3][8], pf[3][8], g[3][8], d[3][12], hm[3][4];
            for (int c = 0; c < 3; ++c) {
                for (int j = 0; j < 8; ++j) X[c][j] = x[c][j];
                geom::elem_differences(X[c], d[c]);
                geom::hourglass_modes(X[c], hm[c]);
            }
            geom::node_normals_x8_diff(pf[0], pf[1], pf[2], d[0], d[1], d[2]);
            geom::volume_gradient_x12_diff(d[0], d[1], d[2], g[0], g[1], g[2]);
            const R vi = 1.0L / (12.0L * (R)det);
            for (int c = 0; c < 3; ++c) {
                R h[4], umax = 0;
                for (int j = 0; j < 8; ++j) umax = std::fmax(umax, std::fabs((R)u[c][j]));
                R shape[8][4];
                for (int m = 0; m < 4; ++m) {
                    h[m] = 0;
                    for (int k = 0; k < 8; ++k) {
                        shape[k][m] = geom::gam<R>(m, k) -
                                      vi * (g[0][k] * hm[0][m] + g[1][k] * hm[1][m] + g[2][k] * hm[2][m]);
                        h[m] += shape[k][m] * (R)u[c][k];
                    }
                }
                R ext[2];
                for (int o = 0; o < 2; ++o) {
                    ext[o] = 0;
                    for (int j = 1; j < 8; ++j)
                        ext[o] = std::fmax(ext[o], std::fabs(X[(c + 1 + o) % 3][j] - X[(c + 1 + o) % 3][0]));
                }
                const R scale = std::ldexp(1.0L, -47) * std::fabs((R)k2) * umax +
                                std::ldexp(1.0L, -51) * (R)pq * 0.125L * 4 * ext[0] * ext[1];
                for (int k = 0; k < 8; ++k) {
                    R f = (R)pq * 0.125L * pf[c][k];
                    R hf = 0;
                    for (int m = 0; m < 4; ++m) hf += shape[k][m] * h[m];
                    f += (R)k2 * hf;
                    const R tol = scale + std::fabs(f) * std::ldexp(1.0L, -51);
                    worst = std::fmax(worst, (double)(std::fabs((R)F[c][k] - f) / tol));
                }
            }
        }
        report("forces", s.name, taken > 2000 ? worst : 9.0, 1.0);
    }
}

// Kinematics.  Volume: three triple products off by 2^-53 of the product of the
// extents, 12 of which are V; areas by 2^-55 of two extents; a direction's
// velocities are exact to 2^-58 of the largest velocity over its extent.
static void kinematics()
{
    for (const Shape &s : kShapes) {
        double worst[4] = {0, 0, 0, 0};
        int taken = 0;
        for (int t = 0; t < 4000; ++t) {
            double x[3][8], u[3][8];
            const double speed = std::exp(uni(-8, 8));
            element(s, x, u, speed, std::exp(uni(-12, 0)));
            if (t % 7 == 0) std::memset(u, 0, sizeof u);
            const double dt2 = 0.02 * s.size * s.az / speed;
            fx::i64 sm[fx::KS_COUNT];
            fx::Op P[3][3], V[3][3];
            int unit[3], lambda[3];
            bool ok = true;
            for (int c = 0; c < 3; ++c) ok = fx::kin_component(x[c], c, sm, 1, P[c], unit[c]) && ok;
            ok = fx::kin_velocities(u, unit, V, lambda) && ok;
            fx::Kinematics k;
            ok = fx::kinematics(sm, 1, P, unit, V, lambda, dt2, k) && ok;
            if (!ok) continue;
            ++taken;
            R X[3][8], U[3][8], ext[3], umax = 0;
            for (int c = 0; c < 3; ++c) {
                ext[c] = 0;
                for (int j = 0; j < 8; ++j) {
                    X[c][j] = x[c][j];
                    U[c][j] = u[c][j];
                    ext[c] = std::fmax(ext[c], std::fabs(X[c][j] - (R)x[c][0]));
                    umax = std::fmax(umax, std::fabs(U[c][j]));
                }
            }
            const R vol = geom::elem_volume(X[0], X[1], X[2]);
            R big = 0;
            const int F[6][4] = {{0, 1, 2, 3}, {4, 7, 6, 5}, {0, 4, 5, 1},
                                 {1, 5, 6, 2}, {2, 3, 7, 6}, {3, 0, 4, 7}};
            for (auto &f : F)
                big = std::fmax(big, geom::area_face_cross(X[0], X[1], X[2], f[0], f[1], f[2], f[3]));
            R D[3][4], Pr[9], Vr[9], g[6];
            for (int c = 0; c < 3; ++c) geom::body_diagonals(X[c], D[c]);
            geom::directions3(D[0], D[1], D[2], Pr);
            for (int c = 0; c < 3; ++c) geom::body_diagonals(U[c], D[c]);
            geom::directions3(D[0], D[1], D[2], Vr);
            const R vdov = geom::velocity_trace_dirs(Pr, Vr, (R)dt2);
            geom::monoq_gradients_dirs(Pr, Vr, vol, g);
            const R box = ext[0] * ext[1] * ext[2], tiny = std::ldexp(1.0L, -51);
            const R least = std::fmin(ext[0], std::fmin(ext[1], ext[2]));
            const R shape = box / vol;  // 1 for a box
            auto rel = [&](double got, R want, R scale) {
                return (double)(std::fabs((R)got - want) / scale);
            };
            worst[0] = std::fmax(worst[0], rel(k.volume, vol, tiny * (vol + box)));
            double r[3][8], rv;
            for (int c = 0; c < 3; ++c)
                for (int j = 0; j < 8; ++j) r[c][j] = x[c][j] - x[c][0];
            worst[0] = std::fmax(worst[0], fx::relative_volume(r, rv) ? rel(rv, vol, tiny * (vol + box)) : 9);
            worst[1] = std::fmax(worst[1], rel(k.arealg, 2 * vol / std::sqrt(big),
                                               8 * tiny * shape * 2 * vol / std::sqrt(big)));
            for (int d = 0; d < 3; ++d)
                worst[2] = std::fmax(worst[2], rel(k.delx[d], g[d], 8 * tiny * shape * g[d]));
            const R rate = 16 * tiny * shape * shape * (umax / least + 1e-30L);
            worst[3] = std::fmax(worst[3], rel(k.vdov, vdov, rate));
            for (int d = 0; d < 3; ++d) worst[3] = std::fmax(worst[3], rel(k.delv[d], g[3 + d], rate));
        }
        const bool some = taken > 2000;
        report("volume", s.name, some ? worst[0] : 9, 1);
        report("length", s.name, some ? worst[1] : 9, 1);
        report("delx", s.name, some ? worst[2] : 9, 1);
        report("rates", s.name, some ? worst[3] : 9, 1);
    }
}

// The EOS of one repetition in long double, branch for branch.
static R sound(R a) { return a <= .1111111e-36L ? .3333333e-18L : std::sqrt(a); }
// (compression + 1 is 1 / v: formed as such, since 1 / v - 1 + 1 would lose the
// leading bits of v in extended precision too)
static R press(R e, R inv, R &b)
{
    b = (R)(2.0 / 3.0) * inv;
    R p = b * e;
    if (std::fabs(p) < (R)1e-7) p = 0;
    return p < 0 ? 0 : p;
}
static void eos_reference(const double a[7], R out[3])
{
    const R e0 = a[0], delv = a[1], pq = (R)a[2] + (R)a[3], qq = a[4], ql = a[5], v = a[6];
    const R inv = 1 / v, half = v - delv * .5L, c = (R)(2.0 / 3.0);
    R e = e0 - .5L * delv * pq, b, q = 0, qt = 0;
    const R ph = press(e, 1 / half, b), w = half;
    if (!(delv > 0)) q = sound(c * e + w * w * b * ph) * ql + qq;
    e += .5L * delv * (3 * pq - 4 * (ph + q));
    if (std::fabs(e) < (R)1e-7) e = 0;
    R p = press(e, inv, b);
    if (!(delv > 0)) qt = sound(c * e + v * v * b * p) * ql + qq;
    e -= (7 * pq - 8 * (ph + q) + (p + qt)) * delv * (R)(1.0 / 6.0);
    if (std::fabs(e) < (R)1e-7) e = 0;
    p = press(e, inv, b);
    if (delv <= 0) {
        q = sound(c * e + v * v * b * p) * ql + qq;
        if (std::fabs(q) < (R)1e-7) q = 0;
    }
    out[0] = p;
    out[1] = e;
    out[2] = q;
}

// Every Num keeps at least 54 bits through the chain of about ten operations:
// results within 2^-49 of the largest term they are summed from.
static void eos()
{
    const char *names[] = {"moving", "rest", "front", "growing", "stretched", "still", "cold"};
    bool fine = true;
    const fx::EosCuts cuts{fx::scale_of(1e-7, fine), fx::scale_of(1e-7, fine),
                           fx::scale_of(1e-7, fine)};
    for (int mode = 0; mode < 7; ++mode) {
        double worst = 0;
        int taken = 0;
        for (int t = 0; t < 20000; ++t) {
            double v = std::exp(uni(-2, 2)), e = std::exp(uni(-10, 20));
            double delv = -std::exp(uni(-25, -1)) * v, p = e / v * .667, q = p * std::exp(uni(-10, 0));
            double qq = q * uni(0, 1), ql = std::sqrt(qq) * uni(0, 1);
            if (mode == 1) { v = 1; e = delv = p = q = qq = ql = 0; }
            if (mode == 2) { e = std::exp(uni(-20, -5)); p = .6 * e; q = qq = std::exp(uni(-5, 15)); ql = std::sqrt(q); }
            if (mode == 3) { delv = -delv; q = qq = ql = 0; }
            if (mode == 4) v = std::exp(uni(3, 18));
            if (mode == 5) delv = uni(-1, 1) * 1e-16;
            if (mode == 6) e = -e * 1e-6;
            const double a[7] = {e, delv, p, q, qq, ql, v};
            fx::EosIn in;
            fx::Num P, E, Q;
            if (!fx::eos_inputs(e, delv, p, q, qq, ql, v, in)) continue;
            if (!fx::eos_repetition(in, cuts, P, E, Q)) continue;
            ++taken;
            R want[3];
            eos_reference(a, want);
            const R scale = std::fabs((R)e) + std::fabs((R)delv) * 8 * (R)(p + q + (double)want[2] + (double)want[0]) + 1e-7L;
            const R tol = std::ldexp(1.0L, -49);
            const R b1 = (R)(2.0 / 3.0) / v;
            worst = std::fmax(worst, (double)(std::fabs((R)fx::real_of(E.m, E.e) - want[1]) / (tol * scale)));
            worst = std::fmax(worst, (double)(std::fabs((R)fx::real_of(P.m, P.e) - want[0]) / (tol * b1 * scale + 1e-30L)));
            worst = std::fmax(worst, (double)(std::fabs((R)fx::real_of(Q.m, Q.e) - want[2]) /
                                              (tol * (want[2] + (R)ql * std::sqrt(scale) + (R)qq + 1e-7L))));
        }
        report("eos", names[mode], taken > 10000 ? worst : 9, 1);
    }
    double r1 = 0, r2 = 0;
    for (int t = 0; t < 400000; ++t) {
        fx::i64 v = (fx::i64)((rng() >> 5) | (1ull << 59)) & ((1ll << 60) - 1);
        if (t % 4 == 1) v = ((fx::i64)1 << 60) - 1 - (fx::i64)(rng() >> (5 + rng() % 59));
        if (t % 4 == 3) v = ((fx::i64)1 << 59) + (fx::i64)(rng() >> (5 + rng() % 59));
        const R got = (R)fx::reciprocal(v), want = std::ldexp(1.0L, 119) / (R)v;
        r1 = std::fmax(r1, (double)std::fabs((got - want) / want));
        fx::Num a = fx::num((fx::i64)((rng() >> 4) >> (rng() % 50)) | 1, (int)(rng() % 400) - 200);
        // significands just below and above powers of two, where the halves carry
        if (t % 4 == 1) a.m = ((fx::i64)1 << 60) - 1 - (fx::i64)(rng() >> (4 + rng() % 60));
        if (t % 4 == 3) a.m = ((fx::i64)1 << 59) + (fx::i64)(rng() >> (5 + rng() % 59));
        const fx::Num s = fx::root(a);
        const R w = std::sqrt(std::ldexp((R)a.m, a.e));
        r2 = std::fmax(r2, (double)std::fabs((std::ldexp((R)s.m, s.e) - w) / w));
    }
    report("reciprocal", "all", r1, std::ldexp(1.0, -56));
    report("root", "all", r2, std::ldexp(1.0, -56));
}

// The sum of eight numbers: each is off by one unit of 2^-59 of the largest, the
// result by half a unit in the last place.
static void sums()
{
    const char *names[] = {"alike", "mixed", "cancel", "zero", "tiny"};
    for (int mode = 0; mode < 5; ++mode) {
        double worst = 0;
        for (int t = 0; t < 20000; ++t) {
            double v[8], got;
            R want = 0, top = 0;
            for (int i = 0; i < 8; ++i) {
                v[i] = uni(-1, 1) * (mode == 1 ? std::exp(uni(-40, 40)) : 1.0);
                if (mode == 2 && i % 2) v[i] = -v[i - 1] * (1 + 1e-13 * uni(-1, 1));
                if (mode == 3 && (i || t % 2)) v[i] = i % 2 ? 0.0 : -0.0;
                if (mode == 4) v[i] *= 1e-240;
                want += v[i];
                top = std::fmax(top, std::fabs((R)v[i]));
            }
            if (!fx::sum_of(v, got)) worst = 9;
            const R tol = 8 * std::ldexp(1.0L, -58) * top + std::ldexp(1.0L, -53) * std::fabs(want);
            if (top == 0) worst = std::fmax(worst, got == 0 ? 0 : 9);
            else worst = std::fmax(worst, (double)(std::fabs((R)got - want) / tol));
        }
        report("sum", names[mode], worst, 1.0);
    }
    double v[8] = {0, 1, std::numeric_limits<double>::infinity(), 0, 0, 0, 0, 0}, got;
    if (fx::sum_of(v, got)) fails = 1;
    v[2] = std::nan("");
    if (fx::sum_of(v, got)) fails = 1;
}

// The strict build's reciprocals, quotients and roots are the hardware's, bit for
// bit, over the whole range: significands at random, sparse, and next to the ends
// of a binade; any exponent; zeros, infinities, NaN and subnormals among them.
static double pick()
{
    uint64_t m = rng() & 0xfffffffffffffull;
    switch (rng() % 6) {
    case 0: m &= rng() & rng(); break;
    case 1: m = (m | rng() | rng()) & 0xfffffffffffffull; break;
    case 2: m = rng() % 64; break;
    case 3: m = 0xfffffffffffffull - rng() % 64; break;
    default: break;
    }
    const uint64_t e = rng() % 3 ? 1019 + rng() % 9 : rng() % 64 ? rng() % 2047 : 2047 * (rng() % 2);
    return fx::from_bits((rng() % 2 << 63) | (e << 52) | m);
}
static void same(const char *what, double a, double b, double got, double want)
{
    if (fx::bits(got) == fx::bits(want) || (got != got && want != want)) return;
    std::printf("%s(%a, %a) = %a, not %a  FAIL\n", what, a, b, got, want);
    fails = 1;
}
// The strict build's integer face areas, volume derivatives and mode sums against
// the same sums in double: the same bits (either zero), or the element is refused,
// which ordinary ones are not.
static void elements()
{
    const double jitter[] = {0.0, 1e-12, 1e-3, 0.1, 0.4};
    long refused = 0, ordinary = 0;
    for (long t = 0; t < 300000 && !fails; ++t) {
        double x[3][8];
        const double scale = std::ldexp(1.0 + (rng() % 1000) / 1000.0, (int)(rng() % 41) - 20);
        const double jit = jitter[rng() % 5];
        const bool stretched = rng() % 4 == 0;
        for (int c = 0; c < 3; ++c) {
            const double at = rng() % 3 ? (double)(rng() % 45) : 0.0;
            for (int j = 0; j < 8; ++j) {
                const int one = c == 0 ? (j ^ j >> 1) & 1 : c == 1 ? j >> 1 & 1 : j >> 2;
                const double u = (double)(rng() >> 11) * 0x1p-53 - 0.5;
                x[c][j] = at + one == 0 ? 0.0 : scale * (at + one + jit * u);
                if (stretched && rng() % 8 == 0) x[c][j] = std::ldexp(x[c][j], -(int)(rng() % 9));
                if (rng() % 64 == 0) x[c][j] = -x[c][j];
            }
        }
        fx::i64 n[24];
        unsigned bad = 0;
        int emax[3];
        for (int c = 0; c < 3; ++c) emax[c] = fx::align8<1>(x[c], n + 8 * c, bad);
        if (!stretched) ordinary += 1;
        if (bad) {
            if (!stretched) refused += 1;
            continue;
        }
        double area[18], dv[24], want[3], w[3][8];
        for (int f = 0; f < 6; f += 2) fx::face_areas<1>(n, emax, f, 2, area);
        for (int f = 0; f < 6; ++f) {
            const unsigned q = fx::face_corners(f);
            lg::geom::face_area_x16(x[0], x[1], x[2], q & 7, q >> 3 & 7, q >> 6 & 7, q >> 9, want[0],
                                want[1], want[2]);
            for (int c = 0; c < 3; ++c)
                if (area[3 * f + c] != want[c]) same("area", f, c, area[3 * f + c], want[c]);
        }
        for (int c = 0; c < 3; ++c) fx::volume_derivatives<1>(n, emax, c, dv, bad);
        lg::geom::volume_derivative(x[0], x[1], x[2], w[0], w[1], w[2]);
        for (int i = 0; i < 24 && !bad; ++i)
            if (dv[i] != w[i / 8][i % 8]) same("derivative", i / 8, i % 8, dv[i], w[i / 8][i % 8]);
        for (int m = 0; m < 4; ++m)
            for (int c = 0; c < 3; ++c) {
                double s = x[c][0] * lg::geom::gam(m, 0);
                for (int j = 1; j < 8; ++j) s += x[c][j] * lg::geom::gam(m, j);
                const double got =
                    fx::double_of(fx::hourglass_mode<1>(n + 8 * c, fx::mode_signs(m)), emax[c]);
                if (got != s) same("mode", m, c, got, s);
            }
        unsigned bad2 = 0;
        double volume = fx::volume_triple<1>(n, emax, 0, bad2);
        volume += fx::volume_triple<1>(n, emax, 1, bad2);
        volume += fx::volume_triple<1>(n, emax, 2, bad2);
        if (!bad2) {
            const double got = volume * (1.0 / 12.0);
            const double ref = lg::geom::elem_volume(x[0], x[1], x[2]);
            if (got != ref) same("volume", 0, 0, got, ref);
        }
        double largest = 0.0;
        for (int f = 0; f < 6; f += 2)
            largest = std::fmax(largest, fx::largest_area_face<1>(n, emax, f, 2, bad2));
        if (!bad2) {
            // the length of a volume 1 is 4 / sqrt(largest)
            const double ref = lg::geom::char_length(x[0], x[1], x[2], 1.0);
            if (4.0 / std::sqrt(largest) != ref) same("length", 0, 0, largest, ref);
        }
        static const int S[3][8] = {{1, 2, 6, 5, 0, 3, 7, 4}, {3, 2, 6, 7, 0, 1, 5, 4},
                                    {4, 5, 6, 7, 0, 1, 2, 3}};
        for (int c = 0; c < 3; ++c) {
            double g[3];
            fx::gradient_sums<1>(n + 8 * c, emax[c], g);
            for (int d = 0; d < 3; ++d) {
                const int *q = S[d];
                const double ref = (x[c][q[0]] + x[c][q[1]] + x[c][q[2]] + x[c][q[3]]) -
                                   (x[c][q[4]] + x[c][q[5]] + x[c][q[6]] + x[c][q[7]]);
                if (g[d] != ref) same("gradient", c, d, g[d], ref);
            }
        }
    }
    if (refused * 50 > ordinary) fails = 1;  // a few change sign across six binades
    std::printf("elements: %ld of %ld ordinary ones refused %s\n", refused, ordinary,
                fails ? "FAIL" : "ok");
}

static void exact()
{
    for (long t = 0; t < 4000000 && !fails; ++t) {
        double a = pick(), b = pick();
        if (t % 97 == 0) a = t % 2 ? 0.0 : -0.0;
        same("div", a, b, fx::exact_div(a, b), a / b);
        same("rcp", b, b, fx::exact_rcp(b), 1.0 / b);
        same("sqrt", a, a, fx::exact_sqrt(a), std::sqrt(a));
        same("a / 2", a, a, fx::times_pow2<-1>(a), a * 0.5);
        same("mul", a, b, fx::exact_mul(a, b), a * b);
        same("8 a", a, a, fx::times_pow2<3>(a), a * 8.0);
        {
            unsigned bad = 0;
            const fx::Factor f = fx::factor(a, bad);
            const fx::Factor g = fx::factor(b, bad);
            const double lo = std::fmin(std::fabs(a), std::fabs(b));
            const double hi = std::fmax(std::fabs(a), std::fabs(b));
            if (!bad) same("product", a, b, fx::product(f, g), a * b);
            if (bad && a == a && b == b && lo > 1e-150 && hi < 1e150)
                same("refused", a, b, 0., 1.);
        }
        same("sqrt of square", a, a, fx::exact_sqrt(a * a), std::sqrt(a * a));
    }
    std::printf("exact: %s\n", fails ? "FAIL" : "ok");
}

// What the formats do not hold is refused: the kernels then take the FP64 path.
static void refused()
{
    const double inf = std::numeric_limits<double>::infinity(), nan = std::nan("");
    for (int what = 0; what < 10; ++what) {
        double x[3][8], u[3][8];
        element(kShapes[3], x, u, 1.0, 0.1);
        double det = geom::elem_volume(x[0], x[1], x[2]), k = 1.0, dt2 = 1e-5;
        bool forces_only = false;
        switch (what) {
        case 0: x[1][3] = nan; break;
        case 1: x[2][0] = inf; break;
        case 2: u[0][5] = nan; break;
        case 3: for (int j = 0; j < 4; ++j) std::swap(x[2][j], x[2][j + 4]); break;  // inverted
        case 4: for (int j = 0; j < 8; ++j) x[2][j] = x[2][0]; break;                 // no height
        case 5: k = inf; forces_only = true; break;
        case 6: for (auto &c : x) for (double &a : c) a *= 0x1p70; break;
        case 7: det = -det; forces_only = true; break;
        case 8: det = 0x1p-130; forces_only = true; break;
        case 9: for (auto &c : x) for (double &a : c) a *= 0x1p-40; det *= 0x1p-120; break;
        }
        fx::i64 sm[fx::FS_COUNT];
        int unit[3], lambda[3];
        fx::Op hg[8][4], P[3][3], V[3][3];
        bool ok = fx::seedable(det);
        for (int c = 0; c < 3; ++c) ok = fx::force_component(x[c], c, sm, 1, unit[c]) && ok;
        ok = fx::force_shape(sm, 1, unit, fx::recip(det) * (1.0 / 12.0), hg) && ok;
        const fx::Scale s = fx::scale_of(k, ok);
        double F[8];
        for (int c = 0; c < 3; ++c)
            ok = fx::force_corners(sm, 1, hg, c, s, unit[0] + unit[1] + unit[2] - unit[c], s, u[c], F) && ok;
        bool kin = true;
        for (int c = 0; c < 3; ++c) kin = fx::kin_component(x[c], c, sm, 1, P[c], unit[c]) && kin;
        kin = fx::kin_velocities(u, unit, V, lambda) && kin;
        fx::Kinematics r;
        kin = fx::kinematics(sm, 1, P, unit, V, lambda, dt2, r) && kin;
        const bool good = !ok && (forces_only || !kin);
        std::printf("refused %d: %s\n", what, good ? "ok" : "FAIL");
        if (!good) fails = 1;
    }
    const double bad[][7] = {{nan, 0, 0, 0, 0, 0, 1}, {1, 0, inf, 0, 0, 0, 1}, {1, 0, 0, 0, 0, 0, 0},
                             {1, 0, 0, 0, 0, 0, -1},  {1, 0, 0, 0, 0, 0, 1e-9}, {1, 0, 0, 0, 0, 0, 1e9},
                             {1e20, 0, 0, 0, 0, 0, 1}, {1, 2.5, 0, 0, 0, 0, 1}};
    for (auto &a : bad) {
        fx::EosIn in;
        const bool ok = fx::eos_inputs(a[0], a[1], a[2], a[3], a[4], a[5], a[6], in);
        std::printf("refused eos: %s\n", ok ? "FAIL" : "ok");
        if (ok) fails = 1;
    }
}

int main(int argc, char **argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "forces") forces();
    else if (what == "kinematics") kinematics();
    else if (what == "eos") eos();
    else if (what == "sums") sums();
    else if (what == "exact") exact();
    else if (what == "elements") elements();
    else if (what == "refused") refused();
    else return 2;
    return fails;
}
