// fixed_bounds_selftest.cc -- the fixed-point EOS and geometry of the FMA and mixed builds
// at the bounds of what they admit, against long double on the host.
//
//   fixed_bounds_selftest expanding|floor|sound|rates|quotients
//
// Prints one line for each case and exits 1 when an error exceeds its bound.
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
#include "lg_fixed_eos.cuh"
#include "lg_fixed_geometry.cuh"

using namespace lg;
typedef long double R;

static std::mt19937_64 rng(23);
static double uni(double a, double b) { return std::uniform_real_distribution<double>(a, b)(rng); }
static int fails = 0;
static void report(const char *what, const char *name, double worst, double bound)
{
    const bool ok = worst <= bound;
    std::printf("%s %s: worst %.3e bound %.3e%s\n", what, name, worst, bound, ok ? "" : "  FAIL");
    if (!ok) fails = 1;
}

// One EOS repetition (lulesh.cc:2048-2176 with refdens 1 and pmin 0) in long double, the
// energy floor emin = -1e15 and the sound speed's floor among its branches.
static R sound(R a) { return a <= .1111111e-36L ? .3333333e-18L : std::sqrt(a); }
static R press(R e, R inv, R &b)
{
    b = (R)(2.0 / 3.0) * inv;
    R p = b * e;
    if (std::fabs(p) < (R)1e-7) p = 0;
    return p < 0 ? 0 : p;
}
// terms: the magnitudes that e and q are summed from
static void eos_reference(const double a[7], R out[3], R &e_terms, R &q_terms)
{
    const R e0 = a[0], delv = a[1], pq = (R)a[2] + (R)a[3], qq = a[4], ql = a[5], v = a[6];
    const R apq = std::fabs((R)a[2]) + std::fabs((R)a[3]), ad = std::fabs(delv);
    const R inv = 1 / v, half = v - delv * .5L, c = (R)(2.0 / 3.0), emin = -1e15L;
    R e = e0 - .5L * delv * pq, b, q = 0, qt = 0;
    e_terms = std::fabs(e0) + 4 * ad * apq;
    if (e < emin) e = emin;
    const R ph = press(e, 1 / half, b);
    if (!(delv > 0)) q = sound(c * e + half * half * b * ph) * ql + qq;
    e_terms += 4 * ad * (ph + std::fabs(q));
    e += .5L * delv * (3 * pq - 4 * (ph + q));
    if (std::fabs(e) < (R)1e-7) e = 0;
    if (e < emin) e = emin;
    R p = press(e, inv, b);
    if (!(delv > 0)) qt = sound(c * e + v * v * b * p) * ql + qq;
    e_terms += ad * (p + std::fabs(qt));
    e -= (7 * pq - 8 * (ph + q) + (p + qt)) * delv * (R)(1.0 / 6.0);
    if (std::fabs(e) < (R)1e-7) e = 0;
    if (e < emin) e = emin;
    p = press(e, inv, b);
    q = 0;
    q_terms = 0;
    if (delv <= 0) {
        const R s = sound(c * e + v * v * b * p);
        q = s * ql + qq;
        q_terms = (s + std::sqrt(e_terms)) * std::fabs(ql) + std::fabs(qq);
        if (std::fabs(q) < (R)1e-7) q = 0;
    }
    out[0] = p;
    out[1] = e;
    out[2] = q;
}
static const double kCut = 1e-7;
// false: the repetition is refused (the kernels take the FP64 form)
static bool eos_fixed(const double a[7], double got[3])
{
    bool fine = true;
    const fx::EosCuts cuts{fx::scale_of(kCut, fine), fx::scale_of(kCut, fine),
                           fx::scale_of(kCut, fine)};
    fx::EosIn in;
    fx::Num P, E, Q;
    if (!fx::eos_inputs(a[0], a[1], a[2], a[3], a[4], a[5], a[6], in)) return false;
    if (!fx::eos_repetition(in, cuts, P, E, Q)) return false;
    got[0] = fx::real_of(P.m, P.e);
    got[1] = fx::real_of(E.m, E.e);
    got[2] = fx::real_of(Q.m, Q.e);
    return true;
}
// the error in units of 2^-48 of the summed terms (each of about ten operations in a row
// keeps 54 bits or more: 10 x 2^-54 < 2^-50 of every term; a cut on either side is 1e-7)
static double eos_error(const double a[7], const double got[3])
{
    R want[3], et, qt;
    eos_reference(a, want, et, qt);
    const R tol = std::ldexp(1.0L, -48), cut = 2e-7L;
    const R b = (R)(2.0 / 3.0) / a[6];
    double w = (double)(std::fabs((R)got[1] - want[1]) / (tol * et + cut));
    w = std::fmax(w, (double)(std::fabs((R)got[0] - want[0]) / (b * (tol * et + cut) + cut)));
    // the root of a cancelled energy is off by the root of its error
    const R dq = std::sqrt(2 * (tol * et + cut)) * std::fabs((R)a[5]);
    return std::fmax(w, (double)(std::fabs((R)got[2] - want[2]) / (tol * qt + dq + cut)));
}

// Expanding elements, whose viscosity the EOS drops however large qq and ql are
static void expanding()
{
    double worst = 0;
    int taken = 0;
    for (int t = 0; t < 100000; ++t) {
        const double v = std::exp(uni(-5, 5)), p = std::exp(uni(-5, 10));
        const double a[7] = {uni(-1, 1) * std::exp(uni(-5, 10)), v * std::exp(uni(-12, -.1)), p,
                             p * uni(0, 1), std::exp(uni(0, 32)), std::exp(uni(0, 32)), v};
        double got[3];
        if (!eos_fixed(a, got)) continue;
        ++taken;
        worst = std::fmax(worst, eos_error(a, got));
    }
    report("expanding", "large qq", taken > 90000 ? worst : 9, 1);
}

// Energies far below any floor: p, q and the volume's change near the largest admitted
static void floor_energy()
{
    const double far[][7] = {{0, 31, 1.4e14, 0, 0, 0, 63}, {0, -57, 1e14, 0, 0, 0, 64},
                             {-1.3e14, 40, 1.2e14, 0, 0, 0, 90}, {0, -1e8, 1e13, 1e13, 1e13, 1e3, 1.1e8}};
    for (auto &a : far) {
        double got[3], w = 0;
        const bool taken = eos_fixed(a, got);
        if (taken) w = eos_error(a, got);
        report("floor", taken ? "taken" : "refused", w, 1);
    }
    double worst = 0;
    int taken = 0, ordinary = 0;
    for (int t = 0; t < 400000; ++t) {
        const double v = std::exp(uni(-19, 19));
        double a[7] = {uni(-1, 1) * std::exp(uni(0, 32.5)), uni(-1, 1) * v * std::exp(uni(-6, 0)),
                       std::exp(uni(0, 32.5)), std::exp(uni(0, 32.5)), std::exp(uni(0, 32.5)),
                       std::exp(uni(-10, 10)), v};
        if (t % 3 == 1) a[3] = a[4] = a[5] = 0;
        double got[3];
        if (!eos_fixed(a, got)) continue;
        ++taken;
        worst = std::fmax(worst, eos_error(a, got));
    }
    // a blast's states stay in: energies to 1e12, a third of the volume's change
    for (int t = 0; t < 20000; ++t) {
        const double v = std::exp(uni(-2, 2)), e = std::exp(uni(0, 27.6)), p = e / v * .667;
        const double a[7] = {e, uni(-.3, .3) * v, p, uni(0, 1) * p, uni(0, 1) * p, std::sqrt(p), v};
        double got[3];
        ordinary += eos_fixed(a, got);
    }
    std::printf("floor: %d of 400000 taken, %d of 20000 ordinary\n", taken, ordinary);
    report("floor", "admitted", taken > 40000 && ordinary == 20000 ? worst : 9, 1);
}

// The sound speed's floor: energies around .1111111e-36 and far from it, ahead of its
// square root.  A product of 2^-58, a root of 2^-57 and the rounding to 53 bits: 2^-52.
static void sound_floor()
{
    double worst = 0;
    for (int t = 0; t < 200000; ++t) {
        const double e = t % 8 ? std::exp(std::log(1e-37) + uni(-3, 3)) : std::exp(uni(-200, 30));
        const double q = t % 64 ? e : t % 128 ? 0.0 : -e;
        for (int p = 0; p < 2; ++p) {
            bool ok = true;
            const fx::Num E = fx::scale_of(q, ok);
            const fx::Num r = fx::sound_speed(E, fx::num(p ? 1 : 0, -60), true);
            const R c = (R)(2.0 / 3.0), want = sound((p ? c + c * c : c) * (R)q);
            worst = std::fmax(worst, (double)(std::fabs((R)fx::real_of(r.m, r.e) - want) / want));
        }
    }
    report("sound", "floor", worst, std::ldexp(1.0, -52));
}

// Velocity components of different sizes: a stream or a shear in x beside a compression
// of ratio in y, a plane wave, a moving frame.  Both rates are sums of
// cofactor x velocity difference; with each term's factors at full precision the error
// is that of an evaluation in double: about 16 roundings of 2^-53 (two products and a
// difference for each half-step cofactor, three products, the divisor) of the terms'
// sum of magnitudes.  On a regular mesh no term cancels and the results have it of
// themselves.
struct Flow {
    const char *name;
    int kind;
    double jitter;
};
static void rates()
{
    static const int C[3][8] = {{0, 1, 1, 0, 0, 1, 1, 0}, {0, 0, 1, 1, 0, 0, 1, 1},
                                {0, 0, 0, 0, 1, 1, 1, 1}};
    const Flow flows[] = {{"stream", 0, 0}, {"stream, bent", 0, .02}, {"shear", 1, 0},
                          {"shear, bent", 1, .02}, {"shear, worn", 1, .2}, {"wave, bent", 2, .02},
                          {"frame", 3, 0}, {"frame, bent", 3, .02}};
    const R unit = std::ldexp(1.0L, -53);
    for (const Flow &f : flows) {
        double worst = 0;
        int taken = 0;
        for (int t = 0; t < 12000; ++t) {
            const double ratio = std::pow(10.0, -(double)(t % 13));
            const double h = uni(.5, 1.5) / 64;
            const int at[3] = {2 + (int)(rng() % 60), 2 + (int)(rng() % 60), 2 + (int)(rng() % 60)};
            double x[3][8], u[3][8];
            const double a = uni(.5, 1.5), b = ratio * uni(.5, 1.5);
            for (int j = 0; j < 8; ++j) {
                for (int c = 0; c < 3; ++c) x[c][j] = h * (at[c] + C[c][j] + f.jitter * uni(-1, 1));
                const double frame = f.kind == 3 ? 1 : 0;
                u[0][j] = f.kind == 0 ? 7 * a : f.kind == 1 ? a * x[1][j] : f.kind == 2 ? -a * x[0][j]
                                                                              : 3 * a - b * x[0][j];
                u[1][j] = f.kind == 2 ? 0 : 2 * frame * a - b * x[1][j];
                u[2][j] = frame * a;
            }
            const double dt2 = 1e-4;
            fx::i64 sm[fx::KS_COUNT];
            fx::Op P[3][3], V[3][3];
            int u0[3], lambda[3];
            bool ok = true;
            for (int c = 0; c < 3; ++c) ok = fx::kin_component(x[c], c, sm, 1, P[c], u0[c]) && ok;
            ok = fx::kin_velocities(u, u0, V, lambda) && ok;
            fx::Kinematics k;
            ok = fx::kinematics(sm, 1, P, u0, V, lambda, dt2, k) && ok;
            if (!ok) continue;
            ++taken;
            R X[3][8], U[3][8], D[3][4], Pr[9], Vr[9], g[6], sum[3], ph[3][3];
            for (int c = 0; c < 3; ++c)
                for (int j = 0; j < 8; ++j) {
                    X[c][j] = x[c][j];
                    U[c][j] = u[c][j];
                }
            const R vol = geom::elem_volume(X[0], X[1], X[2]);
            for (int c = 0; c < 3; ++c) geom::body_diagonals(X[c], D[c]);
            geom::directions3(D[0], D[1], D[2], Pr);
            for (int c = 0; c < 3; ++c) {
                geom::body_diagonals(U[c], D[c]);
                sum[c] = 0;
                for (R d : D[c]) sum[c] += std::fabs(d);
            }
            geom::directions3(D[0], D[1], D[2], Vr);
            const R vdov = geom::velocity_trace_dirs(Pr, Vr, (R)dt2);
            geom::monoq_gradients_dirs(Pr, Vr, vol, g);
            R det = 0, trace_terms = 0;
            for (int c = 0; c < 3; ++c)
                for (int d = 0; d < 3; ++d) ph[c][d] = Pr[3 * c + d] - dt2 * Vr[3 * c + d];
            for (int c = 0; c < 3; ++c) {
                const int i = (c + 1) % 3, j = (c + 2) % 3;
                det += ph[c][1] * (ph[i][2] * ph[j][0] - ph[i][0] * ph[j][2]);
            }
            double w = 0;
            for (int d = 0; d < 3; ++d) {
                const int p = (d + 1) % 3, q = (d + 2) % 3;
                R terms = 0;
                for (int c = 0; c < 3; ++c) {
                    const int i = (c + 1) % 3, j = (c + 2) % 3;
                    terms += (std::fabs(Pr[3 * i + p] * Pr[3 * j + q]) +
                              std::fabs(Pr[3 * i + q] * Pr[3 * j + p])) * sum[c];
                    trace_terms += (std::fabs(ph[i][p] * ph[j][q]) + std::fabs(ph[i][q] * ph[j][p])) * sum[c];
                }
                terms /= 64 * vol;
                if (f.jitter == 0) terms = std::fabs(g[3 + d]);
                const R err = std::fabs((R)k.delv[d] - g[3 + d]);
                w = std::fmax(w, err == 0 ? 0 : (double)(err / (16 * unit * terms)));
            }
            trace_terms /= std::fabs(det);
            if (f.jitter == 0) trace_terms = std::fabs(vdov);
            const R err = std::fabs((R)k.vdov - vdov);
            w = std::fmax(w, err == 0 ? 0 : (double)(err / (16 * unit * trace_terms)));
            worst = std::fmax(worst, w);
        }
        report("rates", f.name, taken > 11500 ? worst : 9, 1);
    }
}

// The FP64 quotients and roots beside the integer forms: a third-order step from an FP32
// seed leaves 2^-60, and its last operation rounds once (2^-53).  The cube root's residual
// holds the rounding of y^3, a third of which remains.
static void quotients()
{
    const R unit = std::ldexp(1.0L, -53), one = 1 + std::ldexp(1.0L, -6);
    R worst[4] = {0, 0, 0, 0};
    auto err = [&](double got, R want) { return std::fabs(((R)got - want) / want) / unit; };
    for (int t = 0; t < 2000000; ++t) {
        const double b = std::ldexp(1.0 + uni(0, 1), (int)(rng() % 244) - 122);
        const double a = std::ldexp(1.0 + uni(0, 1), (int)(rng() % 100) - 50);
        worst[0] = std::fmax(worst[0], err(fx::recip(b), 1 / (R)b));
        worst[1] = std::fmax(worst[1], err(fx::recip_sqrt(b), 1 / std::sqrt((R)b)));
        worst[2] = std::fmax(worst[2], err(fx::recip_cbrt(b), 1 / std::cbrt((R)b)) / (4.0L / 3));
        worst[3] = std::fmax(worst[3], err(fx::quotient(a, b), (R)a / (R)b));
    }
    const char *names[] = {"recip", "recip_sqrt", "recip_cbrt", "quotient"};
    for (int i = 0; i < 4; ++i) report("quotients", names[i], (double)worst[i], (double)one);
}

int main(int argc, char **argv)
{
    const std::string what = argc > 1 ? argv[1] : "";
    if (what == "expanding") expanding();
    else if (what == "floor") floor_energy();
    else if (what == "sound") sound_floor();
    else if (what == "rates") rates();
    else if (what == "quotients") quotients();
    else return 2;
    return fails;
}
