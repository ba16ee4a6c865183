// ks_cell_check.cu -- host check of the FP64 per-cell path: the Kerr-Schild
// cell in terms of l and H (ks_cell, ks_floors, ks_sources, ks_inverse_dt)
// against the general metric with its derivatives (ks_metric,
// static_sources, char_speeds), and the root solve with overlapped residuals
// (c2p_solve) against the one that evaluates them in turn (con2prim_mixed),
// the limited slope against the nested minmod (equal values), and the face
// flux with shared subexpressions against its separate formulas.
//
// Tolerances.  Metric, sources and speeds: some 200 roundings of 1.1e-16,
// conditioned at r >= 2 by at most 10, of the terms' size: 1e-12.  Pressure:
// both solvers accept an iterate with |f| < 1e-12 where f' >= G/(G-1) - 1,
// so they differ by at most 2e-12 (G - 1), G <= 2, beside the rounding of f.
#include "grhd_device.cuh"

#include <algorithm>
#include <cmath>
#include <cstdio>
#include <limits>
#include <random>

using namespace grhd;

namespace
{
int failures = 0;
std::mt19937_64 rng(20261205);

double uniform(double a, double b)
{
    return a + (b - a) * std::uniform_real_distribution<double>()(rng);
}

void check(bool ok, const char *what, double err)
{
    if (!ok && failures++ < 20)
        std::printf("FAIL %s: %.3g\n", what, err);
}

void near(double a, double b, double scale, const char *what)
{
    const double e = std::fabs(a - b) / scale;
    check(e <= 1e-12, what, e);
}

Options options(double G)
{
    Options o{};
    o.G = G;
    o.rho_floor = 1e-10;
    o.p_floor = 1e-12;
    o.atmo_vmax2 = 0.8;
    o.src_atmo_factor = 1.0;
    o.rec_maxit = 80;
    o.rec_tol = 1e-12;
    o.rec_pfloor = 1e-12;
    o.rec_vmax2 = 0.9;
    return o;
}

void solvers(const Options &o, const Cons &c, const double gUU[6])
{
    Prim a, b;
    int ia, ib;
    double ra, rb;
    const bool oa = con2prim(o, c, gUU, a, &ia, &ra);
    const bool ob = con2prim_mixed(o, c, gUU, b, &ib, &rb);
    check(oa == ob, "recovered by one solver only", c.D);
    if (oa && ob)
    {
        const double size = std::fabs(c.tau) + c.D;
        check(std::fabs(a.p - b.p) <= 2e-12 + 1e-13 * size, "pressure",
              a.p - b.p);
        near(a.rho, b.rho, b.rho * (1.0 + 10.0 / size), "density");
    }
}

void cell(double G)
{
    const Options o = options(G);
    const double a = uniform(0, 1) < 0.1 ? 0.0 : uniform(-0.99, 0.99);
    const double R = uniform(2.0, 40.0);
    const double ct = uniform(0, 1) < 0.1 ? 0.0 : uniform(-1, 1);
    const double st = std::sqrt(1.0 - ct * ct), ph = uniform(0, 6.2831853);
    const double x = R * st * std::cos(ph), y = R * st * std::sin(ph),
                 z = R * ct;
    GeoFull f;
    ks_metric<double, true>(1.0, a, x, y, z, f.g, &f);
    KsCell k;
    ks_cell(1.0, a, x, y, z, k);
    double g[6];
    ks_gLL(k, g);
    for (int q = 0; q < 6; ++q)
        near(g[q], f.g.gLL[q], 1.0, "gamma_ij");
    near(k.alpha, f.g.lapse, 1.0, "lapse");
    for (int d = 0; d < 3; ++d)
        near(k.c * k.l[d], f.g.shift[d], 1.0, "shift");

    Prim p;
    p.rho = std::pow(10.0, uniform(-9, 0));
    p.p = p.rho * std::pow(10.0, uniform(-3, 0));
    p.eps = p.p / ((G - 1.0) * p.rho);
    double n[3] = {uniform(-1, 1), uniform(-1, 1), uniform(-1, 1)};
    const double s = std::sqrt(uniform(0, 0.88) / vsq(n, f.g.gLL));
    for (int d = 0; d < 3; ++d)
        p.v[d] = n[d] * s;
    Cons c = p2c(p, f.g.gLL);
    solvers(o, c, f.g.gUU);

    Prim fl = p, fk = p;
    floors(o, fl, f.g.gLL);
    ks_floors(o, k, fk);
    for (int d = 0; d < 3; ++d)
        near(fk.v[d], fl.v[d], 1.0, "floored velocity");
    // a conserved state that is not quite the floored primitives'
    for (int d = 0; d < 3; ++d)
        c.S[d] *= uniform(0.9, 1.1);
    const Cons A = static_sources(fl, c, f);
    const Cons B = ks_sources(o, a, k, x, y, z, fl, c);
    const double scale = (c.D + std::fabs(c.tau) + p.p) * 10.0 / (R * R);
    near(A.D, B.D, scale, "source D");
    near(A.tau, B.tau, scale, "source tau");
    for (int d = 0; d < 3; ++d)
        near(A.S[d], B.S[d], scale, "source S");
    const double inv[3] = {1.0, 2.0, 3.0};
    double speed = 0.0;
    for (int d = 0; d < 3; ++d)
    {
        double lo, hi;
        char_speeds(o, fl, f.g, d, lo, hi);
        speed += std::max(std::fabs(lo), std::fabs(hi)) * inv[d];
    }
    near(ks_inverse_dt(o, k, fl, inv), speed, 10.0, "speed");
}

// Reconstruction.hpp:16-37
double minmod(double l, double r)
{
    if (l * r <= 0.0)
        return 0.0;
    return l > 0.0 ? std::fmin(l, r) : std::fmax(l, r);
}

void slopes()
{
    const double v[] = {0.0, -0.0, 1.0, -1.0, 1e-12, 1.0 + 1e-15, 2.5, -3e5};
    auto one = [](double l, double c, double r, double theta) {
        const double want = minmod(
            theta * (c - l), minmod(0.5 * (r - l), theta * (r - c)));
        const double got = limited_slope_f64(l, c, r, theta);
        check(got == want, "limited slope", got - want);
    };
    for (double theta : {0.0, 1.0, 1.3, 2.0})
    {
        for (double l : v)
            for (double c : v)
                for (double r : v)
                    one(l, c, r, theta);
        for (int it = 0; it < 20000; ++it)
        {
            const double c = uniform(-1, 1);
            one(c + uniform(-1, 1) * std::pow(10.0, uniform(-16, 0)), c,
                c + uniform(-1, 1) * std::pow(10.0, uniform(-16, 0)), theta);
        }
    }
}

// Faces between states that are subsonic, supersonic either way and above
// the velocity cap, at the floors and far from them.
void face(double G)
{
    const Options o = options(G);
    Geo g;
    ks_geo(1.0, uniform(-0.9, 0.9), uniform(2, 20), uniform(-20, 20),
           uniform(-20, 20), g);
    Prim side[2];
    double q[2][5];
    for (int s = 0; s < 2; ++s)
    {
        Prim &p = side[s];
        p.rho = std::pow(10.0, uniform(-11, 0));
        p.p = p.rho * std::pow(10.0, uniform(-4, 0));
        double n[3] = {uniform(-1, 1), uniform(-1, 1), uniform(-1, 1)};
        const double w = std::sqrt(uniform(0, 0.95) / vsq(n, g.gLL));
        for (int d = 0; d < 3; ++d)
            p.v[d] = n[d] * w;
        q[s][0] = p.rho;
        q[s][1] = p.p;
        for (int d = 0; d < 3; ++d)
            q[s][2 + d] = p.v[d];
        floors(o, p, g.gLL);
    }
    for (int d = 0; d < 3; ++d)
    {
        const Cons c[2] = {p2c(side[0], g.gLL), p2c(side[1], g.gLL)};
        const Cons f[2] = {phys_flux(side[0], c[0], d, g.lapse, g.shift),
                           phys_flux(side[1], c[1], d, g.lapse, g.shift)};
        double lo[2], hi[2];
        for (int s = 0; s < 2; ++s)
            char_speeds(o, side[s], g, d, lo[s], hi[s]);
        const double sl = std::fmin(0.0, std::fmin(lo[0], lo[1]));
        const double su = std::fmax(0.0, std::fmax(hi[0], hi[1]));
        auto hlle = [&](double fl, double fr, double cl, double cr) {
            if (sl >= 0.0)
                return fl;
            if (su <= 0.0)
                return fr;
            return (su * fl - sl * fr + sl * su * (cr - cl)) / (su - sl);
        };
        const Cons got =
            state_flux(make_face_opt<double>(o), q[0], q[1], g, d);
        // W^2 <= 5 amplifies rounding, at most ten-fold through the speeds
        const double D = c[0].D + c[1].D;
        const double E = D + c[0].tau + c[1].tau + side[0].p + side[1].p;
        near(got.D, hlle(f[0].D, f[1].D, c[0].D, c[1].D), D, "flux D");
        near(got.tau, hlle(f[0].tau, f[1].tau, c[0].tau, c[1].tau), E,
             "flux tau");
        for (int m = 0; m < 3; ++m)
            near(got.S[m], hlle(f[0].S[m], f[1].S[m], c[0].S[m], c[1].S[m]),
                 5.0 * E, "flux S");
    }
}

// States the recovery meets at its limits.
void limits(double G)
{
    const Options o = options(G);
    const double gUU[6] = {1, 0, 0, 1, 0, 1};
    const double inf = std::numeric_limits<double>::infinity();
    const double nan = std::numeric_limits<double>::quiet_NaN();
    const double Ds[] = {1e-10, 1e-3, 1.0, 50.0, 0.0, -1.0, inf, nan};
    const double taus[] = {1.5e-12, 0.0, -1e-13, -0.5, 1e-3, 0.7, 30.0, inf,
                           nan};
    const double Ss[] = {0.0, 1e-12, 0.1, 3.0, 1e3, inf, nan};
    for (double D : Ds)
        for (double tau : taus)
            for (double S : Ss)
            {
                Cons c;
                c.D = D;
                c.tau = tau;
                c.S[0] = S;
                c.S[1] = c.S[2] = 0.0;
                solvers(o, c, gUU);
            }
}
} // namespace

int main()
{
    for (double G : {4.0 / 3.0, 5.0 / 3.0, 1.9, 2.0})
    {
        for (int it = 0; it < 20000; ++it)
            cell(G);
        for (int it = 0; it < 20000; ++it)
            face(G);
        limits(G);
    }
    slopes();
    std::printf("%d failures\n", failures);
    return failures != 0;
}
