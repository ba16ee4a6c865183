// ks_cell_check.cu -- host check of the FP64 per-cell path: the Kerr-Schild
// cell in terms of l and H (ks_cell, ks_floors, ks_sources, ks_inverse_dt)
// against the general metric with its derivatives (ks_metric,
// static_sources, char_speeds), and the root solve with overlapped residuals
// (c2p_solve) against the one that evaluates them in turn (con2prim_mixed).
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
        limits(G);
    }
    std::printf("%d failures\n", failures);
    return failures != 0;
}
