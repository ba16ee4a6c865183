// face_limits_check.cu -- host check of the FP64 face flux next to states
// that are not numbers or not finite (frozen primitives of an excised
// region): the HLLE flux of a face whose every wave runs away from such a
// state is the other side's physical flux, bit for bit; the limited slope
// beside such a neighbour is the nested minmod's, equal; and without
// reconstruction a cell's face states are its own whatever is beside it.
#include "grhd_device.cuh"

#include <cmath>
#include <cstdio>
#include <limits>
#include <random>

using namespace grhd;

namespace
{
int failures = 0;
std::mt19937_64 rng(20261206);

double uniform(double a, double b)
{
    return a + (b - a) * std::uniform_real_distribution<double>()(rng);
}

bool same(double a, double b)
{
    return a == b || (std::isnan(a) && std::isnan(b));
}

void check(bool ok, const char *what, double got, double want)
{
    if (!ok && failures++ < 20)
        std::printf("FAIL %s: %.17g, not %.17g\n", what, got, want);
}

Options options()
{
    Options o{};
    o.G = 5.0 / 3.0;
    o.rho_floor = 1e-10;
    o.p_floor = 1e-12;
    o.atmo_vmax2 = 0.8;
    o.theta = 2.0;
    o.use_recon = 1;
    return o;
}

// Faces along d = 0 deep inside the horizon (r << 2 M), where every wave runs
// towards the hole: on the +x side of it the right state is upwind, on the
// -x side the left one.
void supersonic_face()
{
    const FaceOpt<double> o = make_face_opt<double>(options());
    const double bad[] = {std::numeric_limits<double>::quiet_NaN(),
                          std::numeric_limits<double>::infinity(),
                          -std::numeric_limits<double>::infinity()};
    const double x = uniform(0.2, 0.4) * (uniform(0, 1) < 0.5 ? -1.0 : 1.0);
    Geo g;
    ks_geo(1.0, 0.0, x, uniform(-0.05, 0.05), uniform(-0.05, 0.05), g);
    double q[5] = {std::pow(10.0, uniform(-6, 0)), 0.0, uniform(-0.1, 0.1),
                   uniform(-0.1, 0.1), uniform(-0.1, 0.1)};
    q[1] = q[0] * uniform(1e-3, 0.3);
    FaceSide up;
    face_side(o, q, g, 0, up);
    check(x > 0.0 ? up.hi < 0.0 : up.lo > 0.0, "upwind speeds", up.lo, up.hi);
    for (double v : bad)
        for (int c = 0; c < 5; ++c)
        {
            double w[5] = {q[0], q[1], q[2], q[3], q[4]};
            w[c] = v;
            const Cons f = x > 0.0 ? state_flux(o, w, q, g, 0)
                                   : state_flux(o, q, w, g, 0);
            check(same(f.D, up.f.D), "upwind flux D", f.D, up.f.D);
            check(same(f.tau, up.f.tau), "upwind flux tau", f.tau, up.f.tau);
            for (int m = 0; m < 3; ++m)
                check(same(f.S[m], up.f.S[m]), "upwind flux S", f.S[m],
                      up.f.S[m]);
        }
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
    const double inf = std::numeric_limits<double>::infinity();
    const double nan = std::numeric_limits<double>::quiet_NaN();
    const double centre[] = {0.0, -0.0, 1.0, -1.0, 2.5e-7, -3e5};
    const double beside[] = {0.0, 1.0, -1.0, 1.0 + 1e-15, 2.5e-7, -3e5,
                             inf, -inf, nan, -nan};
    for (double theta : {1.0, 1.3, 2.0})
        for (double c : centre)
            for (double l : beside)
                for (double r : beside)
                {
                    double want =
                        minmod(theta * (c - l),
                               minmod(0.5 * (r - l), theta * (r - c)));
                    // a plateau's slope is zero: minmod(0, inf) compares
                    // their product, which is not a number, with zero
                    if (l == c && !std::isnan(r))
                        want = 0.0;
                    const double got = limited_slope_f64(l, c, r, theta);
                    check(same(got, want), "limited slope", got, want);
                }
    // differences equal and opposite after rounding
    for (int it = 0; it < 20000; ++it)
    {
        const double c = uniform(-1, 1), h = std::pow(10.0, uniform(-18, 0));
        const double l = c - h, r = c - h * (1.0 + uniform(-1e-16, 1e-16));
        const double want =
            minmod(2.0 * (c - l), minmod(0.5 * (r - l), 2.0 * (r - c)));
        const double got = limited_slope_f64(l, c, r, 2.0);
        check(got == want, "slope at an extremum", got, want);
    }
    Options o = options();
    for (int how = 0; how < 2; ++how)
    {
        o.use_recon = how;
        o.theta = how ? 0.0 : 2.0;
        for (double l : beside)
            for (double r : beside)
            {
                PV pl, pc, pr;
                for (int q = 0; q < 5; ++q)
                {
                    pl.q[q] = l;
                    pc.q[q] = 0.1 + q;
                    pr.q[q] = r;
                }
                const FaceOpt<double> fo = make_face_opt<double>(o);
                double lower[5], upper[5], unused[5];
                cell_states(fo, fo.reach ? pl : pc, pc, pr, unused, upper);
                cell_states(fo, pl, pc, fo.reach ? pr : pc, lower, unused);
                for (int q = 0; q < 5; ++q)
                {
                    check(lower[q] == pc.q[q], "piecewise constant", lower[q],
                          pc.q[q]);
                    check(upper[q] == pc.q[q], "piecewise constant", upper[q],
                          pc.q[q]);
                }
            }
    }
}
} // namespace

int main()
{
    slopes();
    for (int it = 0; it < 2000; ++it)
        supersonic_face();
    std::printf("%d failures\n", failures);
    return failures != 0;
}
