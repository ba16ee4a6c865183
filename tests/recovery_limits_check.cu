// recovery_limits_check.cu -- host check of what the two root solves
// (c2p_solve with overlapped residuals, con2prim_mixed evaluating them in
// turn) report at the recovery's limits: the same outcome, number of
// iterations and, where they fail, residual (both not a number, or equal to
// within the solver's tolerance), conserved variables that are not finite
// among them.
#include "grhd_device.cuh"

#include <cmath>
#include <cstdio>
#include <limits>

using namespace grhd;

int main()
{
    const double inf = std::numeric_limits<double>::infinity();
    const double nan = std::numeric_limits<double>::quiet_NaN();
    const double gUU[6] = {1, 0, 0, 1, 0, 1};
    Options o{};
    o.rec_tol = 1e-12;
    o.rec_pfloor = 1e-12;
    o.rec_vmax2 = 0.9;
    int failures = 0;
    for (int maxit : {0, 1, 80})
        for (double G : {4.0 / 3.0, 5.0 / 3.0, 1.9, 2.0})
            for (double D : {1e-10, 1e-3, 1.0, 50.0, 0.0, -1.0, inf, nan})
                for (double tau : {1.5e-12, 0.0, -1e-13, -0.5, 1e-3, 0.7, 30.0,
                                   inf, nan})
                    for (double S : {0.0, 1e-12, 0.1, 3.0, 1e3, inf, nan})
                    {
                        o.G = G;
                        o.rec_maxit = maxit;
                        const Cons c = {D, {S, 0.0, 0.0}, tau};
                        Prim a, b;
                        int ia, ib;
                        double ra, rb;
                        const bool oa = con2prim(o, c, gUU, a, &ia, &ra);
                        const bool ob = con2prim_mixed(o, c, gUU, b, &ib, &rb);
                        const bool same_residual =
                            (std::isnan(ra) && std::isnan(rb)) || ra == rb ||
                            std::fabs(ra - rb) <= 1e-12 * (1.0 + std::fabs(rb));
                        if ((oa != ob || ia != ib || !same_residual) &&
                            failures++ < 20)
                            std::printf("FAIL G %g D %g tau %g S %g: ok %d %d, "
                                        "iterations %d %d, residual %g %g\n",
                                        G, D, tau, S, oa, ob, ia, ib, ra, rb);
                    }
    std::printf("%d failures\n", failures);
    return failures != 0;
}
