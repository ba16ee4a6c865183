// adjoint_floors_check.cu -- host check that the reverse of a recovery
// decides at the floors as the recorded forward did.  Cells are put where an
// ulp decides: the conserved variables of a density or a squared velocity
// exactly at its bound, so that the recovered one falls a few ulp to either
// side.  For every cell that the taping stage resets, the adjoint that the
// reverse work item gives is compared with the reverse of the forward's own
// recovered primitives; a floor decided the other way changes it by its own
// size.  Tolerance 1e-6 of that size (some 100 roundings amplified by at most
// 1e6 through the pressure's derivative).
#include "grhd_adjoint_items.cuh"

#include <cmath>
#include <cstdio>
#include <random>
#include <vector>

using namespace grhd;
using namespace grhd::adj;

namespace
{
std::mt19937_64 rng(20261206);

double uniform(double a, double b)
{
    return a + (b - a) * std::uniform_real_distribution<double>()(rng);
}
} // namespace

int main()
{
    const double M = 1.0, a = 0.7;
    Options o{};
    o.G = 5.0 / 3.0;
    o.rho_floor = 1e-3;
    o.p_floor = 1e-5;
    o.atmo_vmax2 = 0.3;
    o.src_atmo_factor = 1.0;
    o.rec_maxit = 80;
    o.rec_tol = 1e-12;
    o.rec_pfloor = 1e-12;
    o.rec_vmax2 = 0.9;
    o.theta = 2.0;
    o.use_recon = 1;
    o.dx = 0.5;
    const int n = 16;
    BoxDev b{};
    for (int d = 0; d < 3; ++d)
    {
        b.lo[d] = 0;
        b.hi[d] = n - 1;
        b.in[d] = n;
        b.glo[d] = -2;
        b.ghi[d] = n + 1;
        b.gn[d] = n + 4;
        b.dlo[d] = 0;
        b.dhi[d] = n - 1;
        o.center[d] = -3.1 - 0.7 * d; // the hole lies outside the box
    }
    const int64_t ni = n * n * n;
    b.cs = b.pcs = (int64_t)b.gn[0] * b.gn[1] * b.gn[2];
    b.rcs = ni;
    std::vector<double> un(11 * b.cs), kv(5 * ni, 0.0), acc(5 * ni, 0.0),
        out(11 * b.cs), Y(5 * ni), pY(ni), lam(5 * ni, 0.0), A(5 * ni),
        ra(5 * ni), lamk(5 * ni);
    std::vector<unsigned char> br(ni);
    for (int k = 0; k < n; ++k)
        for (int j = 0; j < n; ++j)
            for (int i = 0; i < n; ++i)
            {
                double x, y, z;
                cell_xyz(o, i, j, k, x, y, z);
                Geo g;
                ks_metric<double, false>(M, a, x, y, z, g, nullptr);
                Prim p;
                p.rho = i % 2 ? o.rho_floor : o.rho_floor * uniform(1, 9);
                p.p = uniform(0, 1) < 0.5 ? o.p_floor * uniform(0.1, 0.9)
                                          : o.p_floor * uniform(1, 9);
                p.eps = p.p / ((o.G - 1.0) * p.rho);
                double v[3] = {uniform(-1, 1), uniform(-1, 1), uniform(-1, 1)};
                const double v2 = i % 2 ? uniform(0.01, 0.2) : o.atmo_vmax2;
                const double s = std::sqrt(v2 / vsq(v, g.gLL));
                for (int d = 0; d < 3; ++d)
                    p.v[d] = s * v[d];
                const Cons c = p2c(p, g.gLL);
                const int64_t q = b.gidx(i, j, k);
                un[kD * b.cs + q] = c.D;
                for (int d = 0; d < 3; ++d)
                    un[(kS1 + d) * b.cs + q] = c.S[d];
                un[kTau * b.cs + q] = c.tau;
            }
    for (double &v : lam)
        v = uniform(-1, 1);
    int reset = 0, near = 0, failures = 0;
    for (int64_t t = 0; t < ni; ++t)
    {
        // stage 3 with k = 0: out = recovery of un
        stage_tape_item(b, o, M, a, un.data(), kv.data(), acc.data(), 3, 0.0,
                        out.data(), Y.data(), pY.data(), br.data(), t);
        proj_rev_item(b, o, M, a, 1.0, lam.data(), Y.data(), pY.data(),
                      br.data(), A.data(), ra.data(), lamk.data(), t);
        if (br[t] != 1)
            continue;
        ++reset;
        int c[3];
        interior_of(b, t, b.in, c);
        double x, y, z;
        cell_xyz(o, c[0], c[1], c[2], x, y, z);
        KsCell kc;
        ks_cell(M, a, x, y, z, kc);
        Geo g;
        ks_geo_of(kc, g);
        const Cons Yc = {Y[t], {Y[ni + t], Y[2 * ni + t], Y[3 * ni + t]},
                         Y[4 * ni + t]};
        Prim pr;
        if (!ks_con2prim(o, kc, Yc, pr) || pr.p != pY[t])
        {
            std::printf("FAIL: not the forward's recovery\n");
            ++failures;
            continue;
        }
        const double v2 = ks_vsq(kc, pr.v);
        near += std::fabs(pr.rho / o.rho_floor - 1.0) < 1e-14 ||
                std::fabs(v2 / o.atmo_vmax2 - 1.0) < 1e-14;
        // the reverse of p2c and of the floors, deciding as the forward did
        Prim fl = pr;
        ks_floors(o, kc, fl);
        const ConsBar Ub = {lam[t],
                            {lam[ni + t], lam[2 * ni + t], lam[3 * ni + t]},
                            lam[4 * ni + t]};
        GeoBar gb;
        zero(gb);
        PrimBar flb = zero_prim_bar(), prb = zero_prim_bar();
        p2c_rev(fl, g.gLL, Ub, flb, gb.gLL);
        {
            // floors_rev, written out
            const double ir = 1.0 / fl.rho, gm1 = o.G - 1.0;
            const double pb = flb.p + flb.eps * ir / gm1;
            const double rb = flb.rho - flb.eps * fl.p * ir * ir / gm1;
            prb.rho = pr.rho > o.rho_floor ? rb : 0.0;
            prb.p = pr.p > o.p_floor ? pb : 0.0;
            if (v2 >= o.atmo_vmax2)
            {
                const double s = std::sqrt(o.atmo_vmax2 / v2);
                double vb = 0.0, vL[3];
                for (int d = 0; d < 3; ++d)
                    vb += flb.v[d] * pr.v[d];
                lower(g.gLL, pr.v, vL);
                for (int d = 0; d < 3; ++d)
                    prb.v[d] = s * (flb.v[d] - vb * vL[d] / v2);
            }
            else
                for (int d = 0; d < 3; ++d)
                    prb.v[d] = flb.v[d];
        }
        ConsBar Yb = zero_cons_bar();
        con2prim_rev(o, Yc, g.gUU, pr.p, prb, Yb, gb.gUU);
        const double want[5] = {Yb.D, Yb.S[0], Yb.S[1], Yb.S[2], Yb.tau};
        double size = 0.0, err = 0.0;
        for (int q = 0; q < 5; ++q)
        {
            size = std::fmax(size, std::fabs(want[q]));
            err = std::fmax(err, std::fabs(want[q] - ra[q * ni + t]));
        }
        if (!(err <= 1e-6 * size) && failures++ < 10)
            std::printf("FAIL cell %d %d %d: off by %.3g of %.3g\n", c[0],
                        c[1], c[2], err, size);
    }
    std::printf("%d reset cells, %d within 1e-14 of a bound, %d failures\n",
                reset, near, failures);
    return failures != 0 || near < 100;
}
