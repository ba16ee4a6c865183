// grhd_kitp.cu -- device kernels of the binary-PN disk driver's source terms
// (alpha viscosity, point-mass sinks); see grhd_kitp.cuh.  One thread per
// interior cell; the viscous fluxes of a tile and its rim are evaluated once,
// into shared memory, from primitives read through L1.
#include "grhd_kitp.cuh"

namespace grhd {

namespace {

__device__ __forceinline__ void cell_of_interior(const BoxDev &b, int64_t t,
                                                 int &i, int &j, int &k)
{
    i = b.lo[0] + (int)(t % b.in[0]);
    const int64_t r = t / b.in[0];
    j = b.lo[1] + (int)(r % b.in[1]);
    k = b.lo[2] + (int)(r / b.in[1]);
}

__device__ __forceinline__ int clampi(int v, int lo, int hi)
{
    return v < lo ? lo : (v > hi ? hi : v);
}

// alpha_dynamic_viscosity (:676-698)
__device__ double dynamic_viscosity(const KitpDev &k, const Options &o,
                                    double rho, double p, const double pos[3])
{
    if (k.alpha == 0.0)
        return 0.0;
    double omega2 = 0.0;
    for (int body = 0; body < 2; ++body)
    {
        double r2 = 1.0e-10;
        for (int d = 0; d < 3; ++d)
        {
            const double dd = pos[d] - k.body[body][d];
            r2 += dd * dd;
        }
        const double y = rsqrt_(r2);
        omega2 += k.mass[body] * (y * y * y);
    }
    const double cs2 = div_(o.G * p, fmax(rho, k.rho_floor_cfg));
    return rho * k.alpha * cs2 * rsqrt_(fmax(omega2, 1.0e-300));
}

// The viscous fluxes of cell (i,j,l) in both directions
// (viscous_flux_for_cell, :700-770): f = (F_x[S_x], F_x[S_y] = F_y[S_x],
// F_y[S_y], F_x[tau], F_y[tau]).
__device__ void viscous_fluxes(const double *__restrict__ s, const BoxDev &b,
                               const Options &o, const KitpDev &k, int i,
                               int j, int l, double f[5])
{
    f[0] = f[1] = f[2] = f[3] = f[4] = 0.0;
    const int64_t g = b.gidx(i, j, l);
    const double rho = __ldg(&s[kRho * b.cs + g]);
    if (rho <= 10.0 * k.atmo_rho_floor)
        return;
    double x, y, z;
    cell_xyz(o, i, j, l, x, y, z);
    const double pos[3] = {x, y, z};
    const double mu =
        dynamic_viscosity(k, o, rho, __ldg(&s[kPress * b.cs + g]), pos);
    if (mu == 0.0)
        return;
    const int iv[2] = {i, j};
    const int64_t step[2] = {1, b.gn[0]};
    double gradv[2][2];
    for (int c = 0; c < 2; ++c)
    {
        const int m = clampi(iv[c] - 1, b.dlo[c], b.dhi[c]) - iv[c];
        const int q = clampi(iv[c] + 1, b.dlo[c], b.dhi[c]) - iv[c];
        const int span = q - m;
        const double den = (span > 1 ? span : 1) * o.dx;
        for (int v = 0; v < 2; ++v)
            gradv[v][c] = div_(__ldg(&s[(kV1 + v) * b.cs + g + q * step[c]]) -
                                   __ldg(&s[(kV1 + v) * b.cs + g +
                                            m * step[c]]),
                               den);
    }
    const double divergence = gradv[0][0] + gradv[1][1];
    const double bulk = (k.beta - 2.0 / 3.0) * divergence;
    const double xx = mu * (gradv[0][0] + gradv[0][0] + bulk);
    const double xy = mu * (gradv[0][1] + gradv[1][0]);
    const double yy = mu * (gradv[1][1] + gradv[1][1] + bulk);
    const double vx = __ldg(&s[kV1 * b.cs + g]);
    const double vy = __ldg(&s[(kV1 + 1) * b.cs + g]);
    f[0] = -xx;
    f[1] = -xy;
    f[2] = -yy;
    f[3] = -xx * vx - xy * vy;
    f[4] = -xy * vx - yy * vy;
}

// A block owns 32 x 8 cells of a plane and evaluates the fluxes of its cells
// and their x and y neighbours once, into shared memory (1.3 evaluations a
// cell; one thread per cell evaluating its four neighbours took 141 us at
// 128 x 128 x 48, three quarters of it in pow; now 30).
constexpr int kVX = 32, kVY = 8;

__global__ void __launch_bounds__(kVX *kVY)
    k_kitp_viscous(double *__restrict__ rhs, int64_t rcs,
                   const double *__restrict__ s, BoxDev b, Options o,
                   KitpDev k)
{
    constexpr int W = kVX + 2, n = W * (kVY + 2);
    __shared__ double F[5][n];
    const int i0 = b.lo[0] + blockIdx.x * kVX;
    const int j0 = b.lo[1] + blockIdx.y * kVY;
    const int tid = threadIdx.y * kVX + threadIdx.x;
    const double w = 1.0 / (2.0 * o.dx);
    for (int l = b.lo[2] + blockIdx.z; l <= b.hi[2]; l += gridDim.z)
    {
        for (int q = tid; q < n; q += kVX * kVY)
        {
            const int u = q % W, v = q / W;
            const int i = i0 - 1 + u, j = j0 - 1 + v;
            const bool corner =
                (u == 0 || u == W - 1) && (v == 0 || v == kVY + 1);
            // cells beyond the domain stand for their clamped neighbours,
            // cells beyond the box's neighbours are not read
            if (corner || i < b.dlo[0] || i > b.dhi[0] || j < b.dlo[1] ||
                j > b.dhi[1] || i > b.hi[0] + 1 || j > b.hi[1] + 1)
                continue;
            double f[5];
            viscous_fluxes(s, b, o, k, i, j, l, f);
#pragma unroll
            for (int c = 0; c < 5; ++c)
                F[c][q] = f[c];
        }
        __syncthreads();
        const int i = i0 + threadIdx.x, j = j0 + threadIdx.y;
        if (i <= b.hi[0] && j <= b.hi[1])
        {
            const int at = (threadIdx.y + 1) * W + threadIdx.x + 1;
            const int xl = at + clampi(i - 1, b.dlo[0], b.dhi[0]) - i;
            const int xh = at + clampi(i + 1, b.dlo[0], b.dhi[0]) - i;
            const int yl = at + W * (clampi(j - 1, b.dlo[1], b.dhi[1]) - j);
            const int yh = at + W * (clampi(j + 1, b.dlo[1], b.dhi[1]) - j);
            const int64_t t = b.iidx(i, j, l);
            rhs[1 * rcs + t] = rhs[1 * rcs + t] - (F[0][xh] - F[0][xl]) * w -
                               (F[1][yh] - F[1][yl]) * w;
            rhs[2 * rcs + t] = rhs[2 * rcs + t] - (F[1][xh] - F[1][xl]) * w -
                               (F[2][yh] - F[2][yl]) * w;
            rhs[4 * rcs + t] = rhs[4 * rcs + t] - (F[3][xh] - F[3][xl]) * w -
                               (F[4][yh] - F[4][yl]) * w;
        }
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256)
    k_kitp_sink_rhs(double *__restrict__ rhs, int64_t rcs,
                    const double *__restrict__ s, BoxDev b, Options o,
                    KitpDev k, double r2max0, double r2max1)
{
    const double r2max[2] = {r2max0, r2max1};
    const int64_t n = b.ivol();
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x)
    {
        int i, j, l;
        cell_of_interior(b, t, i, j, l);
        const int64_t g = b.gidx(i, j, l);
        if (s[kRho * b.cs + g] <= 10.0 * k.atmo_rho_floor)
            continue;
        double x, y, z;
        cell_xyz(o, i, j, l, x, y, z);
        const double rate = kitp_sink(k, r2max, x, y, z);
        if (rate == 0.0)
            continue;
        rhs[0 * rcs + t] -= rate * s[kD * b.cs + g];
        rhs[4 * rcs + t] -= rate * s[kTau * b.cs + g];
        for (int d = 0; d < 3; ++d)
            rhs[(1 + d) * rcs + t] -= rate * s[(kS1 + d) * b.cs + g];
    }
}

__global__ void __launch_bounds__(256)
    k_kitp_sink_decay(double *__restrict__ s, BoxDev b, Options o, KitpDev k,
                      double dt, double r2max0, double r2max1)
{
    const double r2max[2] = {r2max0, r2max1};
    const int64_t n = b.ivol();
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x)
    {
        int i, j, l;
        cell_of_interior(b, t, i, j, l);
        const int64_t g = b.gidx(i, j, l);
        if (s[kD * b.cs + g] <= 0.0)
            continue;
        double x, y, z;
        cell_xyz(o, i, j, l, x, y, z);
        const double rate = kitp_sink(k, r2max, x, y, z);
        if (rate == 0.0)
            continue;
        const double decay = exp(-rate * dt);
        s[kD * b.cs + g] *= decay;
        s[kTau * b.cs + g] *= decay;
        for (int d = 0; d < 3; ++d)
            s[(kS1 + d) * b.cs + g] *= decay;
    }
}

// kitp_primitive (:465-520); the modes scale the midplane surface density.
__device__ Prim kitp_disk_prim(const KitpDiskDev &k, const Options &o,
                               const double pos[3], const Geo &g)
{
    Prim pr = atmosphere(o);
    const double radius = sqrt(pos[0] * pos[0] + pos[1] * pos[1]);
    if (radius <= 1.0e-12)
        return pr;
    const double phi = atan2(pos[1], pos[0]);
    const double h = fmax(k.aspect * radius, 1.0e-12);
    const double vprof = exp(-0.5 * (pos[2] / h) * (pos[2] / h));
    const double zero_sigma = o.rho_floor / k.rho_peak;
    // kitp_sigma_midplane (:408-418) with stable_logistic_cutoff (:398-406)
    const double safe_r = fmax(radius, 1.0e-12);
    const double cavity = k.cavity_factor * k.sep;
    const double cprof =
        (1.0 - k.cavity_delta) * exp(-pow(cavity / safe_r, 12.0)) +
        k.cavity_delta;
    const double arg = -2.0 * (radius - k.outer_cutoff);
    const double cut =
        arg > 700.0 ? 1.0 : (arg < -700.0 ? 0.0 : 1.0 - 1.0 / (1.0 + exp(arg)));
    double sigma = cprof * cut;
    double modes = 1.0;
    for (int m = 0; m < 4; ++m)
        modes += k.amp[m] * cos((m + 1) * phi + k.phase[m]);
    sigma *= modes;
    pr.rho = fmax(o.rho_floor, k.rho_peak * (sigma * vprof + zero_sigma));
    // binary_point_mass_potential (:444-463)
    double pot = 0.0;
    for (int b = 0; b < 2; ++b)
    {
        double r2 = k.soft * k.soft;
        for (int d = 0; d < 3; ++d)
        {
            const double dd = pos[d] - k.body[b][d];
            r2 += dd * dd;
        }
        pot -= k.mass[b] / sqrt(r2);
    }
    const double cs2 =
        fmax(o.p_floor / pr.rho, -pot / (k.mach * k.mach));
    pr.p = fmax(o.p_floor, pr.rho * cs2 / o.G);
    pr.eps = pr.p / ((o.G - 1.0) * pr.rho);
    // kitp_radial_velocity (:420-427), kitp_phi_velocity (:429-442)
    const double v0 = 1.0e-4 * k.omega_bin * k.sep;
    const double vr = v0 * sin(phi) * (radius / k.sep) *
                      exp(-pow(radius / (3.5 * k.sep), 6.0));
    const double total = k.mass[0] + k.mass[1];
    const double wg = sqrt(total / (safe_r * safe_r * safe_r) *
                           fmax(0.0, 1.0 - 1.0 / (k.mach * k.mach)));
    double vphi = 0.0;
    if (wg > 0.0)
        vphi = pow(pow(k.omega_bin, -4.0) + pow(wg, -4.0), -0.25) * safe_r;
    const double cv[3] = {vr * cos(phi) - vphi * sin(phi),
                          vr * sin(phi) + vphi * cos(phi), 0.0};
    for (int d = 0; d < 3; ++d)
        pr.v[d] = (cv[d] + g.shift[d]) / g.lapse;
    floors(o, pr, g.gLL);
    return pr;
}

// fill_kitp_level_data (:522-555): every ghosted cell.
__global__ void __launch_bounds__(256)
    k_kitp_disk_fill(double *__restrict__ s, BoxDev b, Background bg,
                     Options o, KitpDiskDev k)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
         t < b.gvol(); t += (int64_t)gridDim.x * blockDim.x)
    {
        const int i = b.glo[0] + (int)(t % b.gn[0]);
        const int64_t r = t / b.gn[0];
        const int j = b.glo[1] + (int)(r % b.gn[1]);
        const int l = b.glo[2] + (int)(r / b.gn[1]);
        double pos[3];
        cell_xyz(o, i, j, l, pos[0], pos[1], pos[2]);
        Geo g;
        background_metric<false>(bg, pos[0], pos[1], pos[2], g, nullptr);
        const Prim pr = kitp_disk_prim(k, o, pos, g);
        s[kRho * b.cs + t] = pr.rho;
        s[kEps * b.cs + t] = pr.eps;
        s[kPress * b.cs + t] = pr.p;
        for (int d = 0; d < 3; ++d)
            s[(kV1 + d) * b.cs + t] = pr.v[d];
        const Cons c = p2c(pr, g.gLL);
        s[kD * b.cs + t] = c.D;
        s[kTau * b.cs + t] = c.tau;
        for (int d = 0; d < 3; ++d)
            s[(kS1 + d) * b.cs + t] = c.S[d];
    }
}

int blocks_for(int64_t n)
{
    int64_t g = (n + 255) / 256;
    if (g > 148 * 32)
        g = 148 * 32;
    return (int)(g < 1 ? 1 : g);
}

} // namespace

void launch_kitp_viscous_rhs(double *rhs, int64_t rcs, const double *state,
                             const BoxDev &b, const Options &o,
                             const KitpDev &k, cudaStream_t s)
{
    const dim3 grid((b.in[0] + kVX - 1) / kVX, (b.in[1] + kVY - 1) / kVY,
                    b.in[2] < 65535 ? b.in[2] : 65535);
    k_kitp_viscous<<<grid, dim3(kVX, kVY), 0, s>>>(rhs, rcs, state, b, o, k);
}

void launch_kitp_sink_rhs(double *rhs, int64_t rcs, const double *state,
                          const BoxDev &b, const Options &o, const KitpDev &k,
                          cudaStream_t s)
{
    double r2max[2];
    kitp_sink_reach(k, r2max);
    k_kitp_sink_rhs<<<blocks_for(b.ivol()), 256, 0, s>>>(
        rhs, rcs, state, b, o, k, r2max[0], r2max[1]);
}

void launch_kitp_sink_decay(double *state, const BoxDev &b, const Options &o,
                            const KitpDev &k, double dt, cudaStream_t s)
{
    double r2max[2];
    kitp_sink_reach(k, r2max);
    k_kitp_sink_decay<<<blocks_for(b.ivol()), 256, 0, s>>>(
        state, b, o, k, dt, r2max[0], r2max[1]);
}

void launch_kitp_disk_fill(double *state, const BoxDev &b,
                           const Background &bg, const Options &o,
                           const KitpDiskDev &k, cudaStream_t s)
{
    k_kitp_disk_fill<<<blocks_for(b.gvol()), 256, 0, s>>>(state, b, bg, o, k);
}

} // namespace grhd
