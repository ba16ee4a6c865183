// grhd_kitp.cuh -- source terms of the reference's binary-PN disk production
// driver (Examples/GRHDLevelDataBinaryPNKITPDisk/
// Main_GRHDLevelDataBinaryPNKITPDisk.cpp): the alpha-viscosity stress
// divergence (:676-806) and the two point-mass sinks (:557-662), on the
// device, FP64.
#pragma once

#include "grhd_kernels.cuh"

#include <cmath>

namespace grhd {

// The driver's SimulationConfig fields these terms read (:63, :67-71), the
// binary's masses and body positions at the evaluation time, and the
// atmosphere floor that switches them off.
struct KitpDev
{
    double alpha, beta, rho_floor_cfg, sink_size, sink_rate, sink_shape;
    double mass[2];
    double body[2][3];
    double atmo_rho_floor;
};

// Squared distance of each body beyond which its sink kernel
// exp(-(r / R)^shape) is exactly zero (the exponent passes 746, where exp
// underflows).
inline void kitp_sink_reach(const KitpDev &k, double r2max[2])
{
    for (int b = 0; b < 2; ++b)
    {
        const double radius = k.sink_size * k.mass[b];
        r2max[b] = k.sink_shape > 0.0
                       ? radius * radius * pow(746.0, 2.0 / k.sink_shape)
                       : HUGE_VAL;
    }
}

// sink_kernel (:557-565) summed over both bodies (:584-597); r2max as
// kitp_sink_reach gives it.
__device__ __forceinline__ double kitp_sink(const KitpDev &k,
                                            const double r2max[2], double x,
                                            double y, double z)
{
    const double pos[3] = {x, y, z};
    double rate = 0.0;
    for (int body = 0; body < 2; ++body)
    {
        double r2 = 0.0;
        for (int d = 0; d < 3; ++d)
        {
            const double dd = pos[d] - k.body[body][d];
            r2 += dd * dd;
        }
        const double radius = k.sink_size * k.mass[body];
        double kern = 0.0;
        if (radius > 0.0 && k.sink_rate != 0.0 && !(r2 > r2max[body]))
            kern = exp(-pow(r2 / (radius * radius), 0.5 * k.sink_shape));
        rate += k.sink_rate * kern;
    }
    return rate;
}

// rhs (interior, 5 components, stride rcs) -= d/dx F_x + d/dy F_y of the
// viscous stress flux (add_kitp_viscous_rhs, :772-806).
void launch_kitp_viscous_rhs(double *rhs, int64_t rcs, const double *state,
                             const BoxDev &b, const Options &o,
                             const KitpDev &k, cudaStream_t s);
// rhs -= rate * conserved (add_kitp_sink_rhs, :567-610).
void launch_kitp_sink_rhs(double *rhs, int64_t rcs, const double *state,
                          const BoxDev &b, const Options &o, const KitpDev &k,
                          cudaStream_t s);
// conserved *= exp(-rate dt) (apply_kitp_sink_decay, :612-662).
void launch_kitp_sink_decay(double *state, const BoxDev &b, const Options &o,
                            const KitpDev &k, double dt, cudaStream_t s);

// The end of the driver's step (advance_kitp_ssprk2, :842-876) on the
// interior: s = (s + u1 + dt k) / 2 (combine_ssprk2_conserved_state,
// FArrayBoxFiniteVolume.hpp:942-969), the sink decay with the bodies of `kd`
// when `sinks`, and the recovery with atmosphere on the background `bg`.
void launch_kitp_finish(double *state, const BoxDev &b, const double *u1,
                        int64_t u1_cs, const double *k, int64_t rcs,
                        const Background &bg, const Options &o,
                        const KitpDev &kd, bool sinks, double dt,
                        DevStatus *st, cudaStream_t s);

// The disk drivers' Keplerian disk (kitp_primitive, :398-520) with the
// azimuthal density modes m = 1..4 (new): the binary (masses, separation,
// softening, orbital frequency, body positions at the fill time) and the
// disk settings of SimulationConfig (:56-61).
struct KitpDiskDev
{
    double mach, aspect, cavity_factor, cavity_delta, outer_cutoff, rho_peak;
    double amp[4], phase[4];
    double sep, mass[2], soft, omega_bin;
    double body[2][3];
};

// Primitives and conserved variables of every ghosted cell.
void launch_kitp_disk_fill(double *state, const BoxDev &b,
                           const Background &bg, const Options &o,
                           const KitpDiskDev &k, cudaStream_t s);

} // namespace grhd
