// grhd_device.cuh -- pointwise device physics of the fixed-background
// Valencia GRHD operator, templated on the arithmetic type T.
//
// T = double is the FP64 path (parity with the reference); T = float is the
// arithmetic of the mixed path's reconstruction, Riemann solver, metric and
// sources.  The con2prim root solve is FP64 in both paths.  Each function
// names the reference function whose result it reproduces (paths relative
// to the GRDzhadzha source tree).  The metric is evaluated in closed form
// rather than through the reference's generic symmetric inverse +
// Christoffel route; the two agree to rounding.
#pragma once

#include <cuda_runtime.h>
#include <stdint.h>

// Pointwise functions of the FP64 path are also host-callable (the host
// test of the adjoint's reverse-mode functions runs them on the CPU); the
// FP32 overloads use device intrinsics and stay device-only.
#define GRHD_HD __host__ __device__

namespace grhd {

// Symmetric 3x3 packing: 00 01 02 11 12 22.
__host__ __device__ constexpr int sym(int i, int j)
{
    return (i <= j) ? (i == 0 ? j : (i == 1 ? 2 + j : 5))
                    : (j == 0 ? i : (j == 1 ? 2 + i : 5));
}

// ------------------------------------------------------------- arithmetic
// FP64 on the device: division, reciprocal and square root from the
// hardware's approximate reciprocal (square root) refined by Newton-Raphson
// steps, within about one ulp of the IEEE result (checked against it by
// grhd_eval_arith's test) and without the IEEE operations' special-case
// branches, which the face and stage kernels pay on every call.  Their
// domain is that of the quantities they are used on -- densities,
// enthalpies, metric functions, speed differences and squared norms:
// normal numbers up to 2^1021, and 0 for the square root; a zero divisor
// or a quotient that overflows gives NaN (not +-inf), and a subnormal
// operand is flushed to zero.  The oracle and the host keep IEEE
// division.  FP32: the SFU
// reciprocal / reciprocal square root (a few ulp), which is what makes the
// FP32 path cheap.

#ifdef __CUDA_ARCH__
// 1/a: the approximate reciprocal (rcp.approx.ftz.f64, about 20 correct
// bits) and two Newton-Raphson steps y <- y + y (1 - a y), each of which
// squares the relative error.
__device__ __forceinline__ double rcp_newton(double a)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
#pragma unroll
    for (int it = 0; it < 2; ++it)
        y = fma(y, fma(-a, y, 1.0), y);
    return y;
}
#endif

// a / b: the quotient q = a y with y ~ 1/b, corrected once by its exact
// residual r = a - b q (one fused multiply-add): q + r y (Markstein's
// correction, IBM J. Res. Dev. 34 (1990) 111-119).
GRHD_HD __forceinline__ double div_(double a, double b)
{
#ifdef __CUDA_ARCH__
    const double y = rcp_newton(b);
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
#else
    return a / b;
#endif
}
__device__ __forceinline__ float div_(float a, float b)
{
    return __fdividef(a, b);
}
GRHD_HD __forceinline__ double rcp_(double a)
{
#ifdef __CUDA_ARCH__
    const double y = rcp_newton(a);
    return fma(y, fma(-a, y, 1.0), y);
#else
    return 1.0 / a;
#endif
}
__device__ __forceinline__ float rcp_(float a) { return __fdividef(1.0f, a); }
// FP64 reciprocal square root: the hardware's approximate rsqrt
// (rsqrt.approx.ftz.f64, a few ulp of FP32 accuracy) refined by two
// Newton-Raphson steps y <- y + y (1 - a y^2) / 2, each of which squares
// the relative error; the result is within a few ulp of 1/sqrt(a), for
// one MUFU operation and eight FP64 ones instead of an IEEE square root
// followed by an IEEE division.  a > 0 (the callers pass 1 - v^2 with v^2
// below its cap, or a squared norm).
GRHD_HD __forceinline__ double rsqrt_(double a)
{
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
#pragma unroll
    for (int it = 0; it < 2; ++it)
    {
        const double e = fma(-(a * y), y, 1.0);
        y = fma(0.5 * y, e, y);
    }
    return y;
#else
    return 1.0 / sqrt(a);
#endif
}
__device__ __forceinline__ float rsqrt_(float a) { return rsqrtf(a); }
// sqrt(a) = a / sqrt(a): s = a y with y ~ 1/sqrt(a) (rsqrt_), corrected by
// one Newton step on s^2 = a, s + (a - s^2) y / 2; a = 0 returns 0 and a
// negative a NaN.
GRHD_HD __forceinline__ double sqrt_(double a)
{
#ifdef __CUDA_ARCH__
    const double y = rsqrt_(a);
    const double s = a * y;
    const double r = fma(0.5 * y, fma(-s, s, a), s);
    return a > 0.0 ? r
                   : (a == 0.0 ? a : __longlong_as_double(0x7ff8000000000000ll));
#else
    return sqrt(a);
#endif
}
__device__ __forceinline__ float sqrt_(float a) { return sqrtf(a); }
// A product that is never fused into a following sum.  Code shared by
// kernels that must agree bit for bit writes its sums as fma() and its
// products as mul_(), so that no compiler choice of fused pairs is left.
GRHD_HD __forceinline__ double mul_(double a, double b)
{
#ifdef __CUDA_ARCH__
    return __dmul_rn(a, b);
#else
    return a * b;
#endif
}
// 1/a within 0.51 ulp and 1/sqrt(a) within 1.02 (grhd_eval_arith_ulp's test):
// one step of
// the third-order iteration (Householder's) from the approximate value y0 of
// relative error d <= 2^-20: with e = 1 - a y0, 1/a = y0 (1 + e + e^2) up to
// d^3; with e = 1 - a y0^2, a^-1/2 = y0 (1 + e/2 + 3 e^2/8) up to d^3.  Three
// and five FP64 operations instead of the six and eight of two
// Newton-Raphson steps (and rcp_'s correction), with a shorter chain.
GRHD_HD __forceinline__ double rcp_ulp(double a)
{
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-a, y, 1.0);
    return fma(y, fma(e, e, e), y);
#else
    return 1.0 / a;
#endif
}
GRHD_HD __forceinline__ double rsqrt_ulp(double a)
{
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-(a * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
#else
    return 1.0 / sqrt(a);
#endif
}
GRHD_HD __forceinline__ double max_(double a, double b) { return fmax(a, b); }
__device__ __forceinline__ float max_(float a, float b) { return fmaxf(a, b); }
GRHD_HD __forceinline__ double min_(double a, double b) { return fmin(a, b); }
__device__ __forceinline__ float min_(float a, float b) { return fminf(a, b); }
GRHD_HD __forceinline__ double abs_(double a) { return fabs(a); }
__device__ __forceinline__ float abs_(float a) { return fabsf(a); }
// the lapse (1 + 2H)^-1/2 of the Kerr-Schild metric
GRHD_HD __forceinline__ double lapse_rsqrt(double a)
{
#ifdef __CUDA_ARCH__
    return rsqrt(a);
#else
    return 1.0 / sqrt(a);
#endif
}
__device__ __forceinline__ float lapse_rsqrt(float a) { return rsqrtf(a); }

template <typename T> struct PrimT
{
    T rho, eps, p, v[3];
};

template <typename T> struct ConsT
{
    T D, S[3], tau;
};

// Face / cell geometry needed by con2prim, floors and the HLLE flux
// (the members of CellGeometryData, StaticMetric.hpp:19-40, minus K).
template <typename T> struct GeoT
{
    T gLL[6], gUU[6], lapse, shift[3];
};

// Everything the static-metric sources need
// (make_static_metric_derivatives_from_adm, FixedBGMetric.hpp:31-53).
template <typename T> struct GeoFullT
{
    GeoT<T> g;
    T K[6];
    T dlapse[3];
    T dlnsqrtg[3];
    T dgamma[3][6]; // [direction][sym(i,j)]
    T dshift[3][3]; // [i][direction] = d_direction shift^i
};

// Cell primitives as stored for the stencil: rho, p, v (eps is always
// recomputed by the floors before use, Atmosphere.hpp:43-45).
template <typename T> struct PVT
{
    T q[5]; // rho, p, v0, v1, v2
};

using Prim = PrimT<double>;
using Cons = ConsT<double>;
using Geo = GeoT<double>;
using GeoFull = GeoFullT<double>;
using PV = PVT<double>;

// Background constants for one evaluation time.  For the binary the
// orbital state (positions, velocities) is evaluated on the host once per
// call, as CircularBinaryPN::compute_state does per cell (:219-250).
struct Background
{
    int kind; // 0 Kerr-Schild, 1 binary PN
    double M, a;
    double m1, m2, soft2;
    double p1[3], p2[3], v1[3], v2[3];
    // positions at t + h and t - h for the volume-time source FD
    double p1p[3], p2p[3], p1m[3], p2m[3];
    double fd_h;
};

struct Options
{
    double G;           // adiabatic index
    double rho_floor, p_floor, atmo_vmax2, src_atmo_factor;
    int rec_maxit;
    double rec_tol, rec_pfloor, rec_vmax2;
    double theta;
    int use_recon, use_src, use_vol;
    double excision_radius;
    double accretion_radius; // > 0: Mdot through the sphere r < R (new)
    double dx, center[3];
};

// ---------------------------------------------------------------- metric

// Kerr-Schild metric of mass M, spin a at (x,y,z) relative to the hole:
// gamma_ij = delta_ij + 2 H l_i l_j, lapse (1+2H)^-1/2,
// shift^i = 2H l^i/(1 + 2H l.l), gamma^ij by Sherman-Morrison
// (KerrSchild.hpp:64-166; derivatives as get_KS_derivs, :171-242).
template <typename T, bool FULL>
GRHD_HD __forceinline__ void ks_metric(T M, T a, T x, T y, T z,
                                          GeoT<T> &g, GeoFullT<T> *f)
{
    const T a2 = a * a;
    const T rho = max_(sqrt_(x * x + y * y + z * z), T(1.0e-6));
    const T rho2 = rho * rho;
    const T A = rho2 - a2;
    const T Q = sqrt_(T(0.25) * A * A + a2 * z * z);
    const T r2 = T(0.5) * A + Q;
    const T r = sqrt_(r2);
    const T inv_r = rcp_(r);
    const T ct = z * inv_r;
    const T Sigma = r2 + a2 * ct * ct;
    const T H = div_(M * r, Sigma);
    const T inv_ra = rcp_(r2 + a2);
    const T l[3] = {(r * x + a * y) * inv_ra, (r * y - a * x) * inv_ra,
                    z * inv_r};
    const T ll = l[0] * l[0] + l[1] * l[1] + l[2] * l[2];
    const T twoH = T(2) * H;
    const T den = T(1) + twoH * ll;
    const T c = div_(twoH, den); // Sherman-Morrison coefficient
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = i; j < 3; ++j)
        {
            const T ll_ij = l[i] * l[j];
            g.gLL[sym(i, j)] = (i == j ? T(1) : T(0)) + twoH * ll_ij;
            g.gUU[sym(i, j)] = (i == j ? T(1) : T(0)) - c * ll_ij;
        }
    g.lapse = lapse_rsqrt(T(1) + twoH);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        g.shift[i] = c * l[i];
    if (!FULL)
        return;

    // derivatives of r, cos(theta), H and l (derivative index last)
    const T inv_2Q = div_(T(0.5), Q);
    const T xs[3] = {x, y, z};
    T dr[3], dH[3], dl[3][3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
        const T drho = div_(xs[i], rho);
        dr[i] = T(0.5) * inv_r *
                (rho * drho + inv_2Q * (drho * rho * A +
                                        (i == 2 ? T(2) * a2 * z : T(0))));
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
        const T dct = -z * inv_r * inv_r * dr[i] + (i == 2 ? inv_r : T(0));
        dH[i] = H * (dr[i] * inv_r -
                     div_(T(2), Sigma) * (r * dr[i] + a2 * ct * dct));
    }
    const T nx = r * x + a * y, ny = r * y - a * x;
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
        const T two_r_dr = T(2) * r * dr[i];
        dl[0][i] = (x * dr[i] + (i == 0 ? r : T(0)) + (i == 1 ? a : T(0)) -
                    two_r_dr * nx * inv_ra) * inv_ra;
        dl[1][i] = (y * dr[i] + (i == 1 ? r : T(0)) - (i == 0 ? a : T(0)) -
                    two_r_dr * ny * inv_ra) * inv_ra;
        dl[2][i] = -z * dr[i] * inv_r * inv_r + (i == 2 ? inv_r : T(0));
    }
    const T lapse = g.lapse;
    const T lapse2 = lapse * lapse;
    const T lapse3 = lapse2 * lapse;
    // d_k gamma_ij, d ln sqrt(gamma) = 1/2 gUU^ij d gamma_ij
#pragma unroll
    for (int k = 0; k < 3; ++k)
    {
        T trace = T(0);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = i; j < 3; ++j)
            {
                const T d = T(2) * (l[i] * l[j] * dH[k] + H * l[i] * dl[j][k] +
                                    H * l[j] * dl[i][k]);
                f->dgamma[k][sym(i, j)] = d;
                trace += (i == j ? T(1) : T(2)) * g.gUU[sym(i, j)] * d;
            }
        f->dlnsqrtg[k] = T(0.5) * trace;
        f->dlapse[k] = -lapse3 * dH[k];
    }
    // d_j shift^i with shift^i = 2 H lapse^2 l^i (KerrSchild.hpp:177-184)
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            f->dshift[i][j] = T(2) * dH[j] * lapse2 * l[i] +
                              T(4) * H * lapse * f->dlapse[j] * l[i] +
                              T(2) * H * lapse2 * dl[i][j];
    // K_ij = (D_i beta_j + D_j beta_i) / (2 lapse), which for a static
    // metric is the Lie derivative of gamma along beta over 2 lapse:
    //   sum_k gamma_kj d_i b^k + gamma_ki d_j b^k + b^k d_k gamma_ij
    // (the reference's Christoffel form, KerrSchild.hpp:186-207, reduces
    // to this identically).
    const T *b = g.shift;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = i; j < 3; ++j)
        {
            T s = T(0);
#pragma unroll
            for (int k = 0; k < 3; ++k)
            {
                s += g.gLL[sym(k, j)] * f->dshift[k][i] +
                     g.gLL[sym(k, i)] * f->dshift[k][j];
                s += b[k] * f->dgamma[k][sym(i, j)];
            }
            f->K[sym(i, j)] = s * div_(T(0.5), lapse);
        }
    f->g = g;
}

// An FP64 Kerr-Schild cell in terms of its null vector l and H (see "FP64
// Kerr-Schild cell" below).
// T = double, or the dual numbers of the adjoint's spin derivative.
template <typename T> struct KsCellT
{
    T l[3], F, c, alpha, alpha2;
    T r, inv_r, inv_ra, inv_sigma; // 1/r, 1/(r^2 + a^2), 1/Sigma
};
using KsCell = KsCellT<double>;

template <typename T>
GRHD_HD __forceinline__ void ks_cell(double M, T a, double x, double y,
                                     double z, KsCellT<T> &k)
{
    const T a2 = mul_(a, a);
    const double rho2 =
        fmax(fma(x, x, fma(y, y, mul_(z, z))), 1.0e-12); // (1e-6)^2
    const T hA = 0.5 * (rho2 - a2);
    const T az = mul_(a, z);
    const T r2 = hA + sqrt_(fma(hA, hA, mul_(az, az)));
    // r and 1/r from one reciprocal square root, each corrected once
    const T y0 = rsqrt_ulp(r2);
    const T r0 = mul_(r2, y0);
    const T r = fma(fma(-r0, r0, r2), 0.5 * y0, r0);
    k.r = r;
    k.inv_r = fma(fma(-r, y0, 1.0), y0, y0);
    const T ct = mul_(z, k.inv_r);
    const T act = mul_(a, ct);
    k.inv_sigma = rcp_ulp(fma(act, act, r2));
    k.inv_ra = rcp_ulp(r2 + a2);
    k.l[0] = mul_(fma(r, x, mul_(a, y)), k.inv_ra);
    k.l[1] = mul_(fma(r, y, -mul_(a, x)), k.inv_ra);
    k.l[2] = ct;
    k.F = mul_(mul_(2.0 * M, r), k.inv_sigma);
    const T u = 1.0 + k.F;
    k.alpha2 = rcp_ulp(u);
    k.alpha = rsqrt_ulp(u);
    k.c = mul_(k.F, k.alpha2);
}

template <typename T>
GRHD_HD __forceinline__ void ks_gLL(const KsCellT<T> &k, T g[6])
{
    const T f[3] = {mul_(k.F, k.l[0]), mul_(k.F, k.l[1]),
                         mul_(k.F, k.l[2])};
    g[0] = fma(f[0], k.l[0], 1.0);
    g[1] = mul_(f[0], k.l[1]);
    g[2] = mul_(f[0], k.l[2]);
    g[3] = fma(f[1], k.l[1], 1.0);
    g[4] = mul_(f[1], k.l[2]);
    g[5] = fma(f[2], k.l[2], 1.0);
}

// The face geometry of a cell from them: 60 FP64 operations and five special
// functions against some 90 and eight of ks_metric's general sequence.
template <typename T>
GRHD_HD __forceinline__ void ks_geo_of(const KsCellT<T> &k, GeoT<T> &g)
{
    ks_gLL(k, g.gLL);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        g.shift[i] = mul_(k.c, k.l[i]);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = i; j < 3; ++j)
            g.gUU[sym(i, j)] =
                fma(-g.shift[i], k.l[j], T(i == j ? 1.0 : 0.0));
    g.lapse = k.alpha;
}

GRHD_HD __forceinline__ void ks_geo(double M, double a, double x, double y,
                                    double z, Geo &g)
{
    KsCell k;
    ks_cell(M, a, x, y, z, k);
    ks_geo_of(k, g);
}

// Softened circular-binary potentials at `pos` (add_point_potential,
// CircularBinaryPN.hpp:252-297).
template <typename T>
__device__ __forceinline__ void pn_add_point(T mass, T soft2, const double *sp,
                                             const double *sv, const T *pos,
                                             T &U, T &dUdt, T dU[3], T V[3],
                                             T dV[3][3])
{
    T d[3];
    T r2 = soft2;
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
        d[i] = pos[i] - T(sp[i]);
        r2 += d[i] * d[i];
    }
    const T ir = rsqrt_(r2);
    const T ir3 = ir * ir * ir;
    U += mass * ir;
    dUdt += mass * (d[0] * T(sv[0]) + d[1] * T(sv[1]) + d[2] * T(sv[2])) * ir3;
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
        dU[i] += -mass * d[i] * ir3;
        V[i] += mass * T(sv[i]) * ir;
#pragma unroll
        for (int j = 0; j < 3; ++j)
            dV[i][j] += -mass * T(sv[i]) * d[j] * ir3;
    }
}

// Scalar potential only, for the volume-time source (FP64 in both paths).
// The reference takes a central difference in time of ln sqrt(det gamma)
// with step h (FixedBGFArrayBoxFiniteVolume.hpp:616-631), which amplifies
// the rounding of U by ~1/h; the sums here are written with
// round-to-nearest intrinsics so that no multiply-add is fused and U rounds
// as the reference's expression does (sqrt_ and rcp_ give the IEEE results on
// every tested operand, without the IEEE operations' slow-path branches).
__device__ __forceinline__ double pn_scalar(double m1, double m2,
                                            double soft2, const double *p1,
                                            const double *p2,
                                            const double *pos)
{
    double r1 = soft2, r2 = soft2;
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
        const double d1 = __dadd_rn(pos[i], -p1[i]);
        const double d2 = __dadd_rn(pos[i], -p2[i]);
        r1 = __dadd_rn(r1, __dmul_rn(d1, d1));
        r2 = __dadd_rn(r2, __dmul_rn(d2, d2));
    }
    return __dadd_rn(__dmul_rn(m1, rcp_(sqrt_(r1))),
                     __dmul_rn(m2, rcp_(sqrt_(r2))));
}

// CircularBinaryPN::compute_metric_background, CircularBinaryPN.hpp:70-189:
// conformally flat gamma = psi delta with psi = 1 + 2U, lapse^2 =
// 1 - 2U + 2U^2 + 16 V^2/psi, shift = -4 V/psi, and
// K_ij = [psi (d_i b^j + d_j b^i) + delta_ij (b.grad psi - d_t psi)]/(2 lapse).
template <typename T, bool FULL>
__device__ __forceinline__ void pn_metric(const Background &bg, T x, T y, T z,
                                          GeoT<T> &g, GeoFullT<T> *f)
{
    const T pos[3] = {x, y, z};
    T U = T(0), dUdt = T(0), dU[3] = {T(0), T(0), T(0)},
      V[3] = {T(0), T(0), T(0)};
    T dV[3][3] = {{T(0), T(0), T(0)}, {T(0), T(0), T(0)}, {T(0), T(0), T(0)}};
    pn_add_point<T>(T(bg.m1), T(bg.soft2), bg.p1, bg.v1, pos, U, dUdt, dU, V,
                    dV);
    pn_add_point<T>(T(bg.m2), T(bg.soft2), bg.p2, bg.v2, pos, U, dUdt, dU, V,
                    dV);
    const T psi = T(1) + T(2) * U;
    const T ipsi = rcp_(psi);
    const T V2 = V[0] * V[0] + V[1] * V[1] + V[2] * V[2];
    const T lapse2 = T(1) - T(2) * U + T(2) * U * U + T(16) * V2 * ipsi;
    const T lapse = sqrt_(lapse2);
#pragma unroll
    for (int s = 0; s < 6; ++s)
    {
        g.gLL[s] = T(0);
        g.gUU[s] = T(0);
    }
    g.gLL[0] = g.gLL[3] = g.gLL[5] = psi;
    g.gUU[0] = g.gUU[3] = g.gUU[5] = ipsi;
    g.lapse = lapse;
#pragma unroll
    for (int i = 0; i < 3; ++i)
        g.shift[i] = T(-4) * V[i] * ipsi;
    if (!FULL)
        return;
    T bgradpsi = T(0);
#pragma unroll
    for (int d = 0; d < 3; ++d)
    {
        const T dpsi = T(2) * dU[d];
        bgradpsi += g.shift[d] * dpsi;
#pragma unroll
        for (int s = 0; s < 6; ++s)
            f->dgamma[d][s] = (s == 0 || s == 3 || s == 5) ? dpsi : T(0);
        f->dlnsqrtg[d] = T(1.5) * dpsi * ipsi;
        T dV2 = T(0);
#pragma unroll
        for (int c = 0; c < 3; ++c)
        {
            dV2 += T(2) * V[c] * dV[c][d];
            f->dshift[c][d] =
                T(-4) * (dV[c][d] * ipsi - V[c] * dpsi * ipsi * ipsi);
        }
        const T dl2 = (T(-2) + T(4) * U) * dU[d] +
                      T(16) * (dV2 * ipsi - V2 * dpsi * ipsi * ipsi);
        f->dlapse[d] = div_(T(0.5) * dl2, lapse);
    }
    const T dpsidt = T(2) * dUdt;
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = i; j < 3; ++j)
        {
            T s = psi * (f->dshift[j][i] + f->dshift[i][j]);
            if (i == j)
                s += bgradpsi - dpsidt;
            f->K[sym(i, j)] = s * div_(T(0.5), lapse);
        }
    f->g = g;
}

// BGK: the background kind when known at compile time (0 Kerr-Schild,
// 1 binary PN), -1 to read it from bg.kind.
template <bool FULL, int BGK = -1>
__device__ __forceinline__ void background_metric(const Background &bg,
                                                  double x, double y,
                                                  double z, Geo &g,
                                                  GeoFull *f)
{
    if (BGK == 1 || (BGK < 0 && bg.kind == 1))
        pn_metric<double, FULL>(bg, x, y, z, g, f);
    else
        ks_metric<double, FULL>(bg.M, bg.a, x, y, z, g, f);
}

template <typename A, typename B>
GRHD_HD __forceinline__ void convert_geo(const GeoT<A> &s, GeoT<B> &d)
{
#pragma unroll
    for (int q = 0; q < 6; ++q)
    {
        d.gLL[q] = B(s.gLL[q]);
        d.gUU[q] = B(s.gUU[q]);
    }
    d.lapse = B(s.lapse);
#pragma unroll
    for (int q = 0; q < 3; ++q)
        d.shift[q] = B(s.shift[q]);
}

// FP64 Kerr-Schild geometry rounded to FP32 (mixed path, r < 3M).
template <bool FULL>
__device__ __noinline__ void ks_metric_fp64_to_fp32(double M, double a,
                                                    double x, double y,
                                                    double z, GeoT<float> &g,
                                                    GeoFullT<float> *f)
{
    GeoFull fd;
    ks_metric<double, FULL>(M, a, x, y, z, fd.g, FULL ? &fd : nullptr);
    convert_geo(fd.g, g);
    if (FULL)
    {
#pragma unroll
        for (int q = 0; q < 6; ++q)
            f->K[q] = float(fd.K[q]);
#pragma unroll
        for (int d = 0; d < 3; ++d)
        {
            f->dlapse[d] = float(fd.dlapse[d]);
            f->dlnsqrtg[d] = float(fd.dlnsqrtg[d]);
#pragma unroll
            for (int q = 0; q < 6; ++q)
                f->dgamma[d][q] = float(fd.dgamma[d][q]);
#pragma unroll
            for (int q = 0; q < 3; ++q)
                f->dshift[d][q] = float(fd.dshift[d][q]);
        }
        f->g = g;
    }
}

// Mixed-path geometry: FP32 closed forms, except within three gravitational
// radii of a Kerr-Schild hole where the metric (and so its determinant and
// inverse) is evaluated in FP64 -- there r^2 = (rho^2 - a^2)/2 + ... and
// 1 + 2H lose too many FP32 digits.
template <bool FULL, int BGK = -1>
__device__ __forceinline__ void background_metric_mixed(const Background &bg,
                                                        double x, double y,
                                                        double z,
                                                        GeoT<float> &g,
                                                        GeoFullT<float> *f)
{
    if (BGK == 1 || (BGK < 0 && bg.kind == 1))
        pn_metric<float, FULL>(bg, float(x), float(y), float(z), g, f);
    else if (x * x + y * y + z * z < 9.0 * bg.M * bg.M)
    {
        // through temporaries: the call's results live in local memory, and
        // the caller's fields would too, on every path, if it got their
        // address
        GeoT<float> gt;
        GeoFullT<float> ft;
        ks_metric_fp64_to_fp32<FULL>(bg.M, bg.a, x, y, z, gt, &ft);
        g = gt;
        if (FULL)
            *f = ft;
    }
    else
        ks_metric<float, FULL>(float(bg.M), float(bg.a), float(x), float(y),
                               float(z), g, f);
}

template <typename T, bool FULL, int BGK = -1>
__device__ __forceinline__ void metric_T(const Background &bg, double x,
                                         double y, double z, GeoT<T> &g,
                                         GeoFullT<T> *f)
{
    if constexpr (sizeof(T) == sizeof(double) && !FULL)
    {
        if (BGK == 1 || (BGK < 0 && bg.kind == 1))
            pn_metric<double, false>(bg, x, y, z, g, nullptr);
        else
            ks_geo(bg.M, bg.a, x, y, z, g);
    }
    else if constexpr (sizeof(T) == sizeof(double))
        background_metric<FULL, BGK>(bg, x, y, z, g, f);
    else
        background_metric_mixed<FULL, BGK>(bg, x, y, z, g, f);
}

// Coordinates<double>: cell centre (i + 1/2) dx - centre, rounded as the
// reference's separate multiply and subtract (no fused multiply-add), so
// that positions -- and everything the time-difference volume source
// amplifies -- match the reference bit for bit.
GRHD_HD __forceinline__ void cell_xyz(const Options &o, int i, int j,
                                         int k, double &x, double &y,
                                         double &z)
{
#ifdef __CUDA_ARCH__
    x = __dadd_rn(__dmul_rn(i + 0.5, o.dx), -o.center[0]);
    y = __dadd_rn(__dmul_rn(j + 0.5, o.dx), -o.center[1]);
    z = __dadd_rn(__dmul_rn(k + 0.5, o.dx), -o.center[2]);
#else
    // host: a separately rounded multiply and subtract (build the host
    // code without floating-point contraction)
    const volatile double px = (i + 0.5) * o.dx, py = (j + 0.5) * o.dx,
                          pz = (k + 0.5) * o.dx;
    x = px - o.center[0];
    y = py - o.center[1];
    z = pz - o.center[2];
#endif
}

GRHD_HD __forceinline__ bool excised(const Options &o, int i, int j, int k)
{
    if (!(o.excision_radius > 0.0))
        return false;
    double x, y, z;
    cell_xyz(o, i, j, k, x, y, z);
    return sqrt(x * x + y * y + z * z) < o.excision_radius;
}

// spatial_metric_log_sqrt_det for the binary (det = psi^3),
// StaticMetric.hpp:293-302.
__device__ __forceinline__ double pn_log_sqrt_det(double psi)
{
    const double det = __dmul_rn(__dmul_rn(psi, psi), psi);
    if (det <= 0.0 || !isfinite(det))
        return 0.0;
    return 0.5 * log(det);
}

// --------------------------------------------------------- Valencia, EOS

template <typename T>
GRHD_HD __forceinline__ T vsq(const T v[3], const T gLL[6])
{
    return gLL[0] * v[0] * v[0] + gLL[3] * v[1] * v[1] + gLL[5] * v[2] * v[2] +
           T(2) * (gLL[1] * v[0] * v[1] + gLL[2] * v[0] * v[2] +
                   gLL[4] * v[1] * v[2]);
}

// compute_conserved, Valencia.hpp:55-73
template <typename T>
GRHD_HD __forceinline__ ConsT<T> p2c(const PrimT<T> &pr, const T gLL[6])
{
    ConsT<T> c;
    const T vL0 = gLL[0] * pr.v[0] + gLL[1] * pr.v[1] + gLL[2] * pr.v[2];
    const T vL1 = gLL[1] * pr.v[0] + gLL[3] * pr.v[1] + gLL[4] * pr.v[2];
    const T vL2 = gLL[2] * pr.v[0] + gLL[4] * pr.v[1] + gLL[5] * pr.v[2];
    const T v2 = vL0 * pr.v[0] + vL1 * pr.v[1] + vL2 * pr.v[2];
    const T W = rsqrt_(T(1) - v2);
    const T h = T(1) + pr.eps + div_(pr.p, pr.rho);
    const T rhw = pr.rho * h * W * W;
    c.D = pr.rho * W;
    c.tau = rhw - pr.p - c.D;
    c.S[0] = rhw * vL0;
    c.S[1] = rhw * vL1;
    c.S[2] = rhw * vL2;
    return c;
}

// detail::pressure_residual (+ derivative), Valencia.hpp:79-108.  The
// recovery divides with div_ / rcp_ / sqrt_ like the rest of the device
// code; e = tau + D + p equal to zero (which IEEE division would turn into
// a capped v^2) gives a NaN residual and so a failed recovery.
GRHD_HD __forceinline__ double c2p_residual(double p, double D,
                                               double tau, double S2,
                                               double G, double Gfac,
                                               double vmax2, double *deriv)
{
    const double e = tau + D + p;
    const double ie = rcp_(e);
    double v2 = S2 * ie * ie;
    if (v2 > vmax2)
        v2 = vmax2;
    const double W = rsqrt_(1.0 - v2);
    const double W2 = W * W;
    if (deriv)
    {
        const double dW = -W2 * W * v2 * ie;
        *deriv = D * dW + Gfac * (W2 + p * 2.0 * W * dW) - 1.0;
    }
    return D * W + Gfac * p * W2 - e;
}

GRHD_HD __forceinline__ double c2p_S2(const Cons &c, const double gUU[6])
{
    return gUU[0] * c.S[0] * c.S[0] + gUU[3] * c.S[1] * c.S[1] +
           gUU[5] * c.S[2] * c.S[2] +
           2.0 * (gUU[1] * c.S[0] * c.S[1] + gUU[2] * c.S[0] * c.S[2] +
                  gUU[4] * c.S[1] * c.S[2]);
}

// The primitives of a converged pressure, Valencia.hpp:213-226; false when
// the velocity reaches the cap.  mU = gamma^ij S_j, S2 = S_i mU^i.
GRHD_HD __forceinline__ bool c2p_finish(const Options &o, const Cons &c,
                                        const double mU[3], double S2,
                                        double p, Prim &out)
{
    const double e = c.tau + c.D + p;
    const double v2 = div_(S2, mul_(e, e));
    if (!(v2 < o.rec_vmax2))
        return false;
    // W rounded as the reference's 1 / sqrt(1 - v^2) (sqrt_ and rcp_ give
    // the IEEE results, rsqrt_ is up to two ulp off): rho = D / W decides
    // the atmosphere and floor tests bit for bit, and an ulp there switches
    // a cell's sources on or off
    const double W = rcp_(sqrt_(1.0 - v2));
    out.rho = div_(c.D, W);
    out.p = p;
    out.eps = div_(p, mul_(o.G - 1.0, out.rho));
    const double ie = rcp_(e);
    out.v[0] = mul_(mU[0], ie);
    out.v[1] = mul_(mU[1], ie);
    out.v[2] = mul_(mU[2], ie);
    return true;
}

// gamma^ij S_j
GRHD_HD __forceinline__ void raise(const double gUU[6], const double S[3],
                                   double mU[3])
{
    mU[0] = fma(gUU[0], S[0], fma(gUU[1], S[1], mul_(gUU[2], S[2])));
    mU[1] = fma(gUU[1], S[0], fma(gUU[3], S[1], mul_(gUU[4], S[2])));
    mU[2] = fma(gUU[2], S[0], fma(gUU[4], S[1], mul_(gUU[5], S[2])));
}

template <typename A, typename B>
GRHD_HD __forceinline__ auto dot3(const A a[3], const B b[3])
{
    return fma(a[0], b[0], fma(a[1], b[1], mul_(a[2], b[2])));
}

// The residual of c2p_residual and its derivative with one-ulp reciprocals;
// tD = tau + D.
GRHD_HD __forceinline__ double c2p_f(double p, double D, double tD, double S2,
                                     double Gfac, double vmax2, double &deriv)
{
    const double e = tD + p;
    const double ie = rcp_ulp(e);
    double v2 = mul_(mul_(S2, ie), ie);
    if (v2 > vmax2)
        v2 = vmax2;
    const double W = rsqrt_ulp(1.0 - v2);
    const double W2 = mul_(W, W), DW = mul_(D, W), GW2 = mul_(Gfac, W2);
    // dW/dp = -W t with t = W^2 v^2 / e
    const double t = mul_(mul_(W2, v2), ie);
    deriv = fma(-DW, t, fma(GW2, fma(-2.0 * p, t, 1.0), -1.0));
    return fma(GW2, p, DW) - e;
}

// The root solve of recover_primitive, Valencia.hpp:116-228 (bounded loops
// throughout): the reference's bracket, start, steps and acceptance, on a
// residual that rounds differently, so that an iterate with |f| at the
// tolerance may be accepted where the reference takes one step more.  Its
// chain of dependent FP64 operations is what it costs, so the residuals at
// the pressure floor and at the start, which do not depend on one another,
// are evaluated side by side, and the residual at the bracket's upper end
// only where its sign is not known: with u >= |tau| and W >= 1,
// f(u) >= (G/(G-1) - 1) u - tau >= u/4 for G/(G-1) >= 9/4 (G <= 9/5), far
// above rounding.
GRHD_HD __forceinline__ bool c2p_solve(const Options &o, const Cons &c,
                                       double S2, double &p_out, int &iters,
                                       double &resid)
{
    iters = 0;
    resid = 0.0;
    if (!(c.D > 0.0))
        return false;
    const double Gm1 = o.G - 1.0;
    const double Gfac = div_(o.G, Gm1);
    const double vmax2 = o.rec_vmax2;
    const double tol = o.rec_tol;
    const double tD = c.tau + c.D;
    double lower = o.rec_pfloor;
    double upper = fmax(1.0, fabs(c.tau) + c.D);
    double dres, dlow;
    const double f_lower = c2p_f(lower, c.D, tD, S2, Gfac, vmax2, dlow);
    double p = fmin(fmax(mul_(c.tau, Gm1), lower), upper);
    double r = c2p_f(p, c.D, tD, S2, Gfac, vmax2, dres);
    const bool at_floor = fabs(f_lower) <= tol;
    if (!(f_lower < 0.0) && !at_floor)
    {
        // no root above the floor, or not a number: every iteration of the
        // reference's loop stays at the floor
        if (!(f_lower >= 0.0))
        {
            iters = o.rec_maxit;
            resid = f_lower;
        }
        return false;
    }
    const bool bracketed = f_lower < 0.0;
    if (!bracketed)
        upper = lower;
    else if (!(Gfac >= 2.25) || !isfinite(upper))
    {
        double du;
        double f_upper = c2p_f(upper, c.D, tD, S2, Gfac, vmax2, du);
        for (int b = 0; f_upper <= 0.0 && b < o.rec_maxit; ++b)
        {
            upper *= 2.0;
            f_upper = c2p_f(upper, c.D, tD, S2, Gfac, vmax2, du);
        }
        if (!(f_upper > 0.0))
            return false;
        // the start is clamped to the widened bracket
        if (!at_floor)
        {
            p = fmin(fmax(mul_(c.tau, Gm1), lower), upper);
            r = c2p_f(p, c.D, tD, S2, Gfac, vmax2, dres);
        }
    }
    if (at_floor)
    {
        p = lower;
        r = f_lower;
        dres = dlow;
    }
    for (int it = 0; it < o.rec_maxit; ++it)
    {
        iters = it + 1;
        if (fabs(r) < tol)
            break;
        if (bracketed)
        {
            if (r > 0.0)
                upper = p;
            else
                lower = p;
        }
        double np = fma(-r, rcp_ulp(dres), p);
        if (!isfinite(np) || np <= lower || np >= upper)
            np = 0.5 * (lower + upper);
        p = np;
        r = c2p_f(p, c.D, tD, S2, Gfac, vmax2, dres);
    }
    resid = r;
    p_out = p;
    return fabs(r) < tol;
}

// recover_primitive, Valencia.hpp:116-228.
GRHD_HD __forceinline__ bool con2prim(const Options &o, const Cons &c,
                                         const double gUU[6], Prim &out,
                                         int *iters_out, double *resid_out)
{
    double mU[3], p = 0.0, resid;
    int iters;
    raise(gUU, c.S, mU);
    const double S2 = dot3(c.S, mU);
    const bool ok = c2p_solve(o, c, S2, p, iters, resid) &&
                    c2p_finish(o, c, mU, S2, p, out);
    if (iters_out)
        *iters_out = iters;
    if (resid_out)
        *resid_out = resid;
    return ok;
}

GRHD_HD __forceinline__ bool c2p_finish_gUU(const Options &o, const Cons &c,
                                            const double gUU[6], double S2,
                                            double p, Prim &out)
{
    const double mU[3] = {
        gUU[0] * c.S[0] + gUU[1] * c.S[1] + gUU[2] * c.S[2],
        gUU[1] * c.S[0] + gUU[3] * c.S[1] + gUU[4] * c.S[2],
        gUU[2] * c.S[0] + gUU[4] * c.S[1] + gUU[5] * c.S[2]};
    return c2p_finish(o, c, mU, S2, p, out);
}

// The mixed path's bracketed solve: the same root solve one residual at a
// time.  Its kernels that hold three blocks per SM at 80 registers spill with
// c2p_solve's overlapped residuals (stage kernel: 224 -> 356 bytes).
GRHD_HD __forceinline__ bool con2prim_mixed(const Options &o, const Cons &c,
                                         const double gUU[6], Prim &out,
                                         int *iters_out, double *resid_out)
{
    int iters = 0;
    double resid = 0.0;
    bool ok = false;
    if (c.D > 0.0)
    {
        const double G = o.G;
        const double Gfac = div_(G, G - 1.0);
        const double vmax2 = o.rec_vmax2;
        const double tol = o.rec_tol;
        const double S2 = c2p_S2(c, gUU);
        double lower = o.rec_pfloor;
        const double f_lower =
            c2p_residual(lower, c.D, c.tau, S2, G, Gfac, vmax2, nullptr);
        bool bracket_ok = !(f_lower >= 0.0 && fabs(f_lower) > tol);
        double upper = lower;
        if (bracket_ok && f_lower < 0.0)
        {
            upper = fmax(1.0, fabs(c.tau) + c.D);
            double f_upper =
                c2p_residual(upper, c.D, c.tau, S2, G, Gfac, vmax2, nullptr);
            for (int b = 0; f_upper <= 0.0 && b < o.rec_maxit; ++b)
            {
                upper *= 2.0;
                f_upper =
                    c2p_residual(upper, c.D, c.tau, S2, G, Gfac, vmax2, nullptr);
            }
            bracket_ok = f_upper > 0.0;
        }
        if (bracket_ok)
        {
            double p = (fabs(f_lower) <= tol)
                           ? lower
                           : fmin(fmax(c.tau * (G - 1.0), lower), upper);
            double dres;
            double r = c2p_residual(p, c.D, c.tau, S2, G, Gfac, vmax2, &dres);
            for (int it = 0; it < o.rec_maxit; ++it)
            {
                iters = it + 1;
                if (fabs(r) < tol)
                    break;
                if (f_lower < 0.0)
                {
                    if (r > 0.0)
                        upper = p;
                    else
                        lower = p;
                }
                double np = p - div_(r, dres);
                if (!isfinite(np) || np <= lower || np >= upper)
                    np = 0.5 * (lower + upper);
                p = np;
                r = c2p_residual(p, c.D, c.tau, S2, G, Gfac, vmax2, &dres);
            }
            resid = r;
            if (fabs(r) < tol)
                ok = c2p_finish_gUU(o, c, gUU, S2, p, out);
        }
    }
    if (iters_out)
        *iters_out = iters;
    if (resid_out)
        *resid_out = resid;
    return ok;
}

// Mixed path: the same FP64 root solve started from a known nearby
// pressure (the previous stage's), safeguarded Newton on the monotone
// residual; falls back to the full bracketed solve when the guess is not
// usable or a step leaves (p_floor, inf).  Converges to the same root to
// the solver tolerance.
GRHD_HD __forceinline__ bool con2prim_warm(const Options &o, const Cons &c,
                                              const double gUU[6],
                                              double p_guess, Prim &out)
{
    if (c.D > 0.0)
    {
        const double G = o.G;
        const double Gfac = div_(G, G - 1.0);
        const double S2 = c2p_S2(c, gUU);
        // a guess at (or rounded below) the recovery floor: the full solve
        // returns the floor itself when the residual there is within
        // tolerance; only that is tested
        const bool at_floor = !(p_guess > o.rec_pfloor);
        if (at_floor || isfinite(p_guess))
        {
            double p = at_floor ? o.rec_pfloor : p_guess, dres;
            double r =
                c2p_residual(p, c.D, c.tau, S2, G, Gfac, o.rec_vmax2, &dres);
            bool found =
                at_floor ? fabs(r) <= o.rec_tol : fabs(r) < o.rec_tol;
            for (int it = 1; !at_floor && !found && it < 6; ++it)
            {
                p = p - div_(r, dres);
                if (!isfinite(p) || !(p > o.rec_pfloor))
                    break;
                r = c2p_residual(p, c.D, c.tau, S2, G, Gfac, o.rec_vmax2,
                                 &dres);
                found = fabs(r) < o.rec_tol;
            }
            if (found && c2p_finish_gUU(o, c, gUU, S2, p, out))
                return true;
        }
    }
    return con2prim_mixed(o, c, gUU, out, nullptr, nullptr);
}

// enforce_primitive_floors, Atmosphere.hpp:24-46 (eps recomputed always);
// Gm1 = G - 1.
template <typename T>
GRHD_HD __forceinline__ void floors_k(T rho_floor, T p_floor, T vmax2, T Gm1,
                                      PrimT<T> &pr, const T gLL[6])
{
    pr.rho = max_(pr.rho, rho_floor);
    pr.p = max_(pr.p, p_floor);
    const T v2 = vsq(pr.v, gLL);
    if (v2 >= vmax2)
    {
        const T s = sqrt_(div_(vmax2, v2));
        pr.v[0] *= s;
        pr.v[1] *= s;
        pr.v[2] *= s;
    }
    pr.eps = div_(pr.p, Gm1 * pr.rho);
}

template <typename T>
GRHD_HD __forceinline__ void floors(const Options &o, PrimT<T> &pr,
                                       const T gLL[6])
{
    floors_k(T(o.rho_floor), T(o.p_floor), T(o.atmo_vmax2), T(o.G) - T(1), pr,
             gLL);
}

// make_atmosphere_primitive, Atmosphere.hpp:48-60
GRHD_HD __forceinline__ Prim atmosphere(const Options &o)
{
    Prim pr;
    pr.rho = o.rho_floor;
    pr.p = o.p_floor;
    pr.eps = pr.p / ((o.G - 1.0) * pr.rho);
    pr.v[0] = pr.v[1] = pr.v[2] = 0.0;
    return pr;
}

// is_atmosphere_primitive, FArrayBoxFiniteVolume.hpp:118-126
template <typename T>
GRHD_HD __forceinline__ bool is_atmo(const Options &o, const PrimT<T> &pr,
                                        double factor)
{
    const double f = fmax(1.0, factor);
    return pr.rho <= T(f * o.rho_floor) && pr.p <= T(f * o.p_floor);
}

// compute_flux, Valencia.hpp:230-259
template <typename T>
GRHD_HD __forceinline__ ConsT<T> phys_flux(const PrimT<T> &pr,
                                              const ConsT<T> &c, int d,
                                              T lapse, const T shift[3])
{
    ConsT<T> f;
    const T tv = lapse * pr.v[d] - shift[d];
    const T ap = lapse * pr.p;
    f.D = c.D * tv;
    f.tau = c.tau * tv + ap * pr.v[d];
#pragma unroll
    for (int j = 0; j < 3; ++j)
        f.S[j] = c.S[j] * tv + (j == d ? ap : T(0));
    return f;
}

// compute_characteristic_speeds (shifted), RiemannSolvers.hpp:23-67
template <typename T>
GRHD_HD __forceinline__ void char_speeds_k(T G, const PrimT<T> &pr,
                                           const GeoT<T> &g, int d, T &lo,
                                           T &hi)
{
    const T v2 = vsq(pr.v, g.gLL);
    const T h = T(1) + pr.eps + div_(pr.p, pr.rho);
    const T cs2 = div_(G * pr.p, pr.rho * h);
    const T cs = sqrt_(cs2);
    const T vel = pr.v[d];
    const T den = T(1) - v2 * cs2;
    const T rad =
        (T(1) - v2) * (g.gUU[sym(d, d)] * den - vel * vel * (T(1) - cs2));
    const T root = cs * sqrt_(max_(T(0), rad));
    const T base = vel * (T(1) - cs2);
    const T iden = rcp_(den);
    lo = g.lapse * ((base - root) * iden) - g.shift[d];
    hi = g.lapse * ((base + root) * iden) - g.shift[d];
}

template <typename T>
GRHD_HD __forceinline__ void char_speeds(const Options &o,
                                            const PrimT<T> &pr,
                                            const GeoT<T> &g, int d, T &lo,
                                            T &hi)
{
    char_speeds_k(T(o.G), pr, g, d, lo, hi);
}

// The constants of a face flux in its arithmetic type, made once per launch
// (as kernel parameters they are operands in the constant bank; the options'
// FP64 members cost the FP32 path a conversion at each use).
template <typename T> struct FaceOpt
{
    T theta; // > 0
    // cells from a cell to its outer neighbour in a slope: 0 without
    // reconstruction, where that difference, and so the slope, is zero
    // whatever the other neighbour holds
    int reach;
    T rho_floor, p_floor, vmax2, G, Gm1;
    T Gfac; // G / (G - 1): h = 1 + Gfac p / rho
};

template <typename T>
GRHD_HD __forceinline__ FaceOpt<T> make_face_opt(const Options &o)
{
    FaceOpt<T> f;
    // (minmod of slopes scaled by theta <= 0 is zero too)
    f.reach = o.use_recon && o.theta > 0.0;
    f.theta = f.reach ? T(o.theta) : T(1);
    f.rho_floor = T(o.rho_floor);
    f.p_floor = T(o.p_floor);
    f.vmax2 = T(o.atmo_vmax2);
    f.G = T(o.G);
    f.Gm1 = T(o.G) - T(1);
    f.Gfac = T(o.G / (o.G - 1.0));
    return f;
}

// FP64 limited slope of compute_limited_slope (Reconstruction.hpp:16-37),
// minmod(theta (c - l), minmod((r - l) / 2, theta (r - c))): zero unless the
// two one-sided differences have the same sign, else the smallest magnitude
// of the three with that sign -- the nested minmod's value bit for bit
// (multiplying by theta > 0 keeps the order).  As there, a neighbour that is
// not a number (an excised cell's frozen primitives may be) leaves the other
// side's difference.  Without a branch that costs 1 % of a step (256^3
// torus, RK4: 12.8 -> 12.9 ms); a second form behind a test for tiles that
// touch excised cells took 13.5, a test for no reconstruction 13.3.
GRHD_HD __forceinline__ double limited_slope_f64(double l, double c, double r,
                                                 double theta)
{
    const double dl = c - l, dr = r - c, dc = 0.5 * (r - l);
    const bool no_r = dr != dr;
    const double m = theta * (no_r || fabs(dl) < fabs(dr) ? dl : dr);
    // dl with the sign of dr flipped in, off the FP64 pipe
#ifdef __CUDA_ARCH__
    const double x = __hiloint2double(
        __double2hiint(dl) ^ (__double2hiint(dr) & (int)0x80000000),
        __double2loint(dl));
#else
    const double x = copysign(1.0, dr) < 0.0 ? -dl : dl;
#endif
    const double q = fabs(dc) < fabs(m) ? dc : m;
    return x < 0.0 && !no_r ? 0.0 : q;
}

// One side of an FP64 face: conserved state, physical flux along d and
// characteristic speeds of the reconstructed primitives q = (rho, p, v)
// after the floors (Atmosphere.hpp:24-46).  The reference's formulas
// (Valencia.hpp:55-73, 230-259, RiemannSolvers.hpp:23-67) share their
// subexpressions here: with y = p / rho, c = G y and h = 1 + G y / (G - 1)
// the speeds' numerators and denominators are multiplied through by h
// (c_s^2 = c / h), which leaves one reciprocal of rho, one reciprocal square
// root for W, one square root and one reciprocal for the speeds -- four
// special functions per side where the separate formulas take eight.  The
// face kernel is bound by issue and FP64 latency, so the operations removed
// are time removed: with a cheaper limiter and HLLE flux an RK4 step of the
// 256^3 torus went from 29.8 to 24.9 ms, the 64^3 Michel step from 0.81 to
// 0.68 ms.
struct FaceSide
{
    Cons c, f;
    double lo, hi;
};

GRHD_HD __forceinline__ void face_side(const FaceOpt<double> &o,
                                       const double q[5], const Geo &g, int d,
                                       FaceSide &s)
{
    const double rho = q[0] > o.rho_floor ? q[0] : o.rho_floor;
    const double p = q[1] > o.p_floor ? q[1] : o.p_floor;
    double v0 = q[2], v1 = q[3], v2 = q[4];
    double l0 = g.gLL[0] * v0 + g.gLL[1] * v1 + g.gLL[2] * v2;
    double l1 = g.gLL[1] * v0 + g.gLL[3] * v1 + g.gLL[4] * v2;
    double l2 = g.gLL[2] * v0 + g.gLL[4] * v1 + g.gLL[5] * v2;
    double vv = l0 * v0 + l1 * v1 + l2 * v2;
    if (vv >= o.vmax2)
    {
        const double r = sqrt_(div_(o.vmax2, vv));
        v0 *= r;
        v1 *= r;
        v2 *= r;
        l0 *= r;
        l1 *= r;
        l2 *= r;
        vv = l0 * v0 + l1 * v1 + l2 * v2;
    }
    const double vd = d == 0 ? v0 : (d == 1 ? v1 : v2);
    const double u = 1.0 - vv; // 1 / W^2
    const double y = p * rcp_ulp(rho);
    const double W = rsqrt_ulp(u);
    const double c = o.G * y;
    const double h = fma(o.Gfac, y, 1.0);
    const double rhw = rho * h * (W * W);
    s.c.D = rho * W;
    s.c.tau = rhw - p - s.c.D;
    s.c.S[0] = rhw * l0;
    s.c.S[1] = rhw * l1;
    s.c.S[2] = rhw * l2;
    // flux
    const double shift = g.shift[d];
    const double tv = g.lapse * vd - shift;
    const double ap = g.lapse * p;
    s.f.D = s.c.D * tv;
    s.f.tau = s.c.tau * tv + ap * vd;
#pragma unroll
    for (int j = 0; j < 3; ++j)
        s.f.S[j] = s.c.S[j] * tv + (j == d ? ap : 0.0);
    // speeds, numerator and denominator times h
    const double hc = h - c;
    const double den = fma(-vv, c, h);
    const double rad = (c * u) * (g.gUU[sym(d, d)] * den - vd * vd * hc);
    const double root = rad > 0.0 ? rad * rsqrt_ulp(rad) : 0.0;
    const double base = vd * hc;
    const double k = g.lapse * rcp_ulp(den);
    s.lo = (base - root) * k - shift;
    s.hi = (base + root) * k - shift;
}

// The HLLE flux (RiemannSolvers.hpp:69-118) of the two sides.  A comparison
// with a speed that is not a number keeps the other side's, and where every
// wave runs one way the flux is the upwind side's alone: frozen primitives of
// an excised region may be anything, and inside a horizon they must not reach
// the fluid through a term weighted with zero.
GRHD_HD __forceinline__ Cons hlle_flux(const FaceSide &l, const FaceSide &r)
{
    double sl = l.lo < 0.0 ? l.lo : 0.0;
    double su = l.hi > 0.0 ? l.hi : 0.0;
    sl = r.lo < sl ? r.lo : sl;
    su = r.hi > su ? r.hi : su;
    if (!(sl < 0.0))
        return l.f;
    if (!(su > 0.0))
        return r.f;
    const double inv = rcp_ulp(su - sl);
    const double a = su * inv, b = -sl * inv, ss = sl * a;
    Cons f;
    f.D = a * l.f.D + b * r.f.D + ss * (r.c.D - l.c.D);
    f.tau = a * l.f.tau + b * r.f.tau + ss * (r.c.tau - l.c.tau);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        f.S[i] = a * l.f.S[i] + b * r.f.S[i] + ss * (r.c.S[i] - l.c.S[i]);
    return f;
}

GRHD_HD __forceinline__ double slope_of(double l, double c, double r,
                                        double theta)
{
    return limited_slope_f64(l, c, r, theta);
}
// The same in FP32 (the nested minmod's value bit for bit while the products
// of two slopes do not underflow, 1e-45): 15 instructions instead of 21; the
// mixed face kernel, issue-bound, went from 1.66 to 1.43 ms at 256^3.
__device__ __forceinline__ float slope_of(float l, float c, float r,
                                          float theta)
{
    const float tl = theta * (c - l), tr = theta * (r - c),
                dc = 0.5f * (r - l);
    const float q = fminf(fminf(fabsf(tl), fabsf(tr)), fabsf(dc));
    return tl * dc <= 0.0f || dc * tr <= 0.0f ? 0.0f
                                              : copysignf(q, fmaxf(tl, tr));
}

// The reconstructed values of cell c on its lower and upper faces (MUSCL,
// Reconstruction.hpp:39-58) from its neighbours l and r along the direction
// (of which one is the cell itself where o.reach is 0).
template <typename T>
GRHD_HD __forceinline__ void cell_states(const FaceOpt<T> &o,
                                         const PVT<T> &l, const PVT<T> &c,
                                         const PVT<T> &r, T lower[5],
                                         T upper[5])
{
#pragma unroll
    for (int q = 0; q < 5; ++q)
    {
        const T s = slope_of(l.q[q], c.q[q], r.q[q], o.theta);
        upper[q] = c.q[q] + T(0.5) * s;
        lower[q] = c.q[q] - T(0.5) * s;
    }
}

// The HLLE flux between the states ql and qr of a face with geometry g.
GRHD_HD __forceinline__ ConsT<double>
state_flux(const FaceOpt<double> &o, const double ql[5], const double qr[5],
           const GeoT<double> &g, int d)
{
    FaceSide l, r;
    face_side(o, ql, g, d, l);
    face_side(o, qr, g, d, r);
    return hlle_flux(l, r);
}

// The mixed path's, in the reference's separate formulas.
__device__ __forceinline__ ConsT<float>
state_flux(const FaceOpt<float> &o, const float ql[5], const float qr[5],
           const GeoT<float> &g, int d)
{
    using T = float;
    PrimT<T> lp, rp;
    lp.rho = ql[0];
    lp.p = ql[1];
    rp.rho = qr[0];
    rp.p = qr[1];
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
        lp.v[i] = ql[2 + i];
        rp.v[i] = qr[2 + i];
    }
    floors_k(o.rho_floor, o.p_floor, o.vmax2, o.Gm1, lp, g.gLL);
    floors_k(o.rho_floor, o.p_floor, o.vmax2, o.Gm1, rp, g.gLL);
    const ConsT<T> lc = p2c(lp, g.gLL);
    const ConsT<T> rc = p2c(rp, g.gLL);
    // compute_hlle_flux, RiemannSolvers.hpp:69-118
    const ConsT<T> lf = phys_flux(lp, lc, d, g.lapse, g.shift);
    const ConsT<T> rf = phys_flux(rp, rc, d, g.lapse, g.shift);
    T llo, lhi, rlo, rhi;
    char_speeds_k(o.G, lp, g, d, llo, lhi);
    char_speeds_k(o.G, rp, g, d, rlo, rhi);
    const T sl = min_(T(0), min_(llo, rlo));
    const T su = max_(T(0), max_(lhi, rhi));
    if (sl >= T(0))
        return lf;
    if (su <= T(0))
        return rf;
    const T inv = rcp_(su - sl);
    const T ss = sl * su;
    ConsT<T> f;
    f.D = (su * lf.D - sl * rf.D + ss * (rc.D - lc.D)) * inv;
    f.tau = (su * lf.tau - sl * rf.tau + ss * (rc.tau - lc.tau)) * inv;
#pragma unroll
    for (int i = 0; i < 3; ++i)
        f.S[i] = (su * lf.S[i] - sl * rf.S[i] + ss * (rc.S[i] - lc.S[i])) * inv;
    return f;
}

// One MUSCL-HLLE face flux between cells L and R (compute_muscl_hlle_flux,
// FiniteVolume.hpp:63-98, with the face geometry of average_geometry,
// FArrayBoxFiniteVolume.hpp:194-216).  LL, L, R, RR are the cells
// i-1, i, i+1, i+2 around face i+1/2, with o.reach = 0 L, L, R and R.
template <typename T>
GRHD_HD __forceinline__ ConsT<T>
face_flux(const FaceOpt<T> &o, const PVT<T> &LL, const PVT<T> &L,
          const PVT<T> &R, const PVT<T> &RR, const GeoT<T> &g, int d)
{
    T ql[5], qr[5], unused[5];
    cell_states(o, LL, L, R, unused, ql);
    cell_states(o, L, R, RR, qr, unused);
    return state_flux(o, ql, qr, g, d);
}

template <typename T>
GRHD_HD __forceinline__ ConsT<T> face_flux(const Options &o, const PVT<T> &LL,
                                           const PVT<T> &L, const PVT<T> &R,
                                           const PVT<T> &RR, const GeoT<T> &g,
                                           int d)
{
    const FaceOpt<T> fo = make_face_opt<T>(o);
    return fo.reach ? face_flux(fo, LL, L, R, RR, g, d)
                    : face_flux(fo, L, L, R, R, g, d);
}

template <typename T>
GRHD_HD __forceinline__ void average_geo(const GeoT<T> &a, const GeoT<T> &b,
                                            GeoT<T> &g)
{
#pragma unroll
    for (int s = 0; s < 6; ++s)
    {
        g.gLL[s] = T(0.5) * (a.gLL[s] + b.gLL[s]);
        g.gUU[s] = T(0.5) * (a.gUU[s] + b.gUU[s]);
    }
    g.lapse = T(0.5) * (a.lapse + b.lapse);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        g.shift[i] = T(0.5) * (a.shift[i] + b.shift[i]);
}

// compute_static_metric_source_terms, StaticMetric.hpp:193-275
template <typename T>
GRHD_HD __forceinline__ ConsT<T> static_sources(const PrimT<T> &pr,
                                                   const ConsT<T> &c,
                                                   const GeoFullT<T> &f)
{
    const GeoT<T> &g = f.g;
    const T W = rsqrt_(T(1) - vsq(pr.v, g.gLL));
    const T h = T(1) + pr.eps + div_(pr.p, pr.rho);
    const T rhw = pr.rho * h * W * W;
    T st[6];
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = i; j < 3; ++j)
            st[sym(i, j)] = rhw * pr.v[i] * pr.v[j] + pr.p * g.gUU[sym(i, j)];
    const T E = c.D + c.tau;
    T mU[3];
#pragma unroll
    for (int i = 0; i < 3; ++i)
        mU[i] = g.gUU[sym(i, 0)] * c.S[0] + g.gUU[sym(i, 1)] * c.S[1] +
                g.gUU[sym(i, 2)] * c.S[2];
    ConsT<T> F[3];
#pragma unroll
    for (int d = 0; d < 3; ++d)
        F[d] = phys_flux(pr, c, d, g.lapse, g.shift);
    ConsT<T> s;
    s.D = T(0);
    s.tau = T(0);
#pragma unroll
    for (int d = 0; d < 3; ++d)
    {
        s.D -= F[d].D * f.dlnsqrtg[d];
        s.tau -= F[d].tau * f.dlnsqrtg[d];
        s.tau -= mU[d] * f.dlapse[d];
    }
    T sk = T(0);
#pragma unroll
    for (int i = 0; i < 3; ++i)
#pragma unroll
        for (int j = 0; j < 3; ++j)
            sk += st[sym(i, j)] * f.K[sym(i, j)];
    s.tau += g.lapse * sk;
#pragma unroll
    for (int m = 0; m < 3; ++m)
    {
        T ms = -E * f.dlapse[m];
        T sg = T(0);
#pragma unroll
        for (int i = 0; i < 3; ++i)
#pragma unroll
            for (int j = 0; j < 3; ++j)
                sg += st[sym(i, j)] * f.dgamma[m][sym(i, j)];
        ms += T(0.5) * g.lapse * sg;
#pragma unroll
        for (int sd = 0; sd < 3; ++sd)
            ms += c.S[sd] * f.dshift[sd][m];
#pragma unroll
        for (int d = 0; d < 3; ++d)
            ms -= F[d].S[m] * f.dlnsqrtg[d];
        s.S[m] = ms;
    }
    return s;
}

// -------------------------------------------- FP64 Kerr-Schild cell
// The per-cell work of the FP64 path on a Kerr-Schild hole in terms of the
// null vector l and H: gamma_ij = delta_ij + F l_i l_j (F = 2H),
// gamma^ij = delta^ij - c l_i l_j, beta^i = c l^i, with alpha^2 = 1/(1 + F)
// and c = F alpha^2 (l.l = 1).  Ten numbers instead of the 55 of GeoFullT
// are live across the recovery, and the sources contract the derivatives of
// H and l with the fluid directly (ks_sources).  Sums are fma() and products
// mul_(): every kernel that calls these gets the same bits.
// The stage kernel was bound by the spills of those 55 values (580 MB of
// local stores at 128^3) and by the length of the recovery's chain.  With
// this, c2p_solve and 32-bit cell indices it took 1.55 ms per launch at 256^3
// instead of 2.77 at two blocks per SM (bytes alone: 0.72), and fits three
// blocks of 80 registers (262 MB of local stores into L2 at 128^3), with which
// and its prefetched inputs it takes 1.20.

// gamma^ij S_j
template <typename T>
GRHD_HD __forceinline__ void ks_raise(const KsCellT<T> &k, const double S[3],
                                      T mU[3])
{
    const T t = mul_(k.c, dot3(k.l, S));
    mU[0] = fma(-t, k.l[0], S[0]);
    mU[1] = fma(-t, k.l[1], S[1]);
    mU[2] = fma(-t, k.l[2], S[2]);
}

GRHD_HD __forceinline__ double ks_vsq(const KsCell &k, const double v[3])
{
    const double lv = dot3(k.l, v);
    return fma(mul_(k.F, lv), lv, dot3(v, v));
}

// enforce_primitive_floors (floors), Atmosphere.hpp:24-46
GRHD_HD __forceinline__ void ks_floors(const Options &o, const KsCell &k,
                                       Prim &pr)
{
    pr.rho = fmax(pr.rho, o.rho_floor);
    pr.p = fmax(pr.p, o.p_floor);
    const double v2 = ks_vsq(k, pr.v);
    if (v2 >= o.atmo_vmax2)
    {
        const double s = sqrt_(div_(o.atmo_vmax2, v2));
        pr.v[0] = mul_(pr.v[0], s);
        pr.v[1] = mul_(pr.v[1], s);
        pr.v[2] = mul_(pr.v[2], s);
    }
    pr.eps = div_(pr.p, mul_(o.G - 1.0, pr.rho));
}

GRHD_HD __forceinline__ bool ks_con2prim(const Options &o, const KsCell &k,
                                         const Cons &c, Prim &out)
{
    double mU[3], p, resid;
    int iters;
    ks_raise(k, c.S, mU);
    const double S2 = dot3(c.S, mU);
    return c2p_solve(o, c, S2, p, iters, resid) &&
           c2p_finish(o, c, mU, S2, p, out);
}

// compute_static_metric_source_terms (static_sources, StaticMetric.hpp:
// 193-275) at a Kerr-Schild cell, contracted by hand.  With D_i = d_i H:
//   d_i alpha = -alpha^3 D_i, d_i beta^j = 2 alpha^4 D_i l^j + c d_i l^j,
//   d_i ln sqrt(gamma) = alpha^2 D_i,
//   d_m gamma_ij = 2 D_m l_i l_j + F (l_i d_m l_j + l_j d_m l_i),
//   l.d_m l = 0, l^m d_m l_i = 0 (l is unit and geodesic),
// and d_i r = (r x_i + a^2 z delta_iz / r) / Sigma, so that for any vector u
//   u.d_i l = d_i r w(u) + ((r u_x - a u_y) delta_ix + (r u_y + a u_x)
//             delta_iy) / (r^2 + a^2) + u_z delta_iz / r,
//   w(u) = (u_x (x - 2 r l_x) + u_y (y - 2 r l_y)) / (r^2 + a^2)
//          - u_z l_z / r.
template <typename T>
GRHD_HD __forceinline__ ConsT<T> ks_sources(const Options &o, T a,
                                            const KsCellT<T> &k, double x,
                                            double y, double z,
                                            const Prim &pr, const Cons &c)
{
    const T a2 = mul_(a, a);
    const T *l = k.l;
    const double *v = pr.v;
    // d r, d H
    const T rs = mul_(k.r, k.inv_sigma);
    const T ias = mul_(k.inv_r, k.inv_sigma);
    const T dr[3] = {mul_(rs, x), mul_(rs, y),
                          mul_(fma(a2, ias, rs), z)};
    const T H = 0.5 * k.F;
    const T a2ct = mul_(a2, l[2]);
    // r - a^2 ct^2 / r
    const T rm = fma(-mul_(a2ct, l[2]), k.inv_r, k.r);
    const T hk = mul_(H, fma(mul_(-2.0, k.inv_sigma), rm, k.inv_r));
    const T dH[3] = {mul_(hk, dr[0]), mul_(hk, dr[1]),
                          fma(hk, dr[2], -mul_(mul_(k.F, a2ct), ias))};
    const T vH = dot3(v, dH), lH = dot3(l, dH);
    T mU[3];
    ks_raise(k, c.S, mU);
    const T mH = dot3(mU, dH), Sl = dot3(c.S, l);
    // rho h W^2, v.l
    const T lv = dot3(l, v);
    const T vv = fma(mul_(k.F, lv), lv, dot3(v, v));
    const T rhw = mul_(mul_(pr.rho, fma(o.G, pr.eps, 1.0)),
                            rcp_ulp(1.0 - vv));
    const T rl = mul_(rhw, lv);
    // l_i T^ij l_j of the stress T^ij = rhw v^i v^j + p gamma^ij
    const T lTl = fma(rl, lv, mul_(pr.p, k.alpha2));
    // transport velocity along d ln sqrt(gamma)
    const T tv =
        mul_(k.alpha2, fma(k.alpha, vH, -mul_(k.c, lH)));
    // w(u), v.dl.v and div l
    const T tr = 2.0 * k.r;
    const T wx = mul_(fma(-tr, l[0], x), k.inv_ra);
    const T wy = mul_(fma(-tr, l[1], y), k.inv_ra);
    const T wz = -mul_(l[2], k.inv_r);
    const T ri = mul_(k.r, k.inv_ra);
    const T wv = fma(v[0], wx, fma(v[1], wy, mul_(v[2], wz)));
    const T vA =
        fma(dot3(v, dr), wv,
            fma(ri, fma(v[0], v[0], mul_(v[1], v[1])),
                mul_(mul_(v[2], v[2]), k.inv_r)));
    const T div = fma(dr[0], wx, fma(dr[1], wy, fma(dr[2], wz,
                           fma(2.0, ri, k.inv_r))));
    ConsT<T> s;
    s.D = -mul_(c.D, tv);
    const T aa2 = mul_(k.alpha, k.alpha2);
    // alpha T^ij K_ij
    const T db = 2.0 * k.alpha2; // d_i beta^j = db alpha^2 D_i l^j + ...
    const T TK =
        fma(mul_(lTl, k.c), lH,
            fma(rl, mul_(db, vH),
                fma(mul_(rhw, k.c), vA,
                    mul_(pr.p, fma(mul_(db, k.alpha2), lH,
                                   mul_(k.c, div))))));
    s.tau = fma(aa2, fma(-pr.p, vH, mH), fma(-c.tau, tv, TK));
    // momentum: u.d_m l with u = alpha F rhw (v.l) v + c S
    const T X =
        fma(aa2, T((c.D + c.tau) - pr.p),
            fma(k.alpha, lTl, mul_(mul_(db, k.alpha2), Sl)));
    const T q = mul_(mul_(k.alpha, k.F), rl);
    const T u[3] = {fma(q, v[0], mul_(k.c, c.S[0])),
                         fma(q, v[1], mul_(k.c, c.S[1])),
                         fma(q, v[2], mul_(k.c, c.S[2]))};
    const T wu = fma(u[0], wx, fma(u[1], wy, mul_(u[2], wz)));
    const T ai = mul_(a, k.inv_ra);
    const T g[3] = {fma(ri, u[0], -mul_(ai, u[1])),
                         fma(ri, u[1], mul_(ai, u[0])),
                         mul_(u[2], k.inv_r)};
#pragma unroll
    for (int m = 0; m < 3; ++m)
        s.S[m] = fma(dH[m], X,
                     fma(dr[m], wu, fma(-c.S[m], tv, g[m])));
    return s;
}

// Sum over directions of max |characteristic speed| / dx of a cell with
// floored primitives (char_speeds, multiplied through by h as face_side).
GRHD_HD __forceinline__ double ks_inverse_dt(const Options &o,
                                             const KsCell &k, const Prim &pr,
                                             const double inv[3])
{
    const double vv = ks_vsq(k, pr.v);
    const double cg = mul_(o.G * (o.G - 1.0), pr.eps); // G p / rho
    const double h = fma(o.G, pr.eps, 1.0);
    const double hc = h - cg, den = fma(-vv, cg, h);
    const double cu = mul_(cg, 1.0 - vv);
    const double kk = mul_(k.alpha, rcp_ulp(den));
    double cell = 0.0;
#pragma unroll
    for (int d = 0; d < 3; ++d)
    {
        const double shift = mul_(k.c, k.l[d]);
        const double guu = fma(-shift, k.l[d], 1.0);
        const double vd = pr.v[d];
        const double base = mul_(vd, hc);
        const double rad = mul_(cu, fma(guu, den, -mul_(vd, base)));
        const double root = rad > 0.0 ? mul_(rad, rsqrt_ulp(rad)) : 0.0;
        const double lo = fma(base - root, kk, -shift);
        const double hi = fma(base + root, kk, -shift);
        cell = fma(fmax(fabs(lo), fabs(hi)), inv[d], cell);
    }
    return cell;
}

template <typename A, typename B>
GRHD_HD __forceinline__ PrimT<B> convert_prim(const PrimT<A> &s)
{
    PrimT<B> d;
    d.rho = B(s.rho);
    d.eps = B(s.eps);
    d.p = B(s.p);
    d.v[0] = B(s.v[0]);
    d.v[1] = B(s.v[1]);
    d.v[2] = B(s.v[2]);
    return d;
}

template <typename A, typename B>
GRHD_HD __forceinline__ ConsT<B> convert_cons(const ConsT<A> &s)
{
    ConsT<B> d;
    d.D = B(s.D);
    d.S[0] = B(s.S[0]);
    d.S[1] = B(s.S[1]);
    d.S[2] = B(s.S[2]);
    d.tau = B(s.tau);
    return d;
}

} // namespace grhd
