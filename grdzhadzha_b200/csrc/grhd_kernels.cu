// grhd_kernels.cu -- sm_100a kernels of the fixed-background Valencia GRHD
// operator.
//
// The kernels are templated on the arithmetic type T of the primitive
// cache, the face fluxes, the sources and the RHS: T = double is the FP64
// path, T = float the mixed path (the conserved state, the RK accumulator
// and con2prim stay FP64 in both).
//
// One RHS evaluation is three launches:
//   fill_ghosts : physical (outflow) ghost cells of the box, as
//                 fill_conserved_outflow_boundaries_from_fixed_background
//                 (FixedBGFArrayBoxFiniteVolume.hpp:113-177), then the
//                 ghost cells' con2prim into the primitive cache;
//   cells       : interior cells: metric + con2prim into the primitive
//                 cache (recover_primitives_from_fixed_background, :33-58)
//                 and the static-metric and volume-time sources (:255-298,
//                 :616-675);
//   faces       : the face fluxes -- MUSCL slopes, floors, p2c, HLLE --
//                 with the flux divergence and the sources written straight
//                 to the RHS (:179-253, :300-363).
// Inside the RK integrators the per-cell work of the next RHS is fused into
// the stage kernel, so `cells` runs once per step.  The reference evaluates
// every face twice and every direction in a separate pass over the box;
// here the interface states never leave registers / shared memory.
#include "grhd_kernels.cuh"
#include "grhd_kitp.cuh"

#include <atomic>

namespace grhd {

namespace {

constexpr int kWhereShift = 56;

__device__ __forceinline__ void record_error(DevStatus *st, int where,
                                             int64_t order)
{
    const unsigned long long key =
        ((unsigned long long)where << kWhereShift) | (unsigned long long)order;
    atomicMin(&st->err_key, key);
}

// Resident blocks per SM the register budget is sized for: the FP32
// (mixed) kernels fit three 256-thread blocks (80 registers, small
// spills; measured 13 % faster than two), the FP64 ones two (the FP64 face
// tile's 111 KB of shared memory allows no more).
template <typename T> constexpr int kMinBlocks = sizeof(T) == 4 ? 3 : 2;

// The stage kernel's blocks: where its state fits 80 registers with few
// spills, a third block hides more latency than they cost (ms per launch:
// FP64 Kerr-Schild at 256^3 1.36 with three, 1.53 with two; mixed binary at
// 320^3 3.2 and 3.9); the other two keep two (mixed Kerr-Schild at 256^3
// 1.49 with two, 1.63 with three; FP64 binary at 128^3 0.24 and 0.26).
constexpr int kStageThreads = 256;
template <typename T, int BGK>
constexpr int kStageBlocks = (sizeof(T) == 8) == (BGK == 0) ? 3 : 2;

// Loads of data that a persistent launch wrote itself in an earlier phase
// (CG = true) go through L2 (ld.global.cg): the non-coherent read-only path
// (__ldg) is only valid for data left unchanged for a whole launch.
template <bool CG, typename T> __device__ __forceinline__ T rd(const T *p)
{
    return CG ? __ldcg(p) : *p;
}
template <bool CG, typename T> __device__ __forceinline__ T rdro(const T *p)
{
    return CG ? __ldcg(p) : __ldg(p);
}

template <bool CG = false>
__device__ __forceinline__ Cons load_cons(const double *s, int64_t cs,
                                          int64_t idx)
{
    Cons c;
    c.D = rd<CG>(&s[kD * cs + idx]);
    c.S[0] = rd<CG>(&s[(kS1 + 0) * cs + idx]);
    c.S[1] = rd<CG>(&s[(kS1 + 1) * cs + idx]);
    c.S[2] = rd<CG>(&s[(kS1 + 2) * cs + idx]);
    c.tau = rd<CG>(&s[kTau * cs + idx]);
    return c;
}

__device__ __forceinline__ void store_cons(double *s, int64_t cs, int64_t idx,
                                           const Cons &c)
{
    s[kD * cs + idx] = c.D;
    s[(kS1 + 0) * cs + idx] = c.S[0];
    s[(kS1 + 1) * cs + idx] = c.S[1];
    s[(kS1 + 2) * cs + idx] = c.S[2];
    s[kTau * cs + idx] = c.tau;
}

__device__ __forceinline__ void store_prim(double *s, int64_t cs, int64_t idx,
                                           const Prim &p)
{
    s[kRho * cs + idx] = p.rho;
    s[kEps * cs + idx] = p.eps;
    s[kPress * cs + idx] = p.p;
    s[(kV1 + 0) * cs + idx] = p.v[0];
    s[(kV1 + 1) * cs + idx] = p.v[1];
    s[(kV1 + 2) * cs + idx] = p.v[2];
}

template <bool CG = false>
__device__ __forceinline__ Prim load_prim(const double *s, int64_t cs,
                                          int64_t idx)
{
    Prim p;
    p.rho = rd<CG>(&s[kRho * cs + idx]);
    p.eps = rd<CG>(&s[kEps * cs + idx]);
    p.p = rd<CG>(&s[kPress * cs + idx]);
    p.v[0] = rd<CG>(&s[(kV1 + 0) * cs + idx]);
    p.v[1] = rd<CG>(&s[(kV1 + 1) * cs + idx]);
    p.v[2] = rd<CG>(&s[(kV1 + 2) * cs + idx]);
    return p;
}

__device__ __forceinline__ bool primitive_differs(const Prim &a, const Prim &b)
{
    return a.rho != b.rho || a.eps != b.eps || a.p != b.p ||
           a.v[0] != b.v[0] || a.v[1] != b.v[1] || a.v[2] != b.v[2];
}

template <typename T>
__device__ __forceinline__ void store_pv(T *prim, int64_t pcs, int64_t g,
                                         const Prim &pr)
{
    prim[0 * pcs + g] = T(pr.rho);
    prim[1 * pcs + g] = T(pr.p);
    prim[2 * pcs + g] = T(pr.v[0]);
    prim[3 * pcs + g] = T(pr.v[1]);
    prim[4 * pcs + g] = T(pr.v[2]);
}

template <typename T>
__device__ __forceinline__ void store_src(T *src, int64_t rcs, int64_t ri,
                                          const ConsT<T> &s)
{
    src[0 * rcs + ri] = s.D;
    src[1 * rcs + ri] = s.S[0];
    src[2 * rcs + ri] = s.S[1];
    src[3 * rcs + ri] = s.S[2];
    src[4 * rcs + ri] = s.tau;
}

template <typename T> __device__ __forceinline__ ConsT<T> zero_cons()
{
    ConsT<T> z;
    z.D = z.tau = z.S[0] = z.S[1] = z.S[2] = T(0);
    return z;
}

// con2prim of a cell: the reference's bracketed solve (FP64 path) or the
// warm-started FP64 solve from a nearby pressure (mixed path).
template <typename T>
__device__ __forceinline__ bool cell_con2prim(const Options &o, const Cons &c,
                                              const GeoT<T> &g, double p_guess,
                                              Prim &out)
{
    double gUU[6];
#pragma unroll
    for (int q = 0; q < 6; ++q)
        gUU[q] = double(g.gUU[q]);
    if (sizeof(T) == sizeof(double))
        return con2prim(o, c, gUU, out, nullptr, nullptr);
    return con2prim_warm(o, c, gUU, p_guess, out);
}

// The same without a nearby pressure.
template <typename T>
__device__ __forceinline__ bool cold_con2prim(const Options &o, const Cons &c,
                                              const double gUU[6], Prim &out)
{
    if constexpr (sizeof(T) == sizeof(double))
        return con2prim(o, c, gUU, out, nullptr, nullptr);
    else
        return con2prim_mixed(o, c, gUU, out, nullptr, nullptr);
}

template <typename T>
__device__ __forceinline__ void gLL_double(const GeoT<T> &g, double out[6])
{
#pragma unroll
    for (int q = 0; q < 6; ++q)
        out[q] = double(g.gLL[q]);
}

// The metric of a cell for its con2prim, floors and p2c, widened to FP64
// for the solve: the FP64 metric, or the mixed path's, so that every
// con2prim of a cell within one path sees the same gamma (a state the
// stage recovery accepted at the velocity cap is accepted again by the
// next RHS's boundary fill and CFL speed).
template <typename T>
__device__ __forceinline__ void cell_metric_d(const Background &bg, double x,
                                              double y, double z,
                                              double gLL[6], double gUU[6])
{
    GeoT<T> g;
    metric_T<T, false>(bg, x, y, z, g, nullptr);
#pragma unroll
    for (int q = 0; q < 6; ++q)
    {
        gLL[q] = double(g.gLL[q]);
        gUU[q] = double(g.gUU[q]);
    }
}

// ------------------------------------------------------------ ghost fill

// Enumerates the shell "ghosted box minus interior box" as three slabs:
// z outside the interior; z inside, y outside; z and y inside, x outside.
__device__ __forceinline__ bool shell_cell(const BoxDev &b, int64_t t, int &i,
                                           int &j, int &k)
{
    const int64_t gx = b.gn[0], gy = b.gn[1];
    const int64_t zlo = b.lo[2] - b.glo[2];
    const int64_t nz_out = b.gn[2] - b.in[2];
    const int64_t n1 = nz_out * gx * gy;
    if (t < n1)
    {
        const int64_t kk = t / (gx * gy);
        const int64_t r = t - kk * gx * gy;
        k = (kk < zlo) ? b.glo[2] + (int)kk : b.hi[2] + 1 + (int)(kk - zlo);
        j = b.glo[1] + (int)(r / gx);
        i = b.glo[0] + (int)(r % gx);
        return true;
    }
    t -= n1;
    const int64_t ylo = b.lo[1] - b.glo[1];
    const int64_t ny_out = b.gn[1] - b.in[1];
    const int64_t n2 = (int64_t)b.in[2] * ny_out * gx;
    if (t < n2)
    {
        const int64_t kk = t / (ny_out * gx);
        const int64_t r = t - kk * ny_out * gx;
        const int64_t jj = r / gx;
        k = b.lo[2] + (int)kk;
        j = (jj < ylo) ? b.glo[1] + (int)jj : b.hi[1] + 1 + (int)(jj - ylo);
        i = b.glo[0] + (int)(r % gx);
        return true;
    }
    t -= n2;
    const int64_t xlo = b.lo[0] - b.glo[0];
    const int64_t nx_out = b.gn[0] - b.in[0];
    const int64_t n3 = (int64_t)b.in[2] * b.in[1] * nx_out;
    if (t < n3)
    {
        const int64_t kj = t / nx_out;
        const int64_t ii = t - kj * nx_out;
        k = b.lo[2] + (int)(kj / b.in[1]);
        j = b.lo[1] + (int)(kj % b.in[1]);
        i = (ii < xlo) ? b.glo[0] + (int)ii : b.hi[0] + 1 + (int)(ii - xlo);
        return true;
    }
    return false;
}

// Physical (outflow) ghost fill of the shell "ghosted box minus box"
// (fill_conserved_outflow_boundaries_from_fixed_background, :113-177),
// then, for every shell cell, the ghosted-box con2prim of the RHS into the
// primitive cache (recover_primitives_from_fixed_background, :33-58).  The
// fill itself is FP64 in both paths.  Shell cells inside the domain hold
// the owning boxes' values (after grhd_level_exchange); an excised one of
// them keeps its frozen primitives, as it does as an interior cell, so a
// level's RHS does not depend on how it is cut into boxes.
template <typename T, bool CG = false>
__device__ __forceinline__ void ghost_at(double *__restrict__ state,
                                         T *__restrict__ prim,
                                         const BoxDev &b, const Background &bg,
                                         const Options &o, DevStatus *st,
                                         int i, int j, int k)
{
    {
        const int iv[3] = {i, j, k};
        int srcc[3] = {i, j, k};
        bool ghost = false;
#pragma unroll
        for (int d = 0; d < 3; ++d)
        {
            if (iv[d] < b.dlo[d])
            {
                ghost = true;
                srcc[d] = b.lo[d];
            }
            else if (iv[d] > b.dhi[d])
            {
                ghost = true;
                srcc[d] = b.hi[d];
            }
        }
        double x, y, z;
        const int64_t idx = b.gidx(i, j, k);
        cell_xyz(o, i, j, k, x, y, z);
        double tLL[6], tUU[6];
        cell_metric_d<T>(bg, x, y, z, tLL, tUU);
        Cons c;
        if (ghost)
        {
            double sx, sy, sz;
            cell_xyz(o, srcc[0], srcc[1], srcc[2], sx, sy, sz);
            double sLL[6], sUU[6];
            cell_metric_d<T>(bg, sx, sy, sz, sLL, sUU);
            const Cons sc = load_cons<CG>(state, b.cs,
                                          b.gidx(srcc[0], srcc[1], srcc[2]));
            Prim pr;
            if (!cold_con2prim<T>(o, sc, sUU, pr))
            {
                record_error(st, 1, idx);
                return;
            }
            floors(o, pr, tLL);
            store_prim(state, b.cs, idx, pr);
            c = p2c(pr, tLL);
            store_cons(state, b.cs, idx, c);
        }
        else if (excised(o, i, j, k))
        {
            // a ghost that another box of the level owns: frozen like the
            // owner's interior cell
            store_pv(prim, b.pcs, idx, load_prim<CG>(state, b.cs, idx));
            return;
        }
        else
            c = load_cons<CG>(state, b.cs, idx);
        Prim pr;
        if (!cold_con2prim<T>(o, c, tUU, pr))
        {
            record_error(st, 2, idx);
            pr.rho = pr.p = 1.0;
            pr.v[0] = pr.v[1] = pr.v[2] = 0.0;
        }
        store_pv(prim, b.pcs, idx, pr);
    }
}

template <typename T, bool CG = false>
__device__ __forceinline__ void ghost_item(double *__restrict__ state,
                                           T *__restrict__ prim,
                                           const BoxDev &b,
                                           const Background &bg,
                                           const Options &o, DevStatus *st,
                                           int64_t t)
{
    int i, j, k;
    if (shell_cell(b, t, i, j, k))
        ghost_at<T, CG>(state, prim, b, bg, o, st, i, j, k);
}

template <typename T>
__global__ void __launch_bounds__(256)
    k_fill_ghosts(double *__restrict__ state, T *__restrict__ prim, BoxDev b,
                  Background bg, Options o, DevStatus *st, int64_t nshell)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
         t < nshell; t += (int64_t)gridDim.x * blockDim.x)
        ghost_item<T>(state, prim, b, bg, o, st, t);
}

// The shell cells of the ghosted planes k0..k1 only (plane_shell_cell).
template <typename T>
__global__ void __launch_bounds__(256)
    k_fill_ghost_planes(double *__restrict__ state, T *__restrict__ prim,
                        BoxDev b, Background bg, Options o, DevStatus *st,
                        int k0, int k1, int64_t n)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x)
    {
        int i, j, k;
        plane_shell_cell(b, k0, k1, t, i, j, k);
        ghost_at<T>(state, prim, b, bg, o, st, i, j, k);
    }
}

// Static-metric sources (:255-298) from the floored primitives and, for
// the binary, the volume-time source (:616-675, FP64 in both paths); `pr`
// is the cell's unfloored con2prim result.
template <typename T>
__device__ __forceinline__ ConsT<T> cell_sources(const Options &o,
                                                 const Background &bg,
                                                 double x, double y, double z,
                                                 const Prim &pr, const Cons &c,
                                                 const GeoFullT<T> &f)
{
    ConsT<T> s = zero_cons<T>();
    if (o.use_src)
    {
        // floors and the atmosphere test in FP64 for both paths, so that
        // which cells count as atmosphere does not depend on the type
        double gLL[6];
        gLL_double(f.g, gLL);
        Prim fd = pr;
        floors(o, fd, gLL);
        if (!is_atmo(o, fd, o.src_atmo_factor))
            s = static_sources(convert_prim<double, T>(fd),
                               convert_cons<double, T>(c), f);
    }
    if (o.use_vol && bg.kind == 1)
    {
        const double pos[3] = {x, y, z};
        const double Up = pn_scalar(bg.m1, bg.m2, bg.soft2, bg.p1p, bg.p2p, pos);
        const double Um = pn_scalar(bg.m1, bg.m2, bg.soft2, bg.p1m, bg.p2m, pos);
        const double dl =
            div_(__dadd_rn(pn_log_sqrt_det(__dadd_rn(1.0, 2.0 * Up)),
                           -pn_log_sqrt_det(__dadd_rn(1.0, 2.0 * Um))),
                 2.0 * bg.fd_h);
        s.D = T(double(s.D) + (0.0 - c.D * dl));
        s.tau = T(double(s.tau) + (0.0 - c.tau * dl));
#pragma unroll
        for (int m = 0; m < 3; ++m)
            s.S[m] = T(double(s.S[m]) + (0.0 - c.S[m] * dl));
    }
    return s;
}

// Interior cell t of a box (x fastest).  32-bit division, a fifth of the
// instructions of 64-bit: a box of 2^32 cells would be 378 GB of state.
__device__ __forceinline__ void interior_cell(const BoxDev &b, int64_t t,
                                              int &i, int &j, int &k)
{
    const unsigned u = (unsigned)t, nx = b.in[0], ny = b.in[1];
    const unsigned r = u / nx, q = r / ny;
    i = b.lo[0] + (int)(u - r * nx);
    j = b.lo[1] + (int)(r - q * ny);
    k = b.lo[2] + (int)q;
}

// The per-cell work of the FP64 path on a Kerr-Schild background runs on
// KsCell (grhd_device.cuh).
template <typename T, int BGK>
constexpr bool ks64 = sizeof(T) == sizeof(double) && BGK == 0;

// What the next RHS needs of a cell: con2prim's result `pr` into the
// primitive cache and the sources of its floored primitives.
template <typename T>
__device__ __forceinline__ void
ks_prep(const Options &o, const Background &bg, const KsCell &kc, double x,
        double y, double z, bool ok, Prim pr, const Cons &c, T *prim, T *src,
        const BoxDev &b, int64_t g, int64_t t, DevStatus *st)
{
    Cons s = zero_cons<double>();
    if (!ok)
    {
        record_error(st, 2, g);
        pr.rho = pr.p = 1.0;
        pr.v[0] = pr.v[1] = pr.v[2] = 0.0;
        pr.eps = 1.0;
    }
    store_pv(prim, b.pcs, g, pr);
    if (ok && o.use_src)
    {
        ks_floors(o, kc, pr);
        if (!is_atmo(o, pr, o.src_atmo_factor))
            s = ks_sources(o, bg.a, kc, x, y, z, pr, c);
    }
    store_src(src, b.rcs, t, s);
}

// ------------------------------------------------------- per-cell pass

// Interior cells: con2prim into the primitive cache (the ghosted-box
// recovery of the RHS restricted to the interior; the shell is done by
// k_fill_ghosts) and the sources into the source scratch.  Excised cells
// keep their frozen primitives and get no source.  The mixed path starts
// con2prim from the state's stored pressure.
template <typename T, bool CG = false, int BGK = -1>
__device__ __forceinline__ void cells_item(const double *__restrict__ state,
                                           T *__restrict__ prim,
                                           T *__restrict__ src,
                                           const BoxDev &b,
                                           const Background &bg,
                                           const Options &o, DevStatus *st,
                                           int64_t t)
{
    {
        int i, j, k;
        interior_cell(b, t, i, j, k);
        const int64_t g = b.gidx(i, j, k);
        ConsT<T> s = zero_cons<T>();
        if (excised(o, i, j, k))
        {
            store_pv(prim, b.pcs, g, load_prim<CG>(state, b.cs, g));
            store_src(src, b.rcs, t, s);
            return;
        }
        double x, y, z;
        cell_xyz(o, i, j, k, x, y, z);
        if constexpr (ks64<T, BGK>)
        {
            const Cons c = load_cons<CG>(state, b.cs, g);
            KsCell kc;
            ks_cell(bg.M, bg.a, x, y, z, kc);
            Prim pr;
            const bool ok = ks_con2prim(o, kc, c, pr);
            ks_prep(o, bg, kc, x, y, z, ok, pr, c, prim, src, b, g, t, st);
            return;
        }
        GeoFullT<T> f;
        if (o.use_src)
            metric_T<T, true, BGK>(bg, x, y, z, f.g, &f);
        else
            metric_T<T, false, BGK>(bg, x, y, z, f.g, nullptr);
        const Cons c = load_cons<CG>(state, b.cs, g);
        Prim pr;
        if (!cell_con2prim(o, c, f.g, rd<CG>(&state[kPress * b.cs + g]), pr))
        {
            record_error(st, 2, g);
            pr.rho = pr.p = 1.0;
            pr.v[0] = pr.v[1] = pr.v[2] = 0.0;
            pr.eps = 1.0;
        }
        else
            s = cell_sources<T>(o, bg, x, y, z, pr, c, f);
        store_pv(prim, b.pcs, g, pr);
        store_src(src, b.rcs, t, s);
    }
}

template <typename T, int BGK>
__global__ void __launch_bounds__(256, 3)
    k_cells(const double *__restrict__ state, T *__restrict__ prim,
            T *__restrict__ src, BoxDev b, Background bg, Options o,
            DevStatus *st)
{
    const int64_t n = b.ivol();
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x)
        cells_item<T, false, BGK>(state, prim, src, b, bg, o, st, t);
}

// A first RHS's ghost fill and per-cell pass in one launch, FP64: they do not
// depend on one another (the fill reads interior conserved variables and
// writes ghosts), and on a small box each is a launch of a few microseconds
// (right-hand side of a 16^3 patch 56 -> 46 us, 45x38x31 binary 66 -> 57).
// The first `ghost_blocks` blocks fill ghosts: theirs is the longer chain
// (two recoveries a cell).
template <int BGK>
__global__ void __launch_bounds__(256, 2)
    k_prepare(double *state, double *__restrict__ prim,
              double *__restrict__ src, BoxDev b, Background bg, Options o,
              DevStatus *st, int64_t nshell, int ghost_blocks)
{
    const int64_t first = blockIdx.x < ghost_blocks
                              ? blockIdx.x
                              : blockIdx.x - ghost_blocks;
    const int64_t t0 = first * blockDim.x + threadIdx.x;
    if (blockIdx.x < ghost_blocks)
    {
        const int64_t step = (int64_t)ghost_blocks * blockDim.x;
        for (int64_t t = t0; t < nshell; t += step)
            ghost_item<double>(state, prim, b, bg, o, st, t);
    }
    else
    {
        const int64_t step =
            (int64_t)(gridDim.x - ghost_blocks) * blockDim.x;
        const int64_t n = b.ivol();
        for (int64_t t = t0; t < n; t += step)
            cells_item<double, false, BGK>(state, prim, src, b, bg, o, st, t);
    }
}

// ----------------------------------------------------------- face pass

// The tile keeps half of each geometry field a face reads (gamma_ij, the
// diagonal of gamma^ij, lapse, shift), so the face average of two cells is a
// sum; halving is exact, so it is the average's value bit for bit.
template <typename T>
__device__ __forceinline__ void geo_store_half(T *g, int n, int cell,
                                               const GeoT<T> &v)
{
#pragma unroll
    for (int s = 0; s < 6; ++s)
        g[s * n + cell] = v.gLL[s];
    g[6 * n + cell] = v.gUU[0];
    g[7 * n + cell] = v.gUU[3];
    g[8 * n + cell] = v.gUU[5];
    g[9 * n + cell] = v.lapse;
#pragma unroll
    for (int i = 0; i < 3; ++i)
        g[(10 + i) * n + cell] = v.shift[i];
}

template <typename T>
__device__ __forceinline__ void geo_halve(GeoT<T> &v)
{
#pragma unroll
    for (int s = 0; s < 6; ++s)
    {
        v.gLL[s] *= T(0.5);
        v.gUU[s] *= T(0.5);
    }
    v.lapse *= T(0.5);
#pragma unroll
    for (int i = 0; i < 3; ++i)
        v.shift[i] *= T(0.5);
}

// Face geometry along d from two halved cells of the tile.
template <typename T>
__device__ __forceinline__ void geo_sum(const T *g, int n, int ca, int cb,
                                        int d, GeoT<T> &v)
{
#pragma unroll
    for (int s = 0; s < 6; ++s)
        v.gLL[s] = g[s * n + ca] + g[s * n + cb];
    v.gUU[sym(d, d)] = g[(6 + d) * n + ca] + g[(6 + d) * n + cb];
    v.lapse = g[9 * n + ca] + g[9 * n + cb];
    v.shift[d] = g[(10 + d) * n + ca] + g[(10 + d) * n + cb];
}

// The same from a tile cell and a halved cell in registers (z faces).
template <typename T>
__device__ __forceinline__ void geo_sum_z(const T *g, int n, int ca,
                                          const GeoT<T> &b, GeoT<T> &v)
{
#pragma unroll
    for (int s = 0; s < 6; ++s)
        v.gLL[s] = g[s * n + ca] + b.gLL[s];
    v.gUU[5] = g[8 * n + ca] + b.gUU[5];
    v.lapse = g[9 * n + ca] + b.lapse;
    v.shift[2] = g[12 * n + ca] + b.shift[2];
}

template <typename T, bool CG = false>
__device__ __forceinline__ PVT<T> load_pv_global(const T *__restrict__ prim,
                                                 int64_t pcs, int64_t idx)
{
    PVT<T> p;
#pragma unroll
    for (int c = 0; c < 5; ++c)
        p.q[c] = rdro<CG>(&prim[c * pcs + idx]);
    return p;
}

template <typename T>
__device__ __forceinline__ PVT<T> load_pv_smem(const T *P, int cell)
{
    constexpr int n = kPW * kPW;
    PVT<T> p;
#pragma unroll
    for (int c = 0; c < 5; ++c)
        p.q[c] = P[c * n + cell];
    return p;
}

// Asynchronous global -> shared copy of one element (cp.async, 4 or 8
// bytes, cached in L1) and the wait for all of this thread's copies.
template <typename T>
__device__ __forceinline__ void cp_async_elem(T *dst, const T *src)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst);
    if constexpr (sizeof(T) == 8)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d),
                     "l"(src)
                     : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 4;\n" ::"r"(d),
                     "l"(src)
                     : "memory");
}

__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.wait_all;\n" ::: "memory");
}

// The primitive cross tile of a z march at plane k (clamped to the
// ghosted box): cp.async copies (ASYNC), or loads.
template <typename T, bool CG, bool ASYNC>
__device__ __forceinline__ void load_p_tile(T *P, const T *__restrict__ prim,
                                            const BoxDev &b, int i0, int j0,
                                            int k, int tid)
{
    constexpr int nP = kPW * kPW;
    for (int idx = tid; idx < nP; idx += kTB * kTB)
    {
        const int u = idx % kPW, v = idx / kPW;
        if ((u < 2 || u > kPW - 3) && (v < 2 || v > kPW - 3))
            continue;
        const int gi = min(max(i0 - 2 + u, b.glo[0]), b.ghi[0]);
        const int gj = min(max(j0 - 2 + v, b.glo[1]), b.ghi[1]);
        const int64_t g = b.gidx(gi, gj, k);
#pragma unroll
        for (int c = 0; c < 5; ++c)
        {
            if constexpr (ASYNC)
                cp_async_elem(&P[c * nP + idx], &prim[c * b.pcs + g]);
            else
                P[c * nP + idx] = rdro<CG>(&prim[c * b.pcs + g]);
        }
    }
}

// Rest-mass flux of one face through the voxelised sphere r < R (new):
// the face between cells L and R (R = L + e_d) lies on the sphere's
// boundary when exactly one of them is inside; the outward flux is
// +sqrt(gamma_face) F_D dA when L is inside, and Mdot counts the inward
// flux.
template <typename T>
__device__ __forceinline__ double mdot_face(const Options &o, int il, int jl,
                                            int kl, int d, const GeoT<T> &gf,
                                            T FD)
{
    double x, y, z;
    cell_xyz(o, il, jl, kl, x, y, z);
    const bool in_l = sqrt(x * x + y * y + z * z) < o.accretion_radius;
    cell_xyz(o, il + (d == 0), jl + (d == 1), kl + (d == 2), x, y, z);
    const bool in_r = sqrt(x * x + y * y + z * z) < o.accretion_radius;
    if (in_l == in_r)
        return 0.0;
    double g[6];
    gLL_double(gf, g);
    const double det = g[0] * (g[3] * g[5] - g[4] * g[4]) -
                       g[1] * (g[1] * g[5] - g[4] * g[2]) +
                       g[2] * (g[1] * g[4] - g[3] * g[2]);
    return (in_l ? -1.0 : 1.0) * sqrt(det) * double(FD) * (o.dx * o.dx);
}

// Block sum of `v` into part[block] (fixed order within the block).
__device__ __forceinline__ void block_partial(double v, double *scratch,
                                              double *part, int tid, int nt,
                                              int64_t block)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        v += __shfl_down_sync(0xffffffffu, v, off);
    if ((tid & 31) == 0)
        scratch[tid >> 5] = v;
    __syncthreads();
    if (tid == 0)
    {
        double sum = 0.0;
        for (int w = 0; w < nt / 32; ++w)
            sum += scratch[w];
        part[block] = sum;
    }
}

// 16x16 threads own a 16x16 (x,y) cell tile and march along z over a chunk
// of planes; every face is evaluated once per tile.  Per plane, two phases
// between two barriers:
//   1. the lower x and y face of each thread's cell, from the primitive
//      tile (2-cell halo; the planes k to k+2, copied in asynchronously) and
//      the geometry tile (1-cell halo) in shared memory;
//      the tile's last x faces fall to warp 0 and its last y faces to warp
//      1 (the same code once more);
//   2. the geometry of plane k+1 (own cell in registers and to the tile; the
//      halo cells fall to warps 2 and 3), the z face above the cell from it,
//      and the divergence + sources (copied in a plane ahead) to the RHS.
// The tile needs one geometry buffer: plane k's x and y faces have read it
// when plane k+1's cells overwrite it, and a z face reads its own column
// only.  A cell's z slope serves both its z faces: the upper state is
// carried to the next plane.  Tiles of 16 cells fit boxes whose sides are
// multiples of 16 -- the usual patch and grid sizes -- without idle columns.
// Issue- and latency-bound (FP64 pipe about half busy, DRAM idle): against
// tiles of 15 cells with three barriers, two geometry buffers and the y
// fluxes stored across the banks, an FP64 RK4 step of the 256^3 torus went
// from 24.9 to 21.0 ms (mixed 15.9 to 14.9, results unchanged bit for bit),
// the 64^3 Michel step from 0.68 to 0.55 ms.  With a third plane buffered (z
// faces read their column from shared memory instead of waiting for global
// loads) and the sources prefetched, 2.22 -> 2.00 ms per launch at 256^3.
// The march starts at plane k0-1 (z face only), so the face below k0 comes
// from the same code as the block below's upper face, bit for bit: the RHS
// does not depend on where the z blocks start.
// One tile (bx, by, bz) of the face pass; `smem_raw` holds faces_smem<T>()
// bytes; the tile's accretion sum goes to mdot_part[part].
// With BGK = kGridMetric the geometry comes from a cache of the cells'
// (launch_ccz4_cells) instead of the background.
constexpr int kGridMetric = 2;

// Geometry of cell (i,j,k), clamped into the ghosted box, from the cache
// (gLL[6] gUU[6] lapse shift[3], stride n).
__device__ __forceinline__ void cached_geo(const double *__restrict__ gc,
                                           const BoxDev &b, int i, int j,
                                           int k, Geo &g)
{
    const int64_t n = b.gvol();
    const double *c = gc + b.gidx(min(max(i, b.glo[0]), b.ghi[0]),
                                  min(max(j, b.glo[1]), b.ghi[1]), k);
#pragma unroll
    for (int q = 0; q < 6; ++q)
        g.gLL[q] = __ldg(&c[q * n]);
    g.gUU[0] = __ldg(&c[6 * n]);
    g.gUU[3] = __ldg(&c[9 * n]);
    g.gUU[5] = __ldg(&c[11 * n]);
    g.lapse = __ldg(&c[12 * n]);
#pragma unroll
    for (int d = 0; d < 3; ++d)
        g.shift[d] = __ldg(&c[(13 + d) * n]);
}

template <typename T, bool MDOT, bool CG = false, int BGK = -1>
__device__ __forceinline__ void
faces_tile(const T *__restrict__ prim, const T *__restrict__ src,
           T *__restrict__ rhs, const BoxDev &b, const Background &bg,
           const Options &o, const FaceOpt<T> &fo, double idx0_, double idx1_,
           double idx2_, int zchunk, int bx, int by, int bz,
           unsigned char *smem_raw, double *__restrict__ mdot_part,
           int64_t part, const double *__restrict__ gc = nullptr)
{
    constexpr int nP = kPW * kPW;
    constexpr int nG = kGW * kGW;
    constexpr int nF = kTC * (kTC + 1); // x or y faces of a tile plane
    constexpr int wX = kTC + 1;         // x faces of a row
    T *P = reinterpret_cast<T *>(smem_raw); // [3][5][nP], plane mod 3
    T *G = P + 3 * 5 * nP;                  // [kGeoFields][nG]
    T *Fx = G + kGeoFields * nG;            // [5][nF], row-major rows of wX
    T *Fy = Fx + 5 * nF;                    // [5][nF], kTC + 1 rows of kTC
    T *Sr = Fy + 5 * nF;                    // [5][256], this plane's sources
    const T idx0 = T(idx0_), idx1 = T(idx1_), idx2 = T(idx2_);

    const int a = threadIdx.x, bb = threadIdx.y;
    const int tid = bb * kTB + a;
    const int i0 = b.lo[0] + bx * kTC;
    const int j0 = b.lo[1] + by * kTC;
    const int k0 = b.lo[2] + bz * zchunk;
    const int k1 = min(k0 + zchunk - 1, b.hi[2]);
    const int ci = i0 + a, cj = j0 + bb; // this thread's cell column
    const bool col_ok = ci <= b.hi[0] && cj <= b.hi[1];
    const int64_t plane = (int64_t)b.gn[0] * b.gn[1];
    const int own_p = (bb + 2) * kPW + a + 2, own_g = (bb + 1) * kGW + a + 1;
    const int reach = fo.reach;
    // primitive tiles of planes k0-1, k0 and k0+1; P0, P1, P2 hold the planes
    // k, k+1, k+2 of the march
    T *P0 = P, *P1 = P + 5 * nP, *P2 = P + 2 * 5 * nP;
    load_p_tile<T, CG, !CG>(P0, prim, b, i0, j0, k0 - 1, tid);
    load_p_tile<T, CG, !CG>(P1, prim, b, i0, j0, k0, tid);
    load_p_tile<T, CG, !CG>(P2, prim, b, i0, j0, k0 + 1, tid);
    T up[5]; // upper state of the cell at plane k, for the z face above it
    {
        // this column's primitives from plane k0-2 (clamped into the box)
        const T *pcol =
            prim + b.gidx(min(ci, b.hi[0]), min(cj, b.hi[1]), k0 - 2);
        T unused[5];
        cell_states(fo, load_pv_global<T, CG>(pcol, b.pcs, 0),
                    load_pv_global<T, CG>(pcol, b.pcs, plane),
                    load_pv_global<T, CG>(pcol, b.pcs, (1 + reach) * plane),
                    unused, up);
    }

    ConsT<T> Flo = zero_cons<T>();
    double macc = 0.0;
    // k = k0-2 fills the geometry of plane k0-1 only
#pragma unroll 1
    for (int k = k0 - 2; k <= k1; ++k)
    {
        const bool zface = k >= k0 - 1; // the z face above plane k
        const bool cells = k >= k0;     // plane k's x/y faces and RHS
        if (cells)
        {
            // x face between cells (i0+fa-1, i0+fa) in row j0+fb
#pragma unroll 1
            for (int pass = 0; pass < 2; ++pass)
            {
                const int fa = pass ? kTC : a, fb = pass ? tid : bb;
                if (pass && tid >= kTC)
                    break;
                if (j0 + fb > b.hi[1] || i0 + fa - 1 > b.hi[0])
                    continue;
                const int row = (fb + 2) * kPW + fa;
                GeoT<T> gf;
                geo_sum(G, nG, (fb + 1) * kGW + fa, (fb + 1) * kGW + fa + 1, 0,
                        gf);
                const ConsT<T> f = face_flux(
                    fo, load_pv_smem(P0, row + 1 - reach),
                    load_pv_smem(P0, row + 1), load_pv_smem(P0, row + 2),
                    load_pv_smem(P0, row + 2 + reach), gf, 0);
                const int fi = fb * wX + fa;
                if (MDOT && fa < kTC && i0 + fa <= b.hi[0])
                    macc +=
                        mdot_face(o, i0 + fa - 1, j0 + fb, k, 0, gf, f.D);
                Fx[0 * nF + fi] = f.D;
                Fx[1 * nF + fi] = f.S[0];
                Fx[2 * nF + fi] = f.S[1];
                Fx[3 * nF + fi] = f.S[2];
                Fx[4 * nF + fi] = f.tau;
            }
            // y face between rows (j0+fb-1, j0+fb) in column i0+fa
#pragma unroll 1
            for (int pass = 0; pass < 2; ++pass)
            {
                const int fa = pass ? tid - 32 : a, fb = pass ? kTC : bb;
                if (pass && (unsigned)fa >= (unsigned)kTC)
                    break;
                if (i0 + fa > b.hi[0] || j0 + fb - 1 > b.hi[1])
                    continue;
                const int col = fb * kPW + fa + 2;
                GeoT<T> gf;
                geo_sum(G, nG, fb * kGW + fa + 1, (fb + 1) * kGW + fa + 1, 1,
                        gf);
                const ConsT<T> f = face_flux(
                    fo, load_pv_smem(P0, col + (1 - reach) * kPW),
                    load_pv_smem(P0, col + kPW),
                    load_pv_smem(P0, col + 2 * kPW),
                    load_pv_smem(P0, col + (2 + reach) * kPW), gf, 1);
                const int fi = fb * kTC + fa;
                if (MDOT && fb < kTC && j0 + fb <= b.hi[1])
                    macc +=
                        mdot_face(o, i0 + fa, j0 + fb - 1, k, 1, gf, f.D);
                Fy[0 * nF + fi] = f.D;
                Fy[1 * nF + fi] = f.S[0];
                Fy[2 * nF + fi] = f.S[1];
                Fy[3 * nF + fi] = f.S[2];
                Fy[4 * nF + fi] = f.tau;
            }
        }
        // this column's primitives at plane k, whose tile gives way to
        // plane k+3's
        PVT<T> w1;
        if (zface)
            w1 = load_pv_smem(P0, own_p);
        // plane k+2's tile and plane k's sources, issued one plane ago, have
        // landed
        if (!CG)
            cp_async_wait_all();
        __syncthreads();
        // of the planes above k1 the z faces read their own columns only
        if (zface && k < k1)
            load_p_tile<T, CG, !CG>(P0, prim, b, i0, j0, k + 3, tid);
        // geometry of plane k+1: the halo cells (where the next plane has x
        // and y faces), then the own cell, left in registers
        GeoT<T> gn;
        const int halo = tid - 64;
        const bool has_halo =
            (unsigned)halo < 4u * kTC && zface && k + 1 <= k1;
#pragma unroll 1
        for (int pass = has_halo ? 0 : 1; pass < 2; ++pass)
        {
            int u = a + 1, v = bb + 1;
            if (pass == 0)
            {
                const int at = halo % kTC + 1;
                u = halo < 2 * kTC ? (halo < kTC ? 0 : kGW - 1) : at;
                v = halo < 2 * kTC ? at : (halo < 3 * kTC ? 0 : kGW - 1);
            }
            if constexpr (BGK == kGridMetric)
                cached_geo(gc, b, i0 - 1 + u, j0 - 1 + v, k + 1, gn);
            else
            {
                double x, y, z;
                cell_xyz(o, i0 - 1 + u, j0 - 1 + v, k + 1, x, y, z);
                metric_T<T, false, BGK>(bg, x, y, z, gn, nullptr);
            }
            geo_halve(gn);
            if (pass == 0)
                geo_store_half(G, nG, v * kGW + u, gn);
        }
        // z face at k+1/2 for this column
        ConsT<T> Fhi = zero_cons<T>();
        if (zface && col_ok)
        {
            GeoT<T> gf;
            geo_sum_z(G, nG, own_g, gn, gf);
            T low[5], next[5];
            cell_states(fo, w1, load_pv_smem(P1, own_p),
                        load_pv_smem(reach ? P2 : P1, own_p), low, next);
            Fhi = state_flux(fo, up, low, gf, 2);
#pragma unroll
            for (int c = 0; c < 5; ++c)
                up[c] = next[c];
            // a box counts the sphere faces whose upper cell it holds, in
            // every direction, so the boxes of a level count each once
            if (MDOT && (cells ? k < b.hi[2] : k0 == b.lo[2]))
                macc += mdot_face(o, ci, cj, k, 2, gf, Fhi.D);
        }
        geo_store_half(G, nG, own_g, gn);

        if (cells && col_ok)
        {
            const int fx = bb * wX + a, fy = bb * kTC + a;
            const int64_t ri = b.iidx(ci, cj, k);
            T out[5];
            const T fl[5] = {Flo.D, Flo.S[0], Flo.S[1], Flo.S[2], Flo.tau};
            const T fh[5] = {Fhi.D, Fhi.S[0], Fhi.S[1], Fhi.S[2], Fhi.tau};
#pragma unroll
            for (int c = 0; c < 5; ++c)
            {
                const T rx = -idx0 * (Fx[c * nF + fx + 1] - Fx[c * nF + fx]);
                const T ry =
                    -idx1 * (Fy[c * nF + fy + kTC] - Fy[c * nF + fy]);
                const T rz = -idx2 * (fh[c] - fl[c]);
                out[c] = ((rx + ry) + rz) +
                         (CG ? rdro<CG>(&src[c * b.rcs + ri])
                             : Sr[c * (kTB * kTB) + tid]);
            }
            if (excised(o, ci, cj, k))
            {
#pragma unroll
                for (int c = 0; c < 5; ++c)
                    out[c] = T(0);
            }
#pragma unroll
            for (int c = 0; c < 5; ++c)
                rhs[c * b.rcs + ri] = out[c];
        }
        Flo = Fhi;
        // the next plane's sources of this cell
        if (!CG && zface && k < k1 && col_ok)
        {
            const int64_t ri = b.iidx(ci, cj, k + 1);
#pragma unroll
            for (int c = 0; c < 5; ++c)
                cp_async_elem(&Sr[c * (kTB * kTB) + tid],
                              &src[c * b.rcs + ri]);
        }
        if (zface)
        {
            T *const p = P0;
            P0 = P1;
            P1 = P2;
            P2 = p;
        }
        __syncthreads();
    }
    if (MDOT)
        block_partial(macc, reinterpret_cast<double *>(smem_raw), mdot_part,
                      tid, kTB * kTB, part);
}

template <typename T, bool MDOT, int BGK>
__global__ void __launch_bounds__(kTB *kTB, kMinBlocks<T>)
    k_faces(const T *__restrict__ prim, const T *__restrict__ src,
            T *__restrict__ rhs, BoxDev b, Background bg, Options o,
            FaceOpt<T> fo, double idx0_, double idx1_, double idx2_,
            int zchunk, double *__restrict__ mdot_part)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    faces_tile<T, MDOT, false, BGK>(prim, src, rhs, b, bg, o, fo, idx0_, idx1_,
                                    idx2_, zchunk,
                        blockIdx.x, blockIdx.y, blockIdx.z, smem_raw,
                        mdot_part,
                        blockIdx.x + (int64_t)gridDim.x *
                                         (blockIdx.y + (int64_t)gridDim.y *
                                                           blockIdx.z));
}

// Mdot of one RHS evaluation: the block partials summed in a fixed order;
// acc[0] = Mdot, acc[1] += weight * Mdot (the time integral).
__global__ void k_mdot_sum(const double *__restrict__ part, int64_t n,
                           double weight, double *acc)
{
    __shared__ double w[32];
    double v = 0.0;
    for (int64_t q = threadIdx.x; q < n; q += blockDim.x)
        v += part[q];
    block_partial(v, w, w + 8, threadIdx.x, blockDim.x, 0);
    if (threadIdx.x == 0)
    {
        acc[0] = w[8];
        acc[1] += weight * w[8];
    }
}

// ---------------------------------------------- post-update recovery

// recover_primitives_and_apply_atmosphere_from_fixed_background for one
// cell (FixedBGFArrayBoxFiniteVolume.hpp:60-110); c is the updated
// conserved state.  Writes prims (and reset conserved) to `out`.  With kc the
// root solve is the Kerr-Schild cell's, the FP64 right-hand side's own, which
// therefore recovers the same pressures from this state; the mixed right-hand
// side starts its own solve (con2prim_warm) from them.
__device__ __forceinline__ void recover_cell(const Options &o, const Geo &g,
                                             const KsCell *kc, Cons c,
                                             double *out, int64_t cs,
                                             int64_t idx,
                                             unsigned long long cnt[4])
{
    Prim pr;
    const bool ok = kc ? ks_con2prim(o, *kc, c, pr)
                       : con2prim(o, c, g.gUU, pr, nullptr, nullptr);
    bool reset = !ok;
    cnt[0] += 1;
    if (ok)
    {
        Prim fl = pr;
        floors(o, fl, g.gLL);
        reset = primitive_differs(pr, fl);
        if (reset)
            cnt[2] += 1;
        pr = fl;
    }
    else
    {
        cnt[1] += 1;
        pr = atmosphere(o);
    }
    store_prim(out, cs, idx, pr);
    if (reset)
    {
        cnt[3] += 1;
        c = p2c(pr, g.gLL);
    }
    store_cons(out, cs, idx, c);
}

// Lane of the calling thread in its warp (blocks may be 2-D).
__device__ __forceinline__ int lane_id()
{
    return (int)((threadIdx.x + blockDim.x * threadIdx.y) & 31u);
}

__device__ __forceinline__ void flush_counts(DevStatus *st,
                                             unsigned long long cnt[4])
{
#pragma unroll
    for (int q = 0; q < 4; ++q)
    {
        unsigned long long v = cnt[q];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
            v += __shfl_down_sync(0xffffffffu, v, off);
        if (lane_id() == 0 && v)
            atomicAdd(&st->counts[q], v);
    }
}

// update_conserved: dst = src + dt * rhs on the interior
// (add_scaled_conserved_rhs, FArrayBoxFiniteVolume.hpp:927-940), then the
// post-update recovery when `recover` is set.
__global__ void __launch_bounds__(256)
    k_update(double *dst, int64_t dcs, const double *srcs, int64_t scs,
             const double *__restrict__ rhs, BoxDev b, Background bg,
             Options o, double dt, int recover, DevStatus *st)
{
    unsigned long long cnt[4] = {0, 0, 0, 0};
    const int64_t n = b.ivol();
    const int64_t n_pad = (n + blockDim.x - 1) / blockDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_pad;
         t += (int64_t)gridDim.x * blockDim.x)
    {
        if (t < n)
        {
            int i, j, k;
            interior_cell(b, t, i, j, k);
            const int64_t g = b.gidx(i, j, k);
            if (excised(o, i, j, k))
            {
                if (dst != srcs)
                    for (int c = 0; c < kStateComps; ++c)
                        dst[c * dcs + g] = srcs[c * scs + g];
            }
            else
            {
                Cons c = load_cons(srcs, scs, g);
                c.D += dt * rhs[0 * b.rcs + t];
                c.tau += dt * rhs[4 * b.rcs + t];
                c.S[0] += dt * rhs[1 * b.rcs + t];
                c.S[1] += dt * rhs[2 * b.rcs + t];
                c.S[2] += dt * rhs[3 * b.rcs + t];
                if (recover)
                {
                    double x, y, z;
                    cell_xyz(o, i, j, k, x, y, z);
                    Geo geo;
                    background_metric<false>(bg, x, y, z, geo, nullptr);
                    KsCell kc;
                    if (bg.kind == 0)
                        ks_cell(bg.M, bg.a, x, y, z, kc);
                    recover_cell(o, geo, bg.kind == 0 ? &kc : nullptr, c, dst,
                                 dcs, g, cnt);
                }
                else
                {
                    store_cons(dst, dcs, g, c);
                    if (dst != srcs)
                        store_prim(dst, dcs, g, load_prim(srcs, scs, g));
                }
            }
        }
        flush_counts(st, cnt);
        cnt[0] = cnt[1] = cnt[2] = cnt[3] = 0;
    }
}

__global__ void __launch_bounds__(256)
    k_recover(double *__restrict__ state, BoxDev b, Background bg, Options o,
              DevStatus *st)
{
    unsigned long long cnt[4] = {0, 0, 0, 0};
    const int64_t n = b.ivol();
    const int64_t n_pad = (n + blockDim.x - 1) / blockDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_pad;
         t += (int64_t)gridDim.x * blockDim.x)
    {
        if (t < n)
        {
            int i, j, k;
            interior_cell(b, t, i, j, k);
            if (!excised(o, i, j, k))
            {
                const int64_t g = b.gidx(i, j, k);
                double x, y, z;
                cell_xyz(o, i, j, k, x, y, z);
                Geo geo;
                background_metric<false>(bg, x, y, z, geo, nullptr);
                KsCell kc;
                if (bg.kind == 0)
                    ks_cell(bg.M, bg.a, x, y, z, kc);
                recover_cell(o, geo, bg.kind == 0 ? &kc : nullptr,
                             load_cons(state, b.cs, g), state, b.cs, g, cnt);
            }
        }
        flush_counts(st, cnt);
        cnt[0] = cnt[1] = cnt[2] = cnt[3] = 0;
    }
}

// The end of the disk driver's step: combination, sink decay, recovery
// (launch_kitp_finish; as three kernels they took 93 us at 128 x 128 x 48).
// Excised cells combine and decay like the others and keep their primitives.
__global__ void __launch_bounds__(256)
    k_kitp_finish(double *__restrict__ s, BoxDev b,
                  const double *__restrict__ u1, int64_t ucs,
                  const double *__restrict__ k, int64_t rcs, Background bg,
                  Options o, KitpDev kd, int sinks, double r2max0,
                  double r2max1, double dt, DevStatus *st)
{
    const double r2max[2] = {r2max0, r2max1};
    unsigned long long cnt[4] = {0, 0, 0, 0};
    const int64_t n = b.ivol();
    const int64_t n_pad = (n + blockDim.x - 1) / blockDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_pad;
         t += (int64_t)gridDim.x * blockDim.x)
    {
        if (t < n)
        {
            int i, j, l;
            interior_cell(b, t, i, j, l);
            const int64_t g = b.gidx(i, j, l);
            double u[5];
#pragma unroll
            for (int c = 0; c < 5; ++c)
                u[c] = 0.5 * (s[c * b.cs + g] + u1[c * ucs + g] +
                              dt * k[c * rcs + t]);
            double x, y, z;
            cell_xyz(o, i, j, l, x, y, z);
            if (sinks && u[0] > 0.0)
            {
                const double rate = kitp_sink(kd, r2max, x, y, z);
                if (rate != 0.0)
                {
                    const double decay = exp(-rate * dt);
#pragma unroll
                    for (int c = 0; c < 5; ++c)
                        u[c] *= decay;
                }
            }
            Cons c;
            c.D = u[0];
            c.S[0] = u[1];
            c.S[1] = u[2];
            c.S[2] = u[3];
            c.tau = u[4];
            if (excised(o, i, j, l))
                store_cons(s, b.cs, g, c);
            else
            {
                Geo geo;
                background_metric<false, 1>(bg, x, y, z, geo, nullptr);
                recover_cell(o, geo, nullptr, c, s, b.cs, g, cnt);
            }
        }
        flush_counts(st, cnt);
        cnt[0] = cnt[1] = cnt[2] = cnt[3] = 0;
    }
}

// Characteristic-speed CFL contribution of one cell, sum_d max|lambda|/dx_d
// (compute_max_inverse_dt_from_fixed_background, :398-409) for floored
// primitives that are not atmosphere.
template <typename T>
__device__ __forceinline__ double cell_inverse_dt(const Options &o,
                                                  const PrimT<T> &fp,
                                                  const GeoT<T> &g,
                                                  const double inv[3])
{
    double cell = 0.0;
    if (!is_atmo(o, fp, 1.0 + 1.0e-12))
    {
#pragma unroll
        for (int d = 0; d < 3; ++d)
        {
            T lo, hi;
            char_speeds(o, fp, g, d, lo, hi);
            cell += double(max_(abs_(lo), abs_(hi))) * inv[d];
        }
    }
    return cell;
}

// The CFL speed of a cell from its FP64 con2prim result: floors, the
// atmosphere test and the characteristic speeds in FP64 for both paths
// (the mixed path's metric widened), so that the step size does not hinge
// on whether a near-floor cell rounds to the floor in FP32.
template <typename T>
__device__ __forceinline__ double cfl_speed(const Options &o, const Prim &pr,
                                            const GeoT<T> &g,
                                            const double inv[3])
{
    Geo gd;
#pragma unroll
    for (int q = 0; q < 6; ++q)
    {
        gd.gLL[q] = double(g.gLL[q]);
        gd.gUU[q] = double(g.gUU[q]);
    }
    gd.lapse = double(g.lapse);
#pragma unroll
    for (int q = 0; q < 3; ++q)
        gd.shift[q] = double(g.shift[q]);
    Prim fp = pr;
    floors(o, fp, gd.gLL);
    return cell_inverse_dt(o, fp, gd, inv);
}

__device__ __forceinline__ void flush_max_to(unsigned long long *bits,
                                             double v)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
        v = fmax(v, __shfl_down_sync(0xffffffffu, v, off));
    if (lane_id() == 0 && v > 0.0)
        atomicMax(bits, (unsigned long long)__double_as_longlong(v));
}

__device__ __forceinline__ void flush_max(DevStatus *st, double v)
{
    flush_max_to(&st->maxinv_bits, v);
}

// One stage of an integrator fused with the post-update recovery
// (update_conserved / recover_primitives_and_apply_atmosphere,
// FixedBGFArrayBoxFiniteVolume.hpp:60-110, 522-533) and, optionally, with
// the per-cell work of the next RHS evaluation and of the next CFL speed,
// which both start from con2prim of the state this stage writes:
//   * prep: the next RHS's con2prim (unfloored, :33-58) into the primitive
//     cache and its sources (:255-298, :616-675) into the source scratch;
//   * cfl : the next compute_max_inverse_dt (:364-412) as a device max.
// For a cell whose conserved variables were reset, the next con2prim runs
// on the reset state, as the reference's next call would.
// Modes: 0 RK4 stage `stage` (new): stages 0..2 out = U^n + c dt k with
// acc = k1 (+ 2 k2 + 2 k3), stage 3 out = U^n + dt/6 (acc + k4);
// 1 Euler update out = U^n + dt k (advance_ssprk2 stage, :578);
// 2 SSPRK2 combine out = (U^n + U^1 + dt k)/2 (FArrayBoxFiniteVolume.hpp:
// 942-969).  The stage input k, the primitive cache and the sources are of
// type T; U, the accumulator and con2prim are FP64.  The mixed path starts
// con2prim from the primitive cache's pressure of the same cell.
// What a stage reads of one cell: U^n, the stage input k, a second vector v
// (the accumulator after RK4's first stage, U^1 in mode 2) and the mixed
// path's starting pressure.
template <typename T> struct StageIn
{
    double u[5], v[5];
    T k[5], p;
};

static_assert(kD == 0 && kS1 == 1 && kTau == 4,
              "the conserved components come first, in the RHS's order");

// The ensemble's loads of an RK4 stage.
template <typename T>
__device__ __forceinline__ void
stage_load(StageIn<T> &in, const double *un, int64_t ucs,
           const T *__restrict__ kv, const double *__restrict__ acc,
           const T *__restrict__ prim_in, const BoxDev &b, int stage,
           int64_t g, int64_t t)
{
#pragma unroll
    for (int c = 0; c < 5; ++c)
    {
        in.u[c] = rd<true>(&un[c * ucs + g]);
        in.k[c] = rd<true>(&kv[c * b.rcs + t]);
        if (stage > 0)
            in.v[c] = rd<true>(&acc[c * b.rcs + t]);
    }
    if (sizeof(T) != sizeof(double))
        in.p = prim_in ? rd<true>(&prim_in[1 * b.pcs + g]) : T(0);
}

template <int MODE, typename T, bool CG = false, int BGK = -1>
__device__ __forceinline__ void
stage_item(const StageIn<T> &in, const double *un, int64_t ucs, double *out,
           int64_t ocs, double *__restrict__ acc, T *__restrict__ prim,
           T *__restrict__ src, const BoxDev &b, const Background &bg,
           const Options &o, int stage, double dt, bool prep, bool store_p,
           bool cfl, const double inv[3], DevStatus *st, int64_t t, int i,
           int j, int k, int64_t g, unsigned long long cnt[4],
           double &cell_inv)
{
    const double cst = (stage == 2) ? dt : 0.5 * dt;
    const double dt6 = dt / 6.0;
    const bool mixed = sizeof(T) != sizeof(double);
    if (excised(o, i, j, k))
    {
        if (out != un)
            for (int c = 0; c < kStateComps; ++c)
                out[c * ocs + g] = rd<CG>(&un[c * ucs + g]);
        if (prep)
        {
            store_pv(prim, b.pcs, g, load_prim<CG>(un, ucs, g));
            store_src(src, b.rcs, t, zero_cons<T>());
        }
    }
    else
    {
        double u[5];
#pragma unroll
        for (int c = 0; c < 5; ++c)
        {
            const double kk = double(in.k[c]);
            const double u0 = in.u[c];
            if (MODE == 0)
            {
                double a = (stage == 0) ? kk : in.v[c];
                if (stage == 1 || stage == 2)
                    a = a + 2.0 * kk;
                if (stage < 3)
                {
                    acc[c * b.rcs + t] = a;
                    u[c] = u0 + cst * kk;
                }
                else
                    u[c] = u0 + dt6 * (a + kk);
            }
            else if (MODE == 1)
                u[c] = u0 + dt * kk;
            else
                u[c] = 0.5 * (u0 + in.v[c] + dt * kk);
        }
        Cons c;
        c.D = u[0];
        c.S[0] = u[1];
        c.S[1] = u[2];
        c.S[2] = u[3];
        c.tau = u[4];
        double x, y, z;
        cell_xyz(o, i, j, k, x, y, z);
        if constexpr (ks64<T, BGK>)
        {
            KsCell kc;
            ks_cell(bg.M, bg.a, x, y, z, kc);
            // recovery with atmosphere (:60-110)
            Prim pr, stored;
            bool ok = ks_con2prim(o, kc, c, pr);
            bool reset = !ok;
            cnt[0] += 1;
            if (ok)
            {
                stored = pr;
                ks_floors(o, kc, stored);
                reset = primitive_differs(pr, stored);
                if (reset)
                    cnt[2] += 1;
            }
            else
            {
                cnt[1] += 1;
                stored = atmosphere(o);
            }
            if (store_p)
                store_prim(out, ocs, g, stored);
            if (reset)
            {
                cnt[3] += 1;
                double gLL[6];
                ks_gLL(kc, gLL);
                c = p2c(stored, gLL);
            }
            store_cons(out, ocs, g, c);
            if (prep || cfl)
            {
                // con2prim of the state just written (an unchanged cell's
                // is pr)
                if (reset)
                    ok = ks_con2prim(o, kc, c, pr);
                if (!ok && !prep)
                    record_error(st, 4, b.t0 + t);
                if (cfl && ok)
                {
                    Prim fp = pr;
                    ks_floors(o, kc, fp);
                    if (!is_atmo(o, fp, 1.0 + 1.0e-12))
                        cell_inv = ks_inverse_dt(o, kc, fp, inv);
                }
                if (prep)
                    ks_prep(o, bg, kc, x, y, z, ok, pr, c, prim, src, b, g, t,
                            st);
            }
            return;
        }
        GeoFullT<T> f;
        if (prep && o.use_src)
            metric_T<T, true, BGK>(bg, x, y, z, f.g, &f);
        else
            metric_T<T, false, BGK>(bg, x, y, z, f.g, nullptr);
        double gLL[6];
        gLL_double(f.g, gLL);
        const double p_guess = mixed ? double(in.p) : 0.0;
        // recovery with atmosphere (:60-110)
        Prim pr;
        const bool ok = cell_con2prim(o, c, f.g, p_guess, pr);
        bool reset = !ok;
        Prim stored;
        cnt[0] += 1;
        if (ok)
        {
            stored = pr;
            floors(o, stored, gLL);
            reset = primitive_differs(pr, stored);
            if (reset)
                cnt[2] += 1;
        }
        else
        {
            cnt[1] += 1;
            stored = atmosphere(o);
        }
        if (reset)
        {
            cnt[3] += 1;
            c = p2c(stored, gLL);
        }
        // the RK stage buffer (prep) carries conserved variables
        // only: its primitive components are never read
        if (store_p)
            store_prim(out, ocs, g, stored);
        store_cons(out, ocs, g, c);
        if (prep || cfl)
        {
            // con2prim of the state just written (unchanged cells:
            // the same solve on the same input gives pr again).  The mixed
            // path takes the primitives of a cell reset to the atmosphere
            // or to the density / pressure floors as they are: con2prim of
            // their p2c returns them to within its residual tolerance, far
            // below the FP32 rounding of the primitive cache.  The FP64
            // path re-solves, as the reference's next con2prim does.
            Prim pn = pr;
            bool okn = ok;
            if (reset)
            {
                if (mixed && (!ok || (stored.v[0] == pr.v[0] &&
                                      stored.v[1] == pr.v[1] &&
                                      stored.v[2] == pr.v[2])))
                {
                    pn = stored;
                    okn = true;
                }
                else
                    okn = cell_con2prim(o, c, f.g, stored.p, pn);
            }
            if (!okn)
            {
                record_error(st, cfl && !prep ? 4 : 2,
                             cfl && !prep ? b.t0 + t : g);
                pn.rho = pn.p = 1.0;
                pn.v[0] = pn.v[1] = pn.v[2] = 0.0;
                pn.eps = 1.0;
            }
            if (prep)
            {
                store_pv(prim, b.pcs, g, pn);
                ConsT<T> s = zero_cons<T>();
                if (okn)
                    s = cell_sources<T>(o, bg, x, y, z, pn, c, f);
                store_src(src, b.rcs, t, s);
            }
            if (cfl && okn)
                cell_inv = cfl_speed<T>(o, pn, f.g, inv);
        }
    }
}

template <int MODE, typename T, int BGK>
__global__ void __launch_bounds__(kStageThreads, kStageBlocks<T, BGK>)
    k_stage(const double *un, int64_t ucs, const double *us, int64_t tcs,
            double *out, int64_t ocs, const T *__restrict__ kv,
            double *__restrict__ acc, T *__restrict__ prim,
            T *__restrict__ src, BoxDev b, Background bg, Options o,
            int stage, double dt, int prep_flag, int cfl, double i0,
            double i1, double i2, DevStatus *st, const T *__restrict__ prim_in)
{
    // Each thread's inputs of its next cell arrive in its own shared-memory
    // slots (asynchronous copies) while it works on the current one: the
    // kernel's loads were half of its stalls.  Per launch at 256^3, FP64
    // 1.53 -> 1.20 ms and mixed 1.73 -> 1.45 (the bytes alone take 0.72 and
    // 0.58), mixed binary at 320^3 3.40 -> 3.04.
    constexpr bool mixed = sizeof(T) != sizeof(double);
    __shared__ double sd[10][kStageThreads];
    __shared__ T sk[mixed ? 6 : 5][kStageThreads];
    const int tid = threadIdx.x;
    const T *pg = prim_in ? prim_in : prim;
    const bool want_v = MODE == 2 || (MODE == 0 && stage > 0);
    auto fetch = [&](int64_t g, int64_t t) {
#pragma unroll
        for (int c = 0; c < 5; ++c)
        {
            cp_async_elem(&sd[c][tid], &un[c * ucs + g]);
            cp_async_elem(&sk[c][tid], &kv[c * b.rcs + t]);
            if (MODE == 0 && stage > 0)
                cp_async_elem(&sd[5 + c][tid], &acc[c * b.rcs + t]);
            if (MODE == 2)
                cp_async_elem(&sd[5 + c][tid], &us[c * tcs + g]);
        }
        if constexpr (mixed)
            if (pg)
                cp_async_elem(&sk[5][tid], &pg[1 * b.pcs + g]);
    };
    unsigned long long cnt[4] = {0, 0, 0, 0};
    const int64_t n = b.ivol();
    const int64_t n_pad = (n + blockDim.x - 1) / blockDim.x * blockDim.x;
    const double inv[3] = {i0, i1, i2};
    // prep_flag bit 0: the next RHS's per-cell pass; bit 1: the output
    // keeps its primitives even so (the last RK4 stage of a multi-step call)
    const bool prep = (prep_flag & 1) && prim != nullptr;
    const bool store_p = !prep || (prep_flag & 2);
    const int64_t step = (int64_t)gridDim.x * blockDim.x;
    int64_t t = blockIdx.x * (int64_t)blockDim.x + tid;
    int i, j, k;
    int64_t g = 0;
    if (t < n)
    {
        interior_cell(b, t, i, j, k);
        g = b.gidx(i, j, k);
        fetch(g, t);
    }
    for (; t < n_pad; t += step)
    {
        double cell_inv = 0.0;
        if (t < n)
        {
            const int ci = i, cj = j, ck = k;
            const int64_t cg = g;
            StageIn<T> in;
            cp_async_wait_all();
#pragma unroll
            for (int c = 0; c < 5; ++c)
            {
                in.u[c] = sd[c][tid];
                in.k[c] = sk[c][tid];
                in.v[c] = want_v ? sd[5 + c][tid] : 0.0;
            }
            if constexpr (mixed)
                in.p = pg ? sk[5][tid] : T(0);
            if (t + step < n)
            {
                interior_cell(b, t + step, i, j, k);
                g = b.gidx(i, j, k);
                fetch(g, t + step);
            }
            stage_item<MODE, T, false, BGK>(
                in, un, ucs, out, ocs, acc, prim, src, b, bg, o, stage, dt,
                prep, store_p, cfl != 0, inv, st, t, ci, cj, ck, cg, cnt,
                cell_inv);
        }
        flush_counts(st, cnt);
        cnt[0] = cnt[1] = cnt[2] = cnt[3] = 0;
        if (cfl)
            flush_max(st, cell_inv);
    }
}

// compute_max_inverse_dt_from_fixed_background (:364-412): per cell
// con2prim + floors, skip atmosphere, sum_d max|lambda| / dx_d; block max by
// warp shuffles, one atomicMax per warp on the bit pattern.
// One cell of the CFL speed in the metric and arithmetic of type T (the
// FP64 path, or the mixed path as the fused stage computes it).
template <typename T, bool CG = false, int BGK = -1>
__device__ __forceinline__ double cfl_item(const double *__restrict__ state,
                                           const BoxDev &b,
                                           const Background &bg,
                                           const Options &o,
                                           const double inv[3], DevStatus *st,
                                           int64_t t)
{
    double cell = 0.0;
    int i, j, k;
    interior_cell(b, t, i, j, k);
    if (!excised(o, i, j, k))
    {
        double x, y, z;
        cell_xyz(o, i, j, k, x, y, z);
        if constexpr (ks64<T, BGK>)
        {
            KsCell kc;
            ks_cell(bg.M, bg.a, x, y, z, kc);
            Prim pr;
            if (!ks_con2prim(o, kc,
                             load_cons<CG>(state, b.cs, b.gidx(i, j, k)), pr))
                record_error(st, 4, b.t0 + t);
            else
            {
                ks_floors(o, kc, pr);
                if (!is_atmo(o, pr, 1.0 + 1.0e-12))
                    cell = ks_inverse_dt(o, kc, pr, inv);
            }
            return cell;
        }
        // (the mixed path keeps the run-time background: its results stay as
        // they are)
        GeoT<T> geo;
        metric_T<T, false, sizeof(T) == sizeof(double) ? BGK : -1>(
            bg, x, y, z, geo, nullptr);
        double gUU[6];
#pragma unroll
        for (int q = 0; q < 6; ++q)
            gUU[q] = double(geo.gUU[q]);
        Prim pr;
        if (!cold_con2prim<T>(
                o, load_cons<CG>(state, b.cs, b.gidx(i, j, k)), gUU, pr))
            record_error(st, 4, b.t0 + t);
        else
            cell = cfl_speed<T>(o, pr, geo, inv);
    }
    return cell;
}

template <typename T, int BGK>
__global__ void __launch_bounds__(256)
    k_max_inv_dt(const double *__restrict__ state, BoxDev b, Background bg,
                 Options o, double i0, double i1, double i2, DevStatus *st)
{
    const int64_t n = b.ivol();
    const int64_t n_pad = (n + blockDim.x - 1) / blockDim.x * blockDim.x;
    const double inv[3] = {i0, i1, i2};
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_pad;
         t += (int64_t)gridDim.x * blockDim.x)
    {
        double cell = 0.0;
        if (t < n)
            cell = cfl_item<T, false, BGK>(state, b, bg, o, inv, st, t);
        flush_max(st, cell);
    }
}

// Residual of the failing con2prim at one cell (error reporting only).
__global__ void k_residual_probe(const double *__restrict__ state, BoxDev b,
                                 Background bg, Options o, int i, int j,
                                 int k, double *out)
{
    double x, y, z;
    cell_xyz(o, i, j, k, x, y, z);
    Geo g;
    background_metric<false>(bg, x, y, z, g, nullptr);
    Prim pr;
    double res = 0.0;
    con2prim(o, load_cons(state, b.cs, b.gidx(i, j, k)), g.gUU, pr, nullptr,
             &res);
    *out = res;
}

// float RHS of the mixed path into the caller's FP64 array
__global__ void k_widen(const float *__restrict__ in, int64_t n, double *out,
                        int64_t ocs)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
         t < 5 * n; t += (int64_t)gridDim.x * blockDim.x)
    {
        const int64_t c = t / n, r = t - c * n;
        out[c * ocs + r] = double(in[t]);
    }
}

__global__ void k_eval_background(int64_t n, const double *__restrict__ xyz,
                                  Background bg, double *__restrict__ out)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n)
        return;
    GeoFull f;
    background_metric<true>(bg, xyz[3 * t], xyz[3 * t + 1], xyz[3 * t + 2],
                            f.g, &f);
    double *o = out + 64 * t;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
        {
            o[3 * i + j] = f.g.gLL[sym(i, j)];
            o[9 + 3 * i + j] = f.K[sym(i, j)];
        }
    double K = 0.0;
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            K += f.g.gUU[sym(i, j)] * f.K[sym(i, j)];
    o[18] = K;
    o[19] = f.g.lapse;
    for (int i = 0; i < 3; ++i)
        o[20 + i] = f.g.shift[i];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            for (int k = 0; k < 3; ++k)
                o[23 + 9 * i + 3 * j + k] = f.dgamma[k][sym(i, j)];
    for (int i = 0; i < 3; ++i)
        o[50 + i] = f.dlapse[i];
    for (int i = 0; i < 3; ++i)
        for (int j = 0; j < 3; ++j)
            o[53 + 3 * i + j] = f.dshift[i][j];
    o[62] = 0.0;
    o[63] = 0.0;
}

__global__ void k_eval_con2prim(int64_t n, const double *__restrict__ cons,
                                const double *__restrict__ gUU9, Options o,
                                double *__restrict__ prim, int *ok,
                                int *iters, double *resid)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n)
        return;
    Cons c;
    c.D = cons[5 * t];
    c.S[0] = cons[5 * t + 1];
    c.S[1] = cons[5 * t + 2];
    c.S[2] = cons[5 * t + 3];
    c.tau = cons[5 * t + 4];
    double g[6];
    for (int i = 0; i < 3; ++i)
        for (int j = i; j < 3; ++j)
            g[sym(i, j)] = gUU9[9 * t + 3 * i + j];
    Prim pr;
    pr.rho = pr.eps = pr.p = pr.v[0] = pr.v[1] = pr.v[2] = 0.0;
    int it;
    double r;
    ok[t] = con2prim(o, c, g, pr, &it, &r) ? 1 : 0;
    iters[t] = it;
    resid[t] = r;
    prim[6 * t] = pr.rho;
    prim[6 * t + 1] = pr.eps;
    prim[6 * t + 2] = pr.p;
    for (int i = 0; i < 3; ++i)
        prim[6 * t + 3 + i] = pr.v[i];
}

// The FP64 division, reciprocal, square root and reciprocal square root
// of the kernels at n points: out[4t .. 4t+3] = a/b, 1/b, sqrt(a),
// 1/sqrt(a).
__global__ void k_eval_arith(int64_t n, const double *__restrict__ a,
                             const double *__restrict__ b,
                             double *__restrict__ out)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n)
        return;
    out[4 * t] = div_(a[t], b[t]);
    out[4 * t + 1] = rcp_(b[t]);
    out[4 * t + 2] = sqrt_(a[t]);
    out[4 * t + 3] = rsqrt_(a[t]);
}

__global__ void k_eval_arith_ulp(int64_t n, const double *__restrict__ a,
                                 double *__restrict__ out)
{
    const int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (t >= n)
        return;
    out[2 * t] = rcp_ulp(a[t]);
    out[2 * t + 1] = rsqrt_ulp(a[t]);
}

// ------------------------------------------------------------- ensemble

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

// Grid-wide barrier of the persistent ensemble launch (every block is
// resident: the launch is cooperative and sized by the occupancy query).
// Thread 0 of each block arrives on a counter; the last arrival resets it
// and advances the generation the others wait on.  Each wait is bounded by
// bar_timeout_ns: a block whose wait runs out sets ctl->error (recording
// the phase) and every block leaves the kernel.  False on error.
__device__ bool ens_barrier(const EnsLaunch &a, int phase)
{
    EnsControl *c = a.ctl;
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0)
    {
        volatile unsigned int *gen = &c->bar_gen;
        volatile int *err = &c->error;
        const unsigned int g = *gen;
        __threadfence();
        const unsigned int arrived = atomicAdd(&c->bar_count, 1u) + 1u;
        if (arrived == a.nblocks + a.bar_extra)
        {
            atomicExch(&c->bar_count, 0u);
            __threadfence();
            atomicAdd(&c->bar_gen, 1u);
        }
        else
        {
            const unsigned long long t0 = global_ns();
            while (*gen == g && *err == 0)
            {
                if (global_ns() - t0 > a.bar_timeout_ns)
                {
                    if (atomicCAS(&c->error, 0, 1) == 0)
                        c->error_phase = phase;
                    break;
                }
                __nanosleep(128);
            }
        }
        __threadfence();
    }
    __syncthreads();
    return *(volatile int *)&a.ctl->error == 0;
}

// Next work item of phase `phase` for this block.
__device__ __forceinline__ int64_t ens_next(EnsControl *c, int phase,
                                            int64_t *sh)
{
    __syncthreads();
    if (threadIdx.x == 0 && threadIdx.y == 0)
        *sh = (int64_t)atomicAdd(&c->ctr[phase % 3], 1ull);
    __syncthreads();
    return *sh;
}

// Member owning item `it` of a prefix-sum table off[0..nm].
__device__ __forceinline__ int ens_find(const int64_t *off, int nm,
                                        int64_t it)
{
    int lo = 0, hi = nm;
    while (hi - lo > 1)
    {
        const int mid = (lo + hi) >> 1;
        if (__ldg(&off[mid]) <= it)
            lo = mid;
        else
            hi = mid;
    }
    return lo;
}

// dt of a member's step from the CFL speed of the step's input state, as
// the host driver computes it (cfl / max(speed, 1e-14), capped by max_dt).
__device__ __forceinline__ double ens_dt(const EnsMember &m,
                                         unsigned long long step)
{
    const double mi =
        __longlong_as_double((long long)__ldcg(&m.mi_bits[step & 1ull]));
    double dt = m.cfl / fmax(mi, 1.0e-14);
    if (m.max_dt > 0.0)
        dt = fmin(dt, m.max_dt);
    return dt;
}

// Members are Kerr-Schild boxes (the C entry point checks it), so the phases
// carry that metric's code only (24 mixed members: 21.0 -> 20.6 ms).
constexpr int kEnsBgk = 0;

template <typename T>
__device__ __forceinline__ const FaceOpt<T> &
member_face_opt(const EnsMember &m)
{
    if constexpr (sizeof(T) == sizeof(double))
        return m.fo64;
    else
        return m.fo32;
}

// The persistent ensemble kernel: `steps` RK4 steps of every member.
// Phase 0: the CFL speed (when need_cfl), interior con2prim + sources and
// the ghost fill of every state.  Each stage: ghost fill of the stage input
// (not before the first stage of the launch), face pass into k, stage
// combination with post-stage recovery, the next RHS's con2prim + sources
// and (last stage) the next CFL speed; per member one bookkeeping item sums
// the accretion partials and advances the member time.  The arithmetic of
// every item is that of the single-box kernels.
template <typename T>
__global__ void __launch_bounds__(kEnsItemCells, kMinBlocks<T>)
    k_ensemble(EnsLaunch a)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    // raw storage: the member record is copied in word by word below
    __shared__ __align__(16) unsigned char ms_raw[sizeof(EnsMember)];
    EnsMember &ms = *reinterpret_cast<EnsMember *>(ms_raw);
    __shared__ int64_t item_sh;
    const int tid = threadIdx.y * kTB + threadIdx.x;
    EnsControl *ctl = a.ctl;
    const bool lead = blockIdx.x == 0 && tid == 0;
    const unsigned long long step0 = __ldcg(&ctl->steps_done);
    const bool need_cfl = __ldcg(&ctl->need_cfl) != 0;
    const int64_t ncell = __ldg(&a.off_cell[a.nm]);
    const int64_t nghost = __ldg(&a.off_ghost[a.nm]);
    const int64_t ntile = __ldg(&a.off_tile[a.nm]);
    int cur = -1;
    int ph = 0;
    auto load = [&](int m) {
        if (m != cur)
        {
            const unsigned long long *src =
                reinterpret_cast<const unsigned long long *>(a.m + m);
            unsigned long long *dst =
                reinterpret_cast<unsigned long long *>(&ms);
            for (int w = tid; w < (int)(sizeof(EnsMember) / 8);
                 w += kEnsItemCells)
                dst[w] = __ldg(&src[w]);
            __syncthreads();
            cur = m;
        }
    };
    auto zero_next_mi = [&](unsigned long long step) {
        for (int m = 0; m < a.nm; ++m)
            a.m[m].mi_bits[(step + 1ull) & 1ull] = 0ull;
    };

    // ---- phase 0
    {
        const int64_t ncfl = need_cfl ? ncell : 0;
        if (lead)
        {
            ctl->ctr[(ph + 1) % 3] = 0ull;
            zero_next_mi(step0);
        }
        for (;;)
        {
            int64_t it = ens_next(ctl, ph, &item_sh);
            if (it >= ncfl + ncell + nghost)
                break;
            if (it < ncfl)
            {
                const int m = ens_find(a.off_cell, a.nm, it);
                load(m);
                const int64_t t =
                    (it - __ldg(&a.off_cell[m])) * kEnsItemCells + tid;
                double v = 0.0;
                if (t < ms.b.ivol())
                    v = cfl_item<T, true, kEnsBgk>(ms.state, ms.b, ms.bg, ms.o, ms.inv,
                                          ms.st, t);
                flush_max_to(&ms.mi_bits[step0 & 1ull], v);
            }
            else if (it < ncfl + ncell)
            {
                it -= ncfl;
                const int m = ens_find(a.off_cell, a.nm, it);
                load(m);
                const int64_t t =
                    (it - __ldg(&a.off_cell[m])) * kEnsItemCells + tid;
                if (t < ms.b.ivol())
                    cells_item<T, true, kEnsBgk>(ms.state, static_cast<T *>(ms.prim),
                                        static_cast<T *>(ms.src), ms.b, ms.bg,
                                        ms.o, ms.st, t);
            }
            else
            {
                it -= ncfl + ncell;
                const int m = ens_find(a.off_ghost, a.nm, it);
                load(m);
                const int64_t t =
                    (it - __ldg(&a.off_ghost[m])) * kEnsItemCells + tid;
                if (t < ms.nshell)
                    ghost_item<T, true>(ms.state, static_cast<T *>(ms.prim),
                                        ms.b, ms.bg, ms.o, ms.st, t);
            }
        }
        if (!ens_barrier(a, ph++))
            return;
    }

    for (int n = 0; n < a.steps; ++n)
    {
        const unsigned long long step = step0 + (unsigned long long)n;
        for (int s = 0; s < 4; ++s)
        {
            // ---- ghost fill of the stage input
            if (n > 0 || s > 0)
            {
                if (lead)
                {
                    ctl->ctr[(ph + 1) % 3] = 0ull;
                    if (s == 0)
                        zero_next_mi(step);
                }
                for (;;)
                {
                    const int64_t it = ens_next(ctl, ph, &item_sh);
                    if (it >= nghost)
                        break;
                    const int m = ens_find(a.off_ghost, a.nm, it);
                    load(m);
                    const int64_t t =
                        (it - __ldg(&a.off_ghost[m])) * kEnsItemCells + tid;
                    if (t < ms.nshell)
                        ghost_item<T, true>(s == 0 ? ms.state : ms.stage,
                                            static_cast<T *>(ms.prim),
                                            s == 0 ? ms.b : ms.sb, ms.bg,
                                            ms.o, ms.st, t);
                }
                if (!ens_barrier(a, ph++))
                    return;
            }
            // ---- face pass
            if (lead)
                ctl->ctr[(ph + 1) % 3] = 0ull;
            for (;;)
            {
                const int64_t it = ens_next(ctl, ph, &item_sh);
                if (it >= ntile)
                    break;
                const int m = ens_find(a.off_tile, a.nm, it);
                load(m);
                const int64_t local = it - __ldg(&a.off_tile[m]);
                const int bx = (int)(local % ms.tiles[0]);
                const int64_t r = local / ms.tiles[0];
                const int by = (int)(r % ms.tiles[1]);
                const int bz = (int)(r / ms.tiles[1]);
                const FaceOpt<T> &fo = member_face_opt<T>(ms);
                if (ms.has_mdot)
                    faces_tile<T, true, true, kEnsBgk>(
                        static_cast<const T *>(ms.prim),
                        static_cast<const T *>(ms.src), static_cast<T *>(ms.k),
                        ms.b, ms.bg, ms.o, fo, ms.inv[0], ms.inv[1],
                        ms.inv[2], a.zchunk, bx, by, bz, smem_raw, ms.mdot_part, local);
                else
                    faces_tile<T, false, true, kEnsBgk>(
                        static_cast<const T *>(ms.prim),
                        static_cast<const T *>(ms.src), static_cast<T *>(ms.k),
                        ms.b, ms.bg, ms.o, fo, ms.inv[0], ms.inv[1],
                        ms.inv[2], a.zchunk, bx, by, bz, smem_raw, nullptr, local);
            }
            if (!ens_barrier(a, ph++))
                return;
            // ---- stage combination (+ bookkeeping items)
            if (lead)
                ctl->ctr[(ph + 1) % 3] = 0ull;
            for (;;)
            {
                const int64_t it = ens_next(ctl, ph, &item_sh);
                if (it >= ncell + a.nm)
                    break;
                if (it < ncell)
                {
                    const int m = ens_find(a.off_cell, a.nm, it);
                    load(m);
                    const int64_t t =
                        (it - __ldg(&a.off_cell[m])) * kEnsItemCells + tid;
                    const double dt = ens_dt(ms, step);
                    unsigned long long cnt[4] = {0ull, 0ull, 0ull, 0ull};
                    double ci = 0.0;
                    if (t < ms.b.ivol())
                    {
                        int ic, jc, kc;
                        interior_cell(ms.b, t, ic, jc, kc);
                        const int64_t g = ms.b.gidx(ic, jc, kc);
                        StageIn<T> in;
                        stage_load(in, ms.state, ms.b.cs,
                                   static_cast<const T *>(ms.k), ms.acc,
                                   static_cast<const T *>(ms.prim), ms.b, s,
                                   g, t);
                        stage_item<0, T, true, kEnsBgk>(
                            in, ms.state, ms.b.cs, s < 3 ? ms.stage : ms.state,
                            s < 3 ? ms.sb.cs : ms.b.cs, ms.acc,
                            static_cast<T *>(ms.prim),
                            static_cast<T *>(ms.src), ms.b, ms.bg, ms.o, s,
                            dt, true, s == 3, s == 3, ms.inv, ms.st, t, ic,
                            jc, kc, g, cnt, ci);
                    }
                    flush_counts(ms.st, cnt);
                    if (s == 3)
                        flush_max_to(&ms.mi_bits[(step + 1ull) & 1ull], ci);
                }
                else
                {
                    const int m = (int)(it - ncell);
                    load(m);
                    const double dt = ens_dt(ms, step);
                    if (ms.has_mdot)
                    {
                        // the single-box k_mdot_sum, 256 threads
                        const int64_t np = (int64_t)ms.tiles[0] *
                                           ms.tiles[1] * ms.tiles[2];
                        double v = 0.0;
                        for (int64_t q = tid; q < np; q += kEnsItemCells)
                            v += __ldcg(&ms.mdot_part[q]);
                        double *w = reinterpret_cast<double *>(smem_raw);
                        block_partial(v, w, w + 8, tid, kEnsItemCells, 0);
                        if (tid == 0)
                        {
                            const double wgt =
                                (dt / 6.0) * ((s == 1 || s == 2) ? 2.0 : 1.0);
                            ms.mdot_acc[0] = w[8];
                            ms.mdot_acc[1] += wgt * w[8];
                        }
                    }
                    if (s == 3 && tid == 0)
                        *ms.time += dt;
                }
            }
            if (!ens_barrier(a, ph++))
                return;
        }
    }
    if (lead)
    {
        ctl->steps_done = step0 + (unsigned long long)a.steps;
        ctl->need_cfl = 0;
    }
}

int grid_for(int64_t n, int threads)
{
    int64_t blocks = (n + threads - 1) / threads;
    const int64_t cap = 148 * 32; // grid-stride beyond ~32 waves
    if (blocks > cap)
        blocks = cap;
    return (int)(blocks < 1 ? 1 : blocks);
}

template <typename T> size_t faces_smem()
{
    return sizeof(T) *
           (3 * 5 * kPW * kPW + kGeoFields * kGW * kGW +
            2 * 5 * kTC * (kTC + 1) + 5 * kTB * kTB);
}

// ---------------------------------------------- CCZ4-stored geometry
// LevelDataFiniteVolumeOperator (Source/Matter/GRHD/FArrayBoxFiniteVolume.hpp:
// 1215-1364): the same Valencia operator with the geometry of every cell
// read from GRChombo's CCZ4 variables of the state (chi, h_ij, A_ij, K,
// lapse, shift; components 0..24, the GRHD ones from 25) and the metric
// derivatives of the sources as finite differences.  FP64 only.

constexpr int kCzChi = 0, kCzH = 1, kCzK = 7, kCzA = 8, kCzLapse = 18,
              kCzShift = 19;

// load_ccz4_geometry (:168-192): gamma = h / chi, gamma^-1 = chi h^-1 (the
// symmetric cofactor inverse of GRChombo's TensorAlgebra), K_ij = A_ij /
// chi + gamma_ij K / 3.
__device__ __forceinline__ void ccz4_geo(const double *__restrict__ s,
                                         int64_t cs, int64_t g, Geo &geo,
                                         double *K)
{
    const double chi = s[kCzChi * cs + g];
    double h[6], hu[6];
#pragma unroll
    for (int q = 0; q < 6; ++q)
        h[q] = s[(kCzH + q) * cs + g];
    const double det = h[0] * h[3] * h[5] + 2 * h[1] * h[2] * h[4] -
                       h[0] * h[4] * h[4] - h[3] * h[2] * h[2] -
                       h[5] * h[1] * h[1];
    hu[0] = (h[3] * h[5] - h[4] * h[4]) / det;
    hu[1] = (h[2] * h[4] - h[1] * h[5]) / det;
    hu[2] = (h[1] * h[4] - h[2] * h[3]) / det;
    hu[3] = (h[0] * h[5] - h[2] * h[2]) / det;
    hu[4] = (h[1] * h[2] - h[0] * h[4]) / det;
    hu[5] = (h[0] * h[3] - h[1] * h[1]) / det;
#pragma unroll
    for (int q = 0; q < 6; ++q)
    {
        geo.gLL[q] = h[q] / chi;
        geo.gUU[q] = chi * hu[q];
    }
    if (K)
    {
        const double trK = s[kCzK * cs + g];
#pragma unroll
        for (int q = 0; q < 6; ++q)
            K[q] = s[(kCzA + q) * cs + g] / chi + geo.gLL[q] * trK / 3.0;
    }
    geo.lapse = s[kCzLapse * cs + g];
#pragma unroll
    for (int d = 0; d < 3; ++d)
        geo.shift[d] = s[(kCzShift + d) * cs + g];
}

__device__ __forceinline__ double log_sqrt_det6(const double *g)
{
    const double det = g[0] * g[3] * g[5] + 2 * g[1] * g[2] * g[4] -
                       g[0] * g[4] * g[4] - g[3] * g[2] * g[2] -
                       g[5] * g[1] * g[1];
    return (det <= 0.0 || !isfinite(det)) ? 0.0 : 0.5 * log(det);
}

// The geometry cache: gLL[6] gUU[6] lapse shift[3] ln sqrt(det gamma) per
// ghosted cell (the sources difference the last along each direction).
__device__ __forceinline__ void geo_put(double *gc, int64_t n, int64_t g,
                                        const Geo &v)
{
#pragma unroll
    for (int q = 0; q < 6; ++q)
    {
        gc[q * n + g] = v.gLL[q];
        gc[(6 + q) * n + g] = v.gUU[q];
    }
    gc[12 * n + g] = v.lapse;
#pragma unroll
    for (int d = 0; d < 3; ++d)
        gc[(13 + d) * n + g] = v.shift[d];
    gc[16 * n + g] = log_sqrt_det6(v.gLL);
}

__device__ __forceinline__ Geo geo_get(const double *__restrict__ gc,
                                       int64_t n, int64_t g)
{
    Geo v;
#pragma unroll
    for (int q = 0; q < 6; ++q)
    {
        v.gLL[q] = gc[q * n + g];
        v.gUU[q] = gc[(6 + q) * n + g];
    }
    v.lapse = gc[12 * n + g];
#pragma unroll
    for (int d = 0; d < 3; ++d)
        v.shift[d] = gc[(13 + d) * n + g];
    return v;
}

// fill_conserved_outflow_boundaries (:484-519) and
// fill_ccz4_geometry_outflow_boundaries (:430-473) over the shell of the
// box: a physical ghost copies the conserved variables q and (with a metric
// m) chi, h_ij, lapse, shift of its source cell (the box's end in each
// direction it lies outside in).  With qp, every shell cell also takes its
// stored primitives from there (a stage state's ghosts hold the state's).
__global__ void __launch_bounds__(256)
    k_ccz4_fill(double *__restrict__ m, int64_t mcs, double *__restrict__ q,
                int64_t qcs, const double *__restrict__ qp, int64_t pcs,
                BoxDev b, int64_t nshell)
{
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
         t < nshell; t += (int64_t)gridDim.x * blockDim.x)
    {
        int iv[3];
        shell_cell(b, t, iv[0], iv[1], iv[2]);
        const int64_t g = b.gidx(iv[0], iv[1], iv[2]);
        if (qp)
            for (int c = kRho; c < kStateComps; ++c)
                q[c * qcs + g] = qp[c * pcs + g];
        int src[3] = {iv[0], iv[1], iv[2]};
        bool ghost = false;
#pragma unroll
        for (int d = 0; d < 3; ++d)
        {
            if (iv[d] < b.dlo[d])
            {
                ghost = true;
                src[d] = b.lo[d];
            }
            else if (iv[d] > b.dhi[d])
            {
                ghost = true;
                src[d] = b.hi[d];
            }
        }
        if (!ghost)
            continue;
        const int64_t sg = b.gidx(src[0], src[1], src[2]);
        for (int c = 0; c < 5; ++c)
            q[c * qcs + g] = q[c * qcs + sg];
        if (!m)
            continue;
        for (int c = 0; c < 7; ++c) // chi, h
            m[c * mcs + g] = m[c * mcs + sg];
        for (int c = kCzLapse; c < kCzLapse + 4; ++c) // lapse, shift
            m[c * mcs + g] = m[c * mcs + sg];
    }
}

// recover_primitives_from_ccz4_geometry over the ghosted box (:681-702):
// the primitive cache (rho, p, v) and, unless it holds this metric already
// (fresh = 0), the geometry cache of every cell.
__global__ void __launch_bounds__(256)
    k_ccz4_cells(const double *__restrict__ m, int64_t mcs,
                 const double *__restrict__ q, int64_t qcs, BoxDev b,
                 Options o, double *__restrict__ prim,
                 double *__restrict__ gc, int fresh, DevStatus *st)
{
    const int64_t n = b.gvol();
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n;
         t += (int64_t)gridDim.x * blockDim.x)
    {
        Geo geo;
        if (fresh)
        {
            ccz4_geo(m, mcs, t, geo, nullptr);
            geo_put(gc, n, t, geo);
        }
        else
        {
#pragma unroll
            for (int c = 0; c < 6; ++c)
                geo.gUU[c] = gc[(6 + c) * n + t];
        }
        Prim pr;
        if (!con2prim(o, load_cons(q, qcs, t), geo.gUU, pr, nullptr, nullptr))
        {
            record_error(st, 2, t);
            pr.rho = pr.p = 1.0;
            pr.v[0] = pr.v[1] = pr.v[2] = 0.0;
        }
        store_pv(prim, n, t, pr);
    }
}

// The static-metric sources of an interior cell with finite-difference
// derivatives (add_static_metric_sources_to_conserved_rhs, :367-427;
// one-sided where a neighbour's stored primitives are metric-source
// atmosphere, make_metric_source_derivative_stencil, :283-322).
__global__ void __launch_bounds__(256, 3)
    k_ccz4_src(const double *__restrict__ m, int64_t mcs,
               const double *__restrict__ q, int64_t qcs, BoxDev b, Options o,
               const double *__restrict__ prim, const double *__restrict__ gc,
               double *__restrict__ src, double inv0, double inv1,
               double inv2)
{
    const int64_t n = b.gvol();
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
         t < b.ivol(); t += (int64_t)gridDim.x * blockDim.x)
    {
        int i, j, k;
        interior_cell(b, t, i, j, k);
        const int64_t g = b.gidx(i, j, k);
        const double inv[3] = {inv0, inv1, inv2};
        const int64_t step[3] = {1, (int64_t)b.gn[0],
                                 (int64_t)b.gn[0] * b.gn[1]};
        Cons s = zero_cons<double>();
        const Geo ge = geo_get(gc, n, g);
        const PV pv = load_pv_global<double>(prim, n, g);
        Prim pr;
        pr.rho = pv.q[0];
        pr.p = pv.q[1];
        pr.v[0] = pv.q[2];
        pr.v[1] = pv.q[3];
        pr.v[2] = pv.q[4];
        floors(o, pr, ge.gLL);
        if (o.use_src && !is_atmo(o, pr, o.src_atmo_factor))
        {
            // compute_static_metric_source_terms (static_sources), one
            // direction's derivatives at a time
            const Cons c = load_cons(q, qcs, g);
            const double W = rsqrt_(1.0 - vsq(pr.v, ge.gLL));
            const double h = 1.0 + pr.eps + div_(pr.p, pr.rho);
            const double rhw = pr.rho * h * W * W;
            double T[6], mU[3];
#pragma unroll
            for (int e = 0; e < 3; ++e)
#pragma unroll
                for (int f = e; f < 3; ++f)
                    T[sym(e, f)] = rhw * pr.v[e] * pr.v[f] +
                                   pr.p * ge.gUU[sym(e, f)];
            raise(ge.gUU, c.S, mU);
            const double E = c.D + c.tau;
            {
                const double ichi = 1.0 / m[kCzChi * mcs + g];
                const double tr3 = m[kCzK * mcs + g] / 3.0;
                double sk = 0.0;
#pragma unroll
                for (int e = 0; e < 3; ++e)
#pragma unroll
                    for (int f = e; f < 3; ++f)
                    {
                        const int a = sym(e, f);
                        const double K =
                            m[(kCzA + a) * mcs + g] * ichi + ge.gLL[a] * tr3;
                        sk += (e == f ? 1.0 : 2.0) * T[a] * K;
                    }
                s.tau = ge.lapse * sk;
            }
#pragma unroll
            for (int d = 0; d < 3; ++d)
            {
                const int64_t lo_i = g - step[d], hi_i = g + step[d];
                Prim pl, pu;
                pl.rho = q[kRho * qcs + lo_i];
                pl.p = q[kPress * qcs + lo_i];
                pu.rho = q[kRho * qcs + hi_i];
                pu.p = q[kPress * qcs + hi_i];
                const bool la = !is_atmo(o, pl, o.src_atmo_factor);
                const bool ua = !is_atmo(o, pu, o.src_atmo_factor);
                // no fluid neighbour: zero derivatives
                const int64_t lc = la ? lo_i : g, uc = ua ? hi_i : g;
                const double coef = la && ua ? 0.5 * inv[d]
                                    : la || ua ? inv[d]
                                               : 0.0;
                const auto diff = [&](int field) {
                    return coef *
                           (gc[field * n + uc] - gc[field * n + lc]);
                };
                const double dlapse = diff(12), dlns = diff(16);
                double ms = -E * dlapse, sg = 0.0;
#pragma unroll
                for (int e = 0; e < 3; ++e)
#pragma unroll
                    for (int f = e; f < 3; ++f)
                        sg += (e == f ? 1.0 : 2.0) * T[sym(e, f)] *
                              diff(sym(e, f));
                ms += 0.5 * ge.lapse * sg;
#pragma unroll
                for (int e = 0; e < 3; ++e)
                    ms += c.S[e] * diff(13 + e);
                const Cons F = phys_flux(pr, c, d, ge.lapse, ge.shift);
                s.S[d] += ms;
                s.D -= F.D * dlns;
                s.tau -= F.tau * dlns + mU[d] * dlapse;
#pragma unroll
                for (int e = 0; e < 3; ++e)
                    s.S[e] -= F.S[e] * dlns;
            }
        }
        store_src(src, b.rcs, t, s);
    }
}

// The flux differences and sources of the RHS
// (compute_directional_flux_rhs_from_ccz4_geometry, :784-833): the face pass
// with its geometry from the cache.  One thread per cell evaluating the
// cell's six faces (each face twice, as the reference does) took 254 us at
// 100 x 90 x 70; this and k_ccz4_src take 190.
__global__ void __launch_bounds__(kTB *kTB, 2)
    k_ccz4_faces(const double *__restrict__ prim,
                 const double *__restrict__ src, double *__restrict__ rhs,
                 BoxDev b, Options o, FaceOpt<double> fo, double idx0,
                 double idx1, double idx2, int zchunk,
                 const double *__restrict__ gc)
{
    extern __shared__ __align__(16) unsigned char smem_raw[];
    faces_tile<double, false, false, kGridMetric>(
        prim, src, rhs, b, Background(), o, fo, idx0, idx1, idx2, zchunk,
        blockIdx.x, blockIdx.y, blockIdx.z, smem_raw, nullptr, 0, gc);
}

// One stage of an integrator fused with the recovery: out = in + dt rhs, or
// with u1 the SSPRK2 combination out = (in + u1 + dt rhs) / 2
// (add_scaled_conserved_rhs, :927-940, combine_ssprk2_conserved_state,
// :942-969), then recover_primitives_and_apply_atmosphere_from_ccz4_geometry
// (:713-761) on the cached geometry or (gc null) that of the metric m.  GRHD
// components, FP64.
__global__ void __launch_bounds__(256)
    k_ccz4_advance(double *out, int64_t ocs, const double *in, int64_t ics,
                   const double *u1, int64_t ucs,
                   const double *__restrict__ rhs, int64_t rcs, BoxDev b,
                   Options o, const double *__restrict__ gc,
                   const double *__restrict__ m, int64_t mcs, double dt,
                   DevStatus *st)
{
    unsigned long long cnt[4] = {0, 0, 0, 0};
    const int64_t n = b.ivol();
    const int64_t n_pad = (n + blockDim.x - 1) / blockDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_pad;
         t += (int64_t)gridDim.x * blockDim.x)
    {
        if (t < n)
        {
            int i, j, k;
            interior_cell(b, t, i, j, k);
            const int64_t g = b.gidx(i, j, k);
            double u[5];
#pragma unroll
            for (int c = 0; c < 5; ++c)
            {
                const double x = rhs[c * rcs + t], u0 = in[c * ics + g];
                u[c] = u1 ? 0.5 * (u0 + u1[c * ucs + g] + dt * x)
                          : u0 + dt * x;
            }
            Cons c;
            c.D = u[0];
            c.S[0] = u[1];
            c.S[1] = u[2];
            c.S[2] = u[3];
            c.tau = u[4];
            Geo geo;
            if (gc)
                geo = geo_get(gc, b.gvol(), g);
            else
                ccz4_geo(m, mcs, g, geo, nullptr);
            recover_cell(o, geo, nullptr, c, out, ocs, g, cnt);
        }
        flush_counts(st, cnt);
        cnt[0] = cnt[1] = cnt[2] = cnt[3] = 0;
    }
}

// recover_primitives_and_apply_atmosphere_from_ccz4_geometry (:713-761).
__global__ void __launch_bounds__(256)
    k_ccz4_recover(double *__restrict__ s, BoxDev b, Options o, DevStatus *st)
{
    double *q = s + kCcz4GrhdOffset * b.cs;
    unsigned long long cnt[4] = {0, 0, 0, 0};
    const int64_t n = b.ivol();
    const int64_t n_pad = (n + blockDim.x - 1) / blockDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_pad;
         t += (int64_t)gridDim.x * blockDim.x)
    {
        if (t < n)
        {
            int i, j, k;
            interior_cell(b, t, i, j, k);
            const int64_t g = b.gidx(i, j, k);
            Geo geo;
            ccz4_geo(s, b.cs, g, geo, nullptr);
            recover_cell(o, geo, nullptr, load_cons(q, b.cs, g), q, b.cs, g,
                         cnt);
        }
        flush_counts(st, cnt);
        cnt[0] = cnt[1] = cnt[2] = cnt[3] = 0;
    }
}

// compute_max_inverse_dt_from_ccz4_geometry (:1139-1183).
__global__ void __launch_bounds__(256)
    k_ccz4_max_inv_dt(const double *__restrict__ s, BoxDev b, Options o,
                      double inv0, double inv1, double inv2, DevStatus *st)
{
    const double *q = s + kCcz4GrhdOffset * b.cs;
    const int64_t n = b.ivol();
    const int64_t n_pad = (n + blockDim.x - 1) / blockDim.x * blockDim.x;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; t < n_pad;
         t += (int64_t)gridDim.x * blockDim.x)
    {
        double cell = 0.0;
        if (t < n)
        {
            int i, j, k;
            interior_cell(b, t, i, j, k);
            const int64_t g = b.gidx(i, j, k);
            Geo geo;
            ccz4_geo(s, b.cs, g, geo, nullptr);
            Prim pr;
            if (!con2prim(o, load_cons(q, b.cs, g), geo.gUU, pr, nullptr,
                          nullptr))
                record_error(st, 4, t); // GRHD_WHERE_CFL
            else
            {
                floors(o, pr, geo.gLL);
                if (!is_atmo(o, pr, 1.0 + 1.0e-12))
                {
                    const double inv[3] = {inv0, inv1, inv2};
                    for (int d = 0; d < 3; ++d)
                    {
                        double lo, hi;
                        char_speeds(o, pr, geo, d, lo, hi);
                        cell += fmax(fabs(lo), fabs(hi)) * inv[d];
                    }
                }
            }
        }
        flush_max(st, cell);
    }
}

// add_scaled_conserved_rhs (:927-940) on the GRHD components: s += dt rhs.
__global__ void __launch_bounds__(256)
    k_ccz4_update(double *__restrict__ s, const double *__restrict__ rhs,
                  int64_t rcs, BoxDev b, double dt)
{
    double *q = s + kCcz4GrhdOffset * b.cs;
    for (int64_t t = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
         t < b.ivol(); t += (int64_t)gridDim.x * blockDim.x)
    {
        int i, j, k;
        interior_cell(b, t, i, j, k);
        const int64_t g = b.gidx(i, j, k);
        for (int c = 0; c < 5; ++c)
            q[c * b.cs + g] += dt * rhs[c * rcs + t];
    }
}

__global__ void k_ccz4_probe(const double *__restrict__ s, BoxDev b,
                             Options o, int i, int j, int k, double *out)
{
    const int64_t g = b.gidx(i, j, k);
    Geo geo;
    ccz4_geo(s, b.cs, g, geo, nullptr);
    Prim pr;
    double res = 0.0;
    con2prim(o, load_cons(s + kCcz4GrhdOffset * b.cs, b.cs, g), geo.gUU, pr,
             nullptr, &res);
    *out = res;
}

} // namespace

cudaError_t configure_kernels()
{
    cudaError_t e = cudaSuccess;
    const cudaFuncAttribute attr = cudaFuncAttributeMaxDynamicSharedMemorySize;
    const int d = (int)faces_smem<double>(), f = (int)faces_smem<float>();
    const void *fp64[] = {(const void *)k_faces<double, false, 0>,
                          (const void *)k_faces<double, true, 0>,
                          (const void *)k_faces<double, false, 1>,
                          (const void *)k_faces<double, true, 1>};
    const void *fp32[] = {(const void *)k_faces<float, false, 0>,
                          (const void *)k_faces<float, true, 0>,
                          (const void *)k_faces<float, false, 1>,
                          (const void *)k_faces<float, true, 1>};
    for (const void *k : fp64)
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, attr, d);
    for (const void *k : fp32)
        if (e == cudaSuccess)
            e = cudaFuncSetAttribute(k, attr, f);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_ccz4_faces, attr, d);
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_ensemble<double>, attr,
                                 (int)faces_smem<double>());
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_ensemble<float>, attr,
                                 (int)faces_smem<float>());
    return e;
}

template <typename T> size_t ensemble_smem() { return faces_smem<T>(); }

template <typename T> cudaError_t ensemble_occupancy(int *blocks_per_sm)
{
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(
        blocks_per_sm, k_ensemble<T>, kEnsItemCells, faces_smem<T>());
}

template <typename T>
cudaError_t launch_ensemble(const EnsLaunch &a, int grid, cudaStream_t s)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned)grid);
    cfg.blockDim = dim3(kTB, kTB);
    cfg.dynamicSmemBytes = faces_smem<T>();
    cfg.stream = s;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeCooperative;
    attr[0].val.cooperative = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, k_ensemble<T>, a);
}

template size_t ensemble_smem<double>();
template size_t ensemble_smem<float>();
template cudaError_t ensemble_occupancy<double>(int *);
template cudaError_t ensemble_occupancy<float>(int *);
template cudaError_t launch_ensemble<double>(const EnsLaunch &, int,
                                             cudaStream_t);
template cudaError_t launch_ensemble<float>(const EnsLaunch &, int,
                                            cudaStream_t);

namespace
{
// SMs of the current device (a B200's 148 where it cannot be asked)
int num_sms()
{
    static std::atomic<int> cache[64];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
        return 148;
    int have = cache[dev].load(std::memory_order_relaxed);
    if (have > 0)
        return have;
    if (cudaDeviceGetAttribute(&have, cudaDevAttrMultiProcessorCount, dev) !=
        cudaSuccess)
    {
        (void)cudaGetLastError();
        return 148;
    }
    cache[dev].store(have, std::memory_order_relaxed);
    return have;
}

// resident face-kernel blocks of the current device (SMs x blocks per SM
// at the kernel's registers and shared memory), per precision
int face_slots(bool fp32)
{
    static std::atomic<int> cache[64][2];
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess || dev < 0 || dev >= 64)
        return (fp32 ? 3 : 2) * num_sms();
    std::atomic<int> &c = cache[dev][fp32 ? 1 : 0];
    const int have = c.load(std::memory_order_relaxed);
    if (have > 0)
        return have;
    const int sms = num_sms();
    int per = 0;
    const cudaError_t e =
        fp32 ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                   &per, k_faces<float, false, 0>, kTB * kTB,
                   faces_smem<float>())
             : cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                   &per, k_faces<double, false, 0>, kTB * kTB,
                   faces_smem<double>());
    if (e != cudaSuccess || per < 1)
    {
        (void)cudaGetLastError();
        per = fp32 ? 3 : 2;
    }
    c.store(sms * per, std::memory_order_relaxed);
    return sms * per;
}
} // namespace

// Makespan (in plane-times) of nf blocks of df planes followed by np of dp
// planes on `slots` resident blocks, each block started on the slot that
// frees first in launch order (the last z row of a launch holds the short
// blocks): whole waves of full blocks, then the short blocks on the slots
// left free in the last full wave and on the others as they free.
int64_t face_makespan(int64_t nf, int64_t df, int64_t np, int64_t dp,
                      int64_t slots)
{
    const int64_t t1 = (nf / slots) * df, rem = nf % slots;
    int64_t ta = t1, na = slots - rem;           // free at t1
    int64_t tb = t1 + (rem ? df : 0), nb = rem;  // free after the last full
    int64_t end = rem ? tb : t1;
    for (int64_t left = np; left > 0;)
    {
        if (nb == 0 || ta <= tb)
        {
            left -= std::min(left, na);
            ta += dp;
            end = std::max(end, ta);
        }
        else
        {
            left -= std::min(left, nb);
            tb += dp;
            end = std::max(end, tb);
        }
    }
    return end;
}

// The march length of a launch: of the candidates, the one whose blocks,
// list-scheduled in launch order on the resident slots, finish first (ties
// keep the longer march).  A block costs its planes and, once, the two
// lead-in planes (one z face and two planes' geometry): 0.7 of a plane.
// Marches down to one plane spread a small box over the idle SMs: a plane
// takes one block about 9 us, whatever the box (a 16^3 right-hand side:
// 102 us with at least four planes a block, 58 with one; 45x38x31: 84, 70).
int face_march(int nx, int ny, int nz, int64_t slots)
{
    const int64_t tiles =
        (int64_t)((nx + kTC - 1) / kTC) * ((ny + kTC - 1) / kTC);
    const int cand[] = {48, 40, 32, 24, 20, 16, 13, 12, 11, 10,
                        9,  8,  7,  6,  5,  4,  3,  2,  1};
    int best = 1;
    int64_t best_cost = -1;
    for (int z : cand)
    {
        const int r = nz % z;
        const int64_t cost = face_makespan(tiles * (nz / z), 10 * z + 7,
                                           r ? tiles : 0, 10 * r + 7, slots);
        if (best_cost < 0 || cost < best_cost)
        {
            best = z;
            best_cost = cost;
        }
    }
    return best;
}

int face_zchunk(const BoxDev &b, int zchunk, bool fp32)
{
    return zchunk > 0 ? zchunk
                      : face_march(b.in[0], b.in[1], b.in[2],
                                   face_slots(fp32));
}

int face_zchunk_model(int nx, int ny, int nz, int64_t slots)
{
    const int64_t tiles = (int64_t)((nx + 14) / 15) * ((ny + 14) / 15);
    const int cand[5] = {32, 16, 8, 6, 4};
    int best = cand[0];
    int64_t best_cost = -1;
    for (int z : cand)
    {
        // nz / z full blocks per column of tiles, then one of nz % z
        // planes; every block also marches two lead-in planes
        const int r = nz % z;
        const int64_t cost = face_makespan(tiles * (nz / z), z + 2,
                                           r ? tiles : 0, r + 2, slots);
        if (best_cost < 0 || cost < best_cost)
        {
            best = z;
            best_cost = cost;
        }
    }
    return best;
}

int64_t face_kernel_blocks(const BoxDev &b, int zchunk, bool fp32)
{
    zchunk = face_zchunk(b, zchunk, fp32);
    return (int64_t)((b.in[0] + kTC - 1) / kTC) * ((b.in[1] + kTC - 1) / kTC) *
           ((b.in[2] + zchunk - 1) / zchunk);
}

template <typename T>
void launch_fill_ghosts(double *state, T *prim, const BoxDev &b,
                        const Background &bg, const Options &o, DevStatus *st,
                        cudaStream_t s)
{
    const int64_t nshell = b.gvol() - b.ivol();
    if (nshell <= 0)
        return;
    k_fill_ghosts<T><<<grid_for(nshell, 256), 256, 0, s>>>(state, prim, b, bg,
                                                          o, st, nshell);
}

template <typename T>
void launch_fill_ghost_planes(double *state, T *prim, const BoxDev &b,
                              const Background &bg, const Options &o,
                              DevStatus *st, int k0, int k1, cudaStream_t s)
{
    const int64_t n = plane_shell_count(b, k0, k1);
    if (n <= 0)
        return;
    k_fill_ghost_planes<T><<<grid_for(n, 256), 256, 0, s>>>(state, prim, b, bg,
                                                           o, st, k0, k1, n);
}

template <typename T>
void launch_cells(const double *state, T *prim, T *src, const BoxDev &b,
                  const Background &bg, const Options &o, DevStatus *st,
                  cudaStream_t s)
{
    // (the mixed path keeps the run-time background: its results stay as they
    // are)
    auto go = [&](auto kern) {
        kern<<<grid_for(b.ivol(), 256), 256, 0, s>>>(state, prim, src, b, bg,
                                                     o, st);
    };
    if constexpr (sizeof(T) == sizeof(float))
        go(k_cells<T, -1>);
    else
        bg.kind == 1 ? go(k_cells<T, 1>) : go(k_cells<T, 0>);
}

bool launch_prepare(double *state, double *prim, double *src, const BoxDev &b,
                    const Background &bg, const Options &o, DevStatus *st,
                    cudaStream_t s)
{
    const int64_t nshell = b.gvol() - b.ivol();
    // a box with more cells than the SMs hold at once fills them with either
    // pass alone, and the separate ones keep three blocks per SM
    if (b.ivol() + nshell > (int64_t)num_sms() * 2 * 256 * 4)
        return false;
    const int ghosts = (int)((nshell + 255) / 256);
    const int grid = ghosts + (int)((b.ivol() + 255) / 256);
    auto go = [&](auto kern) {
        kern<<<grid, 256, 0, s>>>(state, prim, src, b, bg, o, st, nshell,
                                  ghosts);
    };
    bg.kind == 1 ? go(k_prepare<1>) : go(k_prepare<0>);
    return true;
}

template <typename T>
void launch_faces(const T *prim, const T *src, T *rhs, const BoxDev &b,
                  const Background &bg, const Options &o,
                  const double inv_dx[3], int zchunk, double *mdot_part,
                  cudaStream_t s)
{
    zchunk = face_zchunk(b, zchunk, sizeof(T) == sizeof(float));
    dim3 grid((b.in[0] + kTC - 1) / kTC, (b.in[1] + kTC - 1) / kTC,
              (b.in[2] + zchunk - 1) / zchunk);
    dim3 block(kTB, kTB);
    // one instantiation per background kind: each carries only its own
    // metric code
    const bool md = o.accretion_radius > 0.0 && mdot_part;
    auto go = [&](auto kern) {
        kern<<<grid, block, faces_smem<T>(), s>>>(
            prim, src, rhs, b, bg, o, make_face_opt<T>(o), inv_dx[0],
            inv_dx[1], inv_dx[2], zchunk, md ? mdot_part : nullptr);
    };
    if (bg.kind == 1)
        md ? go(k_faces<T, true, 1>) : go(k_faces<T, false, 1>);
    else
        md ? go(k_faces<T, true, 0>) : go(k_faces<T, false, 0>);
}

void launch_mdot_sum(const double *part, int64_t n, double weight,
                     double *acc, cudaStream_t s)
{
    k_mdot_sum<<<1, 256, 0, s>>>(part, n, weight, acc);
}

void launch_update(double *dst, int64_t dcs, const double *src_state,
                   int64_t scs, const double *rhs, const BoxDev &b,
                   const Background &bg, const Options &o, double dt,
                   int recover, DevStatus *st, cudaStream_t s)
{
    k_update<<<grid_for(b.ivol(), 256), 256, 0, s>>>(
        dst, dcs, src_state, scs, rhs, b, bg, o, dt, recover, st);
}

void launch_recover(double *state, const BoxDev &b, const Background &bg,
                    const Options &o, DevStatus *st, cudaStream_t s)
{
    k_recover<<<grid_for(b.ivol(), 256), 256, 0, s>>>(state, b, bg, o, st);
}

// Blocks of a stage launch: two cells a thread where that leaves four waves
// of blocks, so that a thread's second cell arrives during its first.  More
// cells a thread lose to the spread of their costs (fluid, atmosphere,
// excised): at 256^3 FP64 1.20 ms with two, 1.38 with 14, 1.80 with one wave
// of blocks; at 64^3, two cells in 1.2 waves take 32 us against 28 with one.
template <typename T> int stage_grid(int64_t n, int kind)
{
    const int64_t blocks = (n + kStageThreads - 1) / kStageThreads;
    const int per = kind == 1 ? kStageBlocks<T, 1> : kStageBlocks<T, 0>;
    return (int)(blocks >= 8 * num_sms() * per ? (blocks + 1) / 2 : blocks);
}

template <typename T>
void launch_stage(int mode, const double *un, int64_t ucs, const double *us,
                  int64_t tcs, double *out, int64_t ocs, const T *k,
                  double *acc, T *prim, T *src, int prep, const BoxDev &b,
                  const Background &bg, const Options &o, int stage,
                  double dt, bool cfl, const double inv_dx[3], DevStatus *st,
                  cudaStream_t s, const T *prim_in)
{
    const int grid = stage_grid<T>(b.ivol(), bg.kind);
    const double i0 = inv_dx ? inv_dx[0] : 0.0, i1 = inv_dx ? inv_dx[1] : 0.0,
                 i2 = inv_dx ? inv_dx[2] : 0.0;
    const int pf = prep, cf = cfl ? 1 : 0;
    auto go = [&](auto kern) {
        kern<<<grid, kStageThreads, 0, s>>>(un, ucs, us, tcs, out, ocs, k, acc, prim, src,
                                  b, bg, o, stage, dt, pf, cf, i0, i1, i2, st,
                                  prim_in);
    };
    // one instantiation per background kind (only its own metric code)
    const bool pn = bg.kind == 1;
    if (mode == 0)
        pn ? go(k_stage<0, T, 1>) : go(k_stage<0, T, 0>);
    else if (mode == 1)
        pn ? go(k_stage<1, T, 1>) : go(k_stage<1, T, 0>);
    else
        pn ? go(k_stage<2, T, 1>) : go(k_stage<2, T, 0>);
}

void launch_max_inv_dt(const double *state, const BoxDev &b,
                       const Background &bg, const Options &o,
                       const double inv_dx[3], DevStatus *st, bool mixed,
                       cudaStream_t s)
{
    auto go = [&](auto kern) {
        kern<<<grid_for(b.ivol(), 256), 256, 0, s>>>(
            state, b, bg, o, inv_dx[0], inv_dx[1], inv_dx[2], st);
    };
    if (mixed)
        go(k_max_inv_dt<float, -1>);
    else
        bg.kind == 1 ? go(k_max_inv_dt<double, 1>)
                     : go(k_max_inv_dt<double, 0>);
}

void launch_kitp_finish(double *state, const BoxDev &b, const double *u1,
                        int64_t u1_cs, const double *k, int64_t rcs,
                        const Background &bg, const Options &o,
                        const KitpDev &kd, bool sinks, double dt,
                        DevStatus *st, cudaStream_t s)
{
    double r2max[2];
    kitp_sink_reach(kd, r2max);
    k_kitp_finish<<<grid_for(b.ivol(), 256), 256, 0, s>>>(
        state, b, u1, u1_cs, k, rcs, bg, o, kd, sinks ? 1 : 0, r2max[0],
        r2max[1], dt, st);
}

void launch_residual_probe(const double *state, const BoxDev &b,
                           const Background &bg, const Options &o, int i,
                           int j, int k, double *out, cudaStream_t s)
{
    k_residual_probe<<<1, 1, 0, s>>>(state, b, bg, o, i, j, k, out);
}

void launch_widen(const float *in, int64_t n, double *out, int64_t ocs,
                  cudaStream_t s)
{
    k_widen<<<grid_for(5 * n, 256), 256, 0, s>>>(in, n, out, ocs);
}

void launch_eval_background(int64_t n, const double *xyz,
                            const Background &bg, double *out, cudaStream_t s)
{
    if (n <= 0)
        return;
    k_eval_background<<<(int)((n + 127) / 128), 128, 0, s>>>(n, xyz, bg, out);
}

void launch_eval_con2prim(int64_t n, const double *cons, const double *gUU,
                          const Options &o, double *prim, int *ok, int *iters,
                          double *resid, cudaStream_t s)
{
    if (n <= 0)
        return;
    k_eval_con2prim<<<(int)((n + 127) / 128), 128, 0, s>>>(n, cons, gUU, o,
                                                           prim, ok, iters,
                                                           resid);
}

void launch_eval_arith(int64_t n, const double *a, const double *b,
                       double *out, cudaStream_t s)
{
    if (n <= 0)
        return;
    k_eval_arith<<<(int)((n + 255) / 256), 256, 0, s>>>(n, a, b, out);
}

void launch_eval_arith_ulp(int64_t n, const double *a, double *out,
                           cudaStream_t s)
{
    if (n > 0)
        k_eval_arith_ulp<<<(int)((n + 255) / 256), 256, 0, s>>>(n, a, out);
}

void launch_ccz4_fill(double *m, int64_t mcs, double *q, int64_t qcs,
                      const double *qp, int64_t pcs, const BoxDev &b,
                      cudaStream_t st)
{
    const int64_t nshell = b.gvol() - b.ivol();
    if (nshell > 0)
        k_ccz4_fill<<<grid_for(nshell, 256), 256, 0, st>>>(m, mcs, q, qcs, qp,
                                                           pcs, b, nshell);
}

void launch_ccz4_cells(const double *m, int64_t mcs, const double *q,
                       int64_t qcs, const BoxDev &b, const Options &o,
                       double *prim, double *gc, bool fresh, DevStatus *st,
                       cudaStream_t stream)
{
    k_ccz4_cells<<<grid_for(b.gvol(), 256), 256, 0, stream>>>(
        m, mcs, q, qcs, b, o, prim, gc, fresh ? 1 : 0, st);
}

void launch_ccz4_rhs(const double *m, int64_t mcs, const double *q,
                     int64_t qcs, const BoxDev &b, const Options &o,
                     const double *prim, const double *gc, double *src,
                     double *rhs, const double inv[3], cudaStream_t stream)
{
    k_ccz4_src<<<grid_for(b.ivol(), 256), 256, 0, stream>>>(
        m, mcs, q, qcs, b, o, prim, gc, src, inv[0], inv[1], inv[2]);
    const int zchunk = face_zchunk(b, 0, false);
    const dim3 grid((b.in[0] + kTC - 1) / kTC, (b.in[1] + kTC - 1) / kTC,
                    (b.in[2] + zchunk - 1) / zchunk);
    // this operator has no excision
    Options of = o;
    of.excision_radius = 0.0;
    k_ccz4_faces<<<grid, dim3(kTB, kTB), faces_smem<double>(), stream>>>(
        prim, src, rhs, b, of, make_face_opt<double>(o), inv[0], inv[1],
        inv[2], zchunk, gc);
}

void launch_ccz4_advance(double *out, int64_t ocs, const double *in,
                         int64_t ics, const double *u1, int64_t ucs,
                         const double *rhs, int64_t rcs, const BoxDev &b,
                         const Options &o, const double *gc, const double *m,
                         int64_t mcs, double dt, DevStatus *st,
                         cudaStream_t stream)
{
    k_ccz4_advance<<<grid_for(b.ivol(), 256), 256, 0, stream>>>(
        out, ocs, in, ics, u1, ucs, rhs, rcs, b, o, gc, m, mcs, dt, st);
}

void launch_ccz4_recover(double *s, const BoxDev &b, const Options &o,
                         DevStatus *st, cudaStream_t stream)
{
    k_ccz4_recover<<<grid_for(b.ivol(), 256), 256, 0, stream>>>(s, b, o, st);
}

void launch_ccz4_max_inv_dt(const double *s, const BoxDev &b,
                            const Options &o, const double inv[3],
                            DevStatus *st, cudaStream_t stream)
{
    k_ccz4_max_inv_dt<<<grid_for(b.ivol(), 256), 256, 0, stream>>>(
        s, b, o, inv[0], inv[1], inv[2], st);
}

void launch_ccz4_update(double *s, const double *rhs, int64_t rcs,
                        const BoxDev &b, double dt, cudaStream_t stream)
{
    k_ccz4_update<<<grid_for(b.ivol(), 256), 256, 0, stream>>>(s, rhs, rcs, b,
                                                                dt);
}

void launch_ccz4_probe(const double *s, const BoxDev &b, const Options &o,
                       int i, int j, int k, double *out, cudaStream_t stream)
{
    k_ccz4_probe<<<1, 1, 0, stream>>>(s, b, o, i, j, k, out);
}

#define GRHD_INSTANTIATE(T)                                                   \
    template void launch_fill_ghosts<T>(double *, T *, const BoxDev &,        \
                                        const Background &, const Options &,  \
                                        DevStatus *, cudaStream_t);           \
    template void launch_fill_ghost_planes<T>(                                \
        double *, T *, const BoxDev &, const Background &, const Options &,   \
        DevStatus *, int, int, cudaStream_t);                                 \
    template void launch_cells<T>(const double *, T *, T *, const BoxDev &,   \
                                  const Background &, const Options &,        \
                                  DevStatus *, cudaStream_t);                 \
    template void launch_faces<T>(const T *, const T *, T *, const BoxDev &,  \
                                  const Background &, const Options &,        \
                                  const double *, int, double *,              \
                                  cudaStream_t);                              \
    template void launch_stage<T>(int, const double *, int64_t,               \
                                  const double *, int64_t, double *, int64_t, \
                                  const T *, double *, T *, T *, int,         \
                                  const BoxDev &, const Background &,         \
                                  const Options &, int, double, bool,         \
                                  const double *, DevStatus *, cudaStream_t,  \
                                  const T *);

GRHD_INSTANTIATE(double)
GRHD_INSTANTIATE(float)

} // namespace grhd
