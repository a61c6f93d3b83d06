/*
 * GPU spacetime scalar CESE solvers: solvcon's spacetime::SolverBase march
 * (cpp/solvcon/spacetime/core.hpp:946-1036) with the LinearScalar and
 * InviscidBurgers solution-element kernels (kernel/linear_scalar.hpp:45-87,
 * kernel/inviscid_burgers.hpp:51-109), one variable, periodic boundary.
 *
 * Grid layout (core.cpp:52-99): coordinates x[0 .. 2*ncelm+4]; solution
 * element i on plane p sits at x index 2 + 2i + p, conservation element i at
 * 3 + 2i + p.  A half step on plane p computes, for each conservation element
 * ic, so0 then so1 at its top solution element (index 3 + 2ic + p) from its
 * two bottom solution elements (2 + 2ic + p and 4 + 2ic + p), which are all on
 * the other parity: the half step has no dependency between elements.  One
 * lane per conservation element runs so0, the periodic ghost copy, the CFL
 * of the top element and so1 (the order of march_half1_alpha and
 * march_half2_alpha, core.hpp:1006-1025), so a full step is two launches;
 * march_alpha replays a captured CUDA graph of 32 steps, or marches a small
 * grid in one launch of one cluster.
 */

#include "../../include/scg.h"
#include "cluster.cuh"
#include "common.hpp"
#include "divide.cuh"

#include <cfloat>
#include <memory>
#include <string>
#include <vector>

namespace
{

struct STArgs
{
    double const * x;
    double const * geo; // [G_COUNT][xsize] grid quantities per point
    double * so0;
    double * so1;
    double * cfl;
    int64_t ncelm, xsize;
    double hdt, qdt;
};

// Grid quantities of solution point xi, stored once (k_st_geo) with the very
// expressions the reference evaluates on every half step
// (SolutionElement::xctr/dxneg/dxpos/xn/xp, core.hpp:300-360; the CFL
// half-width and the conservation-element width of
// update_cfl/march_half_so0, core.hpp:962-980), so the march reads them
// instead of recomputing them and its results stay bit-identical.  The four
// divisors of a half step also get their reciprocals (rcp_fix, the bits kept in
// a double), from which div_fix forms each quotient exactly as the division
// would, on the integer pipe: with its quotients on the FP64 pipe (53
// instructions per element there, 28 without) the half step was bound by it.
// Now, above L2, it waits for DRAM first: the grid quantities, so0, so1 and cfl
// lie point after point and a half step takes every second one, so it moves 252 B
// per element for the 120 that it uses (8M elements 360 us, 5.6 TB/s, 83% of the
// measured copy rate; the FP64 pipe 74% busy).
enum
{
    G_DXNEG = 0, // x - xneg
    G_DXPOS,     // xpos - x
    G_DMNEG,     // 0.5 (x + xneg) - xctr
    G_DMPOS,     // 0.5 (x + xpos) - xctr
    G_DISP,      // x - xctr
    G_HDX,       // min(x - xneg, xpos - x)
    G_WIDTH,     // xpos - xneg (the width of the element whose top is xi)
    G_RDXNEG,    // reciprocals of the four divisors
    G_RDXPOS,
    G_RHDX,
    G_RWIDTH,
    G_CFLLIN,    // the linear solver's CFL number hdt / hdx (set with dt)
    G_COUNT
};

__device__ __forceinline__ double mu(double a, double b) { return __dmul_rn(a, b); }
// The same product by either pipe (mul_int's bits are the multiplication's).
template <bool INT>
__device__ __forceinline__ double mu(double a, double b)
{
    return INT ? scg::dev::mul_int(a, b) : __dmul_rn(a, b);
}
__device__ __forceinline__ double rcp_bits(double d)
{
    return __longlong_as_double(static_cast<long long>(scg::dev::rcp_fix(d)));
}
__device__ __forceinline__ double div_bits(double x, double d, double r)
{
    return scg::dev::div_fix(x, d, static_cast<unsigned long long>(__double_as_longlong(r)));
}

__global__ void k_st_geo(double const * x, int64_t xsize, double * geo)
{
    int64_t const xi = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (xi < 1 || xi >= xsize - 1)
    {
        return;
    }
    double const xm = x[xi - 1], x0 = x[xi], xp = x[xi + 1];
    double const xctr = (xm + xp) / 2;
    double const dn = x0 - xm;
    double const dp = xp - x0;
    geo[G_DXNEG * xsize + xi] = dn;
    geo[G_DXPOS * xsize + xi] = dp;
    geo[G_DMNEG * xsize + xi] = 0.5 * (x0 + xm) - xctr;
    geo[G_DMPOS * xsize + xi] = 0.5 * (x0 + xp) - xctr;
    geo[G_DISP * xsize + xi] = x0 - xctr;
    double const hdx = dn < dp ? dn : dp;
    double const width = xp - xm;
    geo[G_HDX * xsize + xi] = hdx;
    geo[G_WIDTH * xsize + xi] = width;
    geo[G_RDXNEG * xsize + xi] = rcp_bits(dn);
    geo[G_RDXPOS * xsize + xi] = rcp_bits(dp);
    geo[G_RHDX * xsize + xi] = rcp_bits(hdx);
    geo[G_RWIDTH * xsize + xi] = rcp_bits(width);
}

__device__ __forceinline__ double gq(STArgs const & a, int k, int64_t xi) { return a.geo[k * a.xsize + xi]; }

// The grid quantities of solution element xi.
struct SelmGrid
{
    double dxneg, dxpos, dmneg, dmpos, disp;

    __device__ __forceinline__ SelmGrid(STArgs const & a, int64_t xi)
        : dxneg(gq(a, G_DXNEG, xi))
        , dxpos(gq(a, G_DXPOS, xi))
        , dmneg(gq(a, G_DMNEG, xi))
        , dmpos(gq(a, G_DMPOS, xi))
        , disp(gq(a, G_DISP, xi))
    {
    }
};

// The parts of a solution element that the conservation elements on either
// side of it use (LinearScalarSelm / InviscidBurgersSelm, xn, xp, tp, so0p):
// ll = xp + tp (to the element on its right), ur = xn - tp (to the element on
// its left) and the value so0p at the next time level.
template <int KIND, bool INT>
struct SelmParts
{
    double ll, ur, so0p;

    __device__ __forceinline__ SelmParts(STArgs const & a, double u, double ux, SelmGrid const & x)
    {
        double const dux = mu<INT>(x.disp, ux);
        double const xn = mu(x.dxneg, u + mu(x.dmneg, ux));
        double const xp = mu(x.dxpos, u + mu(x.dmpos, ux));
        double tp;
        if constexpr (KIND == 0)
        {
            double r = u;
            r += dux;
            r -= mu<INT>(a.qdt, ux);
            tp = mu(a.hdt, r);
        }
        else
        {
            double const u2 = mu(u, u);
            double r = mu(0.5, u2);
            r += mu(mu(x.disp, u), ux);
            r -= mu(mu(a.qdt, u2), ux);
            tp = mu(a.hdt, r);
        }
        ll = xp + tp;
        ur = xn - tp;
        double q = u;
        q += dux;
        q -= mu<INT>(a.hdt, ux);
        so0p = q;
    }
};

// The linear solver's CFL number at every point, hdt / hdx: it depends on
// the grid and the time increment alone, so it is formed when either is set
// (the same quotient the half step would form) and the half steps copy it.
__global__ void k_st_cfl_tab(double * geo, int64_t xsize, double hdt)
{
    int64_t const xi = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (xi < xsize)
    {
        geo[G_CFLLIN * xsize + xi] = div_bits(hdt, geo[G_HDX * xsize + xi], geo[G_RHDX * xsize + xi]);
    }
}

// update_cfl at point xi of value u.
template <int KIND>
__device__ __forceinline__ double cfl_at(STArgs const & a, int64_t xi, double u)
{
    if constexpr (KIND == 0)
        return gq(a, G_CFLLIN, xi);
    else
        return div_bits(fabs(u) * a.hdt, gq(a, G_HDX, xi), gq(a, G_RHDX, xi));
}

template <int ALPHA, bool INT>
__device__ __forceinline__ double wgrad(double duxn, double duxp)
{
    double fan = fabs(duxn), fap = fabs(duxp);
    if constexpr (ALPHA == 2)
    {
        fan = mu<INT>(fan, fan);
        fap = mu<INT>(fap, fap);
    }
    double const den = fap + fan + DBL_MIN;
    return scg::dev::div_fix(mu<INT>(fap, duxn) + mu<INT>(fan, duxp), den, scg::dev::rcp_fix(den));
}

constexpr int WOUT = 31; // conservation elements per warp

// One half step; STAGE bits: 1 so0, 2 cfl of the top element, 4 so1,
// 8 periodic ghost copies (first half only).  Lane l of warp w derives the
// parts of the lower-left solution element of conservation element
// ic = 31 w + l - odd; lanes 0 .. 30 form the element's top from those and the
// next lane's, by shuffles: warps share nothing.
template <int KIND, int ALPHA, int STAGE, bool INT>
__global__ void __launch_bounds__(128) k_st_half(STArgs a, int odd)
{
    int const lane = static_cast<int>(threadIdx.x) & 31;
    int64_t const w = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / 32;
    int64_t const first = w * WOUT - odd;
    if (first >= a.ncelm)
    {
        return;
    }
    // Solution elements exist for ic <= ncelm (the last one is the lower-right
    // element of conservation element ncelm - 1); lanes past it repeat it.
    int64_t const ic = first + lane < a.ncelm ? first + lane : a.ncelm;
    int64_t const xi = 2 + 2 * ic + odd;
    SelmParts<KIND, INT> const sn(a, a.so0[xi], a.so1[xi], SelmGrid(a, xi));
    double const ur = __shfl_down_sync(0xffffffffu, sn.ur, 1);
    double const so0p = __shfl_down_sync(0xffffffffu, sn.so0p, 1);
    if (lane >= WOUT || ic >= a.ncelm)
    {
        return;
    }
    int64_t const xt = xi + 1;
    int64_t const last = 2 * a.ncelm + 1; // selm(ncelm - 1, odd plane)
    double utp;
    if (STAGE & 1)
    {
        utp = div_bits(sn.ll + ur, gq(a, G_WIDTH, xt), gq(a, G_RWIDTH, xt));
        a.so0[xt] = utp;
        if (STAGE & 8)
        {
            if (xt == last)
                a.so0[1] = utp;
            if (xt == 3)
                a.so0[last + 2] = utp;
        }
    }
    else
    {
        utp = a.so0[xt];
    }
    if (STAGE & 2)
    {
        a.cfl[xt] = cfl_at<KIND>(a, xt, utp);
        if (STAGE & 8)
        {
            if (xt == last)
                a.cfl[1] = cfl_at<KIND>(a, 1, utp);
            if (xt == 3)
                a.cfl[last + 2] = cfl_at<KIND>(a, last + 2, utp);
        }
    }
    if (STAGE & 4)
    {
        double const duxn = div_bits(utp - sn.so0p, gq(a, G_DXPOS, xi), gq(a, G_RDXPOS, xi));
        double const duxp = div_bits(so0p - utp, gq(a, G_DXNEG, xi + 2), gq(a, G_RDXNEG, xi + 2));
        double const g = wgrad<ALPHA, INT>(duxn, duxp);
        a.so1[xt] = g;
        if (STAGE & 8)
        {
            if (xt == last)
                a.so1[1] = g;
            if (xt == 3)
                a.so1[last + 2] = g;
        }
    }
}

// Small grids: a whole march in one launch of one cluster (cluster.cuh), thread
// t keeping the even point 2t and the odd point 2t + 1.  The first half step
// writes the odd points of threads 1 .. ncelm from the even points of t and
// t + 1, and copies the end ones to the ghosts of threads ncelm + 1 and 0; the
// second the even points of threads 1 .. ncelm + 1 from the odd points of t - 1
// and t.  A point's CFL number is overwritten by the next step's, so it is
// formed in the last step.
constexpr int ST_WARPS = 8;

template <int KIND, int ALPHA>
__global__ void __launch_bounds__(32 * ST_WARPS) k_st_cluster(STArgs a, int64_t steps)
{
    using namespace scg::cluster;
    __shared__ double slots[2][ST_WARPS][2];
    __shared__ double ghost[2][2]; // so0 and so1 of the first and of the last odd point
    int64_t const nt = a.ncelm + 2;
    int64_t const t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    int64_t const k = t < nt ? t : nt - 1; // threads past the grid repeat its last pair, and write nothing
    int64_t const e = 2 * k, o = 2 * k + 1;
    int64_t const lo = k > 0 ? e - 1 : o;
    double ue = a.so0[e], xe = a.so1[e], uo = a.so0[o], xo = a.so1[o];
    SelmGrid const ge(a, e), go(a, o);
    double const wide_o = gq(a, G_WIDTH, o), rwide_o = gq(a, G_RWIDTH, o);
    double const wide_e = gq(a, G_WIDTH, e), rwide_e = gq(a, G_RWIDTH, e);
    double const rpe = gq(a, G_RDXPOS, e);
    double const dne = gq(a, G_DXNEG, e + 2), rne = gq(a, G_RDXNEG, e + 2); // of the next even point
    double const dpo = gq(a, G_DXPOS, lo), rpo = gq(a, G_RDXPOS, lo);       // of the odd point before
    double const rno = gq(a, G_RDXNEG, o);
    bool const out1 = t >= 1 && t <= a.ncelm, out2 = t >= 1 && t < nt;
    // The other end's ghost: thread ncelm's odd point is thread 0's, thread 1's
    // is thread ncelm + 1's.
    unsigned const to_lo = slot_of(ghost[0], 0);
    unsigned const to_hi = slot_of(ghost[1], static_cast<unsigned>((nt - 1) / blockDim.x));
    cluster_sync(); // every block runs before any stores to another's slots
    for (int64_t s = 0; s < steps; ++s)
    {
        bool const end = s + 1 == steps;
        {
            SelmParts<KIND, false> const p(a, ue, xe, ge);
            double const v[2] = {p.ur, p.so0p};
            double w[2];
            hand_over<2, 1>(v, w, slots[0]);
            if (out1)
            {
                uo = div_bits(p.ll + w[0], wide_o, rwide_o);
                xo = wgrad<ALPHA, false>(div_bits(uo - p.so0p, ge.dxpos, rpe), div_bits(w[1] - uo, dne, rne));
                if (t == a.ncelm)
                {
                    slot_put(to_lo, uo);
                    slot_put(to_lo + 8u, xo);
                }
                if (t == 1)
                {
                    slot_put(to_hi, uo);
                    slot_put(to_hi + 8u, xo);
                }
            }
            cluster_sync();
            if (t == 0)
            {
                uo = ghost[0][0];
                xo = ghost[0][1];
            }
            else if (t == nt - 1)
            {
                uo = ghost[1][0];
                xo = ghost[1][1];
            }
            if (end && t < nt)
            {
                a.cfl[o] = cfl_at<KIND>(a, o, uo);
            }
        }
        {
            SelmParts<KIND, false> const p(a, uo, xo, go);
            double const v[2] = {p.ll, p.so0p};
            double w[2];
            hand_over<2, 0>(v, w, slots[1]);
            if (out2)
            {
                ue = div_bits(w[0] + p.ur, wide_e, rwide_e);
                xe = wgrad<ALPHA, false>(div_bits(ue - w[1], dpo, rpo), div_bits(p.so0p - ue, go.dxneg, rno));
                if (end)
                {
                    a.cfl[e] = cfl_at<KIND>(a, e, ue);
                }
            }
        }
    }
    if (t < nt)
    {
        if (t > 0)
        {
            a.so0[e] = ue;
            a.so1[e] = xe;
        }
        a.so0[o] = uo;
        a.so1[o] = xo;
    }
}

template <int KIND>
__global__ void k_st_cfl(STArgs a, int odd)
{
    // update_cfl (core.hpp:962-971): selm(ic, odd) for ic in [-odd, nselm).
    int64_t const ic = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x - (odd ? 1 : 0);
    if (ic <= a.ncelm)
    {
        int64_t const xi = 2 + 2 * ic + odd;
        a.cfl[xi] = cfl_at<KIND>(a, xi, a.so0[xi]);
    }
}

// treat_boundary_so0 / treat_boundary_so1 (core.hpp:982-1004).
__global__ void k_st_bnd(STArgs a, int which)
{
    double * s = which == 0 ? a.so0 : a.so1;
    int64_t const last = 2 * a.ncelm + 1;
    double const left_in = s[3];
    double const right_in = s[last];
    s[1] = right_in;
    s[last + 2] = left_in;
}

// Grids above this many elements take 7 of an element's FP64 multiplications on
// the integer pipe (k_st_half's INT, the same bits), which takes the FP64 pipes
// below what the loads allow (1M elements, linear 54.0 -> 49.3 us per half step,
// Burgers 67.9 -> 61.2; 100,000 elements 7.6 -> 7.3).
constexpr int64_t INT_ELEMENTS = 80000;

class Spacetime
{
public:
    Spacetime(int kind, double const * xcoord, int64_t ncelm_in, double dt)
        : kind(kind)
        , ncelm(ncelm_in)
    {
        if (kind != 0 && kind != 1)
        {
            throw std::invalid_argument("spacetime: kind must be 0 (linear scalar) or 1 (inviscid Burgers)");
        }
        if (ncelm < 1)
        {
            throw std::invalid_argument("spacetime: ncelm smaller than 1");
        }
        xsize = 2 * ncelm + 5;
        scg::cuda_check(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");
        x.alloc(static_cast<size_t>(xsize));
        geo.alloc(static_cast<size_t>(G_COUNT * xsize));
        so0.alloc(static_cast<size_t>(xsize));
        so1.alloc(static_cast<size_t>(xsize));
        cfl.alloc(static_cast<size_t>(xsize));
        put(x.ptr, xcoord);
        make_geo();
        std::vector<double> z(static_cast<size_t>(xsize), 0.0);
        put(so0.ptr, z.data());
        put(so1.ptr, z.data());
        put(cfl.ptr, z.data());
        set_dt(dt);
    }

    ~Spacetime()
    {
        if (graph_exec)
            cudaGraphExecDestroy(graph_exec);
        if (stream)
        {
            cudaStreamSynchronize(stream);
            cudaStreamDestroy(stream);
        }
    }

    void set_dt(double dt)
    {
        time_increment = dt;
        if (graph_exec)
        {
            cudaGraphExecDestroy(graph_exec);
            graph_exec = nullptr;
        }
        make_cfl_tab();
    }

    void make_cfl_tab()
    {
        k_st_cfl_tab<<<static_cast<unsigned>((xsize + 255) / 256), 256, 0, stream>>>(geo.ptr, xsize,
                                                                                     0.5 * time_increment);
        scg::launched(stream, "spacetime_cfl_tab");
        sync();
    }

    STArgs args()
    {
        return STArgs{x.ptr, geo.ptr, so0.ptr, so1.ptr, cfl.ptr, ncelm, xsize, 0.5 * time_increment,
                      0.25 * time_increment};
    }

    // The grid quantities, after the coordinates are set.
    void make_geo()
    {
        scg::cuda_check(cudaMemsetAsync(geo.ptr, 0, geo.bytes(), stream), "memset");
        k_st_geo<<<static_cast<unsigned>((xsize + 255) / 256), 256, 0, stream>>>(x.ptr, xsize, geo.ptr);
        scg::launched(stream, "spacetime_geo");
        make_cfl_tab();
    }

    double * field(int which)
    {
        switch (which)
        {
        case 0: return x.ptr;
        case 1: return so0.ptr;
        case 2: return so1.ptr;
        case 3: return cfl.ptr;
        default: throw std::invalid_argument("spacetime: unknown array id " + std::to_string(which));
        }
    }

    template <int STAGE>
    void half_t(int alpha, int odd)
    {
        int64_t const n = ncelm + (odd ? 1 : 0);
        // Blocks of one warp while they all are resident at once, as the 1D
        // Euler core's, beyond that blocks of four.
        int64_t const warps = (n + WOUT - 1) / WOUT;
        int const wpb = warps <= int64_t(scg::sm_count()) * 32 ? 1 : 4;
        unsigned const grid = static_cast<unsigned>((warps + wpb - 1) / wpb);
        int const threads = 32 * wpb;
        bool const big = ncelm > INT_ELEMENTS;
        auto * const kernel =
            kind == 0 ? (alpha == 1 ? (big ? k_st_half<0, 1, STAGE, true> : k_st_half<0, 1, STAGE, false>)
                                    : (big ? k_st_half<0, 2, STAGE, true> : k_st_half<0, 2, STAGE, false>))
                      : (alpha == 1 ? (big ? k_st_half<1, 1, STAGE, true> : k_st_half<1, 1, STAGE, false>)
                                    : (big ? k_st_half<1, 2, STAGE, true> : k_st_half<1, 2, STAGE, false>));
        kernel<<<grid, threads, 0, stream>>>(args(), odd);
        scg::launched(stream, "spacetime_half");
    }

    void step(int alpha)
    {
        half_t<1 | 2 | 4 | 8>(alpha, 0);
        half_t<1 | 2 | 4>(alpha, 1);
    }

    void op(int which, int odd, int alpha)
    {
        switch (which)
        {
        case 0: // update_cfl
        case 5: // setup_march == update_cfl(false)
        {
            int const o = which == 5 ? 0 : odd;
            int64_t const n = ncelm + 1 + o;
            if (kind == 0)
                k_st_cfl<0><<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(args(), o);
            else
                k_st_cfl<1><<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(args(), o);
            scg::launched(stream, "spacetime_cfl");
            break;
        }
        case 1: half_t<1>(alpha, odd); break;
        case 2: half_t<4>(alpha, odd); break;
        case 3:
        case 4:
            k_st_bnd<<<1, 1, 0, stream>>>(args(), which - 3);
            scg::launched(stream, "spacetime_bnd");
            break;
        case 6: // march_half1_alpha
            half_t<1 | 2 | 4 | 8>(alpha, 0);
            break;
        case 7: // march_half2_alpha
            half_t<1 | 2 | 4>(alpha, 1);
            break;
        default: throw std::invalid_argument("spacetime: unknown operation " + std::to_string(which));
        }
        sync();
    }

    void march(int alpha, int64_t steps)
    {
        if (alpha != 1 && alpha != 2)
        {
            throw std::invalid_argument("spacetime: alpha must be 1 or 2");
        }
        if (kind == 0 ? (alpha == 1 ? cluster_march<0, 1>(steps) : cluster_march<0, 2>(steps))
                      : (alpha == 1 ? cluster_march<1, 1>(steps) : cluster_march<1, 2>(steps)))
        {
            return;
        }
        int64_t const chunks = steps / GRAPH_STEPS;
        if (chunks > 0)
        {
            if (!graph_exec || graph_alpha != alpha)
            {
                capture(alpha);
            }
            for (int64_t c = 0; c < chunks; ++c)
            {
                scg::cuda_check(cudaGraphLaunch(graph_exec, stream), "cudaGraphLaunch");
                scg::g_launches.fetch_add(2 * GRAPH_STEPS, std::memory_order_relaxed);
            }
        }
        for (int64_t s = chunks * GRAPH_STEPS; s < steps; ++s)
        {
            step(alpha);
        }
    }

    // A small grid's steps in launches of one cluster.
    template <int KIND, int ALPHA>
    bool cluster_march(int64_t steps)
    {
        using namespace scg::cluster;
        int blocks, warps;
        if (!cluster_shape<k_st_cluster<KIND, ALPHA>, ST_WARPS>(ncelm + 2, blocks, warps))
        {
            return false;
        }
        for (int64_t s = 0; s < steps; s += CLUSTER_STEPS)
        {
            launch_cluster(k_st_cluster<KIND, ALPHA>, blocks, 32 * warps, stream, args(),
                           std::min(CLUSTER_STEPS, steps - s));
            scg::launched(stream, "spacetime_cluster");
        }
        return true;
    }

    void capture(int alpha)
    {
        sync();
        if (graph_exec)
        {
            cudaGraphExecDestroy(graph_exec);
            graph_exec = nullptr;
        }
        cudaGraph_t g = nullptr;
        scg::cuda_check(cudaStreamBeginCapture(stream, cudaStreamCaptureModeThreadLocal), "BeginCapture");
        int64_t const before = scg::g_launches.load();
        for (int s = 0; s < GRAPH_STEPS; ++s)
        {
            step(alpha);
        }
        scg::g_launches.store(before);
        scg::cuda_check(cudaStreamEndCapture(stream, &g), "EndCapture");
        scg::cuda_check(cudaGraphInstantiate(&graph_exec, g, 0), "GraphInstantiate");
        cudaGraphDestroy(g);
        graph_alpha = alpha;
    }

    void get(int which, double * host)
    {
        scg::cuda_check(cudaMemcpyAsync(host, field(which), sizeof(double) * static_cast<size_t>(xsize),
                                        cudaMemcpyDeviceToHost, stream),
                        "D2H");
        sync();
    }
    void set(int which, double const * host)
    {
        put(field(which), host);
        if (which == 0)
        {
            make_geo();
        }
    }

    void sync() { scg::cuda_check(cudaStreamSynchronize(stream), "cudaStreamSynchronize"); }

    int kind;
    int64_t ncelm, xsize;
    double time_increment = 0.0;
    cudaStream_t stream = nullptr;

private:
    static constexpr int GRAPH_STEPS = 32;

    void put(double * dst, double const * src)
    {
        scg::cuda_check(cudaMemcpyAsync(dst, src, sizeof(double) * static_cast<size_t>(xsize),
                                        cudaMemcpyHostToDevice, stream),
                        "H2D");
        sync();
    }

    scg::DevBuf<double> x, geo, so0, so1, cfl;
    cudaGraphExec_t graph_exec = nullptr;
    int graph_alpha = 0;
};

// One quotient per thread, by div_fix from the tabulated reciprocal and by
// the division itself, and the FP64 march's reciprocal of d.
__global__ void k_divide_check(double const * x, double const * d, double * q, double * qdiv, double * rcp,
                               int64_t n)
{
    int64_t const i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n)
    {
        q[i] = scg::dev::div_fix(x[i], d[i], scg::dev::rcp_fix(d[i]));
        qdiv[i] = x[i] / d[i];
        rcp[i] = scg::dev::recip(d[i]);
    }
}

// The FP64 march's reciprocal root and root of x.
__global__ void k_root_check(double const * x, double * r, double * s, int64_t n)
{
    int64_t const i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n)
    {
        r[i] = scg::dev::rsq(x[i]);
        s[i] = scg::dev::sqr_t(x[i]);
    }
}

// The integer pipe's product of a and b.
__global__ void k_product_check(double const * a, double const * b, double * p, int64_t n)
{
    int64_t const i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n)
    {
        p[i] = scg::dev::mul_int(a[i], b[i]);
    }
}

} // namespace

struct scg_st
{
    std::unique_ptr<Spacetime> c;
};

extern "C"
{

int scg_st_create(int kind, const double * xcoord, int64_t ncelm, double time_increment, scg_st ** out)
{
    return scg::guarded([&] {
        auto h = std::make_unique<scg_st>();
        h->c = std::make_unique<Spacetime>(kind, xcoord, ncelm, time_increment);
        *out = h.release();
    });
}

int scg_st_destroy(scg_st * h)
{
    return scg::guarded([&] { delete h; });
}

int scg_st_set_time_increment(scg_st * h, double time_increment)
{
    return scg::guarded([&] { h->c->set_dt(time_increment); });
}

int scg_st_get(scg_st * h, int which, double * host, int64_t count)
{
    return scg::guarded([&] {
        if (count != h->c->xsize)
            throw std::invalid_argument("spacetime: host buffer size mismatch");
        h->c->get(which, host);
    });
}

int scg_st_set(scg_st * h, int which, const double * host, int64_t count)
{
    return scg::guarded([&] {
        if (count != h->c->xsize)
            throw std::invalid_argument("spacetime: host buffer size mismatch");
        h->c->set(which, host);
    });
}

int scg_st_op(scg_st * h, int op, int odd_plane, int alpha)
{
    return scg::guarded([&] { h->c->op(op, odd_plane, alpha); });
}

int scg_st_march(scg_st * h, int alpha, int64_t steps)
{
    return scg::guarded([&] {
        if (steps < 0)
            throw std::invalid_argument("spacetime: steps must be >= 0");
        h->c->march(alpha, steps);
    });
}

int scg_st_sync(scg_st * h)
{
    return scg::guarded([&] { h->c->sync(); });
}

int scg_st_stream(const scg_st * h, void ** out)
{
    return scg::guarded([&] { *out = h->c->stream; });
}

int scg_divide_check(const double * x, const double * d, double * q, double * qdiv, double * rcp, int64_t n)
{
    return scg::guarded([&] {
        if (n < 0 || (n > 0 && (!x || !d || !q || !qdiv || !rcp)))
        {
            throw std::invalid_argument("scg_divide_check: null buffer or negative count");
        }
        if (n == 0)
        {
            return;
        }
        size_t const sz = static_cast<size_t>(n);
        scg::DevBuf<double> dx(sz), dd(sz), dq(sz), dqd(sz), dr(sz);
        scg::cuda_check(cudaMemcpy(dx.ptr, x, dx.bytes(), cudaMemcpyHostToDevice), "H2D");
        scg::cuda_check(cudaMemcpy(dd.ptr, d, dd.bytes(), cudaMemcpyHostToDevice), "H2D");
        k_divide_check<<<static_cast<unsigned>((n + 255) / 256), 256>>>(dx.ptr, dd.ptr, dq.ptr, dqd.ptr, dr.ptr, n);
        scg::launched(nullptr, "divide_check");
        scg::cuda_check(cudaMemcpy(q, dq.ptr, dq.bytes(), cudaMemcpyDeviceToHost), "D2H");
        scg::cuda_check(cudaMemcpy(qdiv, dqd.ptr, dqd.bytes(), cudaMemcpyDeviceToHost), "D2H");
        scg::cuda_check(cudaMemcpy(rcp, dr.ptr, dr.bytes(), cudaMemcpyDeviceToHost), "D2H");
    });
}

int scg_root_check(const double * x, double * r, double * s, int64_t n)
{
    return scg::guarded([&] {
        if (n < 0 || (n > 0 && (!x || !r || !s)))
        {
            throw std::invalid_argument("scg_root_check: null buffer or negative count");
        }
        if (n == 0)
        {
            return;
        }
        size_t const sz = static_cast<size_t>(n);
        scg::DevBuf<double> dx(sz), dr(sz), ds(sz);
        scg::cuda_check(cudaMemcpy(dx.ptr, x, dx.bytes(), cudaMemcpyHostToDevice), "H2D");
        k_root_check<<<static_cast<unsigned>((n + 255) / 256), 256>>>(dx.ptr, dr.ptr, ds.ptr, n);
        scg::launched(nullptr, "root_check");
        scg::cuda_check(cudaMemcpy(r, dr.ptr, dr.bytes(), cudaMemcpyDeviceToHost), "D2H");
        scg::cuda_check(cudaMemcpy(s, ds.ptr, ds.bytes(), cudaMemcpyDeviceToHost), "D2H");
    });
}

int scg_product_check(const double * a, const double * b, double * p, int64_t n)
{
    return scg::guarded([&] {
        if (n < 0 || (n > 0 && (!a || !b || !p)))
        {
            throw std::invalid_argument("scg_product_check: null buffer or negative count");
        }
        if (n == 0)
        {
            return;
        }
        size_t const sz = static_cast<size_t>(n);
        scg::DevBuf<double> da(sz), db(sz), dp(sz);
        scg::cuda_check(cudaMemcpy(da.ptr, a, da.bytes(), cudaMemcpyHostToDevice), "H2D");
        scg::cuda_check(cudaMemcpy(db.ptr, b, db.bytes(), cudaMemcpyHostToDevice), "H2D");
        k_product_check<<<static_cast<unsigned>((n + 255) / 256), 256>>>(da.ptr, db.ptr, dp.ptr, n);
        scg::launched(nullptr, "product_check");
        scg::cuda_check(cudaMemcpy(p, dp.ptr, dp.bytes(), cudaMemcpyDeviceToHost), "D2H");
    });
}

} // extern "C"
