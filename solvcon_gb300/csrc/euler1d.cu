/*
 * GPU 1D Euler CESE core: solvcon's onedim::Euler1DCore
 * (cpp/solvcon/onedim/Euler1DCore.hpp:39-349, Euler1DCore.cpp:22-172) on the
 * device.
 *
 * A half step updates the points of one parity from the solution elements
 * ("kernels") at the points of the other parity.  The reference sweeps the
 * points serially with a two-kernel sliding window so that each kernel is
 * derived once; here each lane derives the kernel at one point and shares
 * the quantities its left neighbour needs (flux_lr, up, x - xneg) by warp
 * shuffles.  The first half step also performs the copy-out boundary treatment
 * (it touches only points the half step neither reads nor writes), and
 * update_cfl (which reads only the kernel points) is folded into the same
 * kernel, so a full march_alpha step is two launches.  The fine-grained methods
 * run the same kernel with less asked of it.  The FP32 core (Euler1D32,
 * not in the reference) keeps its state split by parity in a layout of its
 * own and updates four outputs per thread; see the comment above it.
 */

#include "../../include/scg.h"
#include "cluster.cuh"
#include "common.hpp"
#include "divide.cuh"

#include <algorithm>
#include <cmath>
#include <cstring>
#include <memory>
#include <string>
#include <vector>

namespace
{

using namespace scg::cluster;

// Euler1DKernel::tiny (Euler1DCore.hpp:182) in FP64; it underflows in FP32,
// where the same expressions use the smallest floor that keeps them finite.
template <typename R>
struct Tiny1D;
template <>
struct Tiny1D<double>
{
    static constexpr double V = 1.e-100;
};
template <>
struct Tiny1D<float>
{
    static constexpr float V = 1.e-30f;
};

// The FP64 core's device state: the reference's [n][3] tables, and what depends
// on the grid (and the time increment) alone, formed once per coordinate write.
struct E1DArgs
{
    double const * gamma;
    double * so0; // [n][3]
    double * so1; // [n][3]
    double * cfl;
    int64_t n;
    double hdt, qdt;
    double const * invdx; // 1 / (x[i + 1] - x[i])
    double const * invd2; // 1 / (x[i + 2] - x[i])
    double const * cflr;  // dt / 2 / min(x[i] - x[i - 1], x[i + 1] - x[i])
    // The solution element's offsets, [5][n]: x - xctr, xpos - x,
    // (x + xpos) / 2 - xctr, x - xneg, (x + xneg) / 2 - xctr with
    // xctr = (xpos + xneg) / 2 (Euler1DCore.hpp:210-244).
    double const * seo;
};

// The grid's tables of E1DArgs.
__global__ void k_inv_spacing(double const * coord, int64_t n, double hdt, double * invdx, double * invd2,
                              double * cflr, double * seo)
{
    int64_t const i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < n)
    {
        invdx[i] = i + 1 < n ? 1.0 / (coord[i + 1] - coord[i]) : 0.0;
        invd2[i] = i + 2 < n ? 1.0 / (coord[i + 2] - coord[i]) : 0.0;
        double o[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
        double q = 0.0;
        if (i > 0 && i + 1 < n)
        {
            double const x = coord[i];
            double const xneg = coord[i - 1];
            double const xpos = coord[i + 1];
            double const xctr = __dmul_rn(__dadd_rn(xpos, xneg), 0.5);
            o[0] = __dsub_rn(x, xctr);
            o[1] = __dsub_rn(xpos, x);
            o[2] = __dsub_rn(__dmul_rn(0.5, __dadd_rn(x, xpos)), xctr);
            o[3] = __dsub_rn(x, xneg);
            o[4] = __dsub_rn(__dmul_rn(0.5, __dadd_rn(x, xneg)), xctr);
            q = hdt / (o[1] < o[3] ? o[1] : o[3]);
        }
        cflr[i] = q;
        for (int k = 0; k < 5; ++k)
        {
            seo[k * n + i] = o[k];
        }
    }
}

// The FP64 half step is bound by the FP64 pipe (one instruction per SM every 19
// cycles, see divide.cuh), so its routines take the fewest FP64 instructions: the
// Jacobian products are directional derivatives of the flux from the primitive
// variables, the divisions and the root are integer arithmetic (divide.cuh),
// and what the grid fixes is read from tables: 98 FP64 instructions per output
// point, 82 with half_warp's INT (196 with the Jacobian formed, FP64 Newton
// reciprocals and a library root).  Every operation is written as the instruction it is, so the
// fine-grained methods and the fused march round alike, as the reference
// requires.
__device__ __forceinline__ double fm(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double mu(double a, double b) { return __dmul_rn(a, b); }
// The same product by either pipe (mul_int's bits are the multiplication's).
template <bool INT>
__device__ __forceinline__ double mu(double a, double b)
{
    return INT ? scg::dev::mul_int(a, b) : __dmul_rn(a, b);
}
__device__ __forceinline__ double ad(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double sb(double a, double b) { return __dsub_rn(a, b); }

// The primitive variables of one point, r = 1 / (rho + tiny); for any density
// above ~1e-50 the reference's denominators rho^k + tiny equal rho^k.
struct P1D
{
    double u[3], r, v, p, ga;

    __device__ __forceinline__ P1D(double const * so0, double gamma)
    {
        for (int i = 0; i < 3; ++i)
        {
            u[i] = so0[i];
        }
        ga = gamma;
        r = scg::dev::recip(ad(u[0], Tiny1D<double>::V));
        v = mu(u[1], r);
        p = mu(sb(ga, 1.0), fm(-0.5, mu(u[1], v), u[2]));
    }

    // update_cfl at the point (Euler1DCore.cpp:70-94), times the table's
    // dt / 2 / dx.  The reference's sqrt(m * m) / rho is |v| with the density's
    // sign.
    __device__ __forceinline__ double cfl(double cflr) const
    {
        // (p + |p|) / 2: zero for a negative p, NaN for -infinity and NaN.
        unsigned const hp = static_cast<unsigned>(__double2hiint(p));
        double const pr =
            hp >= 0x80000000u ? (hp >= 0xfff00000u ? __longlong_as_double(0x7ff8000000000000ll) : 0.0) : p;
        double const speed =
            __hiloint2double((__double2hiint(v) & 0x7fffffff) | (__double2hiint(r) & static_cast<int>(0x80000000u)),
                             __double2loint(v));
        return mu(ad(scg::dev::sqr_t(mu(mu(ga, pr), r)), speed), cflr);
    }
};

// The offsets of the solution element at point ic (E1DArgs::seo).
struct Offsets1D
{
    double dxctr, dxl, dml, dxr, dmr;

    __device__ __forceinline__ Offsets1D(E1DArgs const & a, int64_t ic)
        : dxctr(a.seo[0 * a.n + ic])
        , dxl(a.seo[1 * a.n + ic])
        , dml(a.seo[2 * a.n + ic])
        , dxr(a.seo[3 * a.n + ic])
        , dmr(a.seo[4 * a.n + ic])
    {
    }
};

// The solution-element kernel at one point (Euler1DKernel::set_value and
// derive, Euler1DCore.hpp:193-244): the value up at the next half level and the
// two half fluxes of calc_flux_ll/lr (Euler1DCore.hpp:246-266).
struct K1D
{
    double up[3];
    double ll[3]; // flux through the lower-left of the CE to the right
    double lr[3]; // flux through the lower-right of the CE to the left

    __device__ __forceinline__ K1D(E1DArgs const & a, P1D const & q, double const * ux, Offsets1D const & x)
    {
        double const * const u = q.u;
        double jx[3], jj[3]; // J u_x = -u_t and J J u_x = -f_t, J the flux's Jacobian
        double const ga1 = sb(q.ga, 1.0);
        double const hv = mu(mu(0.5, q.v), q.v);
        double const h = ad(u[2], q.p);
        // The flux's change along a change w of the state.
        auto along = [&](double const * w, double * o) {
            double const dp = mu(ga1, fm(-q.v, w[1], fm(hv, w[0], w[2])));
            double const dv = mu(fm(-q.v, w[0], w[1]), q.r);
            o[0] = w[1];
            o[1] = fm(u[1], dv, fm(w[1], q.v, dp));
            o[2] = fm(h, dv, mu(ad(w[2], dp), q.v));
        };
        along(ux, jx);
        along(jx, jj);
        double const f[3] = {u[1], fm(u[1], q.v, q.p), mu(h, q.v)};
        for (int i = 0; i < 3; ++i)
        {
            up[i] = fm(-a.hdt, jx[i], fm(x.dxctr, ux[i], u[i]));
            double const tf = mu(a.hdt, fm(-a.qdt, jj[i], fm(x.dxctr, jx[i], f[i])));
            ll[i] = fm(x.dxl, fm(x.dml, ux[i], u[i]), tf);
            lr[i] = fm(x.dxr, fm(x.dmr, ux[i], u[i]), -tf);
        }
    }
};

// The W-alpha gradient (march_half_so1_alpha, Euler1DCore.hpp:284-320); for
// alpha = 2 its numerator duxp^2 duxn + duxn^2 duxp is duxn duxp (duxn + duxp).
template <bool INT>
__device__ __forceinline__ double wgrad(int alpha, double duxn, double duxp)
{
    double num, den;
    if (alpha == 2)
    {
        num = mu<INT>(mu<INT>(duxn, duxp), ad(duxn, duxp));
        den = fm(duxn, duxn, fm(duxp, duxp, Tiny1D<double>::V));
    }
    else
    {
        num = fm(fabs(duxp), duxn, mu(fabs(duxn), duxp));
        den = ad(ad(fabs(duxp), fabs(duxn)), Tiny1D<double>::V);
    }
    return mu<INT>(num, scg::dev::recip(den));
}

// What a half step does (its mask): so0, cfl, the copy-out boundary
// treatment, and so1 with the W-alpha weights for alpha = (mask >> 8) > 0.
constexpr unsigned H_SO0 = 1u, H_CFL = 2u, H_BND = 4u;
constexpr unsigned h_alpha(int alpha) { return static_cast<unsigned>(alpha) << 8; }

// One warp's part of a half step.  Output j is point start + 2j + 1 for
// j < nout; kernels are at start + 2j for j <= nout.  Lane l of warp w derives
// kernel 31 w + l, and lanes 0 .. 30 update the output to its right, with the
// next lane's kernel by shuffles: warps share nothing, so a small tube spreads
// over the SMs in blocks of one warp, and a kernel is derived once but for the
// one in 32 at the seams.
constexpr int WOUT = 31; // outputs per warp

template <bool INT>
__device__ __forceinline__ void half_warp(E1DArgs const & a, int64_t start, int64_t nout, unsigned mask, int64_t w)
{
    int const alpha = static_cast<int>(mask >> 8);
    int const lane = static_cast<int>(threadIdx.x) & 31;
    int64_t const j = w * WOUT + lane;
    int64_t const ic = start + 2 * (j < nout ? j : nout); // lanes past the end repeat the last kernel
    P1D const q(a.so0 + ic * 3, a.gamma[ic]);
    K1D const k(a, q, a.so1 + ic * 3, Offsets1D(a, ic));
    double const idxr = a.invdx[ic - 1]; // 1 / (x - xneg)
    double lr[3], up[3];
    for (int i = 0; i < 3; ++i)
    {
        lr[i] = __shfl_down_sync(0xffffffffu, k.lr[i], 1);
        up[i] = __shfl_down_sync(0xffffffffu, k.up[i], 1);
    }
    double const idp = __shfl_down_sync(0xffffffffu, idxr, 1);
    if (lane < WOUT && j < nout)
    {
        double v[3];
        if (mask & H_SO0)
        {
            double const idx = a.invd2[ic];
            for (int i = 0; i < 3; ++i)
            {
                v[i] = mu<INT>(ad(k.ll[i], lr[i]), idx);
                a.so0[(ic + 1) * 3 + i] = v[i];
            }
        }
        else
        {
            for (int i = 0; i < 3; ++i)
            {
                v[i] = a.so0[(ic + 1) * 3 + i];
            }
        }
        if (mask & H_CFL)
        {
            a.cfl[ic] = q.cfl(a.cflr[ic]);
        }
        if (alpha > 0)
        {
            double const idn = a.invdx[ic];
            for (int i = 0; i < 3; ++i)
            {
                a.so1[(ic + 1) * 3 + i] =
                    wgrad<INT>(alpha, mu<INT>(sb(v[i], k.up[i]), idn), mu<INT>(sb(up[i], v[i]), idp));
            }
        }
    }
}

// The copy-out boundary treatment (Euler1DCore.cpp:132-172) of points 1 and
// n - 2, which the first half step neither reads nor writes.
__device__ __forceinline__ void copy_out(E1DArgs const & a)
{
    int64_t const l = 1, r = a.n - 2;
    for (int i = 0; i < 3; ++i)
    {
        a.so0[l * 3 + i] = a.so0[(l + 1) * 3 + i];
        a.so0[r * 3 + i] = a.so0[(r - 1) * 3 + i];
        a.so1[l * 3 + i] = a.so1[(l + 1) * 3 + i];
        a.so1[r * 3 + i] = a.so1[(r - 1) * 3 + i];
    }
}

// One half step: so0, cfl and so1 at one parity and the boundary treatment, as
// the mask asks.
template <bool INT>
__global__ void __launch_bounds__(128) k_half(E1DArgs a, int64_t start, int64_t nout, unsigned mask)
{
    int64_t const w = (static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x) / 32;
    if (w * WOUT < nout)
    {
        half_warp<INT>(a, start, nout, mask, w);
    }
    if ((mask & H_BND) && blockIdx.x == 0 && threadIdx.x == 0)
    {
        copy_out(a);
    }
}

// Small tubes: a whole march in one launch of one cluster of at most 16 blocks,
// the tube in the threads' registers (cluster.cuh): thread k keeps the even
// point 2k and the odd point 2k + 1.  A half step of a small tube is latency
// and nothing else, most of it outside the arithmetic: the launch, the loads
// from the L2 and the stores on their way back (201 points FP64: 6.4 us per
// half step in a graph of launches, 8.4 launched singly, 5.7 with one cluster
// marching the state in the L2, 3.9 here).
//
// A block's warps at most: one for each of the SM's four FP64 pipes (measured,
// per half step: 3.9 us up to 2,001 points, 4.35 us at 4,001, against 6.0 to
// 6.4 us in graph launches; a second warp per pipe: 7.6 against 6.2).
constexpr int TUBE_WARPS64 = 4;

__global__ void __launch_bounds__(32 * TUBE_WARPS64) k_tube(E1DArgs a, int alpha, int64_t steps, int64_t nout1,
                                                            int64_t nout2)
{
    __shared__ double slots[2][TUBE_WARPS64][6];
    int64_t const nk = (a.n - 1) / 2; // threads with a point pair
    int64_t const t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    int64_t const k = t < nk ? t : nk - 1; // the others repeat the last pair, and write nothing
    int64_t const e = 2 * k, o = 2 * k + 1;
    int64_t const l = k > 0 ? e - 1 : 0;
    double ue[3], xe[3], uo[3], xo[3];
    for (int i = 0; i < 3; ++i)
    {
        ue[i] = a.so0[e * 3 + i];
        xe[i] = a.so1[e * 3 + i];
        uo[i] = a.so0[o * 3 + i];
        xo[i] = a.so1[o * 3 + i];
    }
    double const ge = a.gamma[e], go = a.gamma[o];
    Offsets1D const oe(a, e), oo(a, o);
    double const il = a.invdx[l], ie = a.invdx[e], io = a.invdx[o];
    double const dl = a.invd2[l], de = a.invd2[e];
    bool const out1 = t >= 1 && t <= nout1, out2 = t >= 1 && t <= nout2;
    cluster_sync(); // every block runs before any stores to another's slots
    for (int64_t s = 0; s < steps; ++s)
    {
        bool const end = s + 1 == steps; // a CFL number is overwritten by the next step's
        // First half step: odd points from the even kernels k and k + 1.
        {
            P1D const q(ue, ge);
            K1D const c(a, q, xe, oe);
            double const v[6] = {c.lr[0], c.lr[1], c.lr[2], c.up[0], c.up[1], c.up[2]};
            double w[6];
            hand_over<6, 1>(v, w, slots[0]);
            // The copy-out boundary: point 1 takes point 2's, n - 2 takes n - 3's.
            for (int i = 0; i < 3; ++i)
            {
                double const un = __shfl_down_sync(0xffffffffu, ue[i], 1);
                double const xn = __shfl_down_sync(0xffffffffu, xe[i], 1);
                if (t == 0)
                {
                    uo[i] = un;
                    xo[i] = xn;
                }
                else if (t == nk - 1)
                {
                    uo[i] = ue[i];
                    xo[i] = xe[i];
                }
            }
            if (out1)
            {
                for (int i = 0; i < 3; ++i)
                {
                    uo[i] = mu(ad(c.ll[i], w[i]), de);
                    xo[i] = wgrad<false>(alpha, mu(sb(uo[i], c.up[i]), ie), mu(sb(w[3 + i], uo[i]), io));
                }
                if (end)
                {
                    a.cfl[e] = q.cfl(a.cflr[e]);
                }
            }
        }
        // Second half step: even points from the odd kernels k - 1 and k.
        {
            P1D const q(uo, go);
            K1D const c(a, q, xo, oo);
            double const v[6] = {c.ll[0], c.ll[1], c.ll[2], c.up[0], c.up[1], c.up[2]};
            double w[6];
            hand_over<6, 0>(v, w, slots[1]);
            if (out2)
            {
                for (int i = 0; i < 3; ++i)
                {
                    ue[i] = mu(ad(w[i], c.lr[i]), dl);
                    xe[i] = wgrad<false>(alpha, mu(sb(ue[i], w[3 + i]), il), mu(sb(c.up[i], ue[i]), ie));
                }
            }
            if (end && t < nout2)
            {
                a.cfl[o] = q.cfl(a.cflr[o]);
            }
        }
    }
    if (t < nk)
    {
        for (int i = 0; i < 3; ++i)
        {
            a.so0[e * 3 + i] = ue[i];
            a.so1[e * 3 + i] = xe[i];
            a.so0[o * 3 + i] = uo[i];
            a.so1[o * 3 + i] = xo[i];
        }
    }
}

// update_cfl alone.
__global__ void k_cfl1d(E1DArgs a, int64_t start, int64_t nout)
{
    int64_t const j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j < nout)
    {
        int64_t const it = start + 2 * j;
        a.cfl[it] = P1D(a.so0 + it * 3, a.gamma[it]).cfl(a.cflr[it]);
    }
}

// treat_boundary_so0 / treat_boundary_so1.
__global__ void k_bnd1d(E1DArgs a, int which)
{
    int64_t const l = 1, r = a.n - 2;
    double * s = which == 0 ? a.so0 : a.so1;
    for (int i = 0; i < 3; ++i)
    {
        s[l * 3 + i] = s[(l + 1) * 3 + i];
        s[r * 3 + i] = s[(r - 1) * 3 + i];
    }
}

// What the C ABI calls on a 1D core of either precision.
struct Euler1DBase
{
    virtual ~Euler1DBase() = default;
    virtual std::unique_ptr<Euler1DBase> clone() = 0;
    virtual int64_t count(int which) const = 0;
    virtual void get(int which, double * host) = 0;
    virtual void set(int which, double const * host) = 0;
    virtual void op(int which, int odd, int alpha) = 0;
    virtual void march(int alpha, int64_t steps) = 0;
    virtual void sync() = 0;
    int64_t n = 0;
    double time_increment = 0.0;
    int precision = SCG_FP64;
    cudaStream_t stream = nullptr;
};

// Tubes above this many points take 18 of a point's FP64 multiplications on the
// integer pipe (half_warp's INT, the same bits): there the FP64 pipes are full
// (2M points 214.6 -> 160.9 us per half step, 100,001 points 12.7 -> 12.1), below
// the longer chain of instructions shows (20,001 points 6.4 -> 8.0).
constexpr int64_t INT_POINTS64 = 60000;

// The FP64 core: the reference's arithmetic on the reference's [n][3] device
// tables.  The FP32 core is Euler1D32 below.
class Euler1D : public Euler1DBase
{
public:
    Euler1D(int64_t ncoord, double dt)
    {
        n = ncoord;
        time_increment = dt;
        precision = SCG_FP64;
        if (ncoord % 2 == 0)
        {
            throw std::invalid_argument("ncoord cannot be even");
        }
        if (ncoord < 5)
        {
            throw std::invalid_argument("Euler1DCore: ncoord must be at least 5");
        }
        scg::cuda_check(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");
        coord.alloc(static_cast<size_t>(n));
        invdx.alloc(static_cast<size_t>(n));
        invd2.alloc(static_cast<size_t>(n));
        cflr.alloc(static_cast<size_t>(n));
        seo.alloc(static_cast<size_t>(5 * n));
        for (auto * b : {&cfl, &gamma})
            b->alloc(static_cast<size_t>(n));
        so0.alloc(static_cast<size_t>(n * 3));
        so1.alloc(static_cast<size_t>(n * 3));
        std::vector<double> g(static_cast<size_t>(n), 1.4);
        std::vector<double> z(static_cast<size_t>(n * 3), 0.0);
        set(4, g.data());
        set(0, z.data());
        set(1, z.data());
        set(2, z.data());
        set(3, z.data());
    }

    ~Euler1D() override
    {
        if (graph_exec)
            cudaGraphExecDestroy(graph_exec);
        if (stream)
        {
            cudaStreamSynchronize(stream);
            cudaStreamDestroy(stream);
        }
    }

    std::unique_ptr<Euler1DBase> clone() override
    {
        auto c = std::make_unique<Euler1D>(n, time_increment);
        scg::cuda_check(cudaMemcpyAsync(c->coord.ptr, coord.ptr, sizeof(double) * static_cast<size_t>(n),
                                        cudaMemcpyDeviceToDevice, stream),
                        "copy");
        sync();
        c->spacing();
        for (int k = 1; k < 5; ++k)
        {
            size_t const cnt = static_cast<size_t>(count(k));
            scg::cuda_check(cudaMemcpyAsync(c->state(k), state(k), cnt * sizeof(double), cudaMemcpyDeviceToDevice, stream),
                            "copy");
        }
        sync();
        return c;
    }

    // 0 coord (FP64), 1 cfl, 2 so0, 3 so1, 4 gamma
    double * state(int which)
    {
        switch (which)
        {
        case 1: return cfl.ptr;
        case 2: return so0.ptr;
        case 3: return so1.ptr;
        case 4: return gamma.ptr;
        default: throw std::invalid_argument("Euler1DCore: unknown array id " + std::to_string(which));
        }
    }
    int64_t count(int which) const override { return (which == 2 || which == 3) ? n * 3 : n; }

    void get(int which, double * host) override
    {
        size_t const cnt = static_cast<size_t>(count(which));
        if (which == 0)
        {
            scg::cuda_check(cudaMemcpyAsync(host, coord.ptr, sizeof(double) * cnt, cudaMemcpyDeviceToHost, stream),
                            "D2H");
            sync();
            return;
        }
        scg::cuda_check(cudaMemcpyAsync(host, state(which), sizeof(double) * cnt, cudaMemcpyDeviceToHost, stream),
                        "D2H");
        sync();
    }
    void set(int which, double const * host) override
    {
        size_t const cnt = static_cast<size_t>(count(which));
        if (which == 0)
        {
            put(coord.ptr, host, cnt);
            spacing();
            return;
        }
        put(state(which), host, cnt);
    }

    // The grid's tables (E1DArgs) from the coordinates.
    void spacing()
    {
        k_inv_spacing<<<static_cast<unsigned>((n + 255) / 256), 256, 0, stream>>>(coord.ptr, n, time_increment / 2.0,
                                                                                   invdx.ptr, invd2.ptr, cflr.ptr,
                                                                                   seo.ptr);
        scg::launched(stream, "e1d_inv_spacing");
        sync();
    }

    E1DArgs args()
    {
        return E1DArgs{gamma.ptr, so0.ptr, so1.ptr, cfl.ptr, n, time_increment / 2.0, time_increment / 4.0,
                       invdx.ptr, invd2.ptr, cflr.ptr, seo.ptr};
    }

    // Loop bounds of a half step (Euler1DCore.cpp:73-74, 99-100).
    void range(bool odd, int64_t & start, int64_t & nout) const
    {
        start = 2 - (odd ? 1 : 0);
        int64_t const stop = n - 2 - (odd ? 0 : 1);
        nout = stop > start ? (stop - start + 1) / 2 : 0;
    }

    void half(unsigned mask, bool odd)
    {
        int64_t start, nout;
        range(odd, start, nout);
        // Blocks of one warp while they all are resident at once (32 blocks
        // on each SM), so that a tube takes the FP64 pipes of as many SMs as it
        // has warps; beyond that blocks of four.
        int64_t const warps = std::max<int64_t>((nout + WOUT - 1) / WOUT, 1);
        int const wpb = warps <= int64_t(scg::sm_count()) * 32 ? 1 : 4;
        unsigned const grid = static_cast<unsigned>((warps + wpb - 1) / wpb);
        if (n > INT_POINTS64)
        {
            k_half<true><<<grid, 32 * wpb, 0, stream>>>(args(), start, nout, mask);
        }
        else
        {
            k_half<false><<<grid, 32 * wpb, 0, stream>>>(args(), start, nout, mask);
        }
        scg::launched(stream, "e1d_half");
    }

    void op(int which, int odd, int alpha) override
    {
        switch (which)
        {
        case 0: // update_cfl
        {
            int64_t start, nout;
            range(odd != 0, start, nout);
            if (nout > 0)
            {
                k_cfl1d<<<static_cast<unsigned>((nout + 255) / 256), 256, 0, stream>>>(args(), start, nout);
                scg::launched(stream, "e1d_cfl");
            }
            break;
        }
        case 1: // march_half_so0
            half(H_SO0, odd != 0);
            break;
        case 2: // march_half_so1_alpha
            half(h_alpha(alpha == 1 ? 1 : 2), odd != 0);
            break;
        case 3: // treat_boundary_so0
        case 4: // treat_boundary_so1
            k_bnd1d<<<1, 1, 0, stream>>>(args(), which - 3);
            scg::launched(stream, "e1d_bnd");
            break;
        case 5: // setup_march
        {
            int64_t start, nout;
            range(false, start, nout);
            if (nout > 0)
            {
                k_cfl1d<<<static_cast<unsigned>((nout + 255) / 256), 256, 0, stream>>>(args(), start, nout);
                scg::launched(stream, "e1d_cfl");
            }
            break;
        }
        case 6: // march_half1_alpha: so0, cfl, so1 at the even kernels
            half(H_SO0 | H_CFL | h_alpha(alpha == 1 ? 1 : 2), false);
            break;
        case 7: // march_half2_alpha
            half(H_SO0 | H_CFL | h_alpha(alpha == 1 ? 1 : 2), true);
            break;
        default:
            throw std::invalid_argument("Euler1DCore: unknown operation " + std::to_string(which));
        }
        sync();
    }

    // One march_alpha step (Euler1DCore.hpp:339-349): half 1 with the
    // boundary treatment fused, then half 2.
    void step(int alpha)
    {
        half(H_SO0 | H_CFL | H_BND | h_alpha(alpha), false);
        half(H_SO0 | H_CFL | h_alpha(alpha), true);
    }

    // march_alpha(steps): a small tube in launches of one cluster, a larger one
    // in chunks of GRAPH_STEPS steps that replay one captured CUDA graph, the
    // remainder launched directly.
    void march(int alpha, int64_t steps) override
    {
        if (alpha != 1 && alpha != 2)
        {
            throw std::invalid_argument("Euler1DCore: alpha must be 1 or 2");
        }
        if (cluster_march(alpha, steps))
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

    bool cluster_march(int alpha, int64_t steps)
    {
        int blocks, warps;
        if (!cluster_shape<k_tube, TUBE_WARPS64>((n - 1) / 2, blocks, warps))
        {
            return false;
        }
        int64_t start, nout1, nout2;
        range(false, start, nout1);
        range(true, start, nout2);
        for (int64_t s = 0; s < steps; s += CLUSTER_STEPS)
        {
            launch_cluster(k_tube, blocks, 32 * warps, stream, args(), alpha, std::min(CLUSTER_STEPS, steps - s), nout1,
                           nout2);
            scg::launched(stream, "e1d_tube");
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
        scg::g_launches.store(before); // captured, not launched
        scg::cuda_check(cudaStreamEndCapture(stream, &g), "EndCapture");
        scg::cuda_check(cudaGraphInstantiate(&graph_exec, g, 0), "GraphInstantiate");
        cudaGraphDestroy(g);
        graph_alpha = alpha;
    }

    void sync() override { scg::cuda_check(cudaStreamSynchronize(stream), "cudaStreamSynchronize"); }

private:
    static constexpr int GRAPH_STEPS = 32;

    template <typename T>
    void put(T * dst, T const * src, size_t cnt)
    {
        scg::cuda_check(cudaMemcpyAsync(dst, src, sizeof(T) * cnt, cudaMemcpyHostToDevice, stream), "H2D");
        sync();
    }

    scg::DevBuf<double> coord;
    scg::DevBuf<double> invdx, invd2, cflr, seo; // see E1DArgs
    scg::DevBuf<double> cfl, so0, so1, gamma;
    cudaGraphExec_t graph_exec = nullptr;
    int graph_alpha = 0;
};

// ---------------------------------------------------------------------------
// The FP32 core (not in the reference): FP32 state, cfl and gamma, the
// coordinates kept in FP64 and the spacing between them formed in FP64 and
// rounded once.  It keeps its state in a device layout of its own: every
// quantity split by the parity of the point into two planes (point i -> plane
// i & 1, index i >> 1).  A half step reads the kernel planes of one parity
// and writes the output planes of the other, so every line it fetches is
// used whole, and one thread updates four consecutive outputs with 16-byte
// loads and stores (the planes are padded to a multiple of four).  The host
// sees the reference's [n][3] FP64 tables, converted on the device.

constexpr int B32 = 128;
enum : int
{
    PL_SO0 = 0, // 3 planes: so0 of each variable
    PL_SO1 = 3, // 3 planes: so1
    PL_GAMMA = 6,
    PL_CFL = 7,
    PL_DXM = 8, // x - xneg
    PL_DXP = 9, // xpos - x
    PL_COUNT = 10
};

struct Planes
{
    float * base; // [2][PL_COUNT][P]
    int64_t P;    // plane stride, a multiple of 4
    int64_t n;
    float hdt, qdt;
    __device__ __forceinline__ float * at(int parity, int q) const
    {
        return base + (static_cast<int64_t>(parity) * PL_COUNT + q) * P;
    }
};

// Warps at most of a block that holds part of a tube in registers (1,024
// threads: 32,769 points over 16 blocks).  Per half step 0.53 us up to 2,001
// points, 0.69 us at 8,001, 1.12 us at 20,001 and 1.56 us at 32,001, against 2.1
// to 2.8 us in graph launches.
constexpr int TUBE_WARPS32 = 32;
// The largest FP32 tubes whose half steps take one output per lane instead of
// four per thread (per half step 2.6 against 3.1 us at 80,001 points, 3.5
// against 4.3 us at 320,001, 4.9 against 4.8 us at 640,001, 8.1 against 7.3 us at
// 1,280,001, where the four outputs' wider loads pay).
constexpr int64_t WARP_POINTS32 = 400000;

// Division in the FP32 core: the approximate quotient (within 2 ulp over the
// normal range; every divisor here is a spacing, a density or a positive sum
// of squares, far inside it).  A correctly rounded FP32 division is a
// multi-instruction sequence, and a half step divides about twelve times per
// output point: 20M-point tube 39.7 -> 88.2 G point-steps/s with it, the
// state within the same bound of the FP64 core as before.
__device__ __forceinline__ float div32(float a, float b) { return __fdividef(a, b); }

// The W-alpha gradient of the FP32 core (wgrad with div32).
template <int ALPHA>
__device__ __forceinline__ float wgrad32(float duxn, float duxp)
{
    float fan = fabsf(duxn);
    float fap = fabsf(duxp);
    if constexpr (ALPHA == 2)
    {
        fan *= fan;
        fap *= fap;
    }
    return div32(fap * duxn + fan * duxp, fap + fan + Tiny1D<float>::V);
}

// The solution-element kernel of one point in FP32 delta form: the state u,
// up - u, and the two half fluxes without their dx * u parts (the caller adds
// those relative to the output point); r = 1 / (rho + tiny) for update_cfl.
struct K32
{
    float u[3], upd[3], llp[3], lrp[3];
    float dm, dp, r, ga;
};

// Euler1DKernel::set_value and derive (Euler1DCore.hpp:193-244) in FP32 from
// the point's state, gamma and spacing dm = x - xneg, dp = xpos - x.
__device__ __forceinline__ void derive32(float const * u, float const * ux, float ga, float dm, float dp, float hdt,
                                         float qdt, K32 & k)
{
    float const r = div32(1.f, u[0] + Tiny1D<float>::V);
    float const r2 = r * r;
    float const m2r2 = u[1] * u[1] * r2;
    float jac[3][3];
    jac[0][0] = 0.f;
    jac[0][1] = 1.f;
    jac[0][2] = 0.f;
    jac[1][0] = (ga - 3.f) / 2.f * m2r2;
    jac[1][1] = -(ga - 3.f) * u[1] * r;
    jac[1][2] = ga - 1.f;
    jac[2][0] = (ga - 1.f) * m2r2 * u[1] * r - ga * u[1] * u[2] * r2;
    jac[2][1] = ga * u[2] * r - 1.5f * (ga - 1.f) * m2r2;
    jac[2][2] = ga * u[1] * r;
    float f[3], ut[3], ft[3];
    f[0] = u[1];
    f[1] = (ga - 1.f) * u[2] + (3.f - ga) / 2.f * u[1] * u[1] * r;
    f[2] = ga * u[1] * u[2] * r - (ga - 1.f) / 2.f * u[1] * m2r2;
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
        ut[i] = -jac[i][0] * ux[0] - jac[i][1] * ux[1] - jac[i][2] * ux[2];
    }
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
        ft[i] = jac[i][0] * ut[0] + jac[i][1] * ut[1] + jac[i][2] * ut[2];
    }
    // x - xctr = (dm - dp) / 2, and the BCE midpoints sit at dm / 2 and
    // -dp / 2 from the centre.
    float const dxctr = 0.5f * (dm - dp);
    float const dml = 0.5f * dm;
    float const dmr = -0.5f * dp;
#pragma unroll
    for (int i = 0; i < 3; ++i)
    {
        k.u[i] = u[i];
        k.upd[i] = dxctr * ux[i] + hdt * ut[i];
        float const tf = f[i] - dxctr * ut[i] + qdt * ft[i];
        k.llp[i] = dp * dml * ux[i] + hdt * tf;
        k.lrp[i] = dm * dmr * ux[i] - hdt * tf;
    }
    k.dm = dm;
    k.dp = dp;
    k.r = r;
    k.ga = ga;
}

// update_cfl at a kernel point (Euler1DCore.cpp:70-94) from its derivation.
__device__ __forceinline__ float cfl32(K32 const & k, float hdt)
{
    float const m = k.u[1];
    float const ke = 0.5f * m * m * k.r;
    float pr = (k.ga - 1.f) * (k.u[2] - ke);
    pr = (pr + fabsf(pr)) / 2.f;
    float const wspd = sqrtf(k.ga * pr * k.r) + fabsf(m) * k.r;
    return div32(hdt * wspd, k.dp < k.dm ? k.dp : k.dm);
}

__device__ __forceinline__ float lane(float4 v, int i)
{
    return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w;
}

// One output between its left and right kernels: the new so0 in delta form
// (DO_SO0: the old value u0 plus a change formed from the kernels' states
// relative to it, so FP32 rounding scales with the change; without it u0 is the
// new value already) and, for ALPHA > 0, so1 by the W-alpha gradient.
template <int ALPHA, bool DO_SO0>
__device__ __forceinline__ void output32(K32 const & L, K32 const & R, float const * u0, float * nso0, float * nso1)
{
    float const dxl = L.dp;
    float const dxr = R.dm;
    float const idx = div32(1.f, dxl + dxr);
#pragma unroll
    for (int v = 0; v < 3; ++v)
    {
        float d;
        if constexpr (DO_SO0)
        {
            d = (dxl * (L.u[v] - u0[v]) + dxr * (R.u[v] - u0[v]) + L.llp[v] + R.lrp[v]) * idx;
            nso0[v] = u0[v] + d;
        }
        else
        {
            d = 0.f;
            nso0[v] = u0[v];
        }
        if constexpr (ALPHA > 0)
        {
            // The gradient's differences v - up_l and up_r - v from small
            // terms: (u0 - u_l) + d - (up_l - u_l), (u_r - u0) + (up_r - u_r) - d.
            float const duxn = div32((u0[v] - L.u[v]) + d - L.upd[v], dxl);
            float const duxp = div32((R.u[v] - u0[v]) + R.upd[v] - d, dxr);
            nso1[v] = wgrad32<ALPHA>(duxn, duxp);
        }
    }
}

// One half step of the FP32 core, outputs of parity Q from the kernels of the
// other parity.  Output o (1 <= o <= nout) sits between its left and right
// kernels: kernel indices o and o + 1 when the outputs are odd points (the
// first half step), o - 1 and o when they are even.  Thread t updates outputs
// 4t .. 4t + 3 from the four kernels at the same indices (16-byte loads) and
// one more (the next index or the previous one), each derived once per
// thread.  DO_SO0: the new so0 in delta form (each output's old value plus a
// change formed from the kernels' states relative to it, so FP32 rounding
// scales with the change); without it so0 is already new and only so1 is
// formed.  ALPHA > 0: so1 by the W-alpha gradient.  DO_CFL: update_cfl at
// each output's left kernel.  k_half32's BND: the copy-out boundary treatment
// of points 1 and n - 2, which the half step neither reads nor writes.
template <int ALPHA, bool DO_SO0, bool DO_CFL, int Q>
__device__ __forceinline__ void half32_four(Planes const & a, int64_t nout, int64_t c)
{
    constexpr int P = 1 - Q; // parity of the kernels
    // The five kernels in index order: Q = 1 uses c .. c + 4, Q = 0 uses
    // c - 1 .. c + 3; the one outside the aligned four is the halo.
    int64_t const h = Q == 1 ? c + 4 : c - 1;
    // Index -1 (thread 0 of the second half step) serves only output 0,
    // which is not written: read kernel 0 in its place.
    int64_t const hc = h < 0 ? 0 : h;
    float4 const g4 = *reinterpret_cast<float4 const *>(a.at(P, PL_GAMMA) + c);
    float4 const m4 = *reinterpret_cast<float4 const *>(a.at(P, PL_DXM) + c);
    float4 const p4 = *reinterpret_cast<float4 const *>(a.at(P, PL_DXP) + c);
    float4 u4[3], x4[3];
    float hu[3], hx[3];
#pragma unroll
    for (int v = 0; v < 3; ++v)
    {
        u4[v] = *reinterpret_cast<float4 const *>(a.at(P, PL_SO0 + v) + c);
        x4[v] = *reinterpret_cast<float4 const *>(a.at(P, PL_SO1 + v) + c);
        hu[v] = a.at(P, PL_SO0 + v)[hc];
        hx[v] = a.at(P, PL_SO1 + v)[hc];
    }
    float const hg = a.at(P, PL_GAMMA)[hc];
    float const hm = a.at(P, PL_DXM)[hc];
    float const hp = a.at(P, PL_DXP)[hc];
    // Kernel s (0 .. 4) in index order, derived.
    auto kernel = [&](int s, K32 & k) {
        float u[3], x[3], ga, dm, dp;
        int const l = Q == 1 ? s : s - 1; // lane of the aligned four, or the halo
        if (l < 0 || l > 3)
        {
            for (int v = 0; v < 3; ++v)
            {
                u[v] = hu[v];
                x[v] = hx[v];
            }
            ga = hg;
            dm = hm;
            dp = hp;
        }
        else
        {
            for (int v = 0; v < 3; ++v)
            {
                u[v] = lane(u4[v], l);
                x[v] = lane(x4[v], l);
            }
            ga = lane(g4, l);
            dm = lane(m4, l);
            dp = lane(p4, l);
        }
        derive32(u, x, ga, dm, dp, a.hdt, a.qdt, k);
    };
    // The outputs' so0: their old values (DO_SO0) or the new ones.
    float4 o4[3];
#pragma unroll
    for (int v = 0; v < 3; ++v)
    {
        o4[v] = *reinterpret_cast<float4 const *>(a.at(Q, PL_SO0 + v) + c);
    }
    float nso0[3][4], nso1[3][4], ncfl[4];
    K32 L; // the left kernel of output k; R its right one
    kernel(0, L);
#pragma unroll
    for (int k = 0; k < 4; ++k)
    {
        K32 R;
        kernel(k + 1, R);
        float const u0[3] = {lane(o4[0], k), lane(o4[1], k), lane(o4[2], k)};
        float n0[3], n1[3];
        output32<ALPHA, DO_SO0>(L, R, u0, n0, n1);
#pragma unroll
        for (int v = 0; v < 3; ++v)
        {
            nso0[v][k] = n0[v];
            if constexpr (ALPHA > 0)
            {
                nso1[v][k] = n1[v];
            }
        }
        if constexpr (DO_CFL)
        {
            ncfl[k] = cfl32(L, a.hdt);
        }
        L = R;
    }
    bool const whole = c >= 1 && c + 3 <= nout;
#pragma unroll
    for (int v = 0; v < 3; ++v)
    {
        float * const s0 = a.at(Q, PL_SO0 + v) + c;
        float * const s1 = a.at(Q, PL_SO1 + v) + c;
        if (whole)
        {
            if constexpr (DO_SO0)
            {
                *reinterpret_cast<float4 *>(s0) = make_float4(nso0[v][0], nso0[v][1], nso0[v][2], nso0[v][3]);
            }
            if constexpr (ALPHA > 0)
            {
                *reinterpret_cast<float4 *>(s1) = make_float4(nso1[v][0], nso1[v][1], nso1[v][2], nso1[v][3]);
            }
        }
        else
        {
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                if (c + k >= 1 && c + k <= nout)
                {
                    if constexpr (DO_SO0)
                    {
                        s0[k] = nso0[v][k];
                    }
                    if constexpr (ALPHA > 0)
                    {
                        s1[k] = nso1[v][k];
                    }
                }
            }
        }
    }
    if constexpr (DO_CFL)
    {
        // The left kernel of output o is kernel o (Q = 1) or o - 1 (Q = 0).
        float * const cf = a.at(P, PL_CFL) + c - (Q == 1 ? 0 : 1);
#pragma unroll
        for (int k = 0; k < 4; ++k)
        {
            if (c + k >= 1 && c + k <= nout)
            {
                cf[k] = ncfl[k];
            }
        }
    }
}

// One warp's part of a half step with one output per lane, for tubes that
// leave the GPU's warps idle, where the latency of a thread's four outputs in
// turn would set the time: lane l derives kernel 31 w + l of those the half
// step reads, and lanes 0 .. 30 update the output to its right, with the next
// lane's kernel by shuffles.
template <int ALPHA, int Q>
__device__ __forceinline__ void half32_warp(Planes const & a, int64_t nout, int64_t w)
{
    constexpr int P = 1 - Q;
    int const ln = static_cast<int>(threadIdx.x) & 31;
    int64_t const j = w * WOUT + ln;           // kernel j, output j + 1
    int64_t const i = (j < nout ? j : nout) + Q; // its index in its plane
    int64_t const o = (j < nout ? j : nout - 1) + 1;
    float u[3], x[3], u0[3];
#pragma unroll
    for (int v = 0; v < 3; ++v)
    {
        u[v] = a.at(P, PL_SO0 + v)[i];
        x[v] = a.at(P, PL_SO1 + v)[i];
        u0[v] = a.at(Q, PL_SO0 + v)[o];
    }
    K32 L, R;
    derive32(u, x, a.at(P, PL_GAMMA)[i], a.at(P, PL_DXM)[i], a.at(P, PL_DXP)[i], a.hdt, a.qdt, L);
#pragma unroll
    for (int v = 0; v < 3; ++v)
    {
        R.u[v] = __shfl_down_sync(0xffffffffu, L.u[v], 1);
        R.upd[v] = __shfl_down_sync(0xffffffffu, L.upd[v], 1);
        R.lrp[v] = __shfl_down_sync(0xffffffffu, L.lrp[v], 1);
    }
    R.dm = __shfl_down_sync(0xffffffffu, L.dm, 1);
    if (ln < WOUT && j < nout)
    {
        float n0[3], n1[3];
        output32<ALPHA, true>(L, R, u0, n0, n1);
#pragma unroll
        for (int v = 0; v < 3; ++v)
        {
            a.at(Q, PL_SO0 + v)[o] = n0[v];
            a.at(Q, PL_SO1 + v)[o] = n1[v];
        }
        a.at(P, PL_CFL)[i] = cfl32(L, a.hdt);
    }
}

// The copy-out boundary treatment of points 1 and n - 2.
__device__ __forceinline__ void copy_out32(Planes const & a)
{
    int64_t const hi = (a.n - 3) / 2;
    for (int v = 0; v < 3; ++v)
    {
        a.at(1, PL_SO0 + v)[0] = a.at(0, PL_SO0 + v)[1];
        a.at(1, PL_SO0 + v)[hi] = a.at(0, PL_SO0 + v)[hi];
        a.at(1, PL_SO1 + v)[0] = a.at(0, PL_SO1 + v)[1];
        a.at(1, PL_SO1 + v)[hi] = a.at(0, PL_SO1 + v)[hi];
    }
}

template <int ALPHA, bool DO_SO0, bool DO_CFL, bool BND, int Q>
__global__ void __launch_bounds__(B32) k_half32(Planes a, int64_t nout)
{
    if (BND && blockIdx.x == 0 && threadIdx.x == 0)
    {
        copy_out32(a);
    }
    int64_t const c = 4 * (static_cast<int64_t>(blockIdx.x) * B32 + threadIdx.x);
    if (c <= nout)
    {
        half32_four<ALPHA, DO_SO0, DO_CFL, Q>(a, nout, c);
    }
}

// A small tube's whole march in one cluster, in registers (see k_tube).
template <int ALPHA>
__global__ void __launch_bounds__(32 * TUBE_WARPS32) k_tube32(Planes a, int64_t steps, int64_t nout1, int64_t nout2)
{
    __shared__ float slots[2][TUBE_WARPS32][10];
    int64_t const nk = (a.n - 1) / 2;
    int64_t const t = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    int64_t const k = t < nk ? t : nk - 1;
    float ue[3], xe[3], uo[3], xo[3];
#pragma unroll
    for (int v = 0; v < 3; ++v)
    {
        ue[v] = a.at(0, PL_SO0 + v)[k];
        xe[v] = a.at(0, PL_SO1 + v)[k];
        uo[v] = a.at(1, PL_SO0 + v)[k];
        xo[v] = a.at(1, PL_SO1 + v)[k];
    }
    float const ge = a.at(0, PL_GAMMA)[k], go = a.at(1, PL_GAMMA)[k];
    float const me = a.at(0, PL_DXM)[k], mo = a.at(1, PL_DXM)[k];
    float const pe = a.at(0, PL_DXP)[k], po = a.at(1, PL_DXP)[k];
    bool const out1 = t >= 1 && t <= nout1, out2 = t >= 1 && t <= nout2;
    cluster_sync(); // every block runs before any stores to another's slots
    for (int64_t s = 0; s < steps; ++s)
    {
        bool const end = s + 1 == steps;
        {
            K32 L, R;
            derive32(ue, xe, ge, me, pe, a.hdt, a.qdt, L);
            float const v[10] = {L.u[0],   L.u[1],   L.u[2],   L.upd[0], L.upd[1],
                                 L.upd[2], L.lrp[0], L.lrp[1], L.lrp[2], L.dm};
            float w[10];
            hand_over<10, 1>(v, w, slots[0]);
#pragma unroll
            for (int i = 0; i < 3; ++i)
            {
                R.u[i] = w[i];
                R.upd[i] = w[3 + i];
                R.lrp[i] = w[6 + i];
                float const un = __shfl_down_sync(0xffffffffu, ue[i], 1);
                float const xn = __shfl_down_sync(0xffffffffu, xe[i], 1);
                if (t == 0)
                {
                    uo[i] = un;
                    xo[i] = xn;
                }
                else if (t == nk - 1)
                {
                    uo[i] = ue[i];
                    xo[i] = xe[i];
                }
            }
            R.dm = w[9];
            if (out1)
            {
                float n0[3], n1[3];
                output32<ALPHA, true>(L, R, uo, n0, n1);
#pragma unroll
                for (int i = 0; i < 3; ++i)
                {
                    uo[i] = n0[i];
                    xo[i] = n1[i];
                }
                if (end)
                {
                    a.at(0, PL_CFL)[k] = cfl32(L, a.hdt);
                }
            }
        }
        {
            K32 L, R;
            derive32(uo, xo, go, mo, po, a.hdt, a.qdt, R);
            float const v[10] = {R.u[0],   R.u[1],   R.u[2],   R.upd[0], R.upd[1],
                                 R.upd[2], R.llp[0], R.llp[1], R.llp[2], R.dp};
            float w[10];
            hand_over<10, 0>(v, w, slots[1]);
#pragma unroll
            for (int i = 0; i < 3; ++i)
            {
                L.u[i] = w[i];
                L.upd[i] = w[3 + i];
                L.llp[i] = w[6 + i];
            }
            L.dp = w[9];
            if (out2)
            {
                float n0[3], n1[3];
                output32<ALPHA, true>(L, R, ue, n0, n1);
#pragma unroll
                for (int i = 0; i < 3; ++i)
                {
                    ue[i] = n0[i];
                    xe[i] = n1[i];
                }
            }
            if (end && t < nout2)
            {
                a.at(1, PL_CFL)[k] = cfl32(R, a.hdt);
            }
        }
    }
    if (t < nk)
    {
#pragma unroll
        for (int v = 0; v < 3; ++v)
        {
            a.at(0, PL_SO0 + v)[k] = ue[v];
            a.at(0, PL_SO1 + v)[k] = xe[v];
            a.at(1, PL_SO0 + v)[k] = uo[v];
            a.at(1, PL_SO1 + v)[k] = xo[v];
        }
    }
}

// The march's half step with one output per lane.
template <int ALPHA, bool BND, int Q>
__global__ void __launch_bounds__(B32) k_half32_warp(Planes a, int64_t nout)
{
    if (BND && blockIdx.x == 0 && threadIdx.x == 0)
    {
        copy_out32(a);
    }
    int64_t const w = (static_cast<int64_t>(blockIdx.x) * B32 + threadIdx.x) / 32;
    if (w * WOUT < nout)
    {
        half32_warp<ALPHA, Q>(a, nout, w);
    }
}

// update_cfl alone at count kernel points of one parity from index i0.
__global__ void k_cfl32(Planes a, int parity, int64_t i0, int64_t count)
{
    int64_t const j = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (j >= count)
    {
        return;
    }
    int64_t const i = i0 + j;
    float u[3], x[3];
    for (int v = 0; v < 3; ++v)
    {
        u[v] = a.at(parity, PL_SO0 + v)[i];
        x[v] = a.at(parity, PL_SO1 + v)[i];
    }
    K32 k;
    derive32(u, x, a.at(parity, PL_GAMMA)[i], a.at(parity, PL_DXM)[i], a.at(parity, PL_DXP)[i], a.hdt, a.qdt, k);
    a.at(parity, PL_CFL)[i] = cfl32(k, a.hdt);
}

// treat_boundary_so0 / so1: points 1 and n - 2 from points 2 and n - 3.
__global__ void k_bnd32(Planes a, int q0)
{
    int64_t const hi = (a.n - 3) / 2;
    for (int v = 0; v < 3; ++v)
    {
        a.at(1, q0 + v)[0] = a.at(0, q0 + v)[1];
        a.at(1, q0 + v)[hi] = a.at(0, q0 + v)[hi];
    }
}

// Host table <-> planes.  Table t[i * width + v] of point i (width 3 for so0
// and so1, 1 for cfl and gamma) goes to plane q0 + v of parity i & 1 at
// index i >> 1.
__global__ void k_planes_from_f64(Planes a, int q0, int width, double const * t)
{
    int64_t const i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < a.n)
    {
        for (int v = 0; v < width; ++v)
        {
            a.at(static_cast<int>(i & 1), q0 + v)[i >> 1] = float(t[i * width + v]);
        }
    }
}

__global__ void k_planes_to_f64(Planes a, int q0, int width, double * t)
{
    int64_t const i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < a.n)
    {
        for (int v = 0; v < width; ++v)
        {
            t[i * width + v] = double(a.at(static_cast<int>(i & 1), q0 + v)[i >> 1]);
        }
    }
}

// The spacing planes from the FP64 coordinates, rounded once (zero where a
// neighbour is missing).
__global__ void k_planes_spacing(Planes a, double const * coord)
{
    int64_t const i = static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i < a.n)
    {
        int const p = static_cast<int>(i & 1);
        a.at(p, PL_DXM)[i >> 1] = i > 0 ? float(coord[i] - coord[i - 1]) : 0.f;
        a.at(p, PL_DXP)[i >> 1] = i + 1 < a.n ? float(coord[i + 1] - coord[i]) : 0.f;
    }
}

class Euler1D32 : public Euler1DBase
{
public:
    Euler1D32(int64_t ncoord, double dt)
    {
        n = ncoord;
        time_increment = dt;
        precision = SCG_FP32;
        if (ncoord % 2 == 0)
        {
            throw std::invalid_argument("ncoord cannot be even");
        }
        if (ncoord < 5)
        {
            throw std::invalid_argument("Euler1DCore: ncoord must be at least 5");
        }
        scg::cuda_check(cudaStreamCreateWithFlags(&stream, cudaStreamNonBlocking), "cudaStreamCreate");
        coord.alloc(static_cast<size_t>(n));
        // Each plane holds (n + 1) / 2 points plus room for the last thread's
        // 16-byte accesses past the end.
        P = (((n + 1) / 2 + 8) + 3) / 4 * 4;
        planes.alloc(static_cast<size_t>(2 * PL_COUNT * P));
        scg::cuda_check(cudaMemsetAsync(planes.ptr, 0, planes.bytes(), stream), "memset");
        std::vector<double> g(static_cast<size_t>(n), 1.4);
        set(4, g.data());
        std::vector<double> z(static_cast<size_t>(n), 0.0);
        set(0, z.data());
    }

    ~Euler1D32() override
    {
        if (graph_exec)
            cudaGraphExecDestroy(graph_exec);
        if (stream)
        {
            cudaStreamSynchronize(stream);
            cudaStreamDestroy(stream);
        }
    }

    std::unique_ptr<Euler1DBase> clone() override
    {
        auto c = std::make_unique<Euler1D32>(n, time_increment);
        scg::cuda_check(cudaMemcpyAsync(c->coord.ptr, coord.ptr, sizeof(double) * static_cast<size_t>(n),
                                        cudaMemcpyDeviceToDevice, stream),
                        "copy");
        scg::cuda_check(cudaMemcpyAsync(c->planes.ptr, planes.ptr, planes.bytes(), cudaMemcpyDeviceToDevice, stream),
                        "copy");
        sync();
        return c;
    }

    Planes args() const
    {
        return Planes{planes.ptr, P, n, float(time_increment / 2.0), float(time_increment / 4.0)};
    }

    int64_t count(int which) const override { return (which == 2 || which == 3) ? n * 3 : n; }

    // 1 cfl, 2 so0, 3 so1, 4 gamma -> first plane and width.
    static void plane_of(int which, int & q0, int & width)
    {
        switch (which)
        {
        case 1: q0 = PL_CFL; width = 1; break;
        case 2: q0 = PL_SO0; width = 3; break;
        case 3: q0 = PL_SO1; width = 3; break;
        case 4: q0 = PL_GAMMA; width = 1; break;
        default: throw std::invalid_argument("Euler1DCore: unknown array id " + std::to_string(which));
        }
    }

    void get(int which, double * host) override
    {
        size_t const cnt = static_cast<size_t>(count(which));
        if (which == 0)
        {
            scg::cuda_check(cudaMemcpyAsync(host, coord.ptr, sizeof(double) * cnt, cudaMemcpyDeviceToHost, stream),
                            "D2H");
            sync();
            return;
        }
        int q0, width;
        plane_of(which, q0, width);
        unsigned const grid = static_cast<unsigned>((n + 255) / 256);
        if (double * const dev = static_cast<double *>(scg::mapped_host(host, sizeof(double) * cnt)))
        {
            k_planes_to_f64<<<grid, 256, 0, stream>>>(args(), q0, width, dev);
            scg::launched(stream, "e1d_planes_to_f64");
        }
        else
        {
            double * const tmp = staging(cnt);
            k_planes_to_f64<<<grid, 256, 0, stream>>>(args(), q0, width, tmp);
            scg::launched(stream, "e1d_planes_to_f64");
            scg::cuda_check(cudaMemcpyAsync(host, tmp, sizeof(double) * cnt, cudaMemcpyDeviceToHost, stream), "D2H");
        }
        sync();
    }

    void set(int which, double const * host) override
    {
        size_t const cnt = static_cast<size_t>(count(which));
        unsigned const grid = static_cast<unsigned>((n + 255) / 256);
        if (which == 0)
        {
            scg::cuda_check(cudaMemcpyAsync(coord.ptr, host, sizeof(double) * cnt, cudaMemcpyHostToDevice, stream),
                            "H2D");
            k_planes_spacing<<<grid, 256, 0, stream>>>(args(), coord.ptr);
            scg::launched(stream, "e1d_planes_spacing");
            sync();
            return;
        }
        int q0, width;
        plane_of(which, q0, width);
        if (double const * const dev = static_cast<double const *>(scg::mapped_host(host, sizeof(double) * cnt)))
        {
            k_planes_from_f64<<<grid, 256, 0, stream>>>(args(), q0, width, dev);
            scg::launched(stream, "e1d_planes_from_f64");
        }
        else
        {
            double * const tmp = staging(cnt);
            scg::cuda_check(cudaMemcpyAsync(tmp, host, sizeof(double) * cnt, cudaMemcpyHostToDevice, stream), "H2D");
            k_planes_from_f64<<<grid, 256, 0, stream>>>(args(), q0, width, tmp);
            scg::launched(stream, "e1d_planes_from_f64");
        }
        sync();
    }

    // Grow-only device table for FP64 host data on its way to or from the
    // planes.
    double * staging(size_t cnt)
    {
        if (m_staging.n < cnt)
        {
            sync();
            m_staging.alloc(cnt);
        }
        return m_staging.ptr;
    }

    // Outputs of a half step (Euler1DCore.cpp:97-100): odd = false writes the
    // odd points 3 .. n - 4, odd = true the even points 2 .. n - 3; either
    // way indices 1 .. nout of the output planes.
    int64_t nout_of(bool odd) const { return odd ? (n - 3) / 2 : (n - 5) / 2; }

    template <int ALPHA, bool SO0, bool CFL, bool BND>
    void half(bool odd)
    {
        int64_t const nout = nout_of(odd);
        if (nout <= 0)
        {
            return;
        }
        if constexpr (SO0 && CFL)
        {
            if (n <= WARP_POINTS32)
            {
                int64_t const warps = (nout + WOUT - 1) / WOUT;
                unsigned const g = static_cast<unsigned>((warps * 32 + B32 - 1) / B32);
                if (odd)
                {
                    k_half32_warp<ALPHA, BND, 0><<<g, B32, 0, stream>>>(args(), nout);
                }
                else
                {
                    k_half32_warp<ALPHA, BND, 1><<<g, B32, 0, stream>>>(args(), nout);
                }
                scg::launched(stream, "e1d_half32_warp");
                return;
            }
        }
        int64_t const threads = nout / 4 + 1;
        unsigned const grid = static_cast<unsigned>((threads + B32 - 1) / B32);
        if (odd)
        {
            k_half32<ALPHA, SO0, CFL, BND, 0><<<grid, B32, 0, stream>>>(args(), nout);
        }
        else
        {
            k_half32<ALPHA, SO0, CFL, BND, 1><<<grid, B32, 0, stream>>>(args(), nout);
        }
        scg::launched(stream, "e1d_half32");
    }

    // update_cfl(odd_plane) (Euler1DCore.cpp:70-94): the kernel points of the
    // half step, the even points 2 .. n - 5 (indices 1 ..) or the odd points
    // 1 .. n - 4 (indices 0 ..).
    void cfl_plane(bool odd)
    {
        int64_t const count = nout_of(odd);
        if (count > 0)
        {
            k_cfl32<<<static_cast<unsigned>((count + 255) / 256), 256, 0, stream>>>(args(), odd ? 1 : 0, odd ? 0 : 1,
                                                                                  count);
            scg::launched(stream, "e1d_cfl32");
        }
    }

    void op(int which, int odd, int alpha) override
    {
        switch (which)
        {
        case 0: // update_cfl
            cfl_plane(odd != 0);
            break;
        case 1: // march_half_so0
            half<0, true, false, false>(odd != 0);
            break;
        case 2: // march_half_so1_alpha
            if (alpha == 1)
                half<1, false, false, false>(odd != 0);
            else
                half<2, false, false, false>(odd != 0);
            break;
        case 3: // treat_boundary_so0
        case 4: // treat_boundary_so1
            k_bnd32<<<1, 1, 0, stream>>>(args(), which == 3 ? PL_SO0 : PL_SO1);
            scg::launched(stream, "e1d_bnd32");
            break;
        case 5: // setup_march
            cfl_plane(false);
            break;
        case 6: // march_half1_alpha
            if (alpha == 1)
                half<1, true, true, false>(false);
            else
                half<2, true, true, false>(false);
            break;
        case 7: // march_half2_alpha
            if (alpha == 1)
                half<1, true, true, false>(true);
            else
                half<2, true, true, false>(true);
            break;
        default:
            throw std::invalid_argument("Euler1DCore: unknown operation " + std::to_string(which));
        }
        sync();
    }

    // One march_alpha step: half 1 with the boundary treatment fused, half 2.
    void step(int alpha)
    {
        if (alpha == 1)
        {
            half<1, true, true, true>(false);
            half<1, true, true, false>(true);
        }
        else
        {
            half<2, true, true, true>(false);
            half<2, true, true, false>(true);
        }
    }

    void march(int alpha, int64_t steps) override
    {
        if (alpha != 1 && alpha != 2)
        {
            throw std::invalid_argument("Euler1DCore: alpha must be 1 or 2");
        }
        if (cluster_march(alpha, steps))
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

    template <int ALPHA>
    bool tube_march(int64_t steps)
    {
        int64_t const nout1 = nout_of(false), nout2 = nout_of(true);
        int blocks, warps;
        if (nout1 <= 0 || !cluster_shape<k_tube32<ALPHA>, TUBE_WARPS32>((n - 1) / 2, blocks, warps))
        {
            return false;
        }
        for (int64_t s = 0; s < steps; s += CLUSTER_STEPS)
        {
            launch_cluster(k_tube32<ALPHA>, blocks, 32 * warps, stream, args(), std::min(CLUSTER_STEPS, steps - s),
                           nout1, nout2);
            scg::launched(stream, "e1d_tube32");
        }
        return true;
    }

    bool cluster_march(int alpha, int64_t steps)
    {
        return alpha == 1 ? tube_march<1>(steps) : tube_march<2>(steps);
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
        scg::g_launches.store(before); // captured, not launched
        scg::cuda_check(cudaStreamEndCapture(stream, &g), "EndCapture");
        scg::cuda_check(cudaGraphInstantiate(&graph_exec, g, 0), "GraphInstantiate");
        cudaGraphDestroy(g);
        graph_alpha = alpha;
    }

    void sync() override { scg::cuda_check(cudaStreamSynchronize(stream), "cudaStreamSynchronize"); }

private:
    static constexpr int GRAPH_STEPS = 32;
    scg::DevBuf<double> coord;
    scg::DevBuf<float> planes;
    int64_t P = 0;
    scg::DevBuf<double> m_staging;
    cudaGraphExec_t graph_exec = nullptr;
    int graph_alpha = 0;
};

} // namespace

struct scg_e1d
{
    std::unique_ptr<Euler1DBase> c;
};

extern "C"
{

int scg_e1d_create(int64_t ncoord, double time_increment, scg_e1d ** out)
{
    return scg_e1d_create_precision(ncoord, time_increment, SCG_FP64, out);
}

int scg_e1d_create_precision(int64_t ncoord, double time_increment, int precision, scg_e1d ** out)
{
    return scg::guarded([&] {
        auto h = std::make_unique<scg_e1d>();
        if (precision == SCG_FP64)
            h->c = std::make_unique<Euler1D>(ncoord, time_increment);
        else if (precision == SCG_FP32)
            h->c = std::make_unique<Euler1D32>(ncoord, time_increment);
        else
            throw std::invalid_argument("Euler1DCore: precision must be SCG_FP64 or SCG_FP32");
        *out = h.release();
    });
}

int scg_e1d_precision(const scg_e1d * h, int * precision)
{
    return scg::guarded([&] { *precision = h->c->precision; });
}

int scg_e1d_destroy(scg_e1d * h)
{
    return scg::guarded([&] { delete h; });
}

int scg_e1d_clone(scg_e1d * h, scg_e1d ** out)
{
    return scg::guarded([&] {
        auto c = std::make_unique<scg_e1d>();
        c->c = h->c->clone();
        *out = c.release();
    });
}

int scg_e1d_info(const scg_e1d * h, int64_t * ncoord, double * time_increment)
{
    return scg::guarded([&] {
        *ncoord = h->c->n;
        *time_increment = h->c->time_increment;
    });
}

int scg_e1d_get(scg_e1d * h, int which, double * host, int64_t count)
{
    return scg::guarded([&] {
        if (count != h->c->count(which))
            throw std::invalid_argument("Euler1DCore: host buffer size mismatch");
        h->c->get(which, host);
    });
}

int scg_e1d_set(scg_e1d * h, int which, const double * host, int64_t count)
{
    return scg::guarded([&] {
        if (count != h->c->count(which))
            throw std::invalid_argument("Euler1DCore: host buffer size mismatch");
        h->c->set(which, host);
    });
}

int scg_e1d_op(scg_e1d * h, int op, int odd_plane, int alpha)
{
    return scg::guarded([&] { h->c->op(op, odd_plane, alpha); });
}

int scg_e1d_march(scg_e1d * h, int alpha, int64_t steps)
{
    return scg::guarded([&] {
        if (steps < 0)
            throw std::invalid_argument("Euler1DCore::march_alpha: steps must be >= 0");
        h->c->march(alpha, steps);
    });
}

int scg_e1d_sync(scg_e1d * h)
{
    return scg::guarded([&] { h->c->sync(); });
}

int scg_e1d_stream(const scg_e1d * h, void ** out)
{
    return scg::guarded([&] { *out = h->c->stream; });
}

} // extern "C"
