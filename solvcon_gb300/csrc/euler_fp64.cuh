#pragma once

/*
 * The FP64 march's per-cell routines: calc_soln, calc_cfl, calc_dsoln and
 * calc_solt of the reference EulerCore (cpp/solvcon/multidim/euler_march.cpp,
 * euler_solution.cpp, euler_gradient.cpp, GradientElement.cpp), arranged for
 * the fewest instructions on the FP64 pipe, which bounds these kernels: with
 * the pipe full a warp's FP64 instruction takes an SM 19 cycles (64 on its
 * sub-partition alone), and all instructions together fill 14 to 23% of the
 * issue slots.
 *
 *  - Flux terms once per cell instead of once per face.  calc_soln's temporal
 *    flux through a face from neighbour j is
 *      sum_d [ f_d(u) + dt/4 J_d u_t ] . N_d + sum_{d,e} [ J_d u_,e ] M_ed,
 *    whose brackets depend on cell j alone.  They are formed by the thread
 *    that makes j's so0t (which is -sum_d J_d u_,d, a sum of some of them) and
 *    kept in j's record; a face then costs (1 + ND) (1 + ND) NEQ fused
 *    multiply-adds, all straight into the sums.  Of the NEQ ND components per
 *    bracket the mass row is the momentum's own (kept in so1) and the momentum
 *    rows are symmetric, so 17 (2D) or 39 (3D) values are kept.
 *  - Triangles and tetrahedra: the displacements of a cell's ND + 1 faces sum
 *    to zero, so all its gradient elements have one determinant, and with the
 *    rows c_f of the inverse over the first ND faces and s the sum of the
 *    solution deltas over all faces, the gradient without face m is
 *    g - s c_m, g = sum_f delta_f c_f being the one without the last face.
 *    The weights sum to one, so their mean needs only g, s and the c_m.
 *  - Reciprocals, roots and comparisons, the gradient elements' norms and
 *    weights, and in 2D some products on the integer pipe (divide.cuh,
 *    weights64).
 *
 * FP64-pipe instructions per cell-substep (ncu), with the neighbours' fluxes
 * formed per face and all of this on the FP64 pipe -> now: triangle 743 -> 340,
 * tetrahedron 1,701 -> 903, hexahedron 3,060 -> 1,903; 500k triangles 694 -> 326 us
 * per launch, 384k tetrahedra 1,199 -> 648 us.
 *
 * Every operation is written as the instruction it is (fused multiply-add,
 * multiply, add), so the kernels that inline these routines (one cell type or
 * any, one mesh or a batch) give the same bits however they are compiled.
 */

#include "euler_device.cuh"

namespace scg
{
namespace dev
{

__device__ __forceinline__ double fm(double a, double b, double c) { return __fma_rn(a, b, c); }
__device__ __forceinline__ double mu(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double ad(double a, double b) { return __dadd_rn(a, b); }
// A product of the loop over equations, E of them: in 2D on the integer pipe,
// the same bits (2M triangles 1252 -> 1198 us, 490,000 quadrilaterals 465 -> 453);
// in 3D the longer loop costs more (64,000 hexahedra 285 -> 310), as it does
// outside the loop (1198 -> 1280 with the flux terms' products).
template <int ND, int E>
__device__ __forceinline__ double mx(double a, double b)
{
    return ND == 2 && E > 1 ? mul_int(a, b) : mu(a, b);
}
__device__ __forceinline__ double sb(double a, double b) { return __dsub_rn(a, b); }

// Layout of a record's flux terms: the time-centred fluxes A_d (f_d + dt/4 J_d
// u_t) of mass, momentum (symmetric) and energy, then the flux gradients
// B_{d,e} = J_d u_,e of momentum and energy (those of mass are so1's).
template <int ND>
struct FluxTerms
{
    static constexpr int NS = ND * (ND + 1) / 2;
    static constexpr int A0 = 0;
    static constexpr int AM = ND;
    static constexpr int AE = AM + NS;
    static constexpr int BM = AE + ND;
    static constexpr int BE = BM + NS * ND;
    static constexpr int N = BE + ND * ND;
    // Place of the momentum pair (k, l) among the NS.
    __host__ __device__ static constexpr int sym(int k, int l)
    {
        int const a = k < l ? k : l;
        int const b = k < l ? l : k;
        return a * ND - a * (a - 1) / 2 + b - a;
    }
};

// Primitive variables of a conserved state, rinv = 1 / (rho + TINY).
template <int ND>
struct Prim64
{
    double r, v[ND], p, h, hv, ga1; // hv = |v|^2 / 2

    __device__ __forceinline__ Prim64(double const * u, double ga, double rinv)
    {
        r = rinv;
        v[0] = mu(u[1], r);
        double ke2 = mu(u[1], v[0]);
#pragma unroll
        for (int d = 1; d < ND; ++d)
        {
            v[d] = mu(u[1 + d], r);
            ke2 = fm(u[1 + d], v[d], ke2);
        }
        hv = mu(mu(0.5, ke2), r);
        ga1 = sb(ga, 1.0);
        p = mu(ga1, fm(-0.5, ke2, u[ND + 1]));
        h = ad(u[ND + 1], p);
    }
};

// The change of velocity (dv), pressure and enthalpy (h = E + p) along a
// change w of the conserved state, w[i * S].
template <int ND, int S>
__device__ __forceinline__ void prim_change(Prim64<ND> const & q, double const * w, double * dv, double & dp,
                                            double & dh)
{
    double const w0 = w[0];
    double const we = w[(ND + 1) * S];
    double s = fm(q.hv, w0, we);
#pragma unroll
    for (int k = 0; k < ND; ++k)
    {
        double const wk = w[(1 + k) * S];
        s = fm(-q.v[k], wk, s);
        dv[k] = mu(fm(-q.v[k], w0, wk), q.r);
    }
    dp = mu(q.ga1, s);
    dh = ad(we, dp);
}

// Flux gradients B of a row from its state u and gradients g[i * ND + e].
template <int ND>
__device__ __forceinline__ void flux_gradients(Prim64<ND> const & q, double const * u, double const * g, double * c)
{
    using F = FluxTerms<ND>;
#pragma unroll
    for (int e = 0; e < ND; ++e)
    {
        double dv[ND], dp, dh;
        prim_change<ND, ND>(q, g + e, dv, dp, dh);
#pragma unroll
        for (int k = 0; k < ND; ++k)
        {
            double const gk = g[(1 + k) * ND + e];
#pragma unroll
            for (int l = k; l < ND; ++l)
            {
                double const x = k == l ? fm(gk, q.v[l], dp) : mu(gk, q.v[l]);
                c[F::BM + F::sym(k, l) * ND + e] = fm(u[1 + k], dv[l], x);
            }
            c[F::BE + k * ND + e] = fm(q.h, dv[k], mu(dh, q.v[k]));
        }
    }
}

// Time-centred fluxes A of a row from its state u and time derivative t.
template <int ND>
__device__ __forceinline__ void centred_fluxes(Prim64<ND> const & q, double const * u, double const * t, double qdt,
                                               double * c)
{
    using F = FluxTerms<ND>;
    constexpr int NEQ = ND + 2;
    double w[NEQ]; // the state's change over dt / 4
#pragma unroll
    for (int i = 0; i < NEQ; ++i)
    {
        w[i] = mu(qdt, t[i]);
    }
    double dv[ND], dp, dh;
    prim_change<ND, 1>(q, w, dv, dp, dh);
    double const p = ad(q.p, dp);
    double const h = ad(q.h, dh);
#pragma unroll
    for (int k = 0; k < ND; ++k)
    {
        double const m = ad(u[1 + k], w[1 + k]);
        c[F::A0 + k] = m;
#pragma unroll
        for (int l = k; l < ND; ++l)
        {
            double const x = k == l ? fm(m, q.v[l], p) : mu(m, q.v[l]);
            c[F::AM + F::sym(k, l)] = fm(u[1 + k], dv[l], x);
        }
        c[F::AE + k] = fm(q.h, dv[k], mu(h, q.v[k]));
    }
}

// calc_solt (euler_march.cpp:160-191) and the flux terms of one row.
template <int ND>
__device__ __forceinline__ void solt_terms(double const * u, double const * g, double ga, double rinv, double qdt,
                                           double * t, double * c)
{
    using F = FluxTerms<ND>;
    Prim64<ND> const q(u, ga, rinv);
    flux_gradients<ND>(q, u, g, c);
    double t0 = g[ND];
    double te = c[F::BE];
#pragma unroll
    for (int d = 1; d < ND; ++d)
    {
        t0 = ad(t0, g[(1 + d) * ND + d]);
        te = ad(te, c[F::BE + d * ND + d]);
    }
    t[0] = -t0;
    t[ND + 1] = -te;
#pragma unroll
    for (int k = 0; k < ND; ++k)
    {
        double s = c[F::BM + F::sym(k, 0) * ND];
#pragma unroll
        for (int d = 1; d < ND; ++d)
        {
            s = ad(s, c[F::BM + F::sym(k, d) * ND + d]);
        }
        t[1 + k] = -s;
    }
    centred_fluxes<ND>(q, u, t, qdt, c);
}

template <int ND>
__device__ __forceinline__ void solt_terms(double const * u, double const * g, double ga, double qdt, double * t,
                                           double * c)
{
    solt_terms<ND>(u, g, ga, recip(ad(u[0], Tiny<double>::JAC)), qdt, t, c);
}

// Load the reals [FROM, TO) of a record (whole aligned pairs).
template <int FROM, int TO>
__device__ __forceinline__ void load_part(double const * base, double * out)
{
#pragma unroll
    for (int k = FROM / 2; k < (TO + 1) / 2; ++k)
    {
        double2 const v = __ldg(reinterpret_cast<double2 const *>(base) + k);
        out[2 * k] = v.x;
        out[2 * k + 1] = v.y;
    }
}

// Store a record: so0, so0t, so1 and the flux terms c.
template <int ND>
__device__ __forceinline__ void store_row(double * base, double const * so0, double const * so0t, double const * so1,
                                          double const * c)
{
    using RC = Rec<ND, double>;
    constexpr int NEQ = ND + 2;
    double v[RC::RS];
#pragma unroll
    for (int i = 0; i < RC::RS; ++i)
    {
        v[i] = i < NEQ ? so0[i]
                       : (i < 2 * NEQ ? so0t[i - NEQ]
                                      : (i < RC::NUSED ? so1[i - 2 * NEQ] : (i < RC::NLOAD ? c[i - RC::OP] : 0.0)));
    }
#pragma unroll
    for (int k = 0; k < (RC::NLOAD + 1) / 2; ++k)
    {
        reinterpret_cast<double2 *>(base)[k] = make_double2(v[2 * k], v[2 * k + 1]);
    }
}

// Whether calc_soln adds the neighbours' so0 times their volumes, most of the
// sum, after all faces' flux and gradient terms instead of face by face: the
// NFC ND (ND + 2) terms then round at their own magnitude and not at the sum's.
// The same operations in another order.  Face by face, a march's error against
// plain 64-bit torch was larger than with every face summed on its own, by 6%
// (so0) and 8% (so1) over 6 steps of 1,728 hexahedra and 2% and 3% of 3,600
// quadrilaterals; in this order it is 0 to 3% smaller.  Face by face -> last, per
// substep: 490k quadrilaterals 448.6 -> 449.2 us, 384k tetrahedra 652.5 -> 652.6, 64k
// hexahedra 285.1 -> 285.3, 65k prisms 255.4 -> 256.7, small meshes alike.  Triangles,
// of the fewest terms, showed no such difference, and would take 1,199 -> 1,212 us
// (2M).
template <int CT>
__host__ __device__ constexpr bool volumes_last()
{
    return !(CellT<CT>::ND == 2 && CellT<CT>::SIMPLEX);
}

// calc_soln of one body cell (euler_march.cpp:197-303).  TERMS: the neighbours'
// records hold their flux terms (the march); else they are formed here from
// each neighbour's so0, so0t and so1 (calc_soln on its own, whose so0t is the
// caller's).
template <int CT, bool TERMS>
__device__ __forceinline__ void soln64(MarchArgs<double, double> const & a, int64_t icl, double * so0n)
{
    constexpr int ND = CellT<CT>::ND;
    constexpr int NEQ = ND + 2;
    constexpr int NFC = CellT<CT>::NFC;
    using D = Geo<ND, double>;
    using RC = Rec<ND, double>;
    using F = FluxTerms<ND>;
    GeoView<double> const gv = geo_view(a, icl);
    double acc[NEQ];
#pragma unroll
    for (int i = 0; i < NEQ; ++i)
    {
        acc[i] = -0.0; // -0 + a = a, zeros of both signs too
    }
    // Not unrolled, as the loops over faces and equations of calc_dsoln (which
    // index uf in local memory for it): a substep's instructions in one stretch
    // are more than the instruction caches hold, and FP64 tetrahedra and
    // hexahedra waited for them a fifth of the time.  384k tetrahedra 740 ->
    // 688 us, 64k hexahedra 323 -> 298, 128k prisms 510 -> 440, 490k quadrilaterals
    // 527 -> 490, 2M triangles 1348 -> 1331; most of it from the equations' loop.
#pragma unroll 1
    for (int f = 0; f < NFC; ++f)
    {
        int64_t const jr = __ldg(a.nbr + f * a.ncell + icl);
        double const * const base = a.cur + jr * RC::RS;
        double rec[RC::RS];
        double ct[TERMS ? 1 : F::N];
        double const * c;
        if constexpr (TERMS)
        {
            if constexpr (!volumes_last<CT>())
            {
                load_part<0, NEQ>(base, rec);
            }
            load_part<2 * NEQ, RC::NLOAD>(base, rec);
            c = rec + RC::OP;
        }
        else
        {
            load_part<0, RC::NUSED>(base, rec);
            Prim64<ND> const q(rec, __ldg(a.gamma + jr), recip(ad(rec[0], Tiny<double>::JAC)));
            flux_gradients<ND>(q, rec, rec + 2 * NEQ, ct);
            centred_fluxes<ND>(q, rec, rec + NEQ, a.qdt, ct);
            c = ct;
        }
        double const * const g = rec + 2 * NEQ;
        if constexpr (!volumes_last<CT>())
        {
            double const bvol = fg<ND>(gv, f, D::K_BVOL);
#pragma unroll
            for (int i = 0; i < NEQ; ++i)
            {
                acc[i] = fm(bvol, rec[i], acc[i]);
            }
        }
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            double const vb = fg<ND>(gv, f, D::K_DB + d);
            double const nh = fg<ND>(gv, f, D::K_NH + d);
            acc[0] = fm(-c[F::A0 + d], nh, fm(vb, g[d], acc[0]));
            acc[NEQ - 1] = fm(-c[F::AE + d], nh, fm(vb, g[(NEQ - 1) * ND + d], acc[NEQ - 1]));
#pragma unroll
            for (int k = 0; k < ND; ++k)
            {
                acc[1 + k] = fm(-c[F::AM + F::sym(k, d)], nh, fm(vb, g[(1 + k) * ND + d], acc[1 + k]));
            }
        }
#pragma unroll
        for (int e = 0; e < ND; ++e)
        {
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                double const m = fg<ND>(gv, f, D::K_MH + e * ND + d);
                acc[0] = fm(-g[(1 + d) * ND + e], m, acc[0]);
                acc[NEQ - 1] = fm(-c[F::BE + d * ND + e], m, acc[NEQ - 1]);
#pragma unroll
                for (int k = 0; k < ND; ++k)
                {
                    acc[1 + k] = fm(-c[F::BM + F::sym(k, d) * ND + e], m, acc[1 + k]);
                }
            }
        }
    }
    if constexpr (volumes_last<CT>())
    {
#pragma unroll 1
        for (int f = 0; f < NFC; ++f)
        {
            int64_t const jr = __ldg(a.nbr + f * a.ncell + icl);
            double u[NEQ + 1];
            load_part<0, NEQ>(a.cur + jr * RC::RS, u);
            double const bvol = fg<ND>(gv, f, D::K_BVOL);
#pragma unroll
            for (int i = 0; i < NEQ; ++i)
            {
                acc[i] = fm(bvol, u[i], acc[i]);
            }
        }
    }
    double const ivol = cg<ND>(gv, 0);
#pragma unroll
    for (int i = 0; i < NEQ; ++i)
    {
        so0n[i] = mu(acc[i], ivol);
    }
}

// calc_cfl of one body cell (euler_solution.cpp:106-160); rinv = 1 / (rho +
// TINY), which the reference's three divisions by rho share (the floor changes
// nothing unless rho is below 1e-44, where the reference itself overflows).
template <int ND>
__device__ __forceinline__ double cfl64(MarchArgs<double, double> const & a, int64_t icl, int64_t row, double * so0n,
                                        double & rinv)
{
    constexpr int NEQ = ND + 2;
    double const ga = __ldg(a.gamma + row);
    double const ga1 = sb(ga, 1.0);
    double const ri = recip(ad(so0n[0], Tiny<double>::JAC));
    rinv = ri;
    double momsq = mu(so0n[1], so0n[1]);
#pragma unroll
    for (int d = 1; d < ND; ++d)
    {
        momsq = fm(so0n[1 + d], so0n[1 + d], momsq);
    }
    double const ke = mu(mu(0.5, momsq), ri);
    double const pr = mu(ga1, sb(so0n[NEQ - 1], ke));
    // (pr + |pr|) / 2: pr, zero for a negative one, NaN for -infinity and NaN.
    unsigned const hp = static_cast<unsigned>(__double2hiint(pr));
    bool const neg = hp >= 0x80000000u;
    double pra = neg ? (hp >= 0xfff00000u ? __longlong_as_double(0x7ff8000000000000ll) : 0.0) : pr;
    double const wspd = fm(sqr_t(momsq), ri, sqr_t(mu(mu(ga, pra), ri)));
    double const cflo = mu(wspd, cg<ND>(geo_view(a, icl), 1));
    // pra / (pra + TINY) is exactly 1 whenever TINY does not change pra, as it
    // does not above 1e-43: the division is taken only below.
    double f = 1.0;
    if (static_cast<unsigned>(__double2hiint(pra)) < 0x37100000u)
    {
        f = pra / ad(pra, Tiny<double>::CFL);
    }
    double const cflc = fm(sb(cflo, 1.0), f, 1.0);
    a.cflo[row] = cflo;
    a.cflc[row] = cflc;
    // The reference stores pra/ga1 + ke + TINY, which for pr > 0 is E + TINY
    // (= E to working precision).
    if (!(static_cast<unsigned long long>(__double_as_longlong(pr)) - 1ull < 0x7ff0000000000000ull))
    {
        so0n[NEQ - 1] = pra / ga1 + ke + Tiny<double>::CFL;
    }
    return cflc;
}

// The W-3/4 cap (euler_gradient.cpp:60-108) of one equation: the gradient
// elements' weights w (inverse gradient magnitudes) become their deviations
// from their mean, u_k, and the result c gives the reference's weights
// 1/n + c u_k.  Scaled by wacc = sum w, the three caps are quotients of known
// sign, T1 = (1 - 1/n) / (max u + TINY wacc), T2 = (1/n) / (TINY wacc - min u)
// and T0 = sigma0 / (|cfl| wacc): the smaller of the first two is chosen by
// cross-multiplication, so is whether it is below T0 (it fires), and only the
// chosen quotient is divided out.
template <int N>
__device__ __forceinline__ double cap64(double * w, double acfl, double sigma0, bool & fire)
{
    double wacc = w[0];
#pragma unroll
    for (int k = 1; k < N; ++k)
    {
        wacc = ad(wacc, w[k]);
    }
    double const wq = mu(1.0 / N, wacc);
    double umax = 0.0;
    double umin = -0.0;
#pragma unroll
    for (int k = 0; k < N; ++k)
    {
        w[k] = sb(w[k], wq);
        umax = max_pos(umax, w[k]);
        umin = min_neg(umin, w[k]);
    }
    double const d1 = fm(Tiny<double>::AZ, wacc, umax);
    double const d2 = fm(Tiny<double>::AZ, wacc, -umin);
    bool const first = !lt_nonneg(d1, mu(double(N - 1), d2));
    double const nn = first ? 1.0 - 1.0 / N : 1.0 / N;
    double const dd = first ? d1 : d2;
    double const cw = mu(acfl, wacc);
    fire = lt_nonneg(mu(nn, cw), mu(sigma0, dd));
    return mu(fire ? nn : sigma0, recip(fire ? dd : cw));
}

// The weights of N gradient elements from their squared magnitudes sq in FP64,
// for operands weights64 does not take.
template <int N>
__device__ __noinline__ bool weights64_plain(double const * sq, double acfl, double sigma0, double * wt)
{
    for (int k = 0; k < N; ++k)
    {
        wt[k] = rsq(sq[k]);
    }
    bool fire;
    double const cc = cap64<N>(wt, acfl, sigma0, fire);
    for (int k = 0; k < N; ++k)
    {
        wt[k] = fm(cc, wt[k], 1.0 / N);
    }
    return fire;
}

// n 2^e for n in [2^63, 2^64), rounded to the nearest double (a half away from
// zero; rounding up to 2^64 carries into the exponent).
__device__ __forceinline__ double compose(unsigned long long n, int e)
{
    return __longlong_as_double(
        static_cast<long long>((n >> 11) + ((n >> 10) & 1ull) + (static_cast<unsigned long long>(1085 + e) << 52)));
}

// The same weights, 1/N + (N-1)/N U_k / max(t S, M), in integers but for one
// multiplication: w_k = w[k] 2^(-62 - h[k]), the inverse gradient magnitudes
// (inverse_norm), aligned to the largest of them, S their sum,
// U_k = N w_k - S, M = max(max U, (N-1) max(-U)), and t = (N-1) acfl / sigma0; the
// cap fires where t S < M.  This is cap64's 1/N + cc (w_k - mean w) with the
// common factors taken out, and w_k's scale with them.  The smallest bit kept
// is 2^-57 of the largest w, a sixteenth of its rounding in FP64.  For t in
// 2^[-400, 400) (cap_in_range).  Some 180 integer
// instructions for 15 FP64 ones (N = 3; 19 at 4, 31 at 8); substep 2M triangles
// 1527 -> 1330 us, 490,000 quadrilaterals 568 -> 524, 384,000 tetrahedra 783 -> 737,
// 64,000 hexahedra 328 -> 322.
__device__ __forceinline__ bool cap_in_range(double t)
{
    return (static_cast<unsigned>(__double2hiint(t)) >> 20) - 623u <= 799u;
}
template <int N>
__device__ __forceinline__ bool weights64(unsigned long long * w, int const * h, double t, double * wt)
{
    // (N-1) N 2^(62-P) < 2^63.
    constexpr int P = N <= 3 ? 2 : (N == 4 ? 3 : (N <= 6 ? 4 : 5));
    static_assert(N <= 8, "P");
    int low = h[0];
#pragma unroll
    for (int k = 1; k < N; ++k)
    {
        low = min(low, h[k]);
    }
    unsigned long long sum = 0;
#pragma unroll
    for (int k = 0; k < N; ++k)
    {
        w[k] = w[k] >> min(P + h[k] - low, 63);
        sum += w[k];
    }
    long long u[N], most = 0, least = 0;
#pragma unroll
    for (int k = 0; k < N; ++k)
    {
        u[k] = static_cast<long long>(w[k] * N - sum);
        most = u[k] > most ? u[k] : most;
        least = u[k] < least ? u[k] : least;
    }
    long long const side = -least * (N - 1);
    unsigned long long const big = static_cast<unsigned long long>(side > most ? side : most);
    int const ls = __clzll(static_cast<long long>(sum));
    double const ts = mu(t, compose(sum << ls, -ls));
    // max(t S, M) = n 2^(e - 63) with n in [2^63, 2^64).
    unsigned const th = static_cast<unsigned>(__double2hiint(ts));
    unsigned long long n = sig53(th, static_cast<unsigned>(__double2loint(ts))) << 11;
    int e = static_cast<int>(th >> 20) - 1023;
    int const lb = __clzll(static_cast<long long>(big));
    unsigned long long const nb = big << (lb & 63);
    int const eb = big == 0 ? -2000 : 63 - lb;
    bool const fire = eb > e || (eb == e && nb > n);
    n = fire ? nb : n;
    e = fire ? eb : e;
    n += n < 0ull - 1024ull ? 1024ull : 0ull; // to 53 bits, to the nearest
    unsigned long long r = rcp_sig(static_cast<unsigned>(n >> 43), static_cast<unsigned>(n >> 11)); // 2^62 / (n 2^-63)
    r -= r / N;
    // |u_k| < 2^(e + 1), so that u_k 2^(61 - e) fits; zero where e < 0.
    int const left = min(max(61 - e, 0), 63), right = min(max(e - 61, 0), 63);
#pragma unroll
    for (int k = 0; k < N; ++k)
    {
        bool const neg = u[k] < 0;
        unsigned long long const m = static_cast<unsigned long long>(neg ? -u[k] : u[k]) << left >> right;
        long long const q = static_cast<long long>(mul_hi64(m, r)); // 2^59
        long long const v = static_cast<long long>((1ull << 59) / N) + (neg ? -q : q);
        int const lv = __clzll(v);
        wt[k] = v > 0 ? compose(static_cast<unsigned long long>(v) << lv, -59 - lv) : 0.0;
    }
    return fire;
}

// What calc_dsoln reads of a neighbour's record for equations q .. q + E - 1:
// their so0 and so0t (u, t) and gradients (g).
template <int ND, int E>
struct RowPart
{
    double u[E], t[E], g[E * ND];

    __device__ __forceinline__ RowPart(double const * base, int q)
    {
        constexpr int NEQ = ND + 2;
        if constexpr (E == NEQ)
        {
            double rec[Rec<ND, double>::NUSED + 1];
            load_part<0, Rec<ND, double>::NUSED>(base, rec);
#pragma unroll
            for (int i = 0; i < NEQ; ++i)
            {
                u[i] = rec[i];
                t[i] = rec[NEQ + i];
            }
#pragma unroll
            for (int k = 0; k < NEQ * ND; ++k)
            {
                g[k] = rec[2 * NEQ + k];
            }
        }
        else
        {
#pragma unroll
            for (int i = 0; i < E; ++i)
            {
                u[i] = __ldg(base + q + i);
                t[i] = __ldg(base + NEQ + q + i);
            }
#pragma unroll
            for (int k = 0; k < E * ND; ++k)
            {
                g[k] = __ldg(base + 2 * NEQ + q * ND + k);
            }
        }
    }
};

// calc_dsoln of one body cell (euler_gradient.cpp:23-130 with the gradient
// element of GradientElement.cpp:137-290) for equations q .. q + E - 1 (so0n
// and so1n: theirs): a triangle or tetrahedron.  Returns their firing bits.
template <int CT, int E>
__device__ __forceinline__ unsigned dsoln64_simplex(MarchArgs<double, double> const & a, int64_t icl, int q,
                                                    double const * so0n, double cflc, double * so1n)
{
    constexpr int ND = CellT<CT>::ND;
    constexpr int N = ND + 1; // faces, and gradient elements
    using D = Geo<ND, double>;
    using RC = Rec<ND, double>;
    constexpr int UF = E > 1 ? 1 : N;
    double const acfl = fabs(cflc);
    double const ts = mu(mu(acfl, double(N - 1)), recip(a.sigma0));
    double const tau = fm(acfl, a.tauscale, a.taumin);
    GeoView<double> const gv = geo_view(a, icl);
    // Solution deltas at the evaluation points: of the first ND faces, and
    // their sum over all.
    double uf[ND][E], us[E];
#pragma unroll
    for (int i = 0; i < E; ++i)
    {
        us[i] = -0.0;
    }
#pragma unroll UF
    for (int f = 0; f < N; ++f)
    {
        int64_t const jr = __ldg(a.nbr + f * a.ncell + icl);
        RowPart<ND, E> const r(a.cur + jr * RC::RS, q);
        double jd[ND];
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            jd[d] = fm(tau, fg<ND>(gv, f, D::K_Q + d), fg<ND>(gv, f, D::K_R + d));
        }
#pragma unroll
        for (int i = 0; i < E; ++i)
        {
            double s = sb(fm(a.hdt, r.t[i], r.u[i]), so0n[i]);
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                s = fm(jd[d], r.g[i * ND + d], s);
            }
            if (f < ND)
            {
                uf[f][i] = s;
            }
            us[i] = ad(us[i], s);
        }
    }
    double x[ND][ND]; // displacements of the first ND faces
#pragma unroll
    for (int f = 0; f < ND; ++f)
    {
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            x[f][d] = fm(tau, fg<ND>(gv, f, D::K_Q + d), fg<ND>(gv, f, D::K_P + d));
        }
    }
    // Columns of the inverse of the displacement rows.
    double c[ND][ND];
    if constexpr (ND == 2)
    {
        double const inv = recip(fm(x[0][0], x[1][1], -mu(x[0][1], x[1][0])));
        c[0][0] = mu(x[1][1], inv);
        c[0][1] = mu(-x[1][0], inv);
        c[1][0] = mu(-x[0][1], inv);
        c[1][1] = mu(x[0][0], inv);
    }
    else
    {
#pragma unroll
        for (int m = 0; m < 3; ++m)
        {
            double const * const b = x[(m + 1) % 3];
            double const * const e = x[(m + 2) % 3];
            c[m][0] = fm(b[1], e[2], -mu(b[2], e[1]));
            c[m][1] = fm(b[2], e[0], -mu(b[0], e[2]));
            c[m][2] = fm(b[0], e[1], -mu(b[1], e[0]));
        }
        double const inv = recip(fm(x[0][0], c[0][0], fm(x[0][1], c[0][1], mu(x[0][2], c[0][2]))));
#pragma unroll
        for (int m = 0; m < 3; ++m)
        {
#pragma unroll
            for (int d = 0; d < 3; ++d)
            {
                c[m][d] = mu(c[m][d], inv);
            }
        }
    }
    unsigned fired = 0;
#pragma unroll 1
    for (int i = 0; i < E; ++i)
    {
        // Element m < ND leaves out face m, element ND the last face.
        double g[ND], w[N];
        unsigned long long r[N];
        int h[N];
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            double s = mx<ND, E>(uf[0][i], c[0][d]);
#pragma unroll
            for (int f = 1; f < ND; ++f)
            {
                s = fm(uf[f][i], c[f][d], s);
            }
            g[d] = s;
        }
        bool fixed = cap_in_range(ts);
        fixed = inverse_norm<ND>(g, r[ND], h[ND]) && fixed; // W-1/2: inverse gradient magnitude
#pragma unroll
        for (int m = 0; m < ND; ++m)
        {
            double s[ND];
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                s[d] = fm(-us[i], c[m][d], g[d]);
            }
            fixed = inverse_norm<ND>(s, r[m], h[m]) && fixed;
        }
        bool fire;
        if (fixed)
        {
            fire = weights64<N>(r, h, ts, w);
        }
        else
        {
            double sq[N], wp[N];
#pragma unroll
            for (int m = 0; m < N; ++m)
            {
                sq[m] = Tiny<double>::AZ;
#pragma unroll
                for (int d = 0; d < ND; ++d)
                {
                    double const s = m < ND ? fm(-us[i], c[m < ND ? m : 0][d], g[d]) : g[d];
                    sq[m] = fm(s, s, sq[m]);
                }
            }
            fire = weights64_plain<N>(sq, acfl, a.sigma0, wp);
#pragma unroll
            for (int m = 0; m < N; ++m)
            {
                w[m] = wp[m];
            }
        }
        fired |= fire ? 1u << (q + i) : 0u;
        // sum_k w_k g_k, the weights summing to one.
#pragma unroll
        for (int m = 0; m < ND; ++m)
        {
            double const ws = mx<ND, E>(w[m], us[i]);
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                g[d] = fm(-ws, c[m][d], g[d]);
            }
        }
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            so1n[i * ND + d] = g[d];
        }
    }
    return fired;
}

// a x b, from the stored product of the lower- and higher-numbered face: each
// pair of faces is shared by two gradient elements.
template <int CT>
struct FacePairs
{
    static constexpr int NFC = CellT<CT>::NFC;
    double v[NFC * (NFC - 1) / 2][3];
    __device__ static constexpr int at(int f, int g)
    {
        return f < g ? f * NFC - f * (f + 1) / 2 + g - f - 1 : g * NFC - g * (g + 1) / 2 + f - g - 1;
    }
    __device__ __forceinline__ void form(double const x[][3], int f, int g)
    {
        double const * const b = x[f < g ? f : g];
        double const * const e = x[f < g ? g : f];
        double * const o = v[at(f, g)];
        o[0] = fm(b[1], e[2], -mu(b[2], e[1]));
        o[1] = fm(b[2], e[0], -mu(b[0], e[2]));
        o[2] = fm(b[0], e[1], -mu(b[1], e[0]));
    }
    __device__ __forceinline__ double get(int f, int g, int d) const { return f < g ? v[at(f, g)][d] : -v[at(f, g)][d]; }
};

// Determinants of the gradient elements' displacement rows.
template <int CT>
__device__ __forceinline__ void dets64(double const x[][CellT<CT>::ND], FacePairs<CT> & pr, double * det)
{
    constexpr int ND = CellT<CT>::ND;
    constexpr int NFGE = CellT<CT>::NFGE;
    if constexpr (ND == 3)
    {
#pragma unroll
        for (int k = 0; k < NFGE; ++k)
        {
#pragma unroll
            for (int v = 0; v < 3; ++v)
            {
                pr.form(x, CellT<CT>::fge(k, v), CellT<CT>::fge(k, (v + 1) % 3));
            }
        }
    }
#pragma unroll
    for (int k = 0; k < NFGE; ++k)
    {
        int const f0 = CellT<CT>::fge(k, 0);
        int const f1 = CellT<CT>::fge(k, 1);
        if constexpr (ND == 2)
        {
            det[k] = fm(x[f0][0], x[f1][1], -mu(x[f0][1], x[f1][0]));
        }
        else
        {
            int const f2 = CellT<CT>::fge(k, 2);
            det[k] = fm(x[f0][0], pr.get(f1, f2, 0),
                        fm(x[f0][1], pr.get(f1, f2, 1), mu(x[f0][2], pr.get(f1, f2, 2))));
        }
    }
}

// calc_dsoln of one body cell that is no simplex, for equations q .. q + E - 1.
template <int CT, int E>
__device__ __forceinline__ unsigned dsoln64_general(MarchArgs<double, double> const & a, int64_t icl, int q,
                                                    double const * so0n, double cflc, double * so1n)
{
    constexpr int ND = CellT<CT>::ND;
    constexpr int NFC = CellT<CT>::NFC;
    constexpr int NFGE = CellT<CT>::NFGE;
    using D = Geo<ND, double>;
    using RC = Rec<ND, double>;
    constexpr int UF = E > 1 ? 1 : NFC;
    double const acfl = fabs(cflc);
    double const ts = mu(mu(acfl, double(NFGE - 1)), recip(a.sigma0));
    double const tau = fm(acfl, a.tauscale, a.taumin);
    GeoView<double> const gv = geo_view(a, icl);
    double x[NFC][ND];
#pragma unroll
    for (int f = 0; f < NFC; ++f)
    {
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            x[f][d] = fm(tau, fg<ND>(gv, f, D::K_Q + d), fg<ND>(gv, f, D::K_P + d));
        }
    }
    FacePairs<CT> pr;
    double det[NFGE];
    double delta[ND];
    {
        // Sub-element centroid of the gradient element about the vertex mean
        // (calc_gge_centroid, GradientElement.cpp:81-133).
        dets64<CT>(x, pr, det);
        double voc = det[0];
#pragma unroll
        for (int k = 1; k < NFGE; ++k)
        {
            voc = ad(voc, det[k]);
        }
        double const inv = recip(mu(voc, double(ND + 1)));
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            // Each face's displacement times the sum of its elements' volumes.
            double s = 0.0;
#pragma unroll
            for (int f = 0; f < NFC; ++f)
            {
                double vf = 0.0;
                bool any = false;
#pragma unroll
                for (int k = 0; k < NFGE; ++k)
                {
#pragma unroll
                    for (int v = 0; v < ND; ++v)
                    {
                        if (CellT<CT>::fge(k, v) == f)
                        {
                            vf = any ? ad(vf, det[k]) : det[k];
                            any = true;
                        }
                    }
                }
                s = f == 0 ? mu(x[f][d], vf) : fm(x[f][d], vf, s);
            }
            delta[d] = mu(s, inv);
        }
#pragma unroll
        for (int f = 0; f < NFC; ++f)
        {
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                x[f][d] = sb(x[f][d], delta[d]);
            }
        }
    }
    // Solution deltas at the evaluation points.
    double uf[NFC][E];
#pragma unroll UF
    for (int f = 0; f < NFC; ++f)
    {
        int64_t const jr = __ldg(a.nbr + f * a.ncell + icl);
        RowPart<ND, E> const r(a.cur + jr * RC::RS, q);
        double jd[ND];
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            jd[d] = sb(fm(tau, fg<ND>(gv, f, D::K_Q + d), fg<ND>(gv, f, D::K_R + d)), delta[d]);
        }
#pragma unroll
        for (int i = 0; i < E; ++i)
        {
            double s = sb(fm(a.hdt, r.t[i], r.u[i]), so0n[i]);
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                s = fm(jd[d], r.g[i * ND + d], s);
            }
            uf[f][i] = s;
        }
    }
    // Columns of each element's inverse: grad = sum_v uf[v] C[k][v].
    dets64<CT>(x, pr, det);
    double C[NFGE][ND][ND];
#pragma unroll
    for (int k = 0; k < NFGE; ++k)
    {
        double const inv = recip(det[k]);
        int const f0 = CellT<CT>::fge(k, 0);
        int const f1 = CellT<CT>::fge(k, 1);
        if constexpr (ND == 2)
        {
            C[k][0][0] = mu(x[f1][1], inv);
            C[k][0][1] = mu(-x[f1][0], inv);
            C[k][1][0] = mu(-x[f0][1], inv);
            C[k][1][1] = mu(x[f0][0], inv);
        }
        else
        {
            int const f2 = CellT<CT>::fge(k, 2);
#pragma unroll
            for (int d = 0; d < 3; ++d)
            {
                C[k][0][d] = mu(pr.get(f1, f2, d), inv);
                C[k][1][d] = mu(pr.get(f2, f0, d), inv);
                C[k][2][d] = mu(pr.get(f0, f1, d), inv);
            }
        }
    }
    unsigned fired = 0;
#pragma unroll 1
    for (int i = 0; i < E; ++i)
    {
        double g[NFGE][ND], w[NFGE];
        unsigned long long r[NFGE];
        int h[NFGE];
        bool fixed = cap_in_range(ts);
#pragma unroll
        for (int k = 0; k < NFGE; ++k)
        {
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                double s = mx<ND, E>(uf[CellT<CT>::fge(k, 0)][i], C[k][0][d]);
#pragma unroll
                for (int v = 1; v < ND; ++v)
                {
                    s = fm(uf[CellT<CT>::fge(k, v)][i], C[k][v][d], s);
                }
                g[k][d] = s;
            }
            fixed = inverse_norm<ND>(g[k], r[k], h[k]) && fixed; // W-1/2: inverse gradient magnitude
        }
        bool fire;
        if (fixed)
        {
            fire = weights64<NFGE>(r, h, ts, w);
        }
        else
        {
            double sq[NFGE], wp[NFGE];
#pragma unroll
            for (int k = 0; k < NFGE; ++k)
            {
                sq[k] = Tiny<double>::AZ;
#pragma unroll
                for (int d = 0; d < ND; ++d)
                {
                    sq[k] = fm(g[k][d], g[k][d], sq[k]);
                }
            }
            fire = weights64_plain<NFGE>(sq, acfl, a.sigma0, wp);
#pragma unroll
            for (int k = 0; k < NFGE; ++k)
            {
                w[k] = wp[k];
            }
        }
        fired |= fire ? 1u << (q + i) : 0u;
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            double s = mx<ND, E>(w[0], g[0][d]);
#pragma unroll
            for (int k = 1; k < NFGE; ++k)
            {
                s = fm(w[k], g[k][d], s);
            }
            so1n[i * ND + d] = s;
        }
    }
    return fired;
}

template <int CT, int E>
__device__ __forceinline__ unsigned dsoln64_part(MarchArgs<double, double> const & a, int64_t icl, int q,
                                                 double const * so0n, double cflc, double * so1n)
{
    if constexpr (CellT<CT>::SIMPLEX)
    {
        return dsoln64_simplex<CT, E>(a, icl, q, so0n, cflc, so1n);
    }
    else
    {
        return dsoln64_general<CT, E>(a, icl, q, so0n, cflc, so1n);
    }
}

template <int CT>
__device__ __forceinline__ void dsoln64(MarchArgs<double, double> const & a, int64_t icl, double const * so0n,
                                        double cflc, double * so1n)
{
    unsigned const fired = dsoln64_part<CT, CellT<CT>::ND + 2>(a, icl, 0, so0n, cflc, so1n);
    if (a.limiter)
    {
        a.limiter[icl] = static_cast<uint8_t>(fired);
    }
}

// ---------------------------------------------------------------------------
// One substep of a cell by LPC lanes, one equation each, for meshes too small to
// fill the GPU.  An FP64 instruction takes a warp 64 cycles however many of its
// lanes work, on its SM sub-partition's pipe, and the GPU has 608 of those: a
// thousand cells at a thread each are 32 warps in which hundreds of
// instructions follow one another.  Lane q takes equation q of calc_soln and
// calc_dsoln; what all equations share (the gradient elements' geometry, the CFL
// number, the flux terms) every lane forms for itself; the lanes of the faces
// 0, 1, ... do the boundary work.  The operations and their order are those of
// the one-thread routines, so the results are the same bits.
template <int ND>
struct Split
{
    static constexpr int LPC = ND == 2 ? 4 : 8; // lanes per cell (equations 0 .. NEQ - 1, the rest repeat the last)
};

// Equation q of calc_soln (soln64<CT, true>).
template <int CT>
__device__ __forceinline__ double soln64_eq(MarchArgs<double, double> const & a, int64_t icl, int q)
{
    constexpr int ND = CellT<CT>::ND;
    constexpr int NEQ = ND + 2;
    using D = Geo<ND, double>;
    using RC = Rec<ND, double>;
    using F = FluxTerms<ND>;
    GeoView<double> const gv = geo_view(a, icl);
    // Where the record keeps this equation's A_d and B_{d,e}.
    int oa[ND], ob[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d)
    {
        int const k = q - 1;
        int const lo = k < d ? k : d, hi = k < d ? d : k;
        int const sym = lo * ND - lo * (lo - 1) / 2 + hi - lo;
        oa[d] = RC::OP + (q == 0 ? F::A0 + d : (q == NEQ - 1 ? F::AE + d : F::AM + sym));
        ob[d] = q == 0 ? 2 * NEQ + (1 + d) * ND : RC::OP + (q == NEQ - 1 ? F::BE + d * ND : F::BM + sym * ND);
    }
    constexpr int NFC = CellT<CT>::NFC;
    double acc = -0.0, bvol[NFC], u[NFC];
#pragma unroll
    for (int f = 0; f < NFC; ++f)
    {
        int64_t const jr = __ldg(a.nbr + f * a.ncell + icl);
        double const * const base = a.cur + jr * RC::RS;
        bvol[f] = fg<ND>(gv, f, D::K_BVOL);
        u[f] = __ldg(base + q);
        if constexpr (!volumes_last<CT>())
        {
            acc = fm(bvol[f], u[f], acc);
        }
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            double const vb = fg<ND>(gv, f, D::K_DB + d);
            double const nh = fg<ND>(gv, f, D::K_NH + d);
            acc = fm(-__ldg(base + oa[d]), nh, fm(vb, __ldg(base + 2 * NEQ + q * ND + d), acc));
        }
#pragma unroll
        for (int e = 0; e < ND; ++e)
        {
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                acc = fm(-__ldg(base + ob[d] + e), fg<ND>(gv, f, D::K_MH + e * ND + d), acc);
            }
        }
    }
    if constexpr (volumes_last<CT>())
    {
#pragma unroll
        for (int f = 0; f < NFC; ++f)
        {
            acc = fm(bvol[f], u[f], acc);
        }
    }
    return mu(acc, cg<ND>(gv, 0));
}

} // namespace dev
} // namespace scg
