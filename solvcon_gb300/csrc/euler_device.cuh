#pragma once

/*
 * Device-side building blocks of the multi-dimensional CESE Euler march.
 *
 * The arithmetic is that of the reference EulerCore (cpp/solvcon/multidim/
 * euler_march.cpp, euler_solution.cpp, euler_gradient.cpp, euler_bc.cpp,
 * GradientElement.cpp) rearranged for a GPU whose FP64 pipe, not its HBM, is
 * the scarce resource:
 *
 *  - The flux Jacobian is never formed.  Every product J_d(u) . w the
 *    reference takes (euler_march.cpp:178-189, 280-292) is the directional
 *    derivative of the Euler flux f_d at u along w, evaluated here directly from
 *    primitive variables (jvp_sum).  Same mathematics, about a third of the
 *    operations.
 *  - The sub-face loop of calc_soln (euler_march.cpp:266-294) is linear in the
 *    sub-face centroids and normals, so each face's sub-faces are folded into
 *    two geometric moments at set-up: N = sum_sf n_sf and
 *    M[e][d] = sum_sf (x_sf - x_j)[e] n_sf[d] (pre-scaled by dt/2).
 *  - The gradient element (GradientElement.cpp:137-213) is linear in tau, so
 *    its displacement vectors are idis = P + tau Q - delta and
 *    jdis = R + tau Q - delta with P, Q, R precomputed per face; for simplices
 *    the sub-element centroid shift delta is exactly zero (the fan of a
 *    simplex about its vertex mean has equal sub-volumes).
 *  - Each fundamental gradient element's 2x2/3x3 solve
 *    (GradientElement.cpp:215-290) uses its inverse's rows once per cell,
 *    instead of an adjugate and determinant per equation.
 *
 * Results equal the reference's up to floating-point round-off.
 *
 * This file holds what both precisions share and the FP32 march's building
 * blocks; euler_fp64.cuh has the FP64 march's.
 *
 * Storage (one record per mesh row, ghost rows first, row = icl + ngstcell):
 *   record[row] = { so0[NEQ], so0t[NEQ], so1[NEQ][ND], terms } padded to RS
 * reals, where terms (FP64 records only) are the row's flux terms: functions
 * of its so0, so1 and so0t that calc_soln reads for each of the row's faces
 * (euler_fp64.cuh).  They are written with so0t, by the same thread and from
 * the same state, so they are valid exactly when so0t is.
 */

#include "divide.cuh"

#include <cstdint>
#include <type_traits>

namespace scg
{
namespace dev
{

template <int ND>
struct Dim
{
    static constexpr int NEQ = ND + 2;
    static constexpr int RS = (ND == 2) ? 16 : 32; // record stride in reals
    static constexpr int OT = NEQ;                 // so0t offset
    static constexpr int O1 = 2 * NEQ;             // so1 offset
    // Cell geometry components: 1/cevol[0], hdt/dist.
    static constexpr int KC = 2;
};

// FP64 geometry rounded once to FP32, when the tables are built: the storage
// of the FP32 form's geometry (precision fp32).  The FP32 march uses every
// geometry value in FP32, so the tables hold the rounding that it would
// otherwise form from an FP64 table at every use, with the same bits and half
// the bytes (see geo_store in euler_setup.cuh).
struct Rounded
{
    float v;
};

// Per-face geometry components, stored as G: bvol, dB[ND] = x_BCE - x_nbr
// (G double: bvol dB), Nh[ND], Mh[ND][ND], then either the gradient-element displacements P[ND],
// Q[ND], R[ND] (geometry computed in FP64: G double or Rounded) or
// mid[ND] = x_BCE - x_cell (fp32-geom32: G float).
// P, Q and R follow from dB and mid with means over the cell's faces:
//   P = mid - mean(mid),  Q = mean(dB) - dB,  R = dB - mean(mid),
// which the fp32-geom32 march forms in registers, in FP32, for 4 (2D) or 6
// (3D) fewer stored values per face; the others read them as formed in FP64.
template <int ND, typename G>
struct Geo
{
    static constexpr bool MID = std::is_same<G, float>::value;
    static constexpr int K_BVOL = 0;
    static constexpr int K_DB = 1;
    static constexpr int K_NH = 1 + ND;
    static constexpr int K_MH = 1 + 2 * ND;
    static constexpr int K_P = 1 + 2 * ND + ND * ND; // FP64-computed geometry
    static constexpr int K_Q = K_P + ND;
    static constexpr int K_R = K_Q + ND;
    static constexpr int K_MID = K_P; // fp32-geom32
    static constexpr int KF = MID ? K_MID + ND : K_R + ND;
};

// Record layout per dimension and state precision.
template <int ND, typename R>
struct Rec
{
    static constexpr int NEQ = ND + 2;
    static constexpr int NUSED = 2 * NEQ + NEQ * ND; // so0, so0t, so1: 16 / 25
    // Flux terms (FP64 only: the FP64 march is bound by the FP64 pipe, the
    // FP32 march by memory, where the extra bytes would cost more); see
    // euler_fp64.cuh.
    static constexpr bool TERMS = sizeof(R) == 8;
    static constexpr int OP = NUSED; // their offset
    static constexpr int NTERM = ND == 2 ? 17 : 39;
    static constexpr int NLOAD = TERMS ? NUSED + NTERM : NUSED;
    // 2D FP64: 33 values in 36 reals (nine whole 32-byte sectors).
    static constexpr int RS = TERMS ? (ND == 2 ? 36 : 64) : (ND == 2 ? 16 : 32);
    static_assert(NLOAD <= RS, "record overflow");
};

// Small constants of the reference, with FP32-safe floors.  The FP64 values
// are the reference's own (euler_march.cpp:30, euler_solution.cpp:108,
// euler_gradient.cpp:28); 1e-60 and 1e-200 underflow in FP32, so the FP32
// march uses the smallest floors that keep the same expressions finite.
template <typename R>
struct Tiny;
template <>
struct Tiny<double>
{
    static constexpr double JAC = 1.e-60;
    static constexpr double CFL = 1.e-60;
    static constexpr double AZ = 1.e-200;
};
template <>
struct Tiny<float>
{
    static constexpr float JAC = 1.e-30f;
    static constexpr float CFL = 1.e-30f;
    static constexpr float AZ = 1.e-37f;
};

// An FP64 geometry value rounded to FP32 for the FP32 form's tables, with
// integer instructions (a double -> float conversion issues on the FP64 pipe).
// In the FP32 normal range the result is IEEE round-to-nearest-even: adding
// 2^28 - 1 plus the kept part's lowest bit to the 64-bit pattern carries
// into bit 29 exactly when the 29 bits to be dropped exceed half, or equal
// half with an odd lowest kept bit; the funnel shift then takes bits 29..60,
// the exponent and the top 23 mantissa bits in place, and subtracting
// (1023 - 127) << 23 modulo 2^32 rebiases the exponent (its high bits
// shifted out cancel).  Values below the FP32 normal range (round-off
// residue in the tables) become a signed zero, by one compare and select.
// Larger ones are not taken here: a core of the FP32 form checks each value
// as it builds its tables and refuses values at 2^128 and beyond, infinities
// and NaNs.
__device__ __forceinline__ float geo_r(double v)
{
    unsigned long long const b = static_cast<unsigned long long>(__double_as_longlong(v));
    unsigned const hi = static_cast<unsigned>(b >> 32);
    unsigned long long const t = b + 0x0FFFFFFFull + ((b >> 29) & 1ull);
    unsigned const r = __funnelshift_l(static_cast<unsigned>(t), static_cast<unsigned>(t >> 32), 3) - 0xC0000000u;
    return __uint_as_float(((hi & 0x7FF00000u) >= (897u << 20) ? r : 0u) | (hi & 0x80000000u));
}

// The geometry values geo_r takes: magnitudes below 2^128 (biased exponent
// up to 1150).
__device__ __forceinline__ bool geo_r_takes(double v)
{
    unsigned const e = (static_cast<unsigned>(__double2hiint(v)) >> 20) & 0x7FFu;
    return e <= 1150u;
}

// The FP32 march's reciprocals and quotients.  2D: the approximate quotient
// (div.approx.f32, one instruction and within 2 ulp for divisors of magnitude
// in [2^-126, 2^126]; a zero divisor gives a signed infinity, or NaN over
// zero, as the division does), where a correctly rounded FP32 division is a
// multi-instruction sequence with a branch and the 2D march divides about a
// dozen times per cell-substep by densities, determinants, weight sums and
// CFL numbers, all far inside that range (2M triangles: 0.2352 -> 0.2155 ms
// per launch).  3D: the division (with the approximate quotient the
// tetrahedron kernel ran 6.45 -> 8.59 ms per launch at the same registers,
// scheduled differently).
template <int ND>
__device__ __forceinline__ float mrecip(float d)
{
    if constexpr (ND == 2)
        return __fdividef(1.0f, d);
    else
        return 1.0f / d;
}
template <int ND>
__device__ __forceinline__ float mquot(float x, float y)
{
    if constexpr (ND == 2)
        return __fdividef(x, y);
    else
        return x / y;
}

// Compensated (Kahan) accumulator for the FP32 flux sums.
struct Acc
{
    float s = 0.f;
    float c = 0.f;
    __device__ __forceinline__ void add(float x)
    {
        float const y = x - c;
        float const t = s + y;
        c = (t - s) - y;
        s = t;
    }
    __device__ __forceinline__ float value() const { return s; }
};

// Primitive quantities of a conserved state u (with the reference's density
// floor TINY, euler_march.cpp:41).
template <int ND, typename R>
struct Prim
{
    R r;     // 1 / (rho + TINY)
    R v[ND]; // velocity
    R p;     // pressure
    R h;     // E + p
    R ga1;   // gamma - 1
    R vsq;   // |v|^2

    __device__ __forceinline__ Prim(R const * u, R ga) : Prim(u, ga, mrecip<ND>(u[0] + Tiny<R>::JAC)) {}

    // With 1/(rho + TINY) already at hand.
    __device__ __forceinline__ Prim(R const * u, R ga, R rinv)
    {
        constexpr int NEQ = ND + 2;
        r = rinv;
        R ke2 = R(0);
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            v[d] = u[1 + d] * r;
            ke2 += u[1 + d] * v[d];
        }
        vsq = ke2 * r;
        ga1 = ga - R(1);
        p = ga1 * (u[NEQ - 1] - R(0.5) * ke2);
        h = u[NEQ - 1] + p;
    }
};

// out[i] = sum_d f_d(u)[i] * n[d]  (the flux of euler_march.cpp:58-61, 120-124).
template <int ND, typename R>
__device__ __forceinline__ void flux_dot(Prim<ND, R> const & q, R const * u, R const * n, R * out)
{
    constexpr int NEQ = ND + 2;
    R mn = R(0);
    R vn = R(0);
#pragma unroll
    for (int d = 0; d < ND; ++d)
    {
        mn += u[1 + d] * n[d];
        vn += q.v[d] * n[d];
    }
    out[0] = mn;
#pragma unroll
    for (int k = 0; k < ND; ++k)
    {
        out[1 + k] = u[1 + k] * vn + q.p * n[k];
    }
    out[NEQ - 1] = q.h * vn;
}

// out[i] += sum_d (J_d(u) . w[:, d])[i], with w indexed w[i * ND + d].  J_d is
// the analytic Euler flux Jacobian of euler_march.cpp:63-81 / 126-156; its
// product with w is taken as the directional derivative of f_d.
template <int ND, typename R>
__device__ __forceinline__ void jvp_sum(Prim<ND, R> const & q, R const * u, R const * w, R * out)
{
    constexpr int NEQ = ND + 2;
#pragma unroll
    for (int d = 0; d < ND; ++d)
    {
        R const w0 = w[0 * ND + d];
        R const we = w[(NEQ - 1) * ND + d];
        R vw = R(0);
#pragma unroll
        for (int k = 0; k < ND; ++k)
        {
            vw += q.v[k] * w[(1 + k) * ND + d];
        }
        R const dp = q.ga1 * (we - vw + R(0.5) * q.vsq * w0);
        R const dvd = (w[(1 + d) * ND + d] - q.v[d] * w0) * q.r;
        out[0] += w[(1 + d) * ND + d];
#pragma unroll
        for (int k = 0; k < ND; ++k)
        {
            out[1 + k] += w[(1 + k) * ND + d] * q.v[d] + u[1 + k] * dvd;
        }
        out[1 + d] += dp;
        out[NEQ - 1] += (we + dp) * q.v[d] + q.h * dvd;
    }
}

// so0t = -(J . so1) for one row (euler_march.cpp:160-191), from the row's
// primitives q.
template <int ND, typename R>
__device__ __forceinline__ void solt_prim(Prim<ND, R> const & q, R const * u, R const * g, R * t)
{
    constexpr int NEQ = ND + 2;
    R o[NEQ];
#pragma unroll
    for (int i = 0; i < NEQ; ++i)
    {
        o[i] = R(0);
    }
    jvp_sum<ND, R>(q, u, g, o);
#pragma unroll
    for (int i = 0; i < NEQ; ++i)
    {
        t[i] = -o[i];
    }
}

// Fundamental gradient element tables (1-based in GradientElement.cpp:
// 16-79, 0-based here), per cell type.
template <int CT>
struct CellT;

template <>
struct CellT<4> // triangle
{
    static constexpr int ND = 2, NFC = 3, NFGE = 3;
    static constexpr bool SIMPLEX = true;
    __device__ static constexpr int fge(int k, int v)
    {
        constexpr int t[3][2] = {{0, 1}, {1, 2}, {2, 0}};
        return t[k][v];
    }
};
template <>
struct CellT<3> // quadrilateral
{
    static constexpr int ND = 2, NFC = 4, NFGE = 4;
    static constexpr bool SIMPLEX = false;
    __device__ static constexpr int fge(int k, int v)
    {
        constexpr int t[4][2] = {{0, 1}, {1, 2}, {2, 3}, {3, 0}};
        return t[k][v];
    }
};
template <>
struct CellT<6> // tetrahedron
{
    static constexpr int ND = 3, NFC = 4, NFGE = 4;
    static constexpr bool SIMPLEX = true;
    __device__ static constexpr int fge(int k, int v)
    {
        constexpr int t[4][3] = {{2, 0, 1}, {1, 0, 3}, {3, 0, 2}, {1, 3, 2}};
        return t[k][v];
    }
};
template <>
struct CellT<5> // hexahedron
{
    static constexpr int ND = 3, NFC = 6, NFGE = 8;
    static constexpr bool SIMPLEX = false;
    __device__ static constexpr int fge(int k, int v)
    {
        constexpr int t[8][3] = {{1, 2, 4}, {5, 2, 1}, {3, 2, 5}, {4, 2, 3},
                                 {4, 0, 1}, {1, 0, 5}, {5, 0, 3}, {3, 0, 4}};
        return t[k][v];
    }
};
template <>
struct CellT<7> // prism
{
    static constexpr int ND = 3, NFC = 5, NFGE = 6;
    static constexpr bool SIMPLEX = false;
    __device__ static constexpr int fge(int k, int v)
    {
        constexpr int t[6][3] = {{4, 1, 3}, {2, 1, 4}, {3, 1, 2}, {3, 0, 4}, {4, 0, 2}, {2, 0, 3}};
        return t[k][v];
    }
};
template <>
struct CellT<8> // pyramid
{
    static constexpr int ND = 3, NFC = 5, NFGE = 6;
    static constexpr bool SIMPLEX = false;
    __device__ static constexpr int fge(int k, int v)
    {
        constexpr int t[6][3] = {{0, 4, 1}, {1, 4, 2}, {2, 4, 3}, {3, 4, 0}, {0, 2, 3}, {2, 0, 1}};
        return t[k][v];
    }
};

// Determinant of the rows a, b (, c).
template <int ND, typename R>
__device__ __forceinline__ R det_rows(R const * a, R const * b, R const * c)
{
    if constexpr (ND == 2)
    {
        (void)c;
        return a[0] * b[1] - a[1] * b[0];
    }
    else
    {
        return a[0] * (b[1] * c[2] - b[2] * c[1]) - a[1] * (b[0] * c[2] - b[2] * c[0]) +
               a[2] * (b[0] * c[1] - b[1] * c[0]);
    }
}

// Kernel argument block shared by the march kernels.
template <typename R, typename G>
struct MarchArgs
{
    R const * cur;        // current records (so0c, so0t, so1c)
    R * nxt;              // new records (so0n, next so0t, so1n)
    R const * gamma;      // [nrow]
    R * cflo;             // [nrow]
    R * cflc;             // [nrow]
    G const * geo;        // [tile of GEO_TILE cells][npl][GEO_TILE], see GeoView
    int32_t const * nbr;  // [NSLOT][ncell] neighbour row
    int8_t const * ctype; // [ncell]
    int8_t const * gkind; // [ngst] BC kind of the ghost row, -1 if none
    double const * gnml;  // [ngst][ND] outward unit normal of the boundary face
    double const * gval;  // [ngst][NEQ] inlet conserved state
    uint8_t * limiter;    // [ncell] W-3/4 firing bits per equation, or null
    // Host blocks (mapped) that also receive every row's new so0n
    // [nrow][NEQ] and so1n [nrow][NEQ][ND] in FP64, or null.
    double * out0;
    double * out1;
    // FP32 march: the rounding residual of each body cell's so0 [NEQ][ncell],
    // fed back into the cell's next value (see fused_cell), or null.
    R * comp;
    int64_t ncell;
    int64_t ngst;
    int64_t npl; // geometry values per cell, KC + slots * KF
    R dt, hdt, qdt;
    R sigma0, taumin, tauscale;
};

template <typename T>
__device__ __forceinline__ T ldg(T const * p)
{
    return __ldg(p);
}

// One cell's geometry values.  The tables are kept in tiles of 32 consecutive
// cells, tile-major: value (plane) k of cell i lies at
//   ((i / 32) npl + k) 32 + i % 32,
// so a warp's loads of one plane are one contiguous piece, and all the values
// of a warp's cells are one too (6 KB for the FP32 form's triangles), which the
// FP32 march copies to shared memory at once (SHARED: p points there).
constexpr int GEO_TILE = 32;

template <typename G, bool SHARED = false>
struct GeoView
{
    G const * p; // the cell's value 0

    __device__ __forceinline__ auto at(int k) const
    {
        if constexpr (std::is_same<G, Rounded>::value)
        {
            float const * const q = &p[k * GEO_TILE].v;
            return SHARED ? *q : ldg(q);
        }
        else
        {
            G const * const q = p + k * GEO_TILE;
            return SHARED ? *q : ldg(q);
        }
    }
};

template <typename R, typename G>
__device__ __forceinline__ GeoView<G> geo_view(MarchArgs<R, G> const & a, int64_t icl)
{
    return GeoView<G>{a.geo + (icl / GEO_TILE) * a.npl * GEO_TILE + icl % GEO_TILE};
}

// Value k of face f, and per-cell value k.
template <int ND, typename G, bool SH>
__device__ __forceinline__ auto fg(GeoView<G, SH> const & gv, int f, int k)
{
    return gv.at(Dim<ND>::KC + f * Geo<ND, G>::KF + k);
}
template <int ND, typename G, bool SH>
__device__ __forceinline__ auto cg(GeoView<G, SH> const & gv, int k)
{
    return gv.at(k);
}

} // namespace dev
} // namespace scg
