#pragma once

/*
 * The CESE march kernels of the multi-dimensional Euler core: per-cell device
 * routines for calc_soln, bc_soln, calc_cfl, calc_dsoln, bc_dsoln and calc_solt,
 * the fused one-kernel substep built from them, and the set-up kernels
 * (prepare_ce and the geometry compaction).  See euler_device.cuh for the data
 * layout and for how the arithmetic relates to the reference's, and
 * euler_fp64.cuh for the FP64 march's own routines.
 */

#include "euler_device.cuh"
#include "euler_fp64.cuh"

#include <type_traits>

namespace scg
{
namespace dev
{

// Load the first N reals of an FP32 record (default: so0, so0t, so1).
template <int ND, int N = Rec<ND, float>::NUSED>
__device__ __forceinline__ void load_rec(float const * base, float * out)
{
    float4 const * p = reinterpret_cast<float4 const *>(base);
#pragma unroll
    for (int k = 0; k < N / 4; ++k)
    {
        float4 const v = __ldg(p + k);
        out[4 * k] = v.x;
        out[4 * k + 1] = v.y;
        out[4 * k + 2] = v.z;
        out[4 * k + 3] = v.w;
    }
#pragma unroll
    for (int k = (N / 4) * 4; k < N; ++k)
    {
        out[k] = __ldg(base + k);
    }
}

// Store an FP32 record: so0, so0t, so1.
template <int ND>
__device__ __forceinline__ void store_rec(float * base, float const * so0, float const * so0t, float const * so1)
{
    constexpr int NEQ = ND + 2;
    constexpr int N = Rec<ND, float>::NUSED;
    float v[N];
#pragma unroll
    for (int i = 0; i < NEQ; ++i)
    {
        v[i] = so0[i];
        v[NEQ + i] = so0t[i];
    }
#pragma unroll
    for (int i = 0; i < NEQ * ND; ++i)
    {
        v[2 * NEQ + i] = so1[i];
    }
    float4 * p = reinterpret_cast<float4 *>(base);
#pragma unroll
    for (int k = 0; k < N / 4; ++k)
    {
        p[k] = make_float4(v[4 * k], v[4 * k + 1], v[4 * k + 2], v[4 * k + 3]);
    }
#pragma unroll
    for (int k = (N / 4) * 4; k < N; ++k)
    {
        base[k] = v[k];
    }
}

// What calc_soln hands to calc_dsoln of the same cell when the neighbour
// records are not gathered twice (FP32 triangles and tetrahedra; see
// min_blocks for the register budget that makes it pay): the solution change at
// face f's gradient-evaluation point is linear in tau,
//   u_j + hdt ut_j + jdis . g_j - u_i  with  jdis = A_f + tau B_f,
// so calc_soln, holding neighbour j's record, keeps
//   p[f] = u_j + hdt ut_j + A_f . g_j  and  q[f] = B_f . g_j
// per equation.  A_f = dB_f - mean(mid), B_f = mean(dB) - dB_f where the tables
// hold mid (fp32-geom32), else the stored R_f and Q_f; delta is zero for simplices.
// Whether the fused substep of cell type CT carries calc_soln's neighbour
// terms to calc_dsoln (FP32 simplices) instead of gathering again.
template <int CT>
__host__ __device__ constexpr bool carries()
{
    return CellT<CT>::SIMPLEX;
}

// Resident blocks of BLOCK threads to ask of the compiler for the fused kernel
// of cell type CT (0: any mix), from the registers per thread that were fastest
// with what the kernel stages (Stage); 0 keeps the one-argument launch bound.
// Per launch, at BLOCK = 128:
//  FP32 form, 2M triangles 156 us at 112 registers, 233 at 96 (spills);
//  fp32-geom32 136 at 80, 138 at 96, 149 at 128.  1.3M tetrahedra 245 us at 128,
//  246 at 96.  490k quadrilaterals 58.7 / 55.7 us (FP32 form / fp32-geom32) at
//  112, 60.9 / 54.3 at 96, 64.8 / 55.4 at 80.  176k hexahedra 82 us at 168, 90 at
//  128, 98 at 254.  Any mix: 176k hexahedra 99 us at 168, 105 at 128, 118 at the
//  243 that the compiler takes; 490k quadrilaterals 62 at 96, 66 at its 126.
//  FP64: enough warps to keep the FP64 pipes fed through their loads, spilling
//  for it where a cell has many faces: 64k hexahedra 284 us at 128 (with its
//  spills), 325 at 168, 314 at 255; 128k prisms (any mix) 430 at 168, 432 at 128,
//  441 at 255; 384k tetrahedra 648 at 128, 657 at the 138 that the compiler takes,
//  655 at 102; 490k quadrilaterals (any mix) 446 at 102, 451 at 124; triangles
//  the same from 85 to 106.
// A batch's tiles of 256 round the quotient down, so the budgets there are looser:
// 128 registers for 96 to 128, none (one block, 255) for 168.  It does not
// cost: 12 meshes of 1,024 to 16,000 prisms (any mix) 41.4 us per substep in
// tiles of 256 against 44.9 in tiles of 128 (FP64 299 against 355), 12 of 512 to
// 13,824 hexahedra 45.6 against 47.6 (FP64 349 against 391).
template <int ND, typename R, int CT, int BLOCK, typename G = R>
__host__ __device__ constexpr int min_blocks()
{
    constexpr int regs = sizeof(R) == 8 ? (CT == 5 || CT == 6  ? 128
                                             : CT == 0 && ND == 3 ? 168
                                             : CT == 0            ? 102
                                                                  : 0)
                         : CT == 0      ? (ND == 2 ? 96 : 168)
                         : CT == 5      ? 168
                         : CT == 6      ? 128
                         : CT == 3      ? (Geo<ND, G>::MID ? 96 : 112)
                                        : (Geo<ND, G>::MID ? 80 : 112);
    return regs > 0 ? 65536 / (BLOCK * regs) : 0;
}

template <int ND, int NFC, typename R>
struct Carry
{
    R mm[ND];
    R mb[ND];
    R p[NFC][ND + 2];
    R q[NFC][ND + 2];
};

// The same sums kept in shared memory instead of registers: one slot per
// thread and component, component-major (SB threads apart), so a warp's
// accesses fall in distinct banks; each thread reads only its own slots, so
// no barrier is needed.  Used for tetrahedra (40 floats per cell), where it
// frees registers at the same budget: 24.6M tetrahedra 6.70 -> 6.44 ms per
// launch at 128 registers (at 96 registers it spills and loses); for
// triangles (24 floats) it was slower at every budget (2D, 2M cells: 0.2356
// ms in registers, 0.2451 / 0.2505 / 0.2734 ms at 96 / 80 / 72 registers).
// The single-mesh and batched kernels carry the same way, so a batched core
// gives the same bits as its own march.
template <int ND>
__host__ __device__ constexpr bool carry_shared()
{
    return ND == 3;
}
template <int ND, int NFC, typename R, int SB>
struct CarrySh
{
    struct Row
    {
        R * b;
        __device__ __forceinline__ R & operator[](int i) const { return b[i * SB]; }
    };
    struct Tab
    {
        R * b;
        __device__ __forceinline__ Row operator[](int f) const { return Row{b + f * (ND + 2) * SB}; }
    };
    R mm[ND];
    R mb[ND];
    Tab p;
    Tab q;
};

// Face means of mid and dB where the tables hold mid (fp32-geom32), else zeros.
template <int CT, typename R, typename G, bool SH>
__device__ __forceinline__ void face_means(GeoView<G, SH> const & gv, R * mm, R * mb)
{
    constexpr int ND = CellT<CT>::ND;
    constexpr int NFC = CellT<CT>::NFC;
    using D = Geo<ND, G>;
#pragma unroll
    for (int d = 0; d < ND; ++d)
    {
        mm[d] = R(0);
        mb[d] = R(0);
    }
    if constexpr (D::MID)
    {
#pragma unroll
        for (int f = 0; f < NFC; ++f)
        {
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                mm[d] += fg<ND>(gv, f, D::K_MID + d);
                mb[d] += fg<ND>(gv, f, D::K_DB + d);
            }
        }
        R const inv = R(1) / R(NFC);
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            mm[d] *= inv;
            mb[d] *= inv;
        }
    }
}

// ---------------------------------------------------------------------------
// calc_soln for one body cell (euler_march.cpp:197-303): the CESE flux
// integral over the cell's BCEs, divided by the CCE volume.
//
// FP32.  With u0 (the cell's own current state; the march) the neighbour
// values enter as differences from u0 and d0 receives so0n - u0: the absolute
// rounding then scales with the change, not with the state (the gradients
// calc_dsoln forms from these differences are O(h) of the state).
// recs.load(f, rec) gives the record of face f's neighbour, nbr[f] its row.
template <int CT, typename R, typename G, bool SH, typename RS, typename CA = Carry<CellT<CT>::ND, CellT<CT>::NFC, R>>
__device__ __forceinline__ void soln_cell(MarchArgs<R, G> const & a, GeoView<G, SH> const & gv, int32_t const * nbr,
                                          RS & recs, R * so0n, CA * carry = nullptr, R const * u0 = nullptr,
                                          R * d0 = nullptr)
{
    constexpr int ND = CellT<CT>::ND;
    constexpr int NEQ = ND + 2;
    constexpr int NFC = CellT<CT>::NFC;
    using D = Geo<ND, G>;
    using RC = Rec<ND, R>;
    Acc acc[NEQ];
#pragma unroll
    for (int f = 0; f < NFC; ++f)
    {
        int64_t const jr = nbr[f];
        R rec[RC::NUSED];
        recs.load(f, rec);
        R const * u = rec;
        R const * t = rec + NEQ;
        R const * g = rec + 2 * NEQ;
        R const ga = ldg(a.gamma + jr);

        R const bvol = fg<ND>(gv, f, D::K_BVOL);
        R dB[ND], nh[ND], qn[ND];
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            dB[d] = fg<ND>(gv, f, D::K_DB + d);
            nh[d] = fg<ND>(gv, f, D::K_NH + d);
            qn[d] = a.qdt * nh[d];
        }
        if (carry)
        {
            R A[ND], B[ND];
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                if constexpr (D::MID)
                {
                    A[d] = dB[d] - carry->mm[d];
                    B[d] = carry->mb[d] - dB[d];
                }
                else
                {
                    A[d] = fg<ND>(gv, f, D::K_R + d);
                    B[d] = fg<ND>(gv, f, D::K_Q + d);
                }
            }
#pragma unroll
            for (int i = 0; i < NEQ; ++i)
            {
                R pp = (u0 ? u[i] - u0[i] : u[i]) + a.hdt * t[i];
                R qq = R(0);
#pragma unroll
                for (int d = 0; d < ND; ++d)
                {
                    pp += A[d] * g[i * ND + d];
                    qq += B[d] * g[i * ND + d];
                }
                carry->p[f][i] = pp;
                carry->q[f][i] = qq;
            }
        }
        // Spatial flux: neighbour solution at the BCE centroid times its volume.
#pragma unroll
        for (int i = 0; i < NEQ; ++i)
        {
            R s = u0 ? u[i] - u0[i] : u[i];
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                s += dB[d] * g[i * ND + d];
            }
            acc[i].add(s * bvol);
        }
        // Temporal flux: sum over sub-faces folded into Nh and Mh.
        R w[NEQ * ND];
#pragma unroll
        for (int i = 0; i < NEQ; ++i)
        {
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                R s = t[i] * qn[d];
#pragma unroll
                for (int e = 0; e < ND; ++e)
                {
                    s += g[i * ND + e] * fg<ND>(gv, f, D::K_MH + e * ND + d);
                }
                w[i * ND + d] = s;
            }
        }
        Prim<ND, R> const q(u, ga);
        R fl[NEQ];
        flux_dot<ND, R>(q, u, nh, fl);
        jvp_sum<ND, R>(q, u, w, fl);
#pragma unroll
        for (int i = 0; i < NEQ; ++i)
        {
            acc[i].add(-fl[i]);
        }
    }
    R const ivol = cg<ND>(gv, 0);
#pragma unroll
    for (int i = 0; i < NEQ; ++i)
    {
        if (u0)
        {
            // Delta form: the CCE volume is the sum of the BCE volumes, so
            // sum_f bvol_f u0 / cevol = u0 and only the change is summed.
            d0[i] = acc[i].value() * ivol;
            so0n[i] = u0[i] + d0[i];
        }
        else
        {
            so0n[i] = acc[i].value() * ivol;
        }
    }
}

// calc_cfl for one body cell in FP32 (euler_solution.cpp:106-160): original and
// clamped CFL, and the energy rewritten from the non-negative pressure.  The
// reference's three divisions by rho use one reciprocal 1/(rho + TINY) (the
// floor changes nothing unless rho is below 1e-23); it is returned in rinv for the
// primitives of the same state.
template <int ND, typename R, typename G, bool SH>
__device__ __forceinline__ R cfl_cell(MarchArgs<R, G> const & a, GeoView<G, SH> const & gv, int64_t row, R * so0n, R & rinv)
{
    constexpr int NEQ = ND + 2;
    R const ga = ldg(a.gamma + row);
    R const ga1 = ga - R(1);
    R const ri = mrecip<ND>(so0n[0] + Tiny<R>::JAC);
    rinv = ri;
    R momsq = R(0);
#pragma unroll
    for (int d = 0; d < ND; ++d)
    {
        momsq += so0n[1 + d] * so0n[1 + d];
    }
    R const ke = R(0.5) * momsq * ri;
    R const pr = ga1 * (so0n[NEQ - 1] - ke);
    R const pra = (pr + fabs(pr)) / R(2);
    R const wspd = sqr_t(ga * pra * ri) + sqr_t(momsq) * ri;
    R const cflo = wspd * cg<ND>(gv, 1);
    // pra / (pra + TINY) is exactly 1 whenever TINY does not change pra (any
    // pressure above ~1e-44 in FP64), so the division is taken only below.
    R const prt = pra + Tiny<R>::CFL;
    R const cflc = (cflo - R(1)) * (prt == pra ? R(1) : pra / prt) + R(1);
    a.cflo[row] = cflo;
    a.cflc[row] = cflc;
    // The reference stores pra/ga1 + ke + TINY.  For pr > 0 that is exactly
    // E + TINY (= E to working precision); re-forming it would only add a
    // rounding error to the energy every substep, which matters in FP32.
    if (!(pr > R(0)))
    {
        so0n[NEQ - 1] = pra / ga1 + ke + Tiny<R>::CFL;
    }
    return cflc;
}

// calc_dsoln for one body cell (euler_gradient.cpp:23-130 with the gradient
// element of GradientElement.cpp:137-290): per fundamental gradient element
// solve, W-1/2 weights, W-3/4 cap, weighted sum.  The neighbour records are
// gathered a second time (calc_soln just read them, so the loads hit in
// cache); carrying calc_soln's neighbour terms over instead costs more FP64
// operations, but pays in FP32 for simplices (carry != nullptr, see Carry).
template <int CT, typename R, typename G, bool SH, typename CA = Carry<CellT<CT>::ND, CellT<CT>::NFC, R>>
__device__ __forceinline__ void dsoln_cell(MarchArgs<R, G> const & a, GeoView<G, SH> const & gv, int64_t icl, R const * so0n, R cflc,
                                           R * so1n, CA const * carry = nullptr,
                                           R const * u0 = nullptr, R const * d0 = nullptr)
{
    constexpr int ND = CellT<CT>::ND;
    constexpr int NEQ = ND + 2;
    constexpr int NFC = CellT<CT>::NFC;
    constexpr int NFGE = CellT<CT>::NFGE;
    using D = Geo<ND, G>;

    R const acfl = fabs(cflc);
    R const sgm0 = mquot<ND>(a.sigma0, acfl);
    R const tau = a.taumin + acfl * a.tauscale;
    R const ofg1 = R(1) / R(NFGE);

    // Gradient-evaluation displacements: idis = dst - delta, dst = P + tau Q.
    // In fp32-geom32 P = mid - mean(mid) and Q = mean(dB) - dB are formed
    // here from the face means (the faces' values are read again rather than
    // held: they hit in L1, and registers bound this kernel's occupancy).
    R mm[ND], mb[ND];
    if (carry)
    {
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            mm[d] = carry->mm[d];
            mb[d] = carry->mb[d];
        }
    }
    else
    {
        face_means<CT, R>(gv, mm, mb);
    }
    R idis[NFC][ND];
#pragma unroll
    for (int f = 0; f < NFC; ++f)
    {
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            if constexpr (D::MID)
            {
                idis[f][d] = (fg<ND>(gv, f, D::K_MID + d) - mm[d]) +
                             tau * (mb[d] - fg<ND>(gv, f, D::K_DB + d));
            }
            else
            {
                idis[f][d] = fg<ND>(gv, f, D::K_P + d) + tau * fg<ND>(gv, f, D::K_Q + d);
            }
        }
    }
    R delta[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d)
    {
        delta[d] = R(0);
    }
    if constexpr (!CellT<CT>::SIMPLEX)
    {
        // Sub-element centroid of the gradient element about the vertex mean
        // (calc_gge_centroid, GradientElement.cpp:81-133).
        R voc = R(0);
#pragma unroll
        for (int k = 0; k < NFGE; ++k)
        {
            int const f0 = CellT<CT>::fge(k, 0);
            int const f1 = CellT<CT>::fge(k, 1);
            int const f2 = (ND == 3) ? CellT<CT>::fge(k, ND - 1) : f1;
            R const vob = det_rows<ND, R>(idis[f0], idis[f1], idis[f2]);
            voc += vob;
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                R s = idis[f0][d] + idis[f1][d];
                if constexpr (ND == 3)
                {
                    s += idis[f2][d];
                }
                delta[d] += s * vob;
            }
        }
        R const inv = mrecip<ND>(voc * R(ND + 1));
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            delta[d] *= inv;
        }
#pragma unroll
        for (int f = 0; f < NFC; ++f)
        {
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                idis[f][d] -= delta[d];
            }
        }
    }

    // Solution deltas at the evaluation points: uf[f][i].
    R uf[NFC][NEQ];
    if (carry)
    {
#pragma unroll
        for (int f = 0; f < NFC; ++f)
        {
#pragma unroll
            for (int i = 0; i < NEQ; ++i)
            {
                // carry->p already has the cell's own change (d0) or new state
                // taken out (see fused_cell).
                uf[f][i] = carry->p[f][i] + tau * carry->q[f][i];
            }
        }
    }
    else
    {
#pragma unroll
        for (int f = 0; f < NFC; ++f)
        {
            int64_t const jr = ldg(a.nbr + f * a.ncell + icl);
            R rec[Rec<ND, R>::NUSED];
            load_rec<ND>(a.cur + jr * Rec<ND, R>::RS, rec);
            R jd[ND];
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                if constexpr (D::MID)
                {
                    R const db = fg<ND>(gv, f, D::K_DB + d);
                    jd[d] = (db - mm[d]) + tau * (mb[d] - db) - delta[d];
                }
                else
                {
                    jd[d] = fg<ND>(gv, f, D::K_R + d) + tau * fg<ND>(gv, f, D::K_Q + d) - delta[d];
                }
            }
#pragma unroll
            for (int i = 0; i < NEQ; ++i)
            {
                R s = u0 ? (rec[i] - u0[i]) + a.hdt * rec[NEQ + i] - d0[i] : rec[i] + a.hdt * rec[NEQ + i] - so0n[i];
#pragma unroll
                for (int d = 0; d < ND; ++d)
                {
                    s += jd[d] * rec[2 * NEQ + i * ND + d];
                }
                uf[f][i] = s;
            }
        }
    }

    // Rows of each element's inverse displacement matrix (prescaled by
    // 1/det): grad = sum_v uf[v] * C[k][v].  Each element divides by its own
    // determinant (a product of all of them could underflow in FP32).
    R dets[NFGE];
    R bcx[NFGE][ND == 3 ? 3 : 1]; // 3D: rb x rc, the first row of the adjugate
#pragma unroll
    for (int k = 0; k < NFGE; ++k)
    {
        R const * ra = idis[CellT<CT>::fge(k, 0)];
        R const * rb = idis[CellT<CT>::fge(k, 1)];
        if constexpr (ND == 2)
        {
            dets[k] = ra[0] * rb[1] - ra[1] * rb[0];
        }
        else
        {
            R const * rc = idis[CellT<CT>::fge(k, ND - 1)];
            bcx[k][0] = rb[1] * rc[2] - rb[2] * rc[1];
            bcx[k][1] = rb[2] * rc[0] - rb[0] * rc[2];
            bcx[k][2] = rb[0] * rc[1] - rb[1] * rc[0];
            dets[k] = ra[0] * bcx[k][0] + ra[1] * bcx[k][1] + ra[2] * bcx[k][2];
        }
    }
    R invs[NFGE];
#pragma unroll
    for (int k = 0; k < NFGE; ++k)
    {
        invs[k] = mrecip<ND>(dets[k]);
    }
    R C[NFGE][ND][ND];
#pragma unroll
    for (int k = 0; k < NFGE; ++k)
    {
        R const * ra = idis[CellT<CT>::fge(k, 0)];
        R const * rb = idis[CellT<CT>::fge(k, 1)];
        R const inv = invs[k];
        if constexpr (ND == 2)
        {
            C[k][0][0] = rb[1] * inv;
            C[k][0][1] = -rb[0] * inv;
            C[k][1][0] = -ra[1] * inv;
            C[k][1][1] = ra[0] * inv;
        }
        else
        {
            R const * rc = idis[CellT<CT>::fge(k, ND - 1)];
            C[k][0][0] = bcx[k][0] * inv;
            C[k][0][1] = bcx[k][1] * inv;
            C[k][0][2] = bcx[k][2] * inv;
            C[k][1][0] = (rc[1] * ra[2] - rc[2] * ra[1]) * inv;
            C[k][1][1] = (rc[2] * ra[0] - rc[0] * ra[2]) * inv;
            C[k][1][2] = (rc[0] * ra[1] - rc[1] * ra[0]) * inv;
            C[k][2][0] = (ra[1] * rb[2] - ra[2] * rb[1]) * inv;
            C[k][2][1] = (ra[2] * rb[0] - ra[0] * rb[2]) * inv;
            C[k][2][2] = (ra[0] * rb[1] - ra[1] * rb[0]) * inv;
        }
    }

    uint8_t fired = 0;
#pragma unroll
    for (int i = 0; i < NEQ; ++i)
    {
        R grad[NFGE][ND];
        R wgt[NFGE];
        R wacc = R(0);
#pragma unroll
        for (int k = 0; k < NFGE; ++k)
        {
            R sq = R(0);
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                R s = R(0);
#pragma unroll
                for (int v = 0; v < ND; ++v)
                {
                    s += uf[CellT<CT>::fge(k, v)][i] * C[k][v][d];
                }
                grad[k][d] = s;
                sq += s * s;
            }
            // W-1/2 weighting: inverse gradient magnitude.
            wgt[k] = rsq(sq + Tiny<R>::AZ);
            wacc += wgt[k];
        }
        {
            R const rw = mrecip<ND>(wacc);
            R wmax = R(0);
            R wmin = R(0);
#pragma unroll
            for (int k = 0; k < NFGE; ++k)
            {
                wgt[k] = wgt[k] * rw - ofg1;
                wmax = fmax(wmax, wgt[k]);
                wmin = fmin(wmin, wgt[k]);
            }
            // W-3/4 cap: sm = min(A / a1, B / a2) with A = 1 - 1/n > 0,
            // a1 = wmax + TINY > 0, B = -1/n < 0, a2 = wmin - TINY < 0.  Both
            // quotients are positive, and A / a1 <= B / a2 exactly when
            // A a2 >= B a1, so the smaller one is chosen first and one
            // division is taken instead of two.
            R const a1 = wmax + Tiny<R>::AZ;
            R const a2 = wmin - Tiny<R>::AZ;
            bool const first = (R(1) - ofg1) * a2 >= -ofg1 * a1;
            R const sm = mquot<ND>(first ? R(1) - ofg1 : -ofg1, first ? a1 : a2);
            R const sig = fmin(sm, sgm0);
            if (sm < sgm0)
            {
                fired |= static_cast<uint8_t>(1u << i);
            }
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                R s = R(0);
#pragma unroll
                for (int k = 0; k < NFGE; ++k)
                {
                    s += (ofg1 + sig * wgt[k]) * grad[k][d];
                }
                so1n[i * ND + d] = s;
            }
        }
    }
    if (a.limiter)
    {
        a.limiter[icl] = fired;
    }
}

// Ghost-row order-0 update of one boundary face (euler_bc.cpp:147-215):
// ghost so0n from the interior's so0n (taken before calc_cfl's rewrite).
template <int ND, typename R>
__device__ __forceinline__ void bc0_ghost(int kind, double const * n, double const * val, R const * in, R * out)
{
    constexpr int NEQ = ND + 2;
    if (kind == 2)
    {
#pragma unroll
        for (int i = 0; i < NEQ; ++i)
        {
            out[i] = R(val[i]);
        }
        return;
    }
#pragma unroll
    for (int i = 0; i < NEQ; ++i)
    {
        out[i] = in[i];
    }
    if (kind == 1)
    {
        // Reflect the momentum: m - 2 (m . n) n.
        R mn = R(0);
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            mn += in[1 + d] * R(n[d]);
        }
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            out[1 + d] = in[1 + d] - R(2) * mn * R(n[d]);
        }
    }
}

// Ghost-row order-1 update of one boundary face (euler_bc.cpp:221-320):
// ghost so1n from the interior's so1c.
template <int ND, typename R>
__device__ __forceinline__ void bc1_ghost(int kind, double const * n, R const * g, R * out)
{
    constexpr int NEQ = ND + 2;
    if (kind == 2)
    {
#pragma unroll
        for (int i = 0; i < NEQ * ND; ++i)
        {
            out[i] = R(0);
        }
        return;
    }
    R nn[ND];
#pragma unroll
    for (int d = 0; d < ND; ++d)
    {
        nn[d] = R(n[d]);
    }
    if (kind == 0)
    {
        // Tangential projection of every gradient: g - (g . n) n.
#pragma unroll
        for (int i = 0; i < NEQ; ++i)
        {
            R gn = R(0);
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                gn += g[i * ND + d] * nn[d];
            }
#pragma unroll
            for (int d = 0; d < ND; ++d)
            {
                out[i * ND + d] = g[i * ND + d] - gn * nn[d];
            }
        }
        return;
    }
    // Slip wall: scalar gradients reflected (I - 2 n n^T) g; momentum
    // gradient tensor reflected on both indices, R G R.
#pragma unroll
    for (int ii = 0; ii < 2; ++ii)
    {
        int const i = ii == 0 ? 0 : NEQ - 1;
        R gn = R(0);
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            gn += g[i * ND + d] * nn[d];
        }
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            out[i * ND + d] = g[i * ND + d] - R(2) * gn * nn[d];
        }
    }
    // RG = G - 2 (G n) n^T then R(RG) = RG - 2 n (n^T RG).
    R gm[ND][ND];
#pragma unroll
    for (int p = 0; p < ND; ++p)
    {
        R gnp = R(0);
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            gnp += g[(1 + p) * ND + d] * nn[d];
        }
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            gm[p][d] = g[(1 + p) * ND + d] - R(2) * gnp * nn[d];
        }
    }
#pragma unroll
    for (int d = 0; d < ND; ++d)
    {
        R ntg = R(0);
#pragma unroll
        for (int p = 0; p < ND; ++p)
        {
            ntg += nn[p] * gm[p][d];
        }
#pragma unroll
        for (int p = 0; p < ND; ++p)
        {
            out[(1 + p) * ND + d] = gm[p][d] - R(2) * nn[p] * ntg;
        }
    }
}

// A row's new so0n and so1n, as FP64, into the host blocks of a march that
// delivers them (out0, out1), in the layout of the host arrays: the bytes
// leave over the host link while the march still computes.
template <int ND, typename R, typename G>
__device__ __forceinline__ void deliver_row(MarchArgs<R, G> const & a, int64_t row, R const * so0, R const * so1)
{
    constexpr int NEQ = ND + 2;
    if (a.out0)
    {
        double * const o = a.out0 + row * NEQ;
        if constexpr (NEQ % 2 == 0)
        {
#pragma unroll
            for (int i = 0; i < NEQ; i += 2)
            {
                *reinterpret_cast<double2 *>(o + i) = make_double2(double(so0[i]), double(so0[i + 1]));
            }
        }
        else
        {
#pragma unroll
            for (int i = 0; i < NEQ; ++i)
            {
                o[i] = double(so0[i]);
            }
        }
    }
    if (a.out1)
    {
        double * const o = a.out1 + row * (NEQ * ND);
        if constexpr ((NEQ * ND) % 2 == 0)
        {
#pragma unroll
            for (int i = 0; i < NEQ * ND; i += 2)
            {
                *reinterpret_cast<double2 *>(o + i) = make_double2(double(so1[i]), double(so1[i + 1]));
            }
        }
        else
        {
#pragma unroll
            for (int i = 0; i < NEQ * ND; ++i)
            {
                o[i] = double(so1[i]);
            }
        }
    }
}

// N values v of each lane's row, into the host block's rows row0 .. row0 + 31
// (those below nrow): the warp's rows are one contiguous piece of the block,
// which its lanes store 16 (N even) or 8 bytes at a time in order, each taking
// its values from their lanes by shuffles.  Whole lines then cross the host
// link; a lane's own 16-byte pieces of its row kept the link below the rate
// that the substep's time allows (2M triangles, the last substep with its
// delivery: 2.7 ms against 1.5 without).
template <int N>
__device__ __forceinline__ void deliver_rows(double * out, int64_t row0, int nrow, double const * v)
{
    constexpr int W = N % 2 == 0 ? 2 : 1; // doubles per store
    constexpr int PER = N / W;
    int const ln = static_cast<int>(threadIdx.x) & 31;
    double * const base = out + row0 * N;
#pragma unroll
    for (int r = 0; r < PER; ++r)
    {
        int const q = r * 32 + ln;
        int const src = q / PER;
        int const p = q % PER;
        double x[W];
#pragma unroll
        for (int k = 0; k < PER; ++k)
        {
#pragma unroll
            for (int w = 0; w < W; ++w)
            {
                double const y = __shfl_sync(0xffffffffu, v[k * W + w], src);
                x[w] = k == 0 || k == p ? y : x[w];
            }
        }
        if (src < nrow)
        {
            if constexpr (W == 2)
            {
                reinterpret_cast<double2 *>(base)[q] = make_double2(x[0], x[1]);
            }
            else
            {
                base[q] = x[0];
            }
        }
    }
}

// What an FP32 cell's substep reads first: its neighbours' rows and its own
// current state.
template <int ND, int NFC>
struct CellHead
{
    int32_t nbr[NFC];
    float u0[ND + 2];

    template <typename G>
    __device__ __forceinline__ CellHead(MarchArgs<float, G> const & a, int64_t icl)
    {
#pragma unroll
        for (int f = 0; f < NFC; ++f)
        {
            nbr[f] = ldg(a.nbr + f * a.ncell + icl);
        }
        load_rec<ND, ND + 2>(a.cur + (icl + a.ngst) * Rec<ND, float>::RS, u0);
    }
};

// Neighbour records read, and a cell's own stored, by its thread.
template <int ND>
struct DirectRecs
{
    float const * cur;
    int32_t const * nbr;

    __device__ __forceinline__ void load(int f, float * rec)
    {
        load_rec<ND>(cur + static_cast<int64_t>(nbr[f]) * Rec<ND, float>::RS, rec);
    }
};
template <int ND>
struct DirectOut
{
    float * row;

    __device__ __forceinline__ void store(float const * so0, float const * so0t, float const * so1)
    {
        store_rec<ND>(row, so0, so0t, so1);
    }
};

__device__ __forceinline__ void copy_async16(unsigned to, void const * from)
{
    asm volatile("cp.async.ca.shared.global [%0], [%1], 16;" ::"r"(to), "l"(from) : "memory");
}
__device__ __forceinline__ void copy_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
// Wait until at most n of the committed groups are still on their way.
__device__ __forceinline__ void copy_wait(int n)
{
    switch (n)
    {
    case 0: asm volatile("cp.async.wait_group 0;" ::: "memory"); break;
    case 1: asm volatile("cp.async.wait_group 1;" ::: "memory"); break;
    case 2: asm volatile("cp.async.wait_group 2;" ::: "memory"); break;
    default: asm volatile("cp.async.wait_group 3;" ::: "memory"); break;
    }
}

// The neighbour records of a warp's cells, fetched together: a record's 64
// (2D) or 128 (3D) bytes by 4 or 8 neighbouring lanes, 16 bytes each, straight
// into shared memory, so that a load instruction touches 8 or 4 whole records
// instead of a piece of 32 (a warp's loads of its own records kept the L1's
// data path 52% busy in 2D and 77% in 3D), and NB faces' records are on their
// way at once without holding registers.  Chunk c of lane i's record lies at
// chunk place c ^ (i's low bits), so neither the copies nor the reads of 8 lanes
// meet in a bank.
template <int ND, int NFC, int NB>
struct StagedRecs
{
    static constexpr int LPR = ND == 2 ? 4 : 8;                       // lanes, and chunk places, per record
    static constexpr int CH = (Rec<ND, float>::NUSED + 3) / 4;        // chunks used
    static constexpr int BUF = 32 * LPR;                              // chunks of one face's records
    static constexpr int BYTES = NB * BUF * 16;                       // per warp
    float const * cur;
    int32_t const * nbr;
    float4 * buf;

    __device__ __forceinline__ static int place(int lane, int c)
    {
        return lane * LPR + (c ^ (ND == 2 ? (lane >> 1) & 3 : lane & 7));
    }
    __device__ __forceinline__ void fetch(int f)
    {
        int const ln = static_cast<int>(threadIdx.x) & 31;
        int const c = ln % LPR;
        float4 * const b = buf + (f % NB) * BUF;
#pragma unroll
        for (int r = 0; r < LPR; ++r)
        {
            int const i = r * (32 / LPR) + ln / LPR;
            int64_t const j = __shfl_sync(0xffffffffu, nbr[f], i);
            if (CH == LPR || c < CH)
            {
                copy_async16(static_cast<unsigned>(__cvta_generic_to_shared(b + place(i, c))),
                             cur + j * Rec<ND, float>::RS + 4 * c);
            }
        }
    }
    // Fetch the first NB faces (the first one's group holds what the caller
    // has copied before).
    __device__ __forceinline__ void begin()
    {
#pragma unroll
        for (int f = 0; f < NB; ++f)
        {
            fetch(f);
            copy_commit();
        }
    }
    __device__ __forceinline__ void load(int f, float * rec)
    {
        int const ln = static_cast<int>(threadIdx.x) & 31;
        float4 const * const b = buf + (f % NB) * BUF;
        copy_wait(f + NB <= NFC ? NB - 1 : NFC - 1 - f);
        __syncwarp();
#pragma unroll
        for (int c = 0; c < CH; ++c)
        {
            float4 const v = b[place(ln, c)];
#pragma unroll
            for (int k = 0; k < 4; ++k)
            {
                if (4 * c + k < Rec<ND, float>::NUSED)
                {
                    rec[4 * c + k] = k == 0 ? v.x : k == 1 ? v.y : k == 2 ? v.z : v.w;
                }
            }
        }
        if (f + NB < NFC)
        {
            __syncwarp(); // every lane has read its record
            fetch(f + NB);
            copy_commit();
        }
    }
};

// A cell's new record into its place in shared memory, for the warp to store
// together.
template <int ND, int LPR>
struct StagedOut
{
    float4 * buf;

    __device__ __forceinline__ void store(float const * so0, float const * so0t, float const * so1)
    {
        constexpr int NEQ = ND + 2;
        constexpr int CH = (Rec<ND, float>::NUSED + 3) / 4;
        int const ln = static_cast<int>(threadIdx.x) & 31;
        float v[4 * CH];
#pragma unroll
        for (int i = 0; i < 4 * CH; ++i)
        {
            v[i] = i < NEQ ? so0[i]
                           : (i < 2 * NEQ ? so0t[i - NEQ] : (i < Rec<ND, float>::NUSED ? so1[i - 2 * NEQ] : 0.f));
        }
#pragma unroll
        for (int c = 0; c < CH; ++c)
        {
            buf[StagedRecs<ND, ND + 1, 1>::place(ln, c)] =
                make_float4(v[4 * c], v[4 * c + 1], v[4 * c + 2], v[4 * c + 3]);
        }
    }
};

// One fused CESE substep for one body cell: soln, bc_soln of its boundary
// faces, cfl, dsoln, bc_dsoln of its boundary faces, and calc_solt of the next
// substep for its own row and its ghost rows.  Reads only the current records
// (neighbours' old values) and writes only rows it owns, so one launch covers
// the whole substep with no grid-wide synchronisation.
// recs: see soln_cell; out.store(so0n, so0t, so1n) keeps the new record.  live:
// false for a lane past the mesh, which takes part in calc_soln (whose records
// the warp may fetch together) for its last cell, and does no more.
template <int CT, typename R, typename G, bool SH, int SB, typename RS, typename OUT>
__device__ __forceinline__ void fused_cell(MarchArgs<R, G> const & a, GeoView<G, SH> const & gv, int64_t icl,
                                           CellHead<CellT<CT>::ND, CellT<CT>::NFC> const & head, RS & recs, OUT & out,
                                           bool live)
{
    constexpr int ND = CellT<CT>::ND;
    constexpr int NEQ = ND + 2;
    constexpr int NFC = CellT<CT>::NFC;
    int64_t const row = icl + a.ngst;

    // FP32 simplices hand calc_soln's neighbour terms to calc_dsoln instead
    // of gathering the neighbour records again (see Carry).
    // The choice depends on the cell type and precision only, never on the
    // kernel, so a core's cells give the same bits in every kernel that
    // marches them (single-type or mixed, alone or batched).
    constexpr bool CARRY = carries<CT>();
    // SB > 0: the carried sums in shared memory, SB threads per block.
    using CA = std::conditional_t<(SB > 0 && CARRY), CarrySh<ND, NFC, R, SB>, Carry<ND, NFC, R>>;
    CA carry;
    if constexpr (SB > 0 && CARRY)
    {
        __shared__ R s_carry[2 * NFC * NEQ * SB];
        carry.p.b = s_carry + threadIdx.x;
        carry.q.b = s_carry + NFC * NEQ * SB + threadIdx.x;
    }
    if constexpr (CARRY)
    {
        face_means<CT, R>(gv, carry.mm, carry.mb);
    }
    // Work relative to the cell's own current state (delta form).
    R const * const u0 = head.u0;
    R d0[NEQ];
    R so0n[NEQ];
    soln_cell<CT>(a, gv, head.nbr, recs, so0n, CARRY ? &carry : nullptr, u0, d0);
    if (!live)
    {
        return;
    }
    // FP32 error feedback: what rounding the new so0 to FP32 drops is kept per
    // cell and equation (comp) and added back to the cell's next new value,
    // the rounding taken by an exact two-sum (Knuth) so the kept residual is
    // exactly the part lost.  A CESE cell's new value is formed from its
    // neighbours' stored values, so without this every substep's FP32
    // roundings of the whole state are lost to the totals for good, and they
    // do not average out (measured: the totals of a 3D blast drift ~1e-8 from
    // FP64's in 200 steps, also with FP64 arithmetic on FP32-rounded states);
    // with the residual fed back they cancel over the mesh, and the totals stay
    // within ~1e-10 of FP64's.  Locally the residual re-added is below half an
    // ulp of the state, the size of the rounding itself.  Neighbours read only
    // the rounded so0; the API's so0n and the totals are so0 + comp; d0 becomes
    // the change including the residual.
    R cnew[NEQ];
    if (a.comp)
    {
#pragma unroll
        for (int i = 0; i < NEQ; ++i)
        {
            R const y = d0[i] + a.comp[i * a.ncell + icl];
            R const t = u0[i] + y;
            R const yb = t - u0[i];
            cnew[i] = (u0[i] - (t - yb)) + (y - yb);
            so0n[i] = t;
            d0[i] = y;
        }
    }

    // Boundary faces: ghost so0n (pre-rewrite), so1n and next so0t.
#pragma unroll
    for (int f = 0; f < NFC; ++f)
    {
        int64_t const jr = head.nbr[f];
        if (jr < a.ngst)
        {
            int const kind = a.gkind[jr];
            if (kind >= 0)
            {
                R own[Rec<ND, R>::NUSED];
                load_rec<ND>(a.cur + row * Rec<ND, R>::RS, own);
                R g0[NEQ], g1[NEQ * ND], gt[NEQ];
                bc0_ghost<ND, R>(kind, a.gnml + jr * ND, a.gval + jr * NEQ, so0n, g0);
                bc1_ghost<ND, R>(kind, a.gnml + jr * ND, own + 2 * NEQ, g1);
                Prim<ND, R> const qg(g0, ldg(a.gamma + jr));
                solt_prim<ND, R>(qg, g0, g1, gt);
                store_rec<ND>(a.nxt + jr * Rec<ND, R>::RS, g0, gt, g1);
            }
        }
    }

    R rinv;
    R const e_soln = so0n[NEQ - 1];
    R const cflc = cfl_cell<ND>(a, gv, row, so0n, rinv);
    if (so0n[NEQ - 1] != e_soln)
    {
        d0[NEQ - 1] = so0n[NEQ - 1] - u0[NEQ - 1]; // calc_cfl rewrote the energy
        cnew[NEQ - 1] = R(0);                      // ... and nothing was dropped
    }
    if (a.comp)
    {
#pragma unroll
        for (int i = 0; i < NEQ; ++i)
        {
            a.comp[i * a.ncell + icl] = cnew[i];
        }
    }
    if constexpr (CARRY)
    {
        // Take the cell's own change (delta form) out of the carried sums
        // now, so it need not stay live through calc_dsoln.
#pragma unroll
        for (int f = 0; f < NFC; ++f)
        {
#pragma unroll
            for (int i = 0; i < NEQ; ++i)
            {
                carry.p[f][i] -= d0[i];
            }
        }
    }
    R so1n[NEQ * ND];
    dsoln_cell<CT>(a, gv, icl, so0n, cflc, so1n, CARRY ? &carry : nullptr, u0, d0);
    R so0t[NEQ];
    Prim<ND, R> const q(so0n, ldg(a.gamma + row), rinv);
    solt_prim<ND, R>(q, so0n, so1n, so0t);
    out.store(so0n, so0t, so1n);
}

// The FP64 ghost row jr of a body cell's boundary face: bc_soln from the cell's
// so0n (before calc_cfl's rewrite), bc_dsoln from its so1c, and calc_solt of the
// next substep.
template <int ND>
__device__ __forceinline__ void ghost64(MarchArgs<double, double> const & a, int64_t jr, int64_t row,
                                        double const * so0n)
{
    constexpr int NEQ = ND + 2;
    using RC = Rec<ND, double>;
    int const kind = a.gkind[jr];
    if (kind >= 0)
    {
        double own[RC::NUSED + 1], g0[NEQ], g1[NEQ * ND], gt[NEQ], gc[FluxTerms<ND>::N];
        load_part<2 * NEQ, RC::NUSED>(a.cur + row * RC::RS, own);
        bc0_ghost<ND, double>(kind, a.gnml + jr * ND, a.gval + jr * NEQ, so0n, g0);
        bc1_ghost<ND, double>(kind, a.gnml + jr * ND, own + 2 * NEQ, g1);
        solt_terms<ND>(g0, g1, ldg(a.gamma + jr), a.qdt, gt, gc);
        store_row<ND>(a.nxt + jr * RC::RS, g0, gt, g1, gc);
        deliver_row<ND>(a, jr, g0, g1);
    }
}

// The same in FP64 (euler_fp64.cuh); the new state is returned too.
template <int CT>
__device__ __forceinline__ void fused_cell64(MarchArgs<double, double> const & a, int64_t icl, double * so0n,
                                             double * so1n)
{
    constexpr int ND = CellT<CT>::ND;
    constexpr int NEQ = ND + 2;
    constexpr int NFC = CellT<CT>::NFC;
    using RC = Rec<ND, double>;
    using F = FluxTerms<ND>;
    int64_t const row = icl + a.ngst;
    soln64<CT, true>(a, icl, so0n);
#pragma unroll 1
    for (int f = 0; f < NFC; ++f)
    {
        int64_t const jr = ldg(a.nbr + f * a.ncell + icl);
        if (jr < a.ngst)
        {
            ghost64<ND>(a, jr, row, so0n);
        }
    }
    double rinv;
    double const cflc = cfl64<ND>(a, icl, row, so0n, rinv);
    dsoln64<CT>(a, icl, so0n, cflc, so1n);
    double so0t[NEQ], c[F::N];
    solt_terms<ND>(so0n, so1n, ldg(a.gamma + row), rinv, a.qdt, so0t, c);
    store_row<ND>(a.nxt + row * RC::RS, so0n, so0t, so1n, c);
}

// A cell's fused substep in either precision (so0n, so1n: the FP64 new state).
template <int CT, typename R, typename G, int SB = 0>
__device__ __forceinline__ void substep_cell(MarchArgs<R, G> const & a, int64_t icl, R * so0n, R * so1n)
{
    if constexpr (sizeof(R) == 8)
    {
        fused_cell64<CT>(a, icl, so0n, so1n);
    }
    else
    {
        constexpr int ND = CellT<CT>::ND;
        CellHead<ND, CellT<CT>::NFC> const head(a, icl);
        DirectRecs<ND> recs{a.cur, head.nbr};
        DirectOut<ND> out{a.nxt + (icl + a.ngst) * Rec<ND, float>::RS};
        fused_cell<CT, R, G, false, SB>(a, geo_view(a, icl), icl, head, recs, out, true);
    }
}

// What the single-type FP32 kernels stage in shared memory (staged_cell): the
// neighbour records of NB faces at a time, and in 2D the geometry (6 KB per
// warp; in 3D it is 13 KB, room for two blocks per SM).  Shared memory and
// registers then set the resident blocks together; measured, 2M triangles, us
// per launch at the best register budget for each: nothing staged 180 (FP32
// form) and 159 (fp32-geom32); geometry alone 163 and 149; records alone
// (one face) 182 and 177; geometry and the records of one, two, three faces
// 161, 156, 157 and 136, 138, 151.  1.3M tetrahedra: nothing staged 271, the
// records of one, two, four faces 245, 300, 372.
template <int CT, typename G>
struct Stage
{
    static constexpr int ND = CellT<CT>::ND;
    static constexpr int NFC = CellT<CT>::NFC;
    static constexpr bool GEO = ND == 2;
    static constexpr int NB = ND == 2 && !Geo<ND, G>::MID ? 2 : 1;
    using Recs = StagedRecs<ND, NFC, NB>;
    static constexpr int NPL = Dim<ND>::KC + NFC * Geo<ND, G>::KF;
    static constexpr int GEO_BYTES = GEO ? NPL * GEO_TILE * 4 : 0;
    static constexpr int WARP_BYTES = Recs::BYTES + GEO_BYTES;
};

// Dynamic shared memory of a fused kernel with blocks of B threads.
template <typename R, typename G, int CT1, int B>
__host__ __device__ constexpr int stage_bytes()
{
    if constexpr (CT1 != 0 && sizeof(R) == 4)
    {
        return B / 32 * Stage<CT1, G>::WARP_BYTES;
    }
    else
    {
        return 0;
    }
}

// An FP32 substep of a warp's cells with their neighbours' records (StagedRecs)
// and, in 2D, their geometry (one contiguous tile, see GeoView) copied to
// shared memory by 16-byte asynchronous copies, and their own new records
// stored together from there.
template <int CT, typename G, int SB>
__device__ __forceinline__ void staged_cell(MarchArgs<float, G> const & a, int64_t t)
{
    using S = Stage<CT, G>;
    constexpr int ND = S::ND;
    constexpr int NFC = S::NFC;
    constexpr int RS = Rec<ND, float>::RS;
    static_assert(sizeof(G) == 4, "a tile of 4-byte values");
    extern __shared__ __align__(16) char s_stage[];
    char * const mine = s_stage + (threadIdx.x / 32) * S::WARP_BYTES;
    int const lane = static_cast<int>(threadIdx.x) & 31;
    int64_t const first = t - lane; // the warp's first cell, a multiple of 32
    int64_t const icl = t < a.ncell ? t : a.ncell - 1;
    CellHead<ND, NFC> const head(a, icl);
    G * const geo = reinterpret_cast<G *>(mine + S::Recs::BYTES);
    if constexpr (S::GEO)
    {
        G const * const tile = a.geo + (first / GEO_TILE) * (S::NPL * GEO_TILE);
        constexpr int N = S::GEO_BYTES / 16;
#pragma unroll
        for (int k = 0; k < N; k += 32)
        {
            if (k + 32 <= N || k + lane < N)
            {
                copy_async16(static_cast<unsigned>(__cvta_generic_to_shared(geo + 4 * (k + lane))),
                             tile + 4 * (k + lane));
            }
        }
    }
    typename S::Recs recs{a.cur, head.nbr, reinterpret_cast<float4 *>(mine)};
    recs.begin();
    StagedOut<ND, S::Recs::LPR> out{recs.buf};
    bool const live = t < a.ncell;
    constexpr int CB = carry_shared<ND>() ? SB : 0;
    if constexpr (S::GEO)
    {
        copy_wait(S::NB - 1); // the geometry and the first face's records
        __syncwarp();
        fused_cell<CT, float, G, true, CB>(a, GeoView<G, true>{geo + lane}, icl, head, recs, out, live);
    }
    else
    {
        fused_cell<CT, float, G, false, CB>(a, geo_view(a, icl), icl, head, recs, out, live);
    }
    __syncwarp();
    int const c = lane % S::Recs::LPR;
#pragma unroll
    for (int r = 0; r < S::Recs::LPR; ++r)
    {
        int const i = r * (32 / S::Recs::LPR) + lane / S::Recs::LPR;
        if ((S::Recs::CH == S::Recs::LPR || c < S::Recs::CH) && first + i < a.ncell)
        {
            reinterpret_cast<float4 *>(a.nxt + (first + i + a.ngst) * RS)[c] = recs.buf[S::Recs::place(i, c)];
        }
    }
}

// A ghost row without a boundary condition keeps its stale state; its next so0t
// is still the Jacobian product of that state.
template <int ND>
__device__ __forceinline__ void stale_ghost64(MarchArgs<double, double> const & a, int64_t g)
{
    constexpr int NEQ = ND + 2;
    using RC = Rec<ND, double>;
    if (a.gkind[g] < 0)
    {
        double * const base = a.nxt + g * RC::RS;
        double rec[RC::NUSED], t[NEQ], c[FluxTerms<ND>::N];
#pragma unroll
        for (int i = 0; i < RC::NUSED; ++i)
        {
            rec[i] = base[i];
        }
        solt_terms<ND>(rec, rec + 2 * NEQ, ldg(a.gamma + g), a.qdt, t, c);
        store_row<ND>(base, rec, t, rec + 2 * NEQ, c);
        deliver_row<ND>(a, g, rec, rec + 2 * NEQ);
    }
}

// The work of thread t of one substep: body cell t for t < ncell, ghost row
// t - ncell after that.  CT1 = 0 dispatches on each cell's type; a nonzero
// CT1 compiles the one cell type of a single-type mesh, whose kernel then
// needs only that type's registers.
template <int ND, typename R, typename G, int CT1, int SB>
__device__ __forceinline__ void fused_thread(MarchArgs<R, G> const & a, int64_t t, int64_t t1)
{
    constexpr int NEQ = ND + 2;
    R so0n[NEQ], so1n[NEQ * ND];
    (void)so0n;
    (void)so1n;
    if constexpr (CT1 != 0 && sizeof(R) == 4)
    {
        if (t - (static_cast<int>(threadIdx.x) & 31) < a.ncell) // the whole warp
        {
            staged_cell<CT1, G, SB>(a, t);
        }
    }
    else if (t < a.ncell && t < t1)
    {
        int const ct = a.ctype[t];
        if constexpr (CT1 != 0)
        {
            (void)ct;
            substep_cell<CT1, R, G, carry_shared<ND>() ? SB : 0>(a, t, so0n, so1n);
        }
        else if constexpr (ND == 2)
        {
            if (ct == 4)
                substep_cell<4, R, G>(a, t, so0n, so1n);
            else
                substep_cell<3, R, G>(a, t, so0n, so1n);
        }
        else
        {
            switch (ct)
            {
            case 6: substep_cell<6, R, G>(a, t, so0n, so1n); break;
            case 5: substep_cell<5, R, G>(a, t, so0n, so1n); break;
            case 7: substep_cell<7, R, G>(a, t, so0n, so1n); break;
            default: substep_cell<8, R, G>(a, t, so0n, so1n); break;
            }
        }
    }
    if constexpr (sizeof(R) == 8)
    {
        if (a.out0 || a.out1)
        {
            __syncwarp();
            int64_t const first = t - (static_cast<int>(threadIdx.x) & 31);
            int64_t const left = (a.ncell < t1 ? a.ncell : t1) - first;
            int const nrow = left >= 32 ? 32 : (left > 0 ? static_cast<int>(left) : 0);
            if (a.out0)
            {
                deliver_rows<NEQ>(a.out0, first + a.ngst, nrow, so0n);
            }
            if (a.out1)
            {
                deliver_rows<NEQ * ND>(a.out1, first + a.ngst, nrow, so1n);
            }
        }
    }
    if (t >= a.ncell && t < a.ncell + a.ngst && t < t1)
    {
        // A ghost row without a boundary condition keeps its stale state; its
        // next so0t is still the Jacobian product of that state.
        int64_t const g = t - a.ncell;
        if constexpr (sizeof(R) == 8)
        {
            stale_ghost64<ND>(a, g);
        }
        else if (a.gkind[g] < 0)
        {
            R * const base = a.nxt + g * Rec<ND, R>::RS;
            R rec[Rec<ND, R>::NUSED], tt[NEQ];
#pragma unroll
            for (int i = 0; i < Rec<ND, R>::NUSED; ++i)
            {
                rec[i] = base[i];
            }
            Prim<ND, R> const q(rec, ldg(a.gamma + g));
            solt_prim<ND, R>(q, rec, rec + 2 * NEQ, tt);
            store_rec<ND>(base, rec, tt, rec + 2 * NEQ);
        }
    }
}

// One cell's substep by the LPC lanes of its group (q: the lane's place in it);
// see Split.
template <int CT>
__device__ __forceinline__ void split_cell(MarchArgs<double, double> const & a, int64_t icl, int q)
{
    constexpr int ND = CellT<CT>::ND;
    constexpr int NEQ = ND + 2;
    constexpr int LPC = Split<ND>::LPC;
    using RC = Rec<ND, double>;
    using F = FluxTerms<ND>;
    int64_t const row = icl + a.ngst;
    int const lane = static_cast<int>(threadIdx.x) & 31;
    int const lead = lane - q; // the group's first lane
    unsigned const group = ((1u << LPC) - 1u) << lead;
    int const eq = q < NEQ ? q : NEQ - 1;
    double const mine = soln64_eq<CT>(a, icl, eq);
    double so0n[NEQ];
#pragma unroll
    for (int i = 0; i < NEQ; ++i)
    {
        so0n[i] = __shfl_sync(group, mine, lead + i);
    }
    if (q < CellT<CT>::NFC)
    {
        int64_t const jr = ldg(a.nbr + q * a.ncell + icl);
        if (jr < a.ngst)
        {
            ghost64<ND>(a, jr, row, so0n);
        }
    }
    double rinv;
    double const cflc = cfl64<ND>(a, icl, row, so0n, rinv);
    // This lane's so0n, as calc_cfl left it.
    double own0 = so0n[0];
#pragma unroll
    for (int i = 1; i < NEQ; ++i)
    {
        own0 = eq == i ? so0n[i] : own0;
    }
    double g[ND];
    unsigned fired = dsoln64_part<CT, 1>(a, icl, eq, &own0, cflc, g);
    double so1n[NEQ * ND];
#pragma unroll
    for (int i = 0; i < NEQ; ++i)
    {
#pragma unroll
        for (int d = 0; d < ND; ++d)
        {
            so1n[i * ND + d] = __shfl_sync(group, g[d], lead + i);
        }
    }
#pragma unroll
    for (int k = 1; k < LPC; k *= 2)
    {
        fired |= __shfl_xor_sync(group, fired, k);
    }
    double so0t[NEQ], c[F::N];
    solt_terms<ND>(so0n, so1n, ldg(a.gamma + row), rinv, a.qdt, so0t, c);
    // The record, its 16-byte pieces dealt to the lanes in turn.
    double * const base = a.nxt + row * RC::RS;
#pragma unroll
    for (int k = 0; k < (RC::NLOAD + 1) / 2; ++k)
    {
        double v[2];
#pragma unroll
        for (int w = 0; w < 2; ++w)
        {
            int const i = 2 * k + w;
            v[w] = i < NEQ ? so0n[i]
                           : (i < 2 * NEQ ? so0t[i - NEQ]
                                          : (i < RC::NUSED ? so1n[i - 2 * NEQ]
                                                           : (i < RC::NLOAD ? c[i - RC::OP] : 0.0)));
        }
        if (k % LPC == q)
        {
            reinterpret_cast<double2 *>(base)[k] = make_double2(v[0], v[1]);
        }
    }
    if (q == 0)
    {
        if (a.limiter)
        {
            a.limiter[icl] = static_cast<uint8_t>(fired);
        }
        deliver_row<ND>(a, row, so0n, so1n);
    }
}

// A whole FP64 substep of a small mesh: LPC lanes per body cell, then (rows up
// to t1 of the work order) one per ghost row.
template <int ND>
__global__ void __launch_bounds__(32) k_fused_split(MarchArgs<double, double> a, int64_t t1)
{
    constexpr int LPC = Split<ND>::LPC;
    int64_t const t = static_cast<int64_t>(blockIdx.x) * 32 + threadIdx.x;
    int64_t const icl = t / LPC;
    int const q = static_cast<int>(t % LPC);
    if (icl < a.ncell)
    {
        int const ct = a.ctype[icl];
        if constexpr (ND == 2)
        {
            if (ct == 4)
                split_cell<4>(a, icl, q);
            else
                split_cell<3>(a, icl, q);
        }
        else
        {
            switch (ct)
            {
            case 6: split_cell<6>(a, icl, q); break;
            case 5: split_cell<5>(a, icl, q); break;
            case 7: split_cell<7>(a, icl, q); break;
            default: split_cell<8>(a, icl, q); break;
            }
        }
    }
    else
    {
        int64_t const g = t - a.ncell * LPC;
        if (g < a.ngst && a.ncell + g < t1)
        {
            stale_ghost64<ND>(a, g);
        }
    }
}

// One substep over the rows [t0, t1) of the work order (body cells 0 ..
// ncell - 1, then the ghost rows): the whole substep is [0, ncell + ngst);
// a march that overlaps its state's upload with its first substep launches
// it in ranges.
template <int ND, typename R, typename G, int CT1 = 0>
__global__ void __launch_bounds__(128) k_fused(MarchArgs<R, G> a, int64_t t0, int64_t t1)
{
    int64_t const t = t0 + static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t - (static_cast<int>(threadIdx.x) & 31) < t1) // whole warps
    {
        fused_thread<ND, R, G, CT1, 128>(a, t, t1);
    }
}

// The same kernel asking the compiler for MINB resident blocks of 128
// (min_blocks).  A stated minimum of 1 would instead free the compiler to use
// up to 255 registers, so the kernels without a budget keep the one-argument
// bound.
template <int ND, typename R, typename G, int CT1, int MINB>
__global__ void __launch_bounds__(128, MINB) k_fused_mb(MarchArgs<R, G> a, int64_t t0, int64_t t1)
{
    int64_t const t = t0 + static_cast<int64_t>(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t - (static_cast<int>(threadIdx.x) & 31) < t1) // whole warps
    {
        fused_thread<ND, R, G, CT1, 128>(a, t, t1);
    }
}

} // namespace dev
} // namespace scg
