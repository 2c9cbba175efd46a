// Hot stencil kernels of a step: J_cell / PV / U_plus / CFL, fluid fluxes with
// the contravariant velocities, face and edge EMF, curl, B_cell with the J
// edges, the cell update, the SSP-RK2 average and the Hall EMF.
//
// Each follows the reference's floating-point operation order; this
// translation unit is compiled with -fmad=false, so the results agree with
// the reference bit for bit.
//
// What bounds them: one to three flops per byte, so HBM; the kernels reach it
// only with enough loads in flight.  Every kernel therefore reads all it needs
// of a phase before its first store: fields may alias as far as the compiler
// knows, so a store between two loads makes the second wait for everything
// the first fed.  Points and addresses cost no global loads (mhd_hot.cuh).
// The minimum CTAs per SM of each default form is the fastest of 1 to 6 by
// whole steps on a 64^3 box, the 6 x 80 x 40 x 40 slab and shell and slab
// sweeps: more registers keep more loads in flight, fewer hide more latency.
// Measured on six shells (2.27 M cells, mixed form), against the kernels that
// loaded views and pointers and stored between loads: PV / CFL 267 -> 191 us,
// mixed flux 241 -> 189, face EMF 104 -> 87, edge EMF 95 -> 73, curl and cell
// update (one pass, before: two) 137 -> 89, B_cell and J edges 127 -> 120 us.
#include "mhd_kernels.cuh"
#include "mhd_hot_launch.cuh"

#include <cfloat>
#include <cmath>

namespace mhd
{

namespace
{
// std::max semantics (returns the first argument unless the second compares
// greater), which differs from fmax on NaN.
__device__ __forceinline__ double smax(double a, double b) { return (a < b) ? b : a; }

constexpr int kHotThreads = 256;

// Start of StepOnce, in the first CTA of the step's first kernel (no kernel of
// the step before the update reads dt): dt = global minimum of the CFL bounds,
// abort check (dt < dt_abort or NaN sets the error word,
// LunarSolver_Timestep.cpp:128-139).
__device__ __forceinline__ void run_begin(const RunClock &rc)
{
    if (rc.dt_key && blockIdx.x == 0 && blockIdx.y == 0)
        for (int r = threadIdx.x; r < rc.nruns; r += blockDim.x)
            begin_run(rc, r);
}

// The run data of StepOnce's end (Z4_Lunar/src/LunarSolver_Driver.cpp:75-79)
// and the arming of the dt reductions, in the first CTA of the update (the
// next reduction runs in the derived-field pass after it)
__device__ __forceinline__ void run_end(const RunClock &rc)
{
    if (rc.dt_key && blockIdx.x == 0 && blockIdx.y == 0)
        for (int r = threadIdx.x; r < rc.nruns; r += blockDim.x)
            end_run(rc, r);
}


// planes of the kernels' L2 prefetch (hot_prefetch)
__constant__ int16_t kPfFlux[] = {int16_t(plane_of(F_U)), int16_t(plane_of(F_PV) + 0), int16_t(plane_of(F_PV) + 1), int16_t(plane_of(F_PV) + 2), int16_t(plane_of(F_PV) + 3), int16_t(plane_of(F_RhoE)), int16_t(plane_of(F_Cs)), int16_t(plane_of(F_JDxi) + 0), int16_t(plane_of(F_JDxi) + 1), int16_t(plane_of(F_JDxi) + 2), int16_t(plane_of(F_JDeta) + 0), int16_t(plane_of(F_JDeta) + 1), int16_t(plane_of(F_JDeta) + 2), int16_t(plane_of(F_JDzeta) + 0), int16_t(plane_of(F_JDzeta) + 1), int16_t(plane_of(F_JDzeta) + 2), int16_t(plane_of(F_NAxi)), int16_t(plane_of(F_NAeta)), int16_t(plane_of(F_NAzeta)), int16_t(plane_of(F_Jac)), int16_t(plane_of(F_Uplus) + 0), int16_t(plane_of(F_Uplus) + 1), int16_t(plane_of(F_Uplus) + 2), int16_t(plane_of(F_Jcell) + 0), int16_t(plane_of(F_Jcell) + 1), int16_t(plane_of(F_Jcell) + 2), int16_t(plane_of(F_Bcell) + 0), int16_t(plane_of(F_Bcell) + 1), int16_t(plane_of(F_Bcell) + 2)};

// the strides of one axis
__device__ __forceinline__ int hot_stride(const HotBlock &b, int a)
{
    return a == 0 ? int(b.si) : a == 1 ? int(b.sj) : 1;
}

// ---------------------------------------------------------------------------
// Scheme_U_ + AddSourceToRHS_Fluid
// (Z4_Lunar/src/physics/LunarSolver_FluidRHS.cpp:3-201, :528-568)
// ---------------------------------------------------------------------------

// a cell's Rusanov face state: density, velocity, pressure, and the total
// energy and sound speed k_pv_uplus_dt formed once per cell
struct FaceState
{
    double rho, u, v, w, p, e, c;
};
__device__ __forceinline__ FaceState face_state(const double *U, const double *PV, const double *E, const double *C,
                                                uint64_t vol, int off)
{
    return FaceState{U[off], PV[off], PV[vol + off], PV[2 * vol + off], PV[3 * vol + off], E[off], C[off]};
}

// One Rusanov face flux (Reconstruction_Rusanov, piecewise-constant states).
// The sound speed sqrt(max(0, gamma p / max(rho, 1e-30))) and the total
// energy p / (gamma - 1) + rho |u|^2 / 2 of each cell, and the face area
// |k|, are the reference's expressions evaluated once (k_pv_uplus_dt,
// k_face_normals) instead of once per face side; the values are identical.
__device__ __forceinline__ void rusanov(const FaceState &L, const FaceState &R, double k1, double k2, double k3,
                                        double area, double out[5])
{
    double UL[5], UR[5];
    UL[0] = L.rho;
    UL[1] = L.rho * L.u;
    UL[2] = L.rho * L.v;
    UL[3] = L.rho * L.w;
    UL[4] = L.e;
    UR[0] = R.rho;
    UR[1] = R.rho * R.u;
    UR[2] = R.rho * R.v;
    UR[3] = R.rho * R.w;
    UR[4] = R.e;

    const double uvwL = k1 * L.u + k2 * L.v + k3 * L.w;
    const double uvwR = k1 * R.u + k2 * R.v + k3 * R.w;
    const double radL = fabs(uvwL) + L.c * area;
    const double radR = fabs(uvwR) + R.c * area;
    const double rad = smax(radL, radR);

    double FL[5], FR[5];
    FL[0] = L.rho * uvwL;
    FL[1] = L.rho * uvwL * L.u + k1 * L.p;
    FL[2] = L.rho * uvwL * L.v + k2 * L.p;
    FL[3] = L.rho * uvwL * L.w + k3 * L.p;
    FL[4] = uvwL * (L.e + L.p);
    FR[0] = R.rho * uvwR;
    FR[1] = R.rho * uvwR * R.u + k1 * R.p;
    FR[2] = R.rho * uvwR * R.v + k2 * R.p;
    FR[3] = R.rho * uvwR * R.w + k3 * R.p;
    FR[4] = uvwR * (R.e + R.p);
#pragma unroll
    for (int m = 0; m < 5; ++m)
        out[m] = 0.5 * (FL[m] + FR[m]) - 0.5 * rad * (UR[m] - UL[m]);
}

// Fluid RHS of the inner cells and contravariant velocities (cell_u_contra,
// LunarSolver_MagExplicit_Ideal.cpp:95-115) of the cells within one ghost
// layer, one axis at a time: both read the axis's face vectors at p and p + 1.
template <class A> __device__ __forceinline__ void fluid_ucontra_body(const A &a, const Consts &c, const RunClock &rc)
{
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND_CELL1>(a, t);
    int i, j, k;
    const bool in_box = hot_point<KIND_CELL1>(b, t, i, j, k, p);
    hot_prefetch<KIND_CELL1>(a, kPfFlux);
    pdl_wait();
    run_begin(rc);
    if (!in_box)
        return;
    const uint64_t v = b.vol;
    const bool inner = hot_inner(b, i, j, k);
    const double *U = hot_at(b, p, F_U), *PV = hot_at(b, p, F_PV), *E = hot_at(b, p, F_RhoE), *C = hot_at(b, p, F_Cs);
    const double jac = *hot_at(b, p, F_Jac);
    const double *Up = hot_at(b, p, F_Uplus);
    const double ux = Up[0], uy = Up[v], uz = Up[2 * v];
    const double inv_jac = 1.0 / (fabs(jac) + 1.0e-30);
    const double invJ = 1.0 / jac;
    FaceState s0{};
    if (inner)
        s0 = face_state(U, PV, E, C, v, 0);
    // each component takes its three flux differences in the reference's
    // order, r -= dx / J, r -= dy / J, r -= dz / J, as each axis completes
    double r[5] = {0.0, 0.0, 0.0, 0.0, 0.0};
    double uc[3];
#pragma unroll
    for (int ax = 0; ax < 3; ++ax)
    {
        const int s = hot_stride(b, ax);
        const double *M = hot_at(b, p, F_JDxi + ax);
        const double m0 = M[0], m1 = M[v], m2 = M[2 * v];
        const double q0 = M[s], q1 = M[v + s], q2 = M[2 * v + s];
        const double kx = 0.5 * (m0 + q0);
        const double ky = 0.5 * (m1 + q1);
        const double kz = 0.5 * (m2 + q2);
        uc[ax] = (kx * ux + ky * uy + kz * uz) * inv_jac;
        if (inner)
        {
            const double *N = hot_at(b, p, F_NAxi + ax);
            const FaceState sm = face_state(U, PV, E, C, v, -s), sp = face_state(U, PV, E, C, v, s);
            double Fm[5], Fp[5];
            rusanov(sm, s0, m0, m1, m2, N[0], Fm);
            rusanov(s0, sp, q0, q1, q2, N[s], Fp);
#pragma unroll
            for (int m = 0; m < 5; ++m)
                r[m] -= (Fp[m] - Fm[m]) * invJ;
        }
    }
    if (inner)
    {
        // J x B force with the Hall_Num_Limiter weight (LunarSolver_Tools.cpp:47-56)
        const double *J = hot_at(b, p, F_Jcell), *B = hot_at(b, p, F_Bcell);
        const double jx = J[0], jy = J[v], jz = J[2 * v];
        const double bx = B[0], by = B[v], bz = B[2 * v];
        const double n_true = smax(s0.rho, 0.0) / c.M_H * c.M_ref;
        const double ne_eff = sqrt(n_true * n_true + c.ne_floor * c.ne_floor);
        const double w = n_true / ne_eff;
        const double fc = c.mom_hall * w;
        const double jxb_x = jy * bz - jz * by;
        const double jxb_y = jz * bx - jx * bz;
        const double jxb_z = jx * by - jy * bx;
        r[1] += fc * jxb_x;
        r[2] += fc * jxb_y;
        r[3] += fc * jxb_z;
        r[4] += fc * (jxb_x * s0.u + jxb_y * s0.v + jxb_z * s0.w);
        double *R = hot_at(b, p, F_RHS);
#pragma unroll
        for (int m = 0; m < 5; ++m)
            R[m * v] = r[m];
    }
    double *UC = hot_at(b, p, F_UC);
    UC[0] = uc[0];
    UC[v] = uc[1];
    UC[2 * v] = uc[2];
}

template <class A, int MINB>
__global__ void __launch_bounds__(kHotThreads, MINB) k_fluid_ucontra_t(const __grid_constant__ A a, Consts c, RunClock rc)
{
    fluid_ucontra_body(a, c, rc);
}

// ---------------------------------------------------------------------------
// AssembleOneDirectionEMF_ (Z4_Lunar/src/physics/LunarSolver_MagExplicit_Ideal.cpp:348-496)
// ---------------------------------------------------------------------------

// transverse transport of the faces of axis fa in direction ba: Rusanov flux
// of the mean face fields of the left (L) and right (R) cell, total (t) and
// induced (i), with the cells' contravariant velocities along fa and ba
__device__ __forceinline__ double emf_flux(double btL, double btR, double biL, double biR, double ufL, double ufR,
                                           double ubL, double ubR, double bff)
{
    const double GL = ufL * btL - ubL * bff;
    const double GR = ufR * btR - ubR * bff;
    const double radius = smax(fabs(ufL), fabs(ufR));
    return 0.5 * (GL + GR) - 0.5 * radius * (biR - biL);
}

template <class A> __device__ __forceinline__ void eface_body(const A &a)
{
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND_STAG>(a, t);
    int i, j, k;
    const bool in_box = hot_point<KIND_STAG>(b, t, i, j, k, p);
    pdl_wait();
    if (!in_box)
        return;
    const uint64_t v = b.vol;
    const int st[3] = {int(b.si), int(b.sj), 1};
    // cells: the point's own and the one below it along each axis
    double u0[3], um[3][3];
    const double *UC = hot_at(b, p, F_UC);
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
        u0[c] = UC[c * v];
#pragma unroll
        for (int ax = 0; ax < 3; ++ax)
            um[ax][c] = UC[c * v - st[ax]];
    }
    // per component ba: its face at p (total), and the mean of its low and
    // high face, total and induced, in the point's cell and in the cells below
    // along the two other axes
    double tot0[3], bt0[3], bi0[3], btm[3][3], bim[3][3];
#pragma unroll
    for (int ba = 0; ba < 3; ++ba)
    {
        const double *B = hot_at(b, p, F_Bxi + ba), *D = hot_at(b, p, F_Baddxi + ba);
        const int s = st[ba];
        const double B0 = B[0], D0 = D[0], B1 = B[s], D1 = D[s];
        tot0[ba] = B0 + D0;
        bt0[ba] = 0.5 * ((B0 + D0) + (B1 + D1));
        bi0[ba] = 0.5 * (B0 + B1);
#pragma unroll
        for (int fa = 0; fa < 3; ++fa)
            if (fa != ba)
            {
                const int q = -st[fa];
                const double Bm = B[q], Dm = D[q], Bp = B[q + s], Dp = D[q + s];
                btm[fa][ba] = 0.5 * ((Bm + Dm) + (Bp + Dp));
                bim[fa][ba] = 0.5 * (Bm + Bp);
            }
    }
#pragma unroll
    for (int fa = 0; fa < 3; ++fa)
        if (hot_face(b, fa, i, j, k))
        {
            const int b1 = (fa + 1) % 3, b2 = (fa + 2) % 3;
            const double g1 = emf_flux(btm[fa][b1], bt0[b1], bim[fa][b1], bi0[b1], um[fa][fa], u0[fa], um[fa][b1],
                                       u0[b1], tot0[fa]);
            const double g2 = emf_flux(btm[fa][b2], bt0[b2], bim[fa][b2], bi0[b2], um[fa][fa], u0[fa], um[fa][b2],
                                       u0[b2], tot0[fa]);
            // (component fa of face axis fa is zero and stays so, k_eface_zero_t)
            *hot_at(b, p, F_Efxi + fa, b1) = g2;
            *hot_at(b, p, F_Efxi + fa, b2) = -g1;
        }
}

// the zero components of Eface: zero in a new pool; written again after an
// upload of Eface or a table that wrote them, in every step while one does
template <class A> __global__ void __launch_bounds__(kHotThreads) k_eface_zero_t(const __grid_constant__ A a)
{
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND_STAG>(a, t);
    int i, j, k;
    const bool in_box = hot_point<KIND_STAG>(b, t, i, j, k, p);
    pdl_wait();
    if (!in_box)
        return;
#pragma unroll
    for (int fa = 0; fa < 3; ++fa)
        if (hot_face(b, fa, i, j, k))
            *hot_at(b, p, F_Efxi + fa, fa) = 0.0;
}

template <class A, int MINB>
__global__ void __launch_bounds__(kHotThreads, MINB) k_eface_t(const __grid_constant__ A a)
{
    eface_body(a);
}

// ---------------------------------------------------------------------------
// AssembleEdgeEMF_FromFaceE_Ideal_ (LunarSolver_MagExplicit_Ideal.cpp:53-287)
// with the zeroing of E_edge over the whole array (LunarSolver_MagneticRHS.cpp:9-28)
// ---------------------------------------------------------------------------

__device__ __forceinline__ double max_abs4(double a0, double a1, double a2, double a3)
{
    double a = 0.0;
    a = smax(a, fabs(a0));
    a = smax(a, fabs(a1));
    a = smax(a, fabs(a2));
    a = smax(a, fabs(a3));
    return a;
}

// inner edges of all three axes; ghost edges keep the zero of
// AssembleRHS_Induction_CT_ except where the Eedge sync writes them
template <class A> __device__ __forceinline__ void eedge_body(const A &a)
{
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND_STAG>(a, t);
    int i, j, k;
    const bool in_box = hot_point<KIND_STAG>(b, t, i, j, k, p);
    pdl_wait();
    if (!in_box)
        return;
    const uint64_t v = b.vol;
    const int si = int(b.si), sj = int(b.sj);
    const double *ux = hot_at(b, p, F_UC), *ue = ux + v, *uz = ux + 2 * v;
    const double *Bx = hot_at(b, p, F_Bxi), *Be = hot_at(b, p, F_Beta), *Bz = hot_at(b, p, F_Bzeta);
    const double *Fx = hot_at(b, p, F_Efxi), *Fe = hot_at(b, p, F_Efeta), *Fz = hot_at(b, p, F_Efzeta);
    double E[3];
    const double Cuct = 0.5;
    const double ux0 = ux[0], uxi = ux[-si], uxj = ux[-sj], uxk = ux[-1], uxij = ux[-si - sj], uxik = ux[-si - 1];
    const double ue0 = ue[0], uei = ue[-si], uej = ue[-sj], uek = ue[-1], ueij = ue[-si - sj], uejk = ue[-sj - 1];
    const double uz0 = uz[0], uzi = uz[-si], uzj = uz[-sj], uzk = uz[-1], uzik = uz[-si - 1], uzjk = uz[-sj - 1];
    const double Bx0 = Bx[0], Be0 = Be[0], Bz0 = Bz[0];
    const double Bxj = Bx[-sj], Bxk = Bx[-1], Bei = Be[-si], Bek = Be[-1], Bzi = Bz[-si], Bzj = Bz[-sj];
    {
        const double Ec = 0.25 * (Fe[0] + Fe[-1] + Fz[0] + Fz[-sj]);
        const double a_eta = max_abs4(ue0, uej, uek, uejk);
        const double a_zeta = max_abs4(uz0, uzj, uzk, uzjk);
        const double dBzeta_eta = Bz0 - Bzj;
        const double dBeta_zeta = Be0 - Bek;
        E[0] = Ec + Cuct * (0.5 * a_eta * dBzeta_eta - 0.5 * a_zeta * dBeta_zeta);
    }
    {
        const double *Fxv = Fx + v, *Fzv = Fz + v;
        const double Ec = 0.25 * (Fxv[0] + Fxv[-1] + Fzv[0] + Fzv[-si]);
        const double a_zeta = max_abs4(uz0, uzi, uzk, uzik);
        const double a_xi = max_abs4(ux0, uxi, uxk, uxik);
        const double dBxi_zeta = Bx0 - Bxk;
        const double dBzeta_xi = Bz0 - Bzi;
        E[1] = Ec + Cuct * (0.5 * a_zeta * dBxi_zeta - 0.5 * a_xi * dBzeta_xi);
    }
    {
        const double *Fxv = Fx + 2 * v, *Fev = Fe + 2 * v;
        const double Ec = 0.25 * (Fxv[0] + Fxv[-sj] + Fev[0] + Fev[-si]);
        const double a_xi = max_abs4(ux0, uxi, uxj, uxij);
        const double a_eta = max_abs4(ue0, uei, uej, ueij);
        const double dBeta_xi = Be0 - Bei;
        const double dBxi_eta = Bx0 - Bxj;
        E[2] = Ec + Cuct * (0.5 * a_xi * dBeta_xi - 0.5 * a_eta * dBxi_eta);
    }
#pragma unroll
    for (int ea = 0; ea < 3; ++ea)
        if (hot_edge(b, ea, i, j, k))
            *hot_at(b, p, F_Exi + ea) = E[ea];
}

template <class A, int MINB>
__global__ void __launch_bounds__(kHotThreads, MINB) k_eedge_t(const __grid_constant__ A a)
{
    eedge_body(a);
}

// ---------------------------------------------------------------------------
// CTOperators::CurlEdgeToFace (Z4_Lunar/src/operators/CTOperators.cpp:6-56)
// with multiplier `mult`, written to RHS_B, optionally followed by the face
// part of ApplyUpdate_Euler_ (LunarSolver_Advance.cpp:95-121): B += dt*RHS_B.
// ---------------------------------------------------------------------------

// the discrete curl of the edge planes at qE on the three faces of a point
__device__ __forceinline__ void point_curl(const HotBlock &b, uint32_t p, int qE, double curl[3])
{
    const int si = int(b.si), sj = int(b.sj);
    const double *Ex = hot_plane(b, p, qE), *Ee = hot_plane(b, p, qE + 1), *Ez = hot_plane(b, p, qE + 2);
    const double x0 = Ex[0], xk = Ex[1], xj = Ex[sj], e0 = Ee[0], ek = Ee[1], ei = Ee[si], z0 = Ez[0], zj = Ez[sj],
                 zi = Ez[si];
    curl[0] = (e0 - ek) + (zj - z0);
    curl[1] = (xk - x0) + (z0 - zi);
    curl[2] = (x0 - xj) + (ei - e0);
}

// the three inner faces at each staggered point: RHS = mult * curl E,
// optionally B += dt * RHS.  qE, qR, qB: first planes of the edge field, of
// RHS_B and of B (qR, qB < 0: not written); with bs the faces are taken from
// a snapshot, B = bs + dt RHS (bs[3 block + axis], in the pool's point layout).
// The snapshot form is the implicit Hall trial's update: the same operands and
// operations as restoring B first, so the same bits, without the copy.
// CELLS: the whole Euler update in one pass, also the cell part (U += dt * RHS_H
// on the inner cells, LunarSolver_Advance.cpp:82-93); one launch instead of two
// and twice the loads in flight.
struct CurlArgs
{
    int qE, qR, qB;
    double mult;
    const double *dtp;
    double dtdiv;
    int mult_is_neg_dt;
    const int *rng;
    const double *const *bs;
};
template <bool CELLS, class A>
__device__ __forceinline__ void curl_body(const A &a, const CurlArgs &x, const RunClock &rc)
{
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND_STAG>(a, t);
    int i, j, k;
    const bool in_box = hot_stagger(b, x.rng, t, i, j, k, p);
    pdl_wait();
    if (CELLS)
        run_end(rc);
    if (!in_box)
        return;
    const uint64_t v = b.vol;
    const double mult = x.mult_is_neg_dt ? -x.dtp[b.run] : x.mult;
    double dtB = 0.0;
    if (x.qB >= 0)
        dtB = x.dtp[b.run] / x.dtdiv;
    double curl[3], B[3], u[5], r[5];
    point_curl(b, p, x.qE, curl);
    if (x.qB >= 0)
    {
#pragma unroll
        for (int fa = 0; fa < 3; ++fa)
            B[fa] = x.bs ? x.bs[3 * b.blk + fa][p] : *hot_plane(b, p, x.qB + fa);
    }
    const bool cell = CELLS && hot_inner(b, i, j, k);
    if (cell)
    {
        const double *U = hot_at(b, p, F_U), *R = hot_at(b, p, F_RHS);
#pragma unroll
        for (int m = 0; m < 5; ++m)
        {
            u[m] = U[m * v];
            r[m] = R[m * v];
        }
    }
#pragma unroll
    for (int fa = 0; fa < 3; ++fa)
        if (hot_face(b, fa, i, j, k))
        {
            const double rhs = mult * curl[fa];
            if (x.qR >= 0)
                *hot_plane(b, p, x.qR + fa) = rhs;
            if (x.qB >= 0)
                *hot_plane(b, p, x.qB + fa) = B[fa] + dtB * rhs;
        }
    if (cell)
    {
        double *U = hot_at(b, p, F_U);
#pragma unroll
        for (int m = 0; m < 5; ++m)
            U[m * v] = u[m] + dtB * r[m];
    }
}

template <bool CELLS, class A, int MINB>
__global__ void __launch_bounds__(kHotThreads, MINB)
    k_curl_e2f_t(const __grid_constant__ A a, const __grid_constant__ CurlArgs x, RunClock rc)
{
    curl_body<CELLS>(a, x, rc);
}

// SSP-RK2 (Shu and Osher, 1988) from two Euler stages at one dt: the state
// of the step's start on the points the Euler update writes (inner cells,
// inner faces), then U^{n+1} = 0.5 (U^n + U2) there.  save = 1 stores,
// save = 0 averages.
template <class A> __global__ void __launch_bounds__(kHotThreads) k_rk2_t(const __grid_constant__ A a, int save)
{
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND_STAG>(a, t);
    int i, j, k;
    const bool in_box = hot_point<KIND_STAG>(b, t, i, j, k, p);
    pdl_wait();
    if (!in_box)
        return;
    const uint64_t v = b.vol;
    double *r = b.rk + p;
    double *U = hot_at(b, p, F_U);
    const bool cell = hot_inner(b, i, j, k);
    double x[8], y[8];
#pragma unroll
    for (int m = 0; m < 8; ++m)
    {
        x[m] = m < 5 ? U[m * v] : *hot_at(b, p, F_Bxi + (m - 5));
        y[m] = save ? 0.0 : r[m * v];
    }
#pragma unroll
    for (int m = 0; m < 8; ++m)
        if (m < 5 ? cell : hot_face(b, m - 5, i, j, k))
        {
            if (save)
                r[m * v] = x[m];
            else if (m < 5)
                U[m * v] = 0.5 * (y[m] + x[m]);
            else
                *hot_at(b, p, F_Bxi + (m - 5)) = 0.5 * (y[m] + x[m]);
        }
}

// ---------------------------------------------------------------------------
// calc_Bcell (Z4_Lunar/src/physics/LunarSolver_Tools.cpp:163-241) and
// Calc_J_Edge: CTOperators::CurlAdjFaceToEdge (CTOperators.cpp:58-110) with
// the face Hodge scale beta, times the edge scale alpha
// (LunarSolver_Tools.cpp:777-835), in one pass over the staggered points:
// both read the face B around the same points (the B_cell sync between them
// in the reference touches neither input)
// ---------------------------------------------------------------------------

// an inner cell's place among the block's cells
__device__ __forceinline__ uint32_t hot_cell(const HotBlock &b, int i, int j, int k)
{
    return (uint32_t(i) * uint32_t(b.nj) + uint32_t(j)) * uint32_t(b.nk) + uint32_t(k);
}
// the least-squares weights of inner cell d, kWTile values apart: the FP64
// field, or its FP32 copy
template <typename WT> __device__ __forceinline__ const WT *hot_weights(const HotBlock &b, uint32_t d, int f, int q32);
template <> __device__ __forceinline__ const double *hot_weights<double>(const HotBlock &b, uint32_t d, int f, int)
{
    return hot_at(b, 0, f) + uint64_t(weight_tile(d, f == F_WB ? 18 : 36));
}
template <> __device__ __forceinline__ const float *hot_weights<float>(const HotBlock &b, uint32_t d, int f, int q32)
{
    return hot_plane32(b, 0, kPlane32W + q32) + uint64_t(weight_tile(d, f == F_WB ? 18 : 36));
}

// WT: double (the reference's weights, FP64 form) or float (their FP32
// copies, mixed form: the products and sums stay FP64); EDGES: with the J
// edges (else B_cell alone); IND: with Bind_cell
template <typename WT, bool EDGES, bool IND, class A> __device__ __forceinline__ void bcell_jedge_body(const A &a)
{
    constexpr int KIND = EDGES ? KIND_STAG : KIND_CELL0;
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND>(a, t);
    int i, j, k;
    const bool in_box = hot_point<KIND>(b, t, i, j, k, p);
    pdl_wait();
    if (!in_box)
        return;
    const uint64_t v = b.vol;
    const int st[3] = {int(b.si), int(b.sj), 1};
    const bool cell = hot_inner(b, i, j, k);
    double B0[3], B1[3], D0[3], D1[3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
        const double *B = hot_at(b, p, F_Bxi + c), *D = hot_at(b, p, F_Baddxi + c);
        B0[c] = B[0];
        B1[c] = B[st[c]];
        D0[c] = D[0];
        D1[c] = D[st[c]];
    }
    double J[3];
    if (EDGES)
    {
        // beta B at the point and below it along the two axes other than the component's
        double h0[3], hm[3][3];
#pragma unroll
        for (int c = 0; c < 3; ++c)
        {
            const double *B = hot_at(b, p, F_Bxi + c), *be = hot_at(b, p, F_betaxi + c);
            h0[c] = be[0] * B0[c];
#pragma unroll
            for (int d = 0; d < 3; ++d)
                if (d != c)
                    hm[d][c] = be[-st[d]] * B[-st[d]];
        }
        const double v0 = (hm[2][1] - h0[1]) + (h0[2] - hm[1][2]);
        const double v1 = (h0[0] - hm[2][0]) + (hm[0][2] - h0[2]);
        const double v2 = (hm[1][0] - h0[0]) + (h0[1] - hm[0][1]);
        J[0] = v0 * *hot_at(b, p, F_alphaxi);
        J[1] = v1 * *hot_at(b, p, F_alphaeta);
        J[2] = v2 * *hot_at(b, p, F_alphazeta);
    }
    if (cell)
    {
        const double tot[6] = {-B0[0] - D0[0], B1[0] + D1[0], -B0[1] - D0[1],
                               B1[1] + D1[1],  -B0[2] - D0[2], B1[2] + D1[2]};
        const double ind[6] = {-B0[0], B1[0], -B0[1], B1[1], -B0[2], B1[2]};
        const WT *W = hot_weights<WT>(b, hot_cell(b, i, j, k), F_WB, W32_B);
        double bt[3] = {0.0, 0.0, 0.0}, bi[3] = {0.0, 0.0, 0.0};
#pragma unroll
        for (int q = 0; q < 6; ++q)
#pragma unroll
            for (int c = 0; c < 3; ++c)
            {
                const double w = double(W[(6 * c + q) * kWTile]);
                bt[c] += w * tot[q];
                if (IND)
                    bi[c] += w * ind[q];
            }
        double *Bc = hot_at(b, p, F_Bcell), *Bi = hot_at(b, p, F_Bind);
#pragma unroll
        for (int c = 0; c < 3; ++c)
        {
            Bc[c * v] = bt[c];
            if (IND)
                Bi[c * v] = bi[c];
        }
    }
    if (EDGES)
    {
#pragma unroll
        for (int ea = 0; ea < 3; ++ea)
            if (hot_edge(b, ea, i, j, k))
                *hot_at(b, p, F_Jxi + ea) = J[ea];
    }
}

template <typename WT, bool EDGES, class A, int MINB, bool IND = true>
__global__ void __launch_bounds__(kHotThreads, MINB) k_bcell_jedge_t(const __grid_constant__ A a)
{
    bcell_jedge_body<WT, EDGES, IND>(a);
}

// the J edges alone: planes qB of the face field, qJ of the edge field
template <class A>
__global__ void __launch_bounds__(kHotThreads) k_jedge_t(const __grid_constant__ A a, int qB, int qJ, const int *rng)
{
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND_STAG>(a, t);
    int i, j, k;
    const bool in_box = hot_stagger(b, rng, t, i, j, k, p);
    pdl_wait();
    if (!in_box)
        return;
    const int st[3] = {int(b.si), int(b.sj), 1};
    double h0[3], hm[3][3], al[3];
#pragma unroll
    for (int c = 0; c < 3; ++c)
    {
        const double *B = hot_plane(b, p, qB + c), *be = hot_at(b, p, F_betaxi + c);
        h0[c] = be[0] * B[0];
        al[c] = *hot_at(b, p, F_alphaxi + c);
#pragma unroll
        for (int d = 0; d < 3; ++d)
            if (d != c)
                hm[d][c] = be[-st[d]] * B[-st[d]];
    }
    const double val[3] = {(hm[2][1] - h0[1]) + (h0[2] - hm[1][2]), (h0[0] - hm[2][0]) + (hm[0][2] - h0[2]),
                           (hm[1][0] - h0[0]) + (h0[1] - hm[0][1])};
#pragma unroll
    for (int ea = 0; ea < 3; ++ea)
        if (hot_edge(b, ea, i, j, k))
            *hot_plane(b, p, qJ + ea) = val[ea] * al[ea];
}

// ---------------------------------------------------------------------------
// calc_Jcell (LunarSolver_Tools.cpp:837-892)
// ---------------------------------------------------------------------------
// ALL: every weight is loaded before the first is used (72 registers; left to
// the compiler, a few at a time)
template <typename WT, bool ALL>
__device__ __forceinline__ void jcell_sum(const HotBlock &b, uint32_t p, uint32_t d, double &jx, double &jy, double &jz)
{
    const int si = int(b.si), sj = int(b.sj);
    const double *Jx = hot_at(b, p, F_Jxi), *Je = hot_at(b, p, F_Jeta), *Jz = hot_at(b, p, F_Jzeta);
    const WT *W = hot_weights<WT>(b, d, F_WJ, W32_J);
    WT w[36];
#pragma unroll
    for (int q = 0; q < 36; ++q)
        w[q] = W[q * kWTile];
    const double s[12] = {Jx[0], Jx[sj], Jx[1], Jx[sj + 1], Je[0], Je[si],
                          Je[1], Je[si + 1], Jz[0], Jz[si], Jz[sj], Jz[si + sj]};
    if (ALL)
        asm volatile("" ::: "memory");
    jx = jy = jz = 0.0;
#pragma unroll
    for (int q = 0; q < 12; ++q)
    {
        jx += double(w[q]) * s[q];
        jy += double(w[12 + q]) * s[q];
        jz += double(w[24 + q]) * s[q];
    }
}

// J_cell in a pass of its own over the inner cells: 51 values read and written
// per cell, 36 of them weights.  A few cells per thread's worth of loads in
// flight bound it: on 6 x 64 x 32 x 32 cells 36.2 us with the weights in planes,
// 31.2 in tiles of the inner cells, 29.0 with every load issued first (3 CTAs per
// SM; 2 and 4 the same); in FP32 weights on 2 x 37 x 21 x 25 cells 10.2 and 7.9.
template <typename WT, class A> __global__ void __launch_bounds__(kHotThreads, 3) k_jcell_t(const __grid_constant__ A a)
{
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND_CELL0>(a, t);
    int i, j, k;
    const bool in_box = hot_point<KIND_CELL0>(b, t, i, j, k, p);
    pdl_wait();
    if (!in_box)
        return;
    double jx, jy, jz;
    jcell_sum<WT, true>(b, p, hot_cell(b, i, j, k), jx, jy, jz);
    const uint64_t v = b.vol;
    double *Jc = hot_at(b, p, F_Jcell);
    Jc[0] = jx;
    Jc[v] = jy;
    Jc[2 * v] = jz;
}

// ---------------------------------------------------------------------------
// calc_PV + calc_Uplus (LunarSolver_Tools.cpp:58-141) on the inner cells
// and one ghost layer (the reference covers the whole array; the rest is
// written at read-out, k_pv_all) and, on inner cells, J_cell and the CFL
// time-step bound of the next Compute_Timestep (LunarSolver_Timestep.cpp:8-140)
// reduced with warp shuffles and one atomicMin per thread block.
// ---------------------------------------------------------------------------

// one face of the CFL bound: (|u . n| + c_f) A with n the outward unit
// normal (A and JD / A precomputed per face, k_face_normals), in the
// arithmetic of the face planes: FP64 with the FP64 planes (the reference's
// values and operations), FP32 with their FP32 copies (the mixed form: the
// speeds in FP32, summed over the faces in FP64)
template <typename T>
__device__ __forceinline__ T cfl_face_term(T Af, T nx, T ny, T nz, bool outward_plus, T ux, T uy, T uz, T Bx, T By,
                                           T Bz, T B2, T rho, T cs2, T inver_MA2)
{
    if (Af <= T(0))
        return T(0);
    if (!outward_plus)
    {
        nx = -nx;
        ny = -ny;
        nz = -nz;
    }
    const T un = ux * nx + uy * ny + uz * nz;
    const T Bn = Bx * nx + By * ny + Bz * nz;
    const T vA2 = inver_MA2 * B2 / rho;
    const T vAn2 = inver_MA2 * (Bn * Bn) / rho;
    const T term = cs2 + vA2;
    T disc = term * term - T(4) * cs2 * vAn2;
    if (disc < T(0))
        disc = T(0);
    const T cf = sqrt(T(0.5) * (term + sqrt(disc)));
    return (fabs(un) + cf) * Af;
}

// plane q of axis a's face data at the thread's point: q = 0 the area, 1..3
// the unit normal (the FP64 field Anorm_*, or its FP32 copies)
template <typename WT> __device__ __forceinline__ const WT *hot_face_plane(const HotBlock &b, uint32_t p, int a, int q);
template <>
__device__ __forceinline__ const double *hot_face_plane<double>(const HotBlock &b, uint32_t p, int a, int q)
{
    return hot_at(b, p, F_NAxi + a, q);
}
template <> __device__ __forceinline__ const float *hot_face_plane<float>(const HotBlock &b, uint32_t p, int a, int q)
{
    return hot_plane32(b, p, q == 0 ? G32_AREA + a : G32_NRM + 3 * a + q - 1);
}

// primitive and face-state quantities of one cell (calc_PV, calc_Uplus)
struct CellState
{
    double rho, u, v, w, pr, up[3], cs, rhoe;
};
__device__ __forceinline__ CellState cell_state(const double U[5], const Consts &c)
{
    CellState s;
    s.rho = smax(U[0], 1e-12);
    s.u = U[1] / s.rho;
    s.v = U[2] / s.rho;
    s.w = U[3] / s.rho;
    const double ke = 0.5 * s.rho * (s.u * s.u + s.v * s.v + s.w * s.w);
    double eint = U[4] - ke;
    if (eint < 0.0)
        eint = 0.0;
    s.pr = (c.gamma - 1.0) * eint;
    s.pr = smax(s.pr, 1e-12);
    const bool has_plasma = U[0] > 1e-20;
    s.up[0] = has_plasma ? s.u : 0.0;
    s.up[1] = has_plasma ? s.v : 0.0;
    s.up[2] = has_plasma ? s.w : 0.0;
    // sound speed and total energy of the Rusanov face states
    // (Reconstruction_Rusanov, LunarSolver_FluidRHS.cpp:34-111)
    s.cs = sqrt(smax(0.0, c.gamma * s.pr / smax(U[0], 1e-30)));
    s.rhoe = s.pr / (c.gamma - 1.0) + 0.5 * U[0] * (s.u * s.u + s.v * s.v + s.w * s.w);
    return s;
}

// WT double: PV_H without its temperature, U_plus and the FP64 face states;
// float (mixed form): U_plus.  No kernel of a step reads the temperature, and
// none of the mixed form PV_H (its flux reads the FP32 face states, its J x B
// source the velocities from U); the read-out pass forms PV_H anew (k_pv_all),
// and runs inside a step where a Sync table copies the temperature.  In a mixed
// context also the FP32 face states, deviations from the reference state
// (formed in FP64), sound speed.
template <typename WT>
__device__ __forceinline__ void store_cell_state(const HotBlock &b, uint32_t p, double U0, const CellState &s)
{
    const uint64_t v = b.vol;
    if (sizeof(WT) == sizeof(double))
    {
        double *PV = hot_at(b, p, F_PV);
        PV[0] = s.u;
        PV[v] = s.v;
        PV[2 * v] = s.w;
        PV[3 * v] = s.pr;
        *hot_at(b, p, F_Cs) = s.cs;
        *hot_at(b, p, F_RhoE) = s.rhoe;
    }
    double *Up = hot_at(b, p, F_Uplus);
    Up[0] = s.up[0];
    Up[v] = s.up[1];
    Up[2 * v] = s.up[2];
    if (b.p32)
    {
        float *q = hot_plane32(b, p, kPlane32Q);
        const double *q0 = b.qref;
        q[Q32_RHO * v] = float(U0 - q0[0]);
        q[(Q32_U + 0) * v] = float(s.u - q0[1]);
        q[(Q32_U + 1) * v] = float(s.v - q0[2]);
        q[(Q32_U + 2) * v] = float(s.w - q0[3]);
        q[Q32_P * v] = float(s.pr - q0[4]);
        q[Q32_RHOE * v] = float(s.rhoe - q0[5]);
        q[Q32_C * v] = float(s.cs);
    }
}

// order-preserving key for non-negative doubles (NaN maps above +inf)
__device__ __forceinline__ unsigned long long dbl_key(double x) { return (unsigned long long)__double_as_longlong(x); }

// smallest key of the CTA into *dt_key
__device__ __forceinline__ void reduce_key(unsigned long long key, unsigned long long *dt_key)
{
#pragma unroll
    for (int off = 16; off > 0; off >>= 1)
    {
        const unsigned long long o = __shfl_xor_sync(0xffffffffu, key, off);
        key = (o < key) ? o : key;
    }
    __shared__ unsigned long long wmin[kHotThreads / 32];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (lane == 0)
        wmin[warp] = key;
    __syncthreads();
    if (warp == 0)
    {
        key = (lane < kHotThreads / 32) ? wmin[lane] : ~0ull;
#pragma unroll
        for (int off = 4; off > 0; off >>= 1)
        {
            const unsigned long long o = __shfl_xor_sync(0xffffffffu, key, off);
            key = (o < key) ? o : key;
        }
        if (lane == 0)
            atomicMin(dt_key, key);
    }
}

template <typename WT, bool JCELL, class A>
__device__ __forceinline__ void pv_uplus_dt_body(const A &a, const Consts &c, unsigned long long *dt_key)
{
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND_CELL1>(a, t);
    int i, j, k;
    double dtc = 1e100;
    const bool in_box = hot_point<KIND_CELL1>(b, t, i, j, k, p);
    pdl_wait();
    if (in_box)
    {
        const uint64_t v = b.vol;
        const bool inner = hot_inner(b, i, j, k);
        // the Pole rings' J_cell is the least squares beside this pass (POLE_JCELL_FIRST)
        const bool jc = JCELL && inner && !((b.poles & 1) && j == 0) && !((b.poles & 2) && j == b.nj - 1);
        double U[5];
#pragma unroll
        for (int m = 0; m < 5; ++m)
            U[m] = hot_at(b, p, F_U)[m * v];
        // FP64: the cell state is stored before the CFL bound and J_cell comes
        // last, so that no phase's results stay live over the next one's loads
        // (12 instead of 88 bytes of spills at 64 registers; 95 -> 87 us on 0.76
        // M cells).  Mixed form: J_cell's loads first, all stores last (195
        // against 201 us on 2.27 M cells; its weights take half the registers).
        // With the weights in tiles the two forms take 82 and 190 us.
        constexpr bool kEarly = sizeof(WT) == sizeof(double);
        double jx, jy, jz;
        if (jc && !kEarly)
            jcell_sum<WT, false>(b, p, hot_cell(b, i, j, k), jx, jy, jz);
        const CellState s = cell_state(U, c);
        if (kEarly)
            store_cell_state<WT>(b, p, U[0], s);
        if (inner)
        {
            const double V = fabs(*hot_at(b, p, F_Jac));
            if (V > 0.0)
            {
                const double rho = smax(U[0], 1e-2);
                // same quotients as the primitive velocities when both floors leave rho alone
                const bool same = (rho == s.rho);
                const double ux = same ? s.u : U[1] / rho, uy = same ? s.v : U[2] / rho, uz = same ? s.w : U[3] / rho;
                const double ke = 0.5 * rho * (ux * ux + uy * uy + uz * uz);
                const double eint = U[4] - ke;
                const double pr = (c.gamma - 1.0) * eint;
                const double cs2 = c.gamma * pr / rho;
                const double *Bc = hot_at(b, p, F_Bcell);
                const double Bx = Bc[0], By = Bc[v], Bz = Bc[2 * v];
                const double B2 = Bx * Bx + By * By + Bz * Bz;
                // the face speeds in the planes' arithmetic (identity casts in FP64)
                const WT uxw = WT(ux), uyw = WT(uy), uzw = WT(uz), Bxw = WT(Bx), Byw = WT(By), Bzw = WT(Bz);
                const WT B2w = WT(B2), rhow = WT(rho), cs2w = WT(cs2), iMA2 = WT(c.inver_MA2);
                double denom = 0.0;
#pragma unroll
                for (int ax = 0; ax < 3; ++ax)
                {
                    const int st = hot_stride(b, ax);
                    WT f0[4], f1[4];
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                    {
                        const WT *P = hot_face_plane<WT>(b, p, ax, q);
                        f0[q] = P[0];
                        f1[q] = P[st];
                    }
                    denom += double(cfl_face_term<WT>(f0[0], f0[1], f0[2], f0[3], false, uxw, uyw, uzw, Bxw, Byw, Bzw,
                                                      B2w, rhow, cs2w, iMA2));
                    denom += double(cfl_face_term<WT>(f1[0], f1[1], f1[2], f1[3], true, uxw, uyw, uzw, Bxw, Byw, Bzw,
                                                      B2w, rhow, cs2w, iMA2));
                }
                // cells with denom <= 0 (or NaN) do not bound dt, as in the reference
                if (denom > 0.0)
                    dtc = c.cfl * V / denom;
            }
            if (jc)
            {
                if (kEarly)
                    jcell_sum<WT, false>(b, p, hot_cell(b, i, j, k), jx, jy, jz);
                double *Jc = hot_at(b, p, F_Jcell);
                Jc[0] = jx;
                Jc[v] = jy;
                Jc[2 * v] = jz;
            }
        }
        if (!kEarly)
            store_cell_state<WT>(b, p, U[0], s);
    }
    reduce_key(dbl_key(dtc), dt_key + b.run);
}

template <typename WT, bool JCELL, class A, int MINB>
__global__ void __launch_bounds__(kHotThreads, MINB)
    k_pv_uplus_dt_t(const __grid_constant__ A a, Consts c, unsigned long long *dt_key)
{
    pv_uplus_dt_body<WT, JCELL>(a, c, dt_key);
}

// PV_H, U_plus and the face states on the whole array (read-out); 2-D launch,
// one grid row per block
template <class A> __global__ void __launch_bounds__(kHotThreads) k_pv_all_t(const __grid_constant__ A a, Consts c, int G)
{
    const HotBlock &b = a.v[blockIdx.y];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n2 = uint32_t(b.nk + 2 * G), n1 = uint32_t(b.nj + 2 * G);
    const uint32_t q = t / n2, ii = q / n1;
    pdl_wait();
    if (ii >= uint32_t(b.ni + 2 * G))
        return;
    const int i = int(ii) - G, j = int(q - ii * n1) - G, k = int(t - q * n2) - G;
    const uint32_t p = b.o + uint32_t(i) * b.si + uint32_t(j) * b.sj + uint32_t(k);
    double U[5];
#pragma unroll
    for (int m = 0; m < 5; ++m)
        U[m] = hot_at(b, p, F_U)[m * uint64_t(b.vol)];
    const CellState s = cell_state(U, c);
    store_cell_state<double>(b, p, U[0], s);
    *hot_at(b, p, F_PV, 4) = s.pr / (s.rho * c.state_coeff);
}

// Explicit resistive edge EMF, AddResistiveEdgeEMF_To_ on a zeroed Eres
// (Z4_Lunar/src/physics/LunarSolver_MagExplicit_Resis.cpp:67-209): on inner
// edges with a non-zero shell profile yita0 (eta_edge_*, from the edge
// midpoint radius), Eres = (inver_Rem yita0) (J_avg . dr) with J_avg the mean
// cell current of the four cells around the edge; zero elsewhere.
template <class A>
__global__ void __launch_bounds__(kHotThreads) k_eres_explicit_t(const __grid_constant__ A a, double inver_Rem)
{
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND_STAG>(a, t);
    int i, j, k;
    const bool in_box = hot_point<KIND_STAG>(b, t, i, j, k, p);
    pdl_wait();
    if (!in_box)
        return;
    const uint64_t v = b.vol;
    const double *Jc = hot_at(b, p, F_Jcell);
    double y[3], E[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int ea = 0; ea < 3; ++ea)
        y[ea] = hot_edge(b, ea, i, j, k) ? *hot_at(b, p, F_etaxi + ea) : 0.0;
#pragma unroll
    for (int ea = 0; ea < 3; ++ea)
        if (y[ea] != 0.0)
        {
            const int s1 = ea == 0 ? int(b.sj) : int(b.si), s2 = ea == 2 ? int(b.sj) : 1;
            const int c[4] = {0, -s1, -s2, -s1 - s2};
            double Jx = 0.0, Jy = 0.0, Jz = 0.0;
#pragma unroll
            for (int q = 0; q < 4; ++q)
            {
                Jx += Jc[c[q]];
                Jy += Jc[v + c[q]];
                Jz += Jc[2 * v + c[q]];
            }
            Jx *= 0.25;
            Jy *= 0.25;
            Jz *= 0.25;
            const double *dr = hot_at(b, p, F_drxi + ea);
            const double Jedge = Jx * dr[0] + Jy * dr[v] + Jz * dr[2 * v];
            E[ea] = 0.0 + (inver_Rem * y[ea]) * Jedge;
        }
#pragma unroll
    for (int ea = 0; ea < 3; ++ea)
        if (hot_edge(b, ea, i, j, k))
            *hot_at(b, p, F_Eresxi + ea) = E[ea];
}

// ---------------------------------------------------------------------------
// Hall edge EMF, BuildHallFaceEMF_Rusanov_diff_
// (Z4_Lunar/src/physics/LunarSolver_MagExplicit_Hall.cpp:8-457)
// ---------------------------------------------------------------------------

// Ehc = alpha (J x B) and beta = |alpha| |B|, with alpha = hall_coef / ne_eff
// (Hall_Num_Limiter)
__device__ __forceinline__ void hall_cell_one(const HotBlock &b, uint32_t p, const Consts &c, double hall_coef)
{
    const uint64_t v = b.vol;
    const double rho = *hot_at(b, p, F_U);
    const double *J = hot_at(b, p, F_Jcell), *B = hot_at(b, p, F_Bcell);
    const double Jx = J[0], Jy = J[v], Jz = J[2 * v];
    const double Bx = B[0], By = B[v], Bz = B[2 * v];
    const double n_true = smax(rho, 0.0) / c.M_H * c.M_ref;
    const double ne = sqrt(n_true * n_true + c.ne_floor * c.ne_floor);
    const double alpha = hall_coef / ne;
    double *E = hot_at(b, p, F_Ehc);
    E[0] = alpha * (Jy * Bz - Jz * By);
    E[v] = alpha * (Jz * Bx - Jx * Bz);
    E[2 * v] = alpha * (Jx * By - Jy * Bx);
    *hot_at(b, p, F_HallBeta) = fabs(alpha) * sqrt(Bx * Bx + By * By + Bz * Bz);
}

// every cell of the array; 2-D launch, one grid row per block
template <class A>
__global__ void __launch_bounds__(kHotThreads)
    k_hall_cell_all_t(const __grid_constant__ A a, Consts c, double hall_coef, int G)
{
    const HotBlock &b = a.v[blockIdx.y];
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n2 = uint32_t(b.nk + 2 * G), n1 = uint32_t(b.nj + 2 * G);
    const uint32_t q = t / n2, ii = q / n1;
    pdl_wait();
    if (ii >= uint32_t(b.ni + 2 * G))
        return;
    const int i = int(ii) - G, j = int(q - ii * n1) - G, k = int(t - q * n2) - G;
    hall_cell_one(b, b.o + uint32_t(i) * b.si + uint32_t(j) * b.sj + uint32_t(k), c, hall_coef);
}

// the cells within one ghost layer
template <class A>
__global__ void __launch_bounds__(kHotThreads) k_hall_cell_t(const __grid_constant__ A a, Consts c, double hall_coef)
{
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND_CELL1>(a, t);
    int i, j, k;
    const bool in_box = hot_point<KIND_CELL1>(b, t, i, j, k, p);
    pdl_wait();
    if (in_box)
        hall_cell_one(b, p, c, hall_coef);
}

// Zero boxes of the Hall edge EMF (Solid_Surface layers and Pole edges): zb[8 q
// ..]: block, edge axis, lo[3], hi[3].  The CTA keeps its block's boxes in
// shared memory (a grid of B blocks has about 3 B, three of them a block's; read
// per edge from global memory they took 60 % of the kernel).
constexpr int kHallBoxes = 24;
struct HallBoxes
{
    int n;               // this block's boxes; more than kHallBoxes: read zb instead
    int b[kHallBoxes][7]; // axis, lo, hi
};
__device__ __forceinline__ void hall_boxes(HallBoxes &s, const int *zb, int nzb, int blk)
{
    if (threadIdx.x == 0)
        s.n = 0;
    __syncthreads();
    for (int q = int(threadIdx.x); q < nzb; q += kHotThreads)
        if (zb[8 * q] == blk)
        {
            const int at = atomicAdd(&s.n, 1);
            if (at < kHallBoxes)
                for (int e = 0; e < 7; ++e)
                    s.b[at][e] = zb[8 * q + 1 + e];
        }
    __syncthreads();
}
__device__ __forceinline__ bool hall_zeroed(const HallBoxes &s, const int *zb, int nzb, int blk, int ea, int i, int j,
                                            int k)
{
    bool zero = false;
    const bool own = s.n <= kHallBoxes;
    for (int q = 0; q < (own ? s.n : nzb) && !zero; ++q)
    {
        const int *z = own ? s.b[q] : zb + 8 * q + 1;
        zero = (own || z[-1] == blk) && z[0] == ea && i >= z[1] && j >= z[2] && k >= z[3] && i < z[4] && j < z[5] &&
               k < z[6];
    }
    return zero;
}

// one edge: 4-cell mean of Ehc along dr, minus the whistler diffusion of the
// two face-B jumps across the edge.  E[q], be[q]: Ehc and beta of the edge's
// cells in the order the reference sums them.
struct HallCell
{
    double e[3], beta;
};
__device__ __forceinline__ double hall_edge_value(const HallCell &c0, const HallCell &c1, const HallCell &c2,
                                                  const HallCell &c3, const double dr[3], double dl, double Am0,
                                                  double Am1, double Ap0, double Ap1, double dB_m, double dB_p)
{
    const double eps = 1e-14, Cwh = 0.1;
    const double Ecx = 0.25 * (c0.e[0] + c1.e[0] + c2.e[0] + c3.e[0]);
    const double Ecy = 0.25 * (c0.e[1] + c1.e[1] + c2.e[1] + c3.e[1]);
    const double Ecz = 0.25 * (c0.e[2] + c1.e[2] + c2.e[2] + c3.e[2]);
    const double Ecen = Ecx * dr[0] + Ecy * dr[1] + Ecz * dr[2];
    const double beta_e = smax(smax(c0.beta, c1.beta), smax(c2.beta, c3.beta));
    const double L = smax(dl, eps);
    const double Abar_m = 0.5 * (Am0 + Am1);
    const double inv_m = L / smax(Abar_m, eps);
    const double mu_m = Cwh * beta_e * inv_m * inv_m;
    const double Abar_p = 0.5 * (Ap0 + Ap1);
    const double inv_p = L / smax(Abar_p, eps);
    const double mu_p = Cwh * beta_e * inv_p * inv_p;
    return Ecen - 0.5 * mu_m * dB_m + 0.5 * mu_p * dB_p;
}

__device__ __forceinline__ HallCell hall_cell_at(const double *E, const double *be, uint64_t v, int off)
{
    return HallCell{{E[off], E[v + off], E[2 * v + off]}, be[off]};
}

// inner Hall edge EMF of all three axes, zero inside the boxes zb; the seven
// cells the three edges share are read once.  At 4 CTAs per SM 42 us on 6 x 64
// x 32 x 32 cells (uncapped 114 registers, 2 CTAs: 47 us).
template <class A, int MINB>
__global__ void __launch_bounds__(kHotThreads, MINB)
    k_hall_edge_t(const __grid_constant__ A a, const int *__restrict__ zb, int nzb)
{
    __shared__ HallBoxes boxes;
    uint32_t t, p;
    const HotBlock &b = hot_block<KIND_STAG>(a, t);
    int i, j, k;
    const bool in_box = hot_point<KIND_STAG>(b, t, i, j, k, p);
    hall_boxes(boxes, zb, nzb, b.blk);
    pdl_wait();
    if (!in_box)
        return;
    const uint64_t v = b.vol;
    const int si = int(b.si), sj = int(b.sj);
    const double *E = hot_at(b, p, F_Ehc), *be = hot_at(b, p, F_HallBeta);
    const HallCell c0 = hall_cell_at(E, be, v, 0), ci = hall_cell_at(E, be, v, -si), cj = hall_cell_at(E, be, v, -sj),
                   ck = hall_cell_at(E, be, v, -1), cij = hall_cell_at(E, be, v, -si - sj),
                   cik = hall_cell_at(E, be, v, -si - 1), cjk = hall_cell_at(E, be, v, -sj - 1);
    const double *Bx = hot_at(b, p, F_Bxi), *Be = hot_at(b, p, F_Beta), *Bz = hot_at(b, p, F_Bzeta);
    const double *Ax = hot_at(b, p, F_Areaxi), *Ae = hot_at(b, p, F_Areaeta), *Az = hot_at(b, p, F_Areazeta);
    double out[3] = {0.0, 0.0, 0.0};
    bool in[3];
#pragma unroll
    for (int ea = 0; ea < 3; ++ea)
    {
        in[ea] = hot_edge(b, ea, i, j, k);
        if (!in[ea] || hall_zeroed(boxes, zb, nzb, b.blk, ea, i, j, k))
            continue;
        const double *r = hot_at(b, p, F_drxi + ea);
        const double dr[3] = {r[0], r[v], r[2 * v]};
        const double dl = *hot_at(b, p, F_dlxi + ea);
        if (ea == 0)
            out[0] = hall_edge_value(cjk, cj, ck, c0, dr, dl, Az[0], Az[-sj], Ae[0], Ae[-1], Bz[0] - Bz[-sj],
                                     Be[0] - Be[-1]);
        else if (ea == 1)
            out[1] = hall_edge_value(cik, ci, ck, c0, dr, dl, Ax[0], Ax[-1], Az[0], Az[-si], Bx[0] - Bx[-1],
                                     Bz[0] - Bz[-si]);
        else
            out[2] = hall_edge_value(cij, ci, cj, c0, dr, dl, Ae[0], Ae[-si], Ax[0], Ax[-sj], Be[0] - Be[-si],
                                     Bx[0] - Bx[-sj]);
    }
#pragma unroll
    for (int ea = 0; ea < 3; ++ea)
        if (in[ea])
            *hot_at(b, p, F_Ehxi + ea) = out[ea];
}

} // namespace

// ---------------------------------------------------------------------------
// launchers: one launch per chunk of blocks (nearly always one); the return
// value is the number of launches, or -1 for an unknown variant
// ---------------------------------------------------------------------------

int launch_k_pv_uplus_dt(int variant, bool w32, const HotGrid &h, cudaStream_t st, Consts c, unsigned long long *dt_key)
{
    if (variant < 0 || variant > 3)
        return -1;
    return hot_for(h, KIND_CELL1, [&](const auto &a, dim3 g) {
        using A = std::decay_t<decltype(a)>;
        auto go = [&](auto kernel) { hot_launch(kernel, g, st, a, c, dt_key); };
        switch (variant)
        {
        case 0:
            w32 ? go(k_pv_uplus_dt_t<float, true, A, 4>) : go(k_pv_uplus_dt_t<double, true, A, 4>);
            break;
        case 1:
            w32 ? go(k_pv_uplus_dt_t<float, true, A, 1>) : go(k_pv_uplus_dt_t<double, true, A, 1>);
            break;
        case 2:
            w32 ? go(k_pv_uplus_dt_t<float, true, A, 5>) : go(k_pv_uplus_dt_t<double, true, A, 5>);
            break;
        default:
            // split: J_cell runs in its own pass (launch_k_jcell) before this one
            w32 ? go(k_pv_uplus_dt_t<float, false, A, 4>) : go(k_pv_uplus_dt_t<double, false, A, 4>);
        }
    });
}

int launch_k_pv_all(const HotGrid &h, cudaStream_t st, Consts c)
{
    return hot_for_padded(h, [&](const auto &a, dim3 g) {
        hot_launch(k_pv_all_t<std::decay_t<decltype(a)>>, g, st, a, c, h.G);
    });
}

int launch_k_fluid_ucontra(int variant, const HotGrid &h, cudaStream_t st, Consts c, RunClock rc)
{
    if (variant < 0 || variant > 1)
        return -1;
    return hot_for(h, KIND_CELL1, [&](const auto &a, dim3 g) {
        using A = std::decay_t<decltype(a)>;
        if (variant == 0)
            hot_launch(k_fluid_ucontra_t<A, 2>, g, st, a, c, rc);
        else
            hot_launch(k_fluid_ucontra_t<A, 3>, g, st, a, c, rc);
        rc = RunClock{}; // the first launch only
    });
}

int launch_k_bcell_jedge(int variant, bool w32, const HotGrid &h, cudaStream_t st, bool ind)
{
    if (variant < 0 || variant > 1)
        return -1;
    return hot_for(h, KIND_STAG, [&](const auto &a, dim3 g) {
        using A = std::decay_t<decltype(a)>;
        auto go = [&](auto kernel) { hot_launch(kernel, g, st, a); };
        if (!ind)
            variant == 0 ? go(k_bcell_jedge_t<double, true, A, 2, false>) : go(k_bcell_jedge_t<double, true, A, 6, false>);
        else if (variant == 0)
            w32 ? go(k_bcell_jedge_t<float, true, A, 2>) : go(k_bcell_jedge_t<double, true, A, 2>);
        else
            w32 ? go(k_bcell_jedge_t<float, true, A, 6>) : go(k_bcell_jedge_t<double, true, A, 6>);
    });
}

int launch_k_bcell(const HotGrid &h, cudaStream_t st)
{
    return hot_for(h, KIND_CELL0, [&](const auto &a, dim3 g) {
        hot_launch(k_bcell_jedge_t<double, false, std::decay_t<decltype(a)>, 1>, g, st, a);
    });
}

int launch_k_jedge(const HotGrid &h, cudaStream_t st, int fB0, int fJ0, const int *rng, int64_t nreg)
{
    const int qB = plane_of(fB0), qJ = plane_of(fJ0);
    return hot_for(
        h, KIND_STAG,
        [&](const auto &a, dim3 g) { hot_launch(k_jedge_t<std::decay_t<decltype(a)>>, g, st, a, qB, qJ, rng); }, nreg);
}

int launch_k_jcell(bool w32, const HotGrid &h, cudaStream_t st)
{
    return hot_for(h, KIND_CELL0, [&](const auto &a, dim3 g) {
        using A = std::decay_t<decltype(a)>;
        if (w32)
            hot_launch(k_jcell_t<float, A>, g, st, a);
        else
            hot_launch(k_jcell_t<double, A>, g, st, a);
    });
}

int launch_k_eface(int variant, const HotGrid &h, cudaStream_t st)
{
    if (variant < 0 || variant > 1)
        return -1;
    return hot_for(h, KIND_STAG, [&](const auto &a, dim3 g) {
        using A = std::decay_t<decltype(a)>;
        if (variant == 0)
            hot_launch(k_eface_t<A, 2>, g, st, a);
        else
            hot_launch(k_eface_t<A, 6>, g, st, a);
    });
}

int launch_k_eface_zero(const HotGrid &h, cudaStream_t st)
{
    return hot_for(h, KIND_STAG,
                   [&](const auto &a, dim3 g) { hot_launch(k_eface_zero_t<std::decay_t<decltype(a)>>, g, st, a); });
}

int launch_k_eedge(int variant, const HotGrid &h, cudaStream_t st)
{
    if (variant < 0 || variant > 1)
        return -1;
    return hot_for(h, KIND_STAG, [&](const auto &a, dim3 g) {
        using A = std::decay_t<decltype(a)>;
        if (variant == 0)
            hot_launch(k_eedge_t<A, 3>, g, st, a);
        else
            hot_launch(k_eedge_t<A, 8>, g, st, a);
    });
}

int launch_k_curl_e2f(int variant, const HotGrid &h, cudaStream_t st, int fE0, int fR0, int fB0, double mult,
                      const double *dtp, double dtdiv, int mult_is_neg_dt, const int *rng, int64_t nreg,
                      const double *const *bs)
{
    if (variant < 0 || variant > 1)
        return -1;
    const CurlArgs x{plane_of(fE0), fR0 >= 0 ? plane_of(fR0) : -1, fB0 >= 0 ? plane_of(fB0) : -1, mult, dtp, dtdiv,
                     mult_is_neg_dt, rng, bs};
    return hot_for(
        h, KIND_STAG,
        [&](const auto &a, dim3 g) {
            using A = std::decay_t<decltype(a)>;
            if (variant == 0)
                hot_launch(k_curl_e2f_t<false, A, 4>, g, st, a, x, RunClock{});
            else
                hot_launch(k_curl_e2f_t<false, A, 6>, g, st, a, x, RunClock{});
        },
        nreg);
}

int launch_k_update(int variant, const HotGrid &h, cudaStream_t st, int fR0, const double *dtp, RunClock rc)
{
    if (variant < 0 || variant > 1)
        return -1;
    const CurlArgs x{plane_of(F_Exi), fR0 >= 0 ? plane_of(fR0) : -1, plane_of(F_Bxi), -1.0, dtp, 1.0, 0, nullptr,
                     nullptr};
    return hot_for(h, KIND_STAG, [&](const auto &a, dim3 g) {
        using A = std::decay_t<decltype(a)>;
        if (variant == 0)
            hot_launch(k_curl_e2f_t<true, A, 4>, g, st, a, x, rc);
        else
            hot_launch(k_curl_e2f_t<true, A, 6>, g, st, a, x, rc);
        rc = RunClock{}; // the first launch only
    });
}

int launch_k_rk2(const HotGrid &h, cudaStream_t st, int save)
{
    return hot_for(h, KIND_STAG,
                   [&](const auto &a, dim3 g) { hot_launch(k_rk2_t<std::decay_t<decltype(a)>>, g, st, a, save); });
}

int launch_k_eres_explicit(const HotGrid &h, cudaStream_t st, double inver_Rem)
{
    return hot_for(h, KIND_STAG, [&](const auto &a, dim3 g) {
        hot_launch(k_eres_explicit_t<std::decay_t<decltype(a)>>, g, st, a, inver_Rem);
    });
}

int launch_k_hall_cell(const HotGrid &h, cudaStream_t st, Consts c, double hall_coef, bool all)
{
    if (all)
        return hot_for_padded(h, [&](const auto &a, dim3 g) {
            hot_launch(k_hall_cell_all_t<std::decay_t<decltype(a)>>, g, st, a, c, hall_coef, h.G);
        });
    return hot_for(h, KIND_CELL1, [&](const auto &a, dim3 g) {
        hot_launch(k_hall_cell_t<std::decay_t<decltype(a)>>, g, st, a, c, hall_coef);
    });
}

int launch_k_hall_edge(int variant, const HotGrid &h, cudaStream_t st, const int *zb, int nzb)
{
    if (variant < 0 || variant > 1)
        return -1;
    return hot_for(h, KIND_STAG, [&](const auto &a, dim3 g) {
        using A = std::decay_t<decltype(a)>;
        if (variant == 0)
            hot_launch(k_hall_edge_t<A, 4>, g, st, a, zb, nzb);
        else
            hot_launch(k_hall_edge_t<A, 2>, g, st, a, zb, nzb);
    });
}

} // namespace mhd
