// FP64 kernels beside the step's hot stencils (mhd_kernels_step.cu): geometry,
// Syncs, run clocks, the persistent resistive solve, the Pole handlers and the
// output diagnostics.
//
// Each evaluates its stage with the same floating-point operation order as
// the reference's loops; this translation unit is compiled with -fmad=false so
// that no multiply-add is contracted, and the results agree with the
// reference bit for bit.
#include "mhd_kernels.cuh"
#include "mhd_hot_launch.cuh"
#include "mhd_basis.cuh"

#include <cfloat>
#include <algorithm>
#include <cmath>

namespace mhd
{

// std::max semantics (returns the first argument unless the second compares
// greater), which differs from fmax on NaN.
__device__ __forceinline__ double smax(double a, double b) { return (a < b) ? b : a; }

// Thread -> (block, i, j, k) over a box [lo, lo + n) with k fastest.
__device__ __forceinline__ bool box_point(const int lo[3], const int n[3], int64_t t, int &i, int &j, int &k)
{
    const int64_t tot = int64_t(n[0]) * n[1] * n[2];
    if (t >= tot)
        return false;
    k = lo[2] + int(t % n[2]);
    t /= n[2];
    j = lo[1] + int(t % n[1]);
    i = lo[0] + int(t / n[1]);
    return true;
}

// Box of a location on block b: inner range [0, n + plus) widened by g.
__device__ __forceinline__ void loc_box(const BlockView &b, int loc, int g, int lo[3], int n[3])
{
    int pi, pj, pk;
    loc_plus(loc, pi, pj, pk);
    lo[0] = lo[1] = lo[2] = -g;
    n[0] = b.ni + pi + 2 * g;
    n[1] = b.nj + pj + 2 * g;
    n[2] = b.nk + pk + 2 * g;
}

// |JD| and JD / |JD| of every face (geometry; once per set-up)
__global__ void k_face_normals(const BlockView *__restrict__ bvs)
{
    const BlockView &b = bvs[blockIdx.y];
    const int fa = blockIdx.z;
    int lo[3], n[3];
    loc_box(b, LOC_FXI + fa, b.G, lo, n);
    int i, j, k;
    if (!box_point(lo, n, int64_t(blockIdx.x) * blockDim.x + threadIdx.x, i, j, k))
        return;
    const int64_t p = pidx(b, i, j, k);
    const int64_t v = b.vol;
    const double *M = b.f[F_JDxi + fa];
    const double ax = M[p], ay = M[v + p], az = M[2 * v + p];
    const double A = sqrt(ax * ax + ay * ay + az * az);
    double *N = b.f[F_NAxi + fa];
    N[p] = A;
    N[v + p] = ax / A;
    N[2 * v + p] = ay / A;
    N[3 * v + p] = az / A;
}

// contravariant velocity of a cell along `axis` (cell_u_contra,
// LunarSolver_MagExplicit_Ideal.cpp:95-115)
__device__ __forceinline__ double u_contra(const BlockView &b, int axis, int i, int j, int k)
{
    const int JD = (axis == 0) ? F_JDxi : (axis == 1) ? F_JDeta : F_JDzeta;
    const int64_t p = pidx(b, i, j, k);
    const int64_t q = pidx(b, i + (axis == 0), j + (axis == 1), k + (axis == 2));
    const int64_t v = b.vol;
    const double *M = b.f[JD];
    const double kx = 0.5 * (M[p] + M[q]);
    const double ky = 0.5 * (M[v + p] + M[v + q]);
    const double kz = 0.5 * (M[2 * v + p] + M[2 * v + q]);
    const double inv_jac = 1.0 / (fabs(b.f[F_Jac][p]) + 1.0e-30);
    const double *Up = b.f[F_Uplus];
    return (kx * Up[p] + ky * Up[v + p] + kz * Up[2 * v + p]) * inv_jac;
}

// the three contravariant velocities of every cell within one layer of the
// inner range, stored once per step instead of being recomputed by every
// face and edge stencil that needs them (up to eight times per point)
__global__ void k_ucontra(const BlockView *__restrict__ bvs)
{
    const BlockView &b = bvs[blockIdx.y];
    int lo[3], n[3];
    loc_box(b, LOC_CELL, 1, lo, n);
    int i, j, k;
    if (!box_point(lo, n, int64_t(blockIdx.x) * blockDim.x + threadIdx.x, i, j, k))
        return;
    const int64_t p = pidx(b, i, j, k);
    double *UC = b.f[F_UC];
    UC[p] = u_contra(b, 0, i, j, k);
    UC[b.vol + p] = u_contra(b, 1, i, j, k);
    UC[2 * b.vol + p] = u_contra(b, 2, i, j, k);
}

// is (i, j, k) an inner point of the face (kind 0) or edge (kind 1) axis a
__device__ __forceinline__ bool inner_of(const BlockView &b, int kind, int a, int i, int j, int k)
{
    int pl[3];
    loc_plus((kind == 0 ? LOC_FXI : LOC_EXI) + a, pl[0], pl[1], pl[2]);
    return i < b.ni + pl[0] && j < b.nj + pl[1] && k < b.nk + pl[2];
}

// calc_divB on inner cells (Z4_Lunar/src/physics/LunarSolver_Tools.cpp:685-775;
// layouts with Pole patches, whose first shell the reference zeroes, are not
// handled here)
__global__ void k_divb(const BlockView *__restrict__ bvs)
{
    const BlockView &b = bvs[blockIdx.y];
    int lo[3], n[3];
    loc_box(b, LOC_CELL, 0, lo, n);
    int i, j, k;
    if (!box_point(lo, n, int64_t(blockIdx.x) * blockDim.x + threadIdx.x, i, j, k))
        return;
    const int64_t p = pidx(b, i, j, k);
    const double *Bx = b.f[F_Bxi], *Be = b.f[F_Beta], *Bz = b.f[F_Bzeta];
    const double num = Bx[pidx(b, i + 1, j, k)] - Bx[p] + Be[pidx(b, i, j + 1, k)] - Be[p] + Bz[pidx(b, i, j, k + 1)] -
                       Bz[p];
    b.f[F_divB][p] = num / b.f[F_Jac][p];
}

// ---------------------------------------------------------------------------
// Calc_J_Edge: CTOperators::CurlAdjFaceToEdge (CTOperators.cpp:58-110) with
// the face Hodge scale beta, times the edge scale alpha
// (LunarSolver_Tools.cpp:777-835).
// ---------------------------------------------------------------------------
__device__ __forceinline__ void jedge_one(const BlockView &b, int ea, int i, int j, int k, int fB0, int fJ0,
                                          double mult)
{
    const double *Fx = b.f[fB0], *Fe = b.f[fB0 + 1], *Fz = b.f[fB0 + 2];
    const double *bx = b.f[F_betaxi], *be = b.f[F_betaeta], *bz = b.f[F_betazeta];
    const int64_t c0 = pidx(b, i, j, k);
    double val;
    if (ea == 0)
    {
        const int64_t a = pidx(b, i, j, k - 1), d = pidx(b, i, j - 1, k);
        val = (be[a] * Fe[a] - be[c0] * Fe[c0]) + (bz[c0] * Fz[c0] - bz[d] * Fz[d]);
    }
    else if (ea == 1)
    {
        const int64_t a = pidx(b, i, j, k - 1), d = pidx(b, i - 1, j, k);
        val = (bx[c0] * Fx[c0] - bx[a] * Fx[a]) + (bz[d] * Fz[d] - bz[c0] * Fz[c0]);
    }
    else
    {
        const int64_t a = pidx(b, i, j - 1, k), d = pidx(b, i - 1, j, k);
        val = (bx[a] * Fx[a] - bx[c0] * Fx[c0]) + (be[c0] * Fe[c0] - be[d] * Fe[d]);
    }
    const double J = mult * val;
    b.f[fJ0 + ea][c0] = J * b.f[F_alphaxi + ea][c0];
}

// Start of StepOnce in a launch of its own (a stage; the step's flux kernel
// does it in its first CTA)
__global__ void k_begin_step(RunClock rc)
{
    for (int r = threadIdx.x; r < rc.nruns; r += blockDim.x)
        begin_run(rc, r);
}

__device__ __forceinline__ unsigned long long dbl_key(double x)
{
    // order-preserving key for non-negative doubles (NaN maps above +inf)
    return (unsigned long long)__double_as_longlong(x);
}

// Arms the dt reductions with the reference's initial bound (dt_local = 1e100).
__global__ void k_arm_dt(unsigned long long *dt_key, int nruns)
{
    for (int r = threadIdx.x; r < nruns; r += blockDim.x)
        dt_key[r] = dbl_key(1e100);
}

// ---------------------------------------------------------------------------
// compiled Sync: dst <- src over the field pool
// ---------------------------------------------------------------------------
__global__ void k_gather(double *__restrict__ pool, const uint64_t *__restrict__ dst, const uint64_t *__restrict__ src,
                         int64_t n)
{
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < n)
        pool[dst[t]] = pool[src[t]];
}

// Copies and fixed values of one or more Syncs in one pass: no destination is
// another's source, so their order does not matter.  The lists are read
// before the wait for the kernel that writes the sources (they never change
// inside a step).
template <typename I>
__global__ void k_sync(double *__restrict__ pool, const I *__restrict__ dst, const I *__restrict__ src, int64_t n,
                       const I *__restrict__ cdst, const double *__restrict__ cval, int64_t nconst)
{
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < n)
    {
        const I d = dst[t], s = src[t];
        pdl_wait();
        pool[d] = pool[s];
    }
    else if (t - n < nconst)
    {
        const I d = cdst[t - n];
        const double v = cval[t - n];
        pdl_wait();
        pool[d] = v;
    }
}
template <typename I>
static void sync_launch(cudaStream_t st, double *pool, const I *dst, const I *src, int64_t n, const I *cdst,
                        const double *cval, int64_t nconst)
{
    pdl_launch(k_sync<I>, dim3(unsigned((n + nconst + 255) / 256)), 256, 0, st, pool, dst, src, n, cdst, cval, nconst);
}
void launch_k_sync(cudaStream_t st, double *pool, const uint64_t *dst, const uint64_t *src, int64_t n,
                   const uint64_t *cdst, const double *cval, int64_t nconst)
{
    sync_launch(st, pool, dst, src, n, cdst, cval, nconst);
}
void launch_k_sync(cudaStream_t st, double *pool, const uint32_t *dst, const uint32_t *src, int64_t n,
                   const uint32_t *cdst, const double *cval, int64_t nconst)
{
    sync_launch(st, pool, dst, src, n, cdst, cval, nconst);
}

// phase A of a Sync: points set to fixed values by physical handlers
// (Farfield states, zero-curl edge EMF, zeroed wall layers)
__global__ void k_set_consts(double *__restrict__ pool, const uint64_t *__restrict__ dst,
                             const double *__restrict__ val, int64_t n)
{
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < n)
        pool[dst[t]] = val[t];
}

// phase A of Sync("Ucell") on a Solid_Surface face: LunarBoundary::BC_Solid_Surface_
// (Z4_Lunar/src/boundary/Boundary_Condition_Fluid.cpp:19-185).  The first inner
// cell layer takes the density of the next cell inwards (floored at 2.5e-3),
// zero velocity and its pressure; every ghost layer then repeats that
// layer's state.  One thread per boundary cell column; dir = +-1, +-2, +-3.
__device__ __forceinline__ void wall_u_one(const BlockView &b, int dir, double gamma, int64_t t);

// all Solid_Surface handlers of a sync in one launch: walls[2 q] = block,
// walls[2 q + 1] = direction of handler q = blockIdx.y
__global__ void k_wall_u_all(const BlockView *__restrict__ bvs, const int *__restrict__ walls, double gamma)
{
    const int q = blockIdx.y;
    pdl_wait();
    wall_u_one(bvs[walls[2 * q]], walls[2 * q + 1], gamma, int64_t(blockIdx.x) * blockDim.x + threadIdx.x);
}

void launch_k_wall_u(dim3 grid, cudaStream_t st, const BlockView *bvs, const int *walls, double gamma)
{
    pdl_launch(k_wall_u_all, grid, 256, 0, st, bvs, walls, gamma);
}

__device__ __forceinline__ void wall_u_one(const BlockView &b, int dir, double gamma, int64_t t)
{
    const int ax = (dir < 0 ? -dir : dir) - 1;
    const int sgn = dir > 0 ? 1 : -1;
    const int n[3] = {b.ni, b.nj, b.nk};
    const int t1 = (ax == 0) ? 1 : 0;
    const int t2 = (ax == 2) ? 1 : 2;
    if (t >= int64_t(n[t1]) * n[t2])
        return;
    int c[3];
    c[t1] = int(t / n[t2]);
    c[t2] = int(t % n[t2]);
    c[ax] = (sgn < 0) ? 0 : n[ax] - 1;
    const double rho_floor = 2.5e-3, p_floor = 1e-12;
    double *U = b.f[F_U];
    const int64_t v = b.vol;
    auto pressure = [&](double rho, double mx, double my, double mz, double E) {
        rho = smax(rho, rho_floor);
        const double ke = 0.5 * (mx * mx + my * my + mz * mz) / rho;
        double eint = E - ke;
        if (eint < 0.0)
            eint = 0.0;
        double p = (gamma - 1.0) * eint;
        return smax(p, p_floor);
    };
    // first layer from the cell one further inside
    int r[3] = {c[0], c[1], c[2]};
    r[ax] -= sgn;
    const int64_t pr = pidx(b, r[0], r[1], r[2]);
    const int64_t p0 = pidx(b, c[0], c[1], c[2]);
    {
        const double rho_r = smax(U[pr], rho_floor);
        const double p_r = pressure(rho_r, U[v + pr], U[2 * v + pr], U[3 * v + pr], U[4 * v + pr]);
        const double vz = 0.0;
        const double ke_g = 0.5 * rho_r * (vz * vz + vz * vz + vz * vz);
        U[p0] = rho_r;
        U[v + p0] = rho_r * vz;
        U[2 * v + p0] = rho_r * vz;
        U[3 * v + p0] = rho_r * vz;
        U[4 * v + p0] = p_r / (gamma - 1.0) + ke_g;
    }
    // ghost layers repeat the (updated) first layer
    const double rho_r = smax(U[p0], rho_floor);
    const double p_r = pressure(rho_r, U[v + p0], U[2 * v + p0], U[3 * v + p0], U[4 * v + p0]);
    const double vz = 0.0;
    const double ke_g = 0.5 * rho_r * (vz * vz + vz * vz + vz * vz);
    for (int ng = 1; ng <= b.G; ++ng)
    {
        int gidx[3] = {c[0], c[1], c[2]};
        gidx[ax] += ng * sgn;
        const int64_t pg = pidx(b, gidx[0], gidx[1], gidx[2]);
        U[pg] = rho_r;
        U[v + pg] = rho_r * vz;
        U[2 * v + pg] = rho_r * vz;
        U[3 * v + pg] = rho_r * vz;
        U[4 * v + pg] = p_r / (gamma - 1.0) + ke_g;
    }
}

// two-phase variant when a source is also a destination
__global__ void k_gather_stage(double *__restrict__ tmp, const double *__restrict__ pool,
                               const uint64_t *__restrict__ src, int64_t n)
{
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < n)
        tmp[t] = pool[src[t]];
}
__global__ void k_scatter_stage(double *__restrict__ pool, const double *__restrict__ tmp,
                                const uint64_t *__restrict__ dst, int64_t n)
{
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t < n)
        pool[dst[t]] = tmp[t];
}

// ---------------------------------------------------------------------------
// AoS (reference host layout) <-> padded SoA, on the device
// ---------------------------------------------------------------------------
__global__ void k_aos_to_soa(const BlockView *__restrict__ bvs, int blk, int fid, int ncomp, int lo0, int lo1,
                             int lo2, int n0, int n1, int n2, const double *__restrict__ aos)
{
    const BlockView &b = bvs[blk];
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t tot = int64_t(n0) * n1 * n2 * ncomp;
    if (t >= tot)
        return;
    int64_t r = t;
    const int m = int(r % ncomp);
    r /= ncomp;
    const int k = lo2 + int(r % n2);
    r /= n2;
    const int j = lo1 + int(r % n1);
    const int i = lo0 + int(r / n1);
    b.f[fid][field_index(b, fid, ncomp, m, i, j, k)] = aos[t];
}

__global__ void k_soa_to_aos(const BlockView *__restrict__ bvs, int blk, int fid, int ncomp, int lo0, int lo1,
                             int lo2, int n0, int n1, int n2, double *__restrict__ aos)
{
    const BlockView &b = bvs[blk];
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    const int64_t tot = int64_t(n0) * n1 * n2 * ncomp;
    if (t >= tot)
        return;
    int64_t r = t;
    const int m = int(r % ncomp);
    r /= ncomp;
    const int k = lo2 + int(r % n2);
    r /= n2;
    const int j = lo1 + int(r % n1);
    const int i = lo0 + int(r / n1);
    aos[t] = b.f[fid][field_index(b, fid, ncomp, m, i, j, k)];
}

// ---------------------------------------------------------------------------
// The implicit resistive solve in one persistent kernel
// (SolveImplicitResistiveDiffusion_, Z4_Lunar/src/implicit/Lunar_ImplicitResistive.cpp:430-491,
// with the operator MatMultImplicitResistive_, :369-427)
//
// Launched cooperatively (every CTA resident), so CTAs can wait for one
// another at grid barriers.  Every barrier wait is bounded: a CTA that gives
// up sets the error word and leaves, and the others give up at their next
// barrier.  Dot products: each CTA writes its partial sums, and after the
// barrier every CTA adds all partials in the same fixed order, so all CTAs
// hold bit-identical results and take the same control decisions without a
// second barrier.  The GMRES scalars (Hessenberg matrix, rotations, counters)
// live in each CTA's shared memory; CTA 0 writes them back at the end.
// ---------------------------------------------------------------------------

constexpr long long kBarrierSpins = 1ll << 22; // about a second of polling

// Grid barrier on a count that only grows: bar[0] arrivals, bar[1] the count
// at which the launch starts (CTA 0 leaves the next launch's when the solve
// ends; every CTA has read it before its first arrival, which CTA 0's exit
// implies), bar[2] the polling limit of every wait (0: kBarrierSpins; a smaller
// limit is set only by the failure-detection hook mhd_test_stall_barrier, and
// the host clears all four words after a solve that gave up).  A CTA arrives
// once per barrier and waits for the count of all, so the last arrival itself
// releases the others: one round trip to L2 less per barrier than a count that
// is reset behind a generation number, and no sleep between polls.  A CTA that
// gives up arrives at no later barrier, so the others give up in turn; they
// look at the error word while they wait.
struct GridBar
{
    unsigned *bar;
    int *err;
    volatile int *h_err;
    unsigned target, limit; // thread 0's
};
__device__ __forceinline__ GridBar grid_bar(unsigned *bar, int *err, volatile int *h_err)
{
    GridBar g{bar, err, h_err, 0u, 0u};
    if (threadIdx.x == 0)
    {
        g.target = *(volatile unsigned *)(bar + 1);
        g.limit = *(volatile unsigned *)(bar + 2);
    }
    return g;
}
__device__ __forceinline__ bool grid_barrier(GridBar &g)
{
    __shared__ int ok; // one decision for the whole CTA
    __syncthreads();
    if (threadIdx.x == 0)
    {
        const long long limit = g.limit ? (long long)g.limit : kBarrierSpins;
        g.target += gridDim.x;
        ok = 1;
        long long spins = 0;
        // release: what the CTA wrote before (cumulative through the barrier
        // above); acquire: what the others wrote before their arrivals
        asm volatile("red.release.gpu.global.add.u32 [%0], %1;" ::"l"(g.bar), "r"(1u) : "memory");
        for (;;)
        {
            unsigned count;
            asm volatile("ld.acquire.gpu.global.u32 %0, [%1];" : "=r"(count) : "l"(g.bar) : "memory");
            if (int(count - g.target) >= 0)
                break;
            ++spins;
            if (spins > limit || ((spins & 255) == 0 && *(volatile int *)g.err == MHD_EKRYLOV))
            {
                atomicExch(g.err, MHD_EKRYLOV);
                *g.h_err = MHD_EKRYLOV;
                ok = 0;
                break;
            }
        }
    }
    __syncthreads();
    return ok != 0;
}

struct GmresScalars
{
    double H[31 * 31], cs[31], sn[31], g[32], hcol[32], y[31], d[32];
    double beta, resid, bnorm, ttol;
    int j, its, reason, breakdown, inner, outer, cycles;
};

// out[c] = V_c . w for c < nv, or out[0] = w . w (V null); with_self also
// out[nv] = w . w in the same reduction; every CTA ends with the same values
// in out (shared memory)
__device__ bool grid_dots(const ResistSolve &a, GridBar &gb, const double *V, int nv, const double *w, double *out,
                          int &pbuf, bool with_self = false)
{
    __shared__ double wred[8][8];
    const int G = gridDim.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // CTAs past the vector's end hold no element: their partial sums are +0,
    // which changes no sum that starts at +0, so they write none
    const int Gn = int(min(int64_t(G), (a.n + int64_t(blockDim.x) - 1) / int64_t(blockDim.x)));
    double *part = a.partial + int64_t(pbuf) * 32 * G;
    pbuf ^= 1;
    const int nd = nv + (with_self ? 1 : 0);
    if (int(blockIdx.x) < Gn)
        for (int c0 = 0; c0 < nd; c0 += 8)
        {
            double acc[8] = {0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0, 0.0};
            for (int64_t t = int64_t(blockIdx.x) * blockDim.x + tid; t < a.n; t += int64_t(G) * blockDim.x)
            {
                const double wt = w[t];
#pragma unroll
                for (int q = 0; q < 8; ++q)
                    if (c0 + q < nd)
                        acc[q] += ((V && c0 + q < nv) ? V[int64_t(c0 + q) * a.n + t] : wt) * wt;
            }
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (c0 + q < nd)
                {
                    for (int off = 16; off > 0; off >>= 1)
                        acc[q] += __shfl_xor_sync(0xffffffffu, acc[q], off);
                    if (lane == 0)
                        wred[warp][q] = acc[q];
                }
            __syncthreads();
            if (tid < 8 && c0 + tid < nd)
            {
                double sum = 0.0;
                for (int wp = 0; wp < int(blockDim.x >> 5); ++wp)
                    sum += wred[wp][tid];
                part[int64_t(c0 + tid) * G + blockIdx.x] = sum;
            }
            __syncthreads();
        }
    if (!grid_barrier(gb))
        return false;
    for (int c = warp; c < nd; c += int(blockDim.x >> 5))
    {
        double sum = 0.0;
        // (loads of a batch in flight together, added in CTA order)
        for (int g = lane; g < Gn; g += 128)
        {
            double y[4];
#pragma unroll
            for (int e = 0; e < 4; ++e)
                y[e] = g + 32 * e < Gn ? __ldcg(&part[int64_t(c) * G + g + 32 * e]) : 0.0;
#pragma unroll
            for (int e = 0; e < 4; ++e)
                sum += y[e];
        }
        for (int off = 16; off > 0; off >>= 1)
            sum += __shfl_xor_sync(0xffffffffu, sum, off);
        if (lane == 0)
            out[c] = sum;
    }
    __syncthreads();
    return true;
}

// fixed values (unless already written) then copies of a point list
__device__ bool grid_apply(const ResistSolve &a, GridBar &gb, const DevCopy &l, bool consts_done)
{
    const int64_t t0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, ts = int64_t(gridDim.x) * blockDim.x;
    if (l.nconst > 0 && !consts_done)
    {
        for (int64_t t = t0; t < l.nconst; t += ts)
            a.pool[l.cdst[t]] = l.cval[t];
        if (!grid_barrier(gb))
            return false;
    }
    if (l.n == 0)
        return true;
    if (l.tmp)
    {
        for (int64_t t = t0; t < l.n; t += ts)
            l.tmp[t] = a.pool[l.src[t]];
        if (!grid_barrier(gb))
            return false;
        for (int64_t t = t0; t < l.n; t += ts)
            a.pool[l.dst[t]] = __ldcg(&l.tmp[t]);
    }
    else
        for (int64_t t = t0; t < l.n; t += ts)
            a.pool[l.dst[t]] = a.pool[l.src[t]];
    return grid_barrier(gb);
}

// discrete curl of the edge planes qE on face axis fa of the point
__device__ __forceinline__ double hot_curl(const HotBlock &b, uint32_t p, int qE, int fa)
{
    const int si = int(b.si), sj = int(b.sj);
    const double *Ex = hot_plane(b, p, qE), *Ee = hot_plane(b, p, qE + 1), *Ez = hot_plane(b, p, qE + 2);
    if (fa == 0)
        return (Ee[0] - Ee[1]) + (Ez[sj] - Ez[0]);
    if (fa == 1)
        return (Ex[1] - Ex[0]) + (Ez[0] - Ez[si]);
    return (Ex[0] - Ex[sj]) + (Ee[si] - Ee[0]);
}

// What a thread's first item of each phase's list needs that no phase writes:
// read once at the start of the solve, because the fence of every barrier
// drops the L1 lines a second read would hit.  The lists hold at most a few
// items per thread, usually one.
struct PreUnknown // an unknown's edge: its point, axis, resistivity, edge and face scales
{
    const HotBlock *b;
    uint32_t p;
    int ea;
    uint64_t e;
    double eta, alpha, beta[4];
};
struct PreFused // an item of a fused list; a curl's point and axis decoded
{
    uint64_t dst;
    int kind, fa;
    int64_t idx;
    double val;
    const HotBlock *b;
    uint32_t p;
};
struct PreRegion // a staggered point of the region and its inner faces
{
    const HotBlock *b;
    uint32_t p;
    int faces;
};

// the other component and offset of each term of the edge circulation of axis
// ea (CTOperators.cpp:58-110): (h1[o1] - h1[0]) + (h2[0] - h2[o2]) for ea = 0 ...
__device__ __forceinline__ void edge_terms(const HotBlock &b, int ea, int &f1, int &o1, int &f2, int &o2)
{
    f1 = ea == 0 ? 1 : 0;
    f2 = ea == 2 ? 1 : 2;
    o1 = ea == 2 ? -int(b.sj) : -1;
    o2 = ea == 0 ? -int(b.sj) : -int(b.si);
}
__device__ __forceinline__ PreUnknown load_unknown(const ResistSolve &a, const HotBlock *hb, int64_t t)
{
    PreUnknown u;
    const int *l = a.uloc + 5 * t;
    u.b = hb + l[0];
    u.ea = l[1];
    u.p = u.b->o + uint32_t(l[2]) * u.b->si + uint32_t(l[3]) * u.b->sj + uint32_t(l[4]);
    u.e = a.e[t];
    u.eta = a.eta[t];
    int f1, o1, f2, o2;
    edge_terms(*u.b, u.ea, f1, o1, f2, o2);
    const double *b1 = hot_at(*u.b, u.p, F_betaxi) + uint64_t(f1) * u.b->vol;
    const double *b2 = hot_at(*u.b, u.p, F_betaxi) + uint64_t(f2) * u.b->vol;
    u.alpha = hot_at(*u.b, u.p, F_alphaxi)[uint64_t(u.ea) * u.b->vol];
    u.beta[0] = b1[0];
    u.beta[1] = b1[o1];
    u.beta[2] = b2[0];
    u.beta[3] = b2[o2];
    return u;
}
// dJ at the unknown's edge (jedge_one's operations), stored; y = Eres - eta dJ
__device__ __forceinline__ double unknown_value(const ResistSolve &a, const PreUnknown &u)
{
    int f1, o1, f2, o2;
    edge_terms(*u.b, u.ea, f1, o1, f2, o2);
    const double *F1 = hot_at(*u.b, u.p, F_dBxi) + uint64_t(f1) * u.b->vol;
    const double *F2 = hot_at(*u.b, u.p, F_dBxi) + uint64_t(f2) * u.b->vol;
    const double h1 = u.beta[0] * F1[0], m1 = u.beta[1] * F1[o1], h2 = u.beta[2] * F2[0], m2 = u.beta[3] * F2[o2];
    const double E = a.pool[u.e];
    const double val = u.ea == 1 ? (h1 - m1) + (m2 - h2) : (m1 - h1) + (h2 - m2);
    const double dJ = val * u.alpha;
    hot_at(*u.b, u.p, F_dJxi)[uint64_t(u.ea) * u.b->vol] = dJ;
    return E - u.eta * dJ;
}
__device__ __forceinline__ PreFused load_fused(const FusedList &l, const HotBlock *hb, int64_t q)
{
    PreFused x;
    x.dst = l.dst[q];
    x.kind = l.kind[q];
    x.idx = l.idx[q];
    x.val = l.val[q];
    x.fa = 0;
    x.b = hb;
    x.p = 0;
    if (x.kind == FUSE_CURL)
    {
        const int k = int(x.idx % 4096) - 64, j = int((x.idx / 4096) % 4096) - 64;
        const int i = int((x.idx / (int64_t(4096) * 4096)) % 4096) - 64;
        x.fa = int(x.idx / (int64_t(4096) * 4096 * 4096));
        x.b = hb + l.blk[q];
        x.p = x.b->o + uint32_t(i) * x.b->si + uint32_t(j) * x.b->sj + uint32_t(k);
    }
    return x;
}
__device__ __forceinline__ PreRegion load_region(const ResistSolve &a, const HotBlock *hb, int64_t q)
{
    PreRegion r{hb, 0u, 0};
    if (a.reg.n >= 0)
    {
        r.b = hb + a.reg.pt[3 * q];
        r.p = a.reg.pt[3 * q + 1];
        r.faces = int(a.reg.pt[3 * q + 2]);
        return r;
    }
    const uint32_t blk = uint32_t(q) / uint32_t(a.nreg);
    r.b = hb + blk;
    int i, j, k;
    if (hot_stagger(*r.b, a.rng, uint32_t(q) - blk * uint32_t(a.nreg), i, j, k, r.p))
        for (int fa = 0; fa < 3; ++fa)
            r.faces |= hot_face(*r.b, fa, i, j, k) ? 1 << fa : 0;
    return r;
}

struct PreItems
{
    PreUnknown u;
    PreFused fa, fb;
    PreRegion r;
};

// y = A src (MatMultImplicitResistive_): Eres at the unknowns and their
// aliases, Sync("Eres1form"), dB = -dt curl Eres on the region, Sync("dB"),
// then per unknown dJ = alpha curlAdj(beta dB) at its edge and y = Eres - eta
// dJ.  What src reads must be complete at entry unless first_barrier: the
// aliases read other threads' elements.  src is the stored basis vector bit
// for bit (the same operations), so the basis vector itself need not be
// complete; y may be the array src reads (it is written after the last
// barrier).  first: the solve's first product, which also writes the points
// whose value no later one changes (the static tails of the lists).
__device__ bool grid_matvec(const ResistSolve &a, GridBar &gb, const HotBlock *hb, const PreItems &pre,
                            const BasisVec &src, bool first_barrier, bool first, double *y)
{
    const int64_t t0 = int64_t(blockIdx.x) * blockDim.x + threadIdx.x, ts = int64_t(gridDim.x) * blockDim.x;
    if (first_barrier && !grid_barrier(gb))
        return false;
    const double mdt = -a.dtp[0];
    if (a.fa.n >= 0)
    {
        // one phase: every Eres point the unknowns, aliases and Sync("Eres1form") set
        for (int64_t q = t0; q < (first ? a.fa.n : a.fa.dyn); q += ts)
        {
            const PreFused x = q == t0 ? pre.fa : load_fused(a.fa, hb, q);
            double v;
            if (x.kind == FUSE_UNKNOWN)
                v = src.at(x.idx);
            else if (x.kind == FUSE_ALIAS)
                v = x.val * src.at(x.idx);
            else if (x.kind == FUSE_CONST)
                v = x.val;
            else
                v = a.pool[x.idx];
            a.pool[x.dst] = v;
        }
        if (!grid_barrier(gb))
            return false;
    }
    else
    {
        for (int64_t t = t0; t < a.n; t += ts)
            a.pool[a.e[t]] = src.at(t);
        for (int64_t q = t0; q < a.nalias; q += ts)
            a.pool[a.alias[q]] = a.sign[q] * src.at(a.alias_of[q]);
        if (a.merge1)
            for (int64_t t = t0; t < a.eres1form.nconst; t += ts)
                a.pool[a.eres1form.cdst[t]] = a.eres1form.cval[t];
        if (!grid_barrier(gb))
            return false;
        if (!grid_apply(a, gb, a.eres1form, a.merge1 != 0))
            return false;
    }
    const int64_t np = a.reg.n >= 0 ? (first ? a.reg.n : a.reg.dyn) : int64_t(a.nblocks) * a.nreg;
    for (int64_t q = t0; q < np; q += ts)
    {
        const PreRegion r = q == t0 ? pre.r : load_region(a, hb, q);
#pragma unroll
        for (int fa = 0; fa < 3; ++fa)
            if (r.faces & (1 << fa))
                *hot_at(*r.b, r.p, F_dBxi + fa) = mdt * hot_curl(*r.b, r.p, plane_of(F_Eresxi), fa);
    }
    // (once per solve where no product writes the points otherwise, as the static tails: the region list is there)
    if (a.merge2 && (first || a.reg.n < 0))
        for (int64_t t = t0; t < a.db.nconst; t += ts)
            a.pool[a.db.cdst[t]] = a.db.cval[t];
    if (a.fb.n >= 0)
    {
        // the Sync("dB") copies in the same phase: each destination takes
        // the curl at its source directly (fixed values were written above)
        for (int64_t q = t0; q < (first ? a.fb.n : a.fb.dyn); q += ts)
        {
            const PreFused x = q == t0 ? pre.fb : load_fused(a.fb, hb, q);
            double v;
            if (x.kind == FUSE_CURL)
                v = mdt * hot_curl(*x.b, x.p, plane_of(F_Eresxi), x.fa);
            else if (x.kind == FUSE_CONST)
                v = x.val;
            else
                v = a.pool[x.idx];
            a.pool[x.dst] = v;
        }
        if (!grid_barrier(gb))
            return false;
    }
    else
    {
        if (!grid_barrier(gb))
            return false;
        if (!grid_apply(a, gb, a.db, a.merge2 != 0))
            return false;
    }
    for (int64_t t = t0; t < a.n; t += ts)
        y[t] = unknown_value(a, t == t0 ? pre.u : load_unknown(a, hb, t));
    return true;
}

// What bounds the solve: the round trips of its phases (a barrier, then the
// dependent loads of the phase's work), with the system resident in L2 and one
// item per thread.  On 6 x 80 x 40 x 40 cells (8440 unknowns, 4 iterations, 21
// barriers) 158 us per solve with a reset barrier, lists read in every phase and
// every point written by every product; 120 with a counting barrier, the lists'
// entries, scales and blocks loaded once into registers and shared memory; 96.6
// with the points that never change written by the first product alone, a CTA
// for every 256 items and release / acquire in place of two fences; 98.6 with the
// elements of other CTAs formed where they are read (BasisVec: before, the
// second pass's result was read without a barrier behind its store).
__global__ void __launch_bounds__(256) k_gmres_resist(ResistSolve a)
{
    __shared__ GmresScalars S;
    __shared__ double dv[32];
    __shared__ HotBlock sblk[kResistBlocks];
    __shared__ int gone;
    GridBar gb = grid_bar(a.bar, a.err, a.h_err);
    const int tid = threadIdx.x;
    if (tid == 0) // a solve of an earlier step gave up: the barrier's words are stale until the host clears them
        gone = *(volatile int *)a.err == MHD_EKRYLOV;
    for (int q = tid; q < min(a.nblocks, kResistBlocks) * int(sizeof(HotBlock) / 4); q += blockDim.x)
        reinterpret_cast<uint32_t *>(sblk)[q] = reinterpret_cast<const uint32_t *>(a.hb)[q];
    __syncthreads();
    if (gone)
        return;
    const HotBlock *hb = a.nblocks <= kResistBlocks ? sblk : a.hb;
    const int64_t t0 = int64_t(blockIdx.x) * blockDim.x + tid, ts = int64_t(gridDim.x) * blockDim.x;
    const int64_t n = a.n;
    int pbuf = 0;
    PreItems pre{};
    if (t0 < n)
        pre.u = load_unknown(a, hb, t0);
    if (t0 < a.fa.n)
        pre.fa = load_fused(a.fa, hb, t0);
    if (t0 < a.fb.n)
        pre.fb = load_fused(a.fb, hb, t0);
    if (t0 < (a.reg.n >= 0 ? a.reg.n : int64_t(a.nblocks) * a.nreg))
        pre.r = load_region(a, hb, t0);
    // right-hand side b = eta J at the unknowns (PackImplicitJedgeToVec_), x = 0
    for (int64_t t = t0; t < n; t += ts)
    {
        a.b[t] = 0.0 + a.eta[t] * a.pool[a.j[t]];
        a.x[t] = 0.0;
    }
    if (!grid_dots(a, gb, nullptr, 1, a.b, dv, pbuf))
        return;
    if (tid == 0)
    {
        S.bnorm = sqrt(dv[0]);
        S.ttol = fmax(a.rtol * S.bnorm, a.atol);
        S.its = 0;
        S.reason = 0;
        S.cycles = 0;
        S.resid = S.bnorm;
    }
    __syncthreads();
    for (;;)
    {
        // cycle start: r = b - A x, beta = ||r||
        if (!grid_matvec(a, gb, hb, pre, BasisVec{a.x, 1.0, nullptr, nullptr, 0, n}, true, S.cycles == 0, a.w))
            return;
        for (int64_t t = t0; t < n; t += ts)
            a.r[t] = a.b[t] - a.w[t];
        if (!grid_dots(a, gb, nullptr, 1, a.r, dv, pbuf))
            return;
        if (tid == 0)
        {
            S.beta = sqrt(dv[0]);
            for (int q = 0; q < 32; ++q)
                S.g[q] = 0.0;
            S.g[0] = S.beta;
            S.resid = S.beta;
            S.breakdown = 0;
            S.j = 0;
            S.inner = 1;
            if (S.beta <= S.ttol)
            {
                S.reason = (S.beta <= a.atol) ? 3 : 2;
                S.inner = 0;
            }
            else if (S.its >= a.maxit)
            {
                S.reason = -3;
                S.inner = 0;
            }
        }
        __syncthreads();
        if (S.inner)
            for (int64_t t = t0; t < n; t += ts)
                a.V[t] = a.r[t] / S.beta;
        while (S.inner)
        {
            const int j = S.j;
            // V_j: r / beta (j = 0), or from the previous step's w', basis
            // and products, complete at the last reduction's barrier
            const BasisVec vj = j == 0 ? BasisVec{a.r, S.beta, nullptr, nullptr, 0, n}
                                       : BasisVec{a.w, S.hcol[j], a.V, S.d, j, n};
            if (!grid_matvec(a, gb, hb, pre, vj, false, false, a.w))
                return;
            // classical Gram-Schmidt, twice
            if (!grid_dots(a, gb, a.V, j + 1, a.w, S.hcol, pbuf))
                return;
            for (int64_t t = t0; t < n; t += ts)
            {
                double s = a.w[t];
                for (int c = 0; c <= j; ++c)
                    s -= S.hcol[c] * a.V[int64_t(c) * n + t];
                a.w[t] = s;
            }
            // second pass, its dots and ||w'||^2 in one reduction: with V
            // orthonormal, ||w' - V d||^2 = ||w'||^2 - ||d||^2; w' itself
            // stays, for the next product's reads of other threads' elements
            if (!grid_dots(a, gb, a.V, j + 1, a.w, S.d, pbuf, true))
                return;
            if (tid <= j)
                S.hcol[tid] += S.d[tid];
            __syncthreads();
            if (tid == 0)
            {
                // new column: rotations, residual estimate
                double dd = 0.0;
                for (int c = 0; c <= j; ++c)
                    dd += S.d[c] * S.d[c];
                const double nw2 = S.d[j + 1] - dd;
                S.hcol[j + 1] = sqrt(nw2 > 0.0 ? nw2 : 0.0);
                for (int i = 0; i <= j + 1; ++i)
                    S.H[i * 31 + j] = S.hcol[i];
                for (int i = 0; i < j; ++i)
                {
                    const double x0 = S.H[i * 31 + j], x1 = S.H[(i + 1) * 31 + j];
                    S.H[i * 31 + j] = S.cs[i] * x0 + S.sn[i] * x1;
                    S.H[(i + 1) * 31 + j] = -S.sn[i] * x0 + S.cs[i] * x1;
                }
                const double x0 = S.H[j * 31 + j], x1 = S.H[(j + 1) * 31 + j];
                const double den = sqrt(x0 * x0 + x1 * x1);
                S.cs[j] = den > 0.0 ? x0 / den : 1.0;
                S.sn[j] = den > 0.0 ? x1 / den : 0.0;
                S.H[j * 31 + j] = den;
                S.H[(j + 1) * 31 + j] = 0.0;
                S.g[j + 1] = -S.sn[j] * S.g[j];
                S.g[j] = S.cs[j] * S.g[j];
                S.resid = fabs(S.g[j + 1]);
                S.breakdown = (S.hcol[j + 1] == 0.0) ? 1 : 0;
            }
            __syncthreads();
            if (!S.breakdown)
            {
                const BasisVec next{a.w, S.hcol[j + 1], a.V, S.d, j + 1, n};
                for (int64_t t = t0; t < n; t += ts)
                    a.V[int64_t(j + 1) * n + t] = next.at(t);
            }
            __syncthreads();
            if (tid == 0)
            {
                S.its += 1;
                S.j += 1;
                S.inner = !(S.resid <= S.ttol || S.breakdown || S.j >= a.m || S.its >= a.maxit);
            }
            __syncthreads();
        }
        // cycle end: H y = g, x += V y
        if (tid == 0)
        {
            const int m = S.j;
            for (int i = m - 1; i >= 0; --i)
            {
                double s = S.g[i];
                for (int q = i + 1; q < m; ++q)
                    s -= S.H[i * 31 + q] * S.y[q];
                S.y[i] = s / S.H[i * 31 + i];
            }
            S.cycles += 1;
        }
        __syncthreads();
        for (int64_t t = t0; t < n; t += ts)
        {
            double s = a.x[t];
            for (int c = 0; c < S.j; ++c)
                s += S.y[c] * a.V[int64_t(c) * n + t];
            a.x[t] = s;
        }
        if (tid == 0)
        {
            S.outer = 0;
            if (S.reason != 0)
                S.outer = 0;
            else if (S.resid <= S.ttol || S.breakdown)
                S.reason = (S.resid <= a.atol) ? 3 : 2;
            else if (S.its >= a.maxit)
                S.reason = -3;
            else
                S.outer = 1;
        }
        __syncthreads();
        if (!S.outer)
            break;
    }
    if (blockIdx.x == 0 && tid == 0)
    {
        GmresState *st = a.st;
        st->its = S.its;
        st->resid = S.resid;
        st->bnorm = S.bnorm;
        st->ttol = S.ttol;
        st->reason = S.reason;
        st->j = S.j;
        st->total_its += S.its;
        st->total_cycles += S.cycles;
        *(volatile unsigned *)(a.bar + 1) = gb.target; // (the count at the next launch's start)
    }
}

// Geometry of one block from its ghost node mesh (mhd_geom.cuh): one thread
// per point of the padded box, one grid row per group (group0, group0 + 1, ...)
__global__ void k_geometry(const BlockView *__restrict__ bvs, int blk, NodeMesh m, int G, int group0, double b0,
                           double b1, double b2)
{
    const BlockView &b = bvs[blk];
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (t >= b.vol)
        return;
    const int k = int(t % b.NK) - b.G;
    const int j = int((t / b.NK) % b.NJ) - b.G;
    const int i = int(t / (int64_t(b.NK) * b.NJ)) - b.G;
    const double gb[3] = {b0, b1, b2};
    geom_point(m, b, group0 + int(blockIdx.y), i, j, k, G, gb);
}

// output-step diagnostics: minima start at +inf, maxima at -inf, max |divB| at 0
__global__ void k_diag_init(unsigned long long *keys)
{
    const int t = threadIdx.x;
    if (t < DIAG_NMIN)
        keys[t] = diag_key(INFINITY);
    else if (t < DIAG_NMIN + DIAG_NQ - 1)
        keys[t] = diag_key(-INFINITY);
    else if (t == DIAG_NMIN + DIAG_NQ - 1)
        keys[t] = diag_key(0.0);
}

// one inner cell per thread, one grid row per block; NaN values are skipped
// (std::min / std::max keep the running value against a NaN)
__global__ void k_diag(const BlockView *__restrict__ bvs, int run, unsigned long long *keys)
{
    const BlockView &b = bvs[blockIdx.y];
    const int64_t t = int64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    unsigned long long kmin[DIAG_NMIN], kmax[DIAG_NQ];
#pragma unroll
    for (int q = 0; q < DIAG_NQ; ++q)
    {
        if (q < DIAG_NMIN)
            kmin[q] = ~0ull;
        kmax[q] = 0ull;
    }
    if ((run < 0 || b.run == run) && t < int64_t(b.ni) * b.nj * b.nk)
    {
        const int k = int(t % b.nk), j = int((t / b.nk) % b.nj), i = int(t / (int64_t(b.nk) * b.nj));
        double v[DIAG_NQ];
        diag_cell(b, i, j, k, v);
#pragma unroll
        for (int q = 0; q < DIAG_NQ; ++q)
            if (v[q] == v[q])
            {
                const unsigned long long key = diag_key(v[q]);
                if (q < DIAG_NMIN)
                    kmin[q] = key;
                kmax[q] = key;
            }
    }
#pragma unroll
    for (int q = 0; q < DIAG_NQ; ++q)
    {
        unsigned long long lo = (q < DIAG_NMIN) ? kmin[q] : ~0ull, hi = kmax[q];
#pragma unroll
        for (int off = 16; off > 0; off >>= 1)
        {
            const unsigned long long olo = __shfl_xor_sync(0xffffffffu, lo, off);
            const unsigned long long ohi = __shfl_xor_sync(0xffffffffu, hi, off);
            lo = (olo < lo) ? olo : lo;
            hi = (ohi > hi) ? ohi : hi;
        }
        if ((threadIdx.x & 31) == 0)
        {
            if (q < DIAG_NMIN && lo != ~0ull)
                atomicMin(&keys[q], lo);
            if (hi != 0ull)
                atomicMax(&keys[DIAG_NMIN + q], hi);
        }
    }
}

// The J edges that read a B_zeta face the Pole rewrite changed (POLE_BZETA
// writes the first cell layer jc at each Pole: J_xi at j = jc, jc + 1 and
// J_eta at j = jc read it): Calc_J_Edge again on the staggered points
// j = jc, jc + 1 of each Pole, after the rewrite.  Every other J edge was
// formed before the rewrite, in the fused B_cell / J-edge pass, from the
// same faces, so the J edges are those of the reference's order (calc_Bcell
// with the rewrite, then Calc_J_Edge) bit for bit.  Work items per Pole:
// (ni + 1) x 2 x (nk + 1).  jeta_ring = 0: without the J_eta ring at jc, which
// POLE_JETA in the same launch overwrites in the reference's order.
__host__ __device__ inline int64_t pole_items(int op, int ni, int nk)
{
    return op == POLE_JEDGE ? int64_t(ni + 1) * 2 * (nk + 1) : pole_work(op == POLE_JCELL_FIRST ? POLE_JCELL : op, ni, nk);
}
__device__ __forceinline__ void pole_jedge_one(const BlockView &b, int side, int64_t t, int jeta_ring)
{
    const int jc = side < 0 ? 0 : b.nj - 1;
    if (t >= pole_items(POLE_JEDGE, b.ni, b.nk))
        return;
    const int k = int(t % (b.nk + 1)), j = jc + int((t / (b.nk + 1)) % 2), i = int(t / (2 * int64_t(b.nk + 1)));
#pragma unroll
    for (int ea = 0; ea < 2; ++ea)
        if (inner_of(b, 1, ea, i, j, k) && (ea == 0 || j != jc || jeta_ring))
            jedge_one(b, ea, i, j, k, F_Bxi, F_Jxi, 1.0);
}

// ---------------------------------------------------------------------------
// The ring sums (POLE_RING_U, POLE_RING_BXI) and ring least squares
// (POLE_BCELL, POLE_EETA_REG / POLE_ERES_REG, POLE_JCELL), a group of threads
// per ring.  The threads form the products of a chunk of k (square roots and
// divisions in parallel, the same operations as pole_one).  Each sum then runs
// in one lane over the pushes in the reference's order (k, then the handler's
// order within k), so it equals the one-thread ring sum bit for bit: a skipped
// push adds +0, which changes no sum that starts at +0.  The normal matrix A
// and the count depend on the geometry only and are summed once per geometry
// (build), nine lanes one entry each; every application sums the right-hand
// side, three lanes one component each, and one lane regularises, solves and
// broadcasts.
// What bounds them: the chain of dependent adds (8 nk for J_cell) and two
// rounds of loads.  J_cell's 8 pushes per k, a square root and four divisions
// each, take a CTA of 128 threads (a warp: 39 us on six shells of 30 to 100
// rings per Pole, the CTA 29); the others, 1 or 3 pushes per k, a warp (U_H and
// B_xi rings 12 us against 25 with a CTA each).
// ---------------------------------------------------------------------------
constexpr int kPoleThreads = 128;
// a ring's group: T threads, K values of k per chunk, at most NQ pushes per k
template <int T> struct PoleGroup
{
    static constexpr int K = T == 32 ? 32 : 64, NQ = T == 32 ? 3 : 8;
    // a row of products is 2 doubles longer than its pushes, so that the lanes
    // that sum read different banks
    static constexpr int ROW = K * NQ + 2;
    static __host__ __device__ constexpr size_t bytes(bool build)
    {
        return ((build ? 9 : 3) * size_t(ROW) + 4) * sizeof(double) + size_t(K) * NQ * sizeof(int);
    }
    static __device__ __forceinline__ int tid() { return int(threadIdx.x) % T; }
    static __device__ __forceinline__ void sync()
    {
        if (T == 32)
            __syncwarp();
        else
            __syncthreads();
    }
};

// One chunk of pushes in shared memory: products (apply: phi s[a] in row a;
// build: s[a] s[c] in row 3 a + c), 0 for a push that is skipped, and its use
// flag.  Push q of k sits at K q + k.
struct PoleChunk
{
    double *p;
    int *ok;
    double *x;   // the solution, three values
    int *status; // 0 solved, 1 no usable push, 2 singular
};

struct PolePush
{
    double s[3], phi;
    bool ok;
};

// the sums of a ring's pushes push(q, k), q < NQ, in order (k, then q): the
// group's lanes < 3 (build: < 9, and lane 9 the count) return them in acc
template <int T, int NQ, class Push>
__device__ __forceinline__ void pole_sum(const PoleChunk &sh, bool build, int nk, Push push, double &acc, int &cnt)
{
    using G = PoleGroup<T>;
    constexpr int K = G::K;
    const int tid = G::tid();
    for (int k0 = 0; k0 < nk; k0 += K)
    {
        const int nl = min(K, (nk - k0 + 7) & ~7); // whole groups of 8; the tail adds zeros
#pragma unroll
        for (int e = tid; e < K * NQ; e += T)
        {
            const int q = e / K, k = k0 + e % K;
            PolePush t{{0.0, 0.0, 0.0}, 0.0, false};
            if (k < nk)
                t = push(q, k);
            sh.ok[e] = t.ok ? 1 : 0;
#pragma unroll
            for (int a = 0; a < 3; ++a)
            {
                if (!build)
                    sh.p[a * G::ROW + e] = t.ok ? t.phi * t.s[a] : 0.0;
                else
#pragma unroll
                    for (int c = 0; c < 3; ++c)
                        sh.p[(3 * a + c) * G::ROW + e] = t.ok ? t.s[a] * t.s[c] : 0.0;
            }
        }
        G::sync();
        if (tid < (build ? 9 : 3))
        {
            const double *x = sh.p + tid * G::ROW;
            constexpr int L = NQ >= 8 ? 1 : NQ >= 3 ? 4 : 8; // k per unrolled group
            for (int l = 0; l < nl; l += L)
            {
                double y[L * NQ];
#pragma unroll
                for (int e = 0; e < L * NQ; ++e)
                    y[e] = x[K * (e % NQ) + l + e / NQ];
#pragma unroll
                for (int e = 0; e < L * NQ; ++e)
                    acc += y[e];
            }
        }
        else if (build && tid == 9)
            for (int e = 0; e < K * NQ; ++e)
                cnt += sh.ok[e];
        G::sync();
    }
}

// k average of a ring (pole_one's POLE_RING_U / POLE_RING_BXI)
__device__ __forceinline__ void pole_ring(const BlockView &b, int side, int op, int64_t t, const PoleChunk &sh)
{
    const bool u = op == POLE_RING_U;
    const int i = u ? int(t / 5) : int(t), m = u ? int(t % 5) : 0, jc = side < 0 ? 0 : b.nj - 1;
    double *F = b.f[u ? F_U : F_Bxi] + int64_t(m) * b.vol + pidx(b, i, jc, 0);
    double acc = 0.0;
    int cnt = 0;
    // phi s = F 1: the value itself
    pole_sum<32, 1>(sh, false, b.nk, [&](int, int k) { return PolePush{{1.0, 0.0, 0.0}, F[k], true}; }, acc, cnt);
    const double avg = __shfl_sync(0xffffffffu, acc, 0) / double(b.nk);
    for (int k = threadIdx.x & 31; k < b.nk; k += 32)
        F[k] = avg;
}

// build: store the ring's A and count (cache[0..8], cache[9]) and return
// false; apply: regularise (trace of |A_aa| or of A_aa), solve, leave x and
// the status in shared memory; true when solved
template <int T>
__device__ bool pole_finish(const PoleChunk &sh, double acc, int cnt, bool build, double *cache, bool trace_abs,
                            bool count_guard)
{
    const int tid = PoleGroup<T>::tid();
    if (build)
    {
        if (tid < 9)
            cache[tid] = acc;
        else if (tid == 9)
            cache[9] = double(cnt);
        if (tid == 0)
            *sh.status = 3;
        PoleGroup<T>::sync();
        return false;
    }
    if (tid < 32)
    {
        const double r0 = __shfl_sync(0xffffffffu, acc, 0), r1 = __shfl_sync(0xffffffffu, acc, 1),
                     r2 = __shfl_sync(0xffffffffu, acc, 2);
        if (tid == 0)
        {
            int st = 0;
            double xs[3] = {0.0, 0.0, 0.0};
            if (count_guard && int(cache[9]) <= 0)
                st = 1;
            else
            {
                double A[3][3] = {
                    {cache[0], cache[1], cache[2]}, {cache[3], cache[4], cache[5]}, {cache[6], cache[7], cache[8]}};
                const double rhs[3] = {r0, r1, r2};
                const double tr =
                    trace_abs ? fabs(A[0][0]) + fabs(A[1][1]) + fabs(A[2][2]) : A[0][0] + A[1][1] + A[2][2];
                const double reg = 1.0e-12 * pole_max1(tr);
                A[0][0] += reg;
                A[1][1] += reg;
                A[2][2] += reg;
                st = pole_solve3(A, rhs, xs) ? 0 : 2;
            }
            *sh.status = st;
            for (int c = 0; c < 3; ++c)
                sh.x[c] = xs[c];
        }
    }
    PoleGroup<T>::sync();
    return *sh.status == 0;
}

__device__ void pole_bcell(const BlockView &b, int side, int64_t t, const PoleChunk &sh, double *cache, bool build)
{
    const int nj = b.nj, nk = b.nk;
    const int64_t v = b.vol;
    const int i = int(t >> 1);
    const bool total = (t & 1) == 0;
    if (build && !total)
        return; // one A per ring, shared by the total and the induced field
    const int jc = side < 0 ? 0 : nj - 1;
    const int jn = side < 0 ? jc + 1 : jc;
    const double sn = side < 0 ? 1.0 : -1.0;
    const double *Aet = b.f[F_JDeta], *Axi = b.f[F_JDxi];
    const double *Bet = b.f[F_Beta], *Bxi = b.f[F_Bxi], *Aadd = b.f[F_Baddeta], *Xadd = b.f[F_Baddxi];
    double acc = 0.0;
    int cnt = 0;
    // outer eta face, low and high xi face of each cell of the ring
    pole_sum<32, 3>(
        sh, build, nk,
        [&](int q, int k) {
            const int64_t p = q == 0 ? pidx(b, i, jn, k) : q == 1 ? pidx(b, i, jc, k) : pidx(b, i + 1, jc, k);
            const double *A = q == 0 ? Aet : Axi;
            const double a0 = A[p], a1 = A[v + p], a2 = A[2 * v + p];
            double f = q == 0 ? Bet[p] : Bxi[p];
            if (total)
                f += q == 0 ? Aadd[p] : Xadd[p];
            PolePush o;
            o.s[0] = q == 0 ? sn * a0 : q == 1 ? -a0 : a0;
            o.s[1] = q == 0 ? sn * a1 : q == 1 ? -a1 : a1;
            o.s[2] = q == 0 ? sn * a2 : q == 1 ? -a2 : a2;
            o.phi = q == 0 ? sn * f : q == 1 ? -f : f;
            o.ok = !((o.s[0] * o.s[0] + o.s[1] * o.s[1] + o.s[2] * o.s[2]) <= 1.0e-300);
            return o;
        },
        acc, cnt);
    // BC_Pole_Bcell_Collapse_ solves whenever the regularised system is regular
    if (!pole_finish<32>(sh, acc, cnt, build, cache, true, false))
        return;
    double *Out = b.f[total ? F_Bcell : F_Bind];
    for (int k = threadIdx.x & 31; k < nk; k += 32)
    {
        const int64_t p = pidx(b, i, jc, k);
        Out[p] = sh.x[0];
        Out[v + p] = sh.x[1];
        Out[2 * v + p] = sh.x[2];
    }
}

// the regulation of E_eta (field F_Eeta) or Eres_eta (F_Ereseta): both are
// eta edges of the same ring, so their normal matrices (from dr_eta) are one
__device__ void pole_eeta(const BlockView &b, int side, int64_t t, const PoleChunk &sh, double *cache, bool build,
                          int field)
{
    const int nj = b.nj, nk = b.nk, tid = threadIdx.x & 31;
    const int64_t v = b.vol;
    const int i = int(t);
    const int jc = side < 0 ? 0 : nj - 1;
    double *E = b.f[field];
    const double *dr = b.f[F_dreta];
    double acc = 0.0;
    int cnt = 0;
    // k = n_k is the same edge as k = 0
    pole_sum<32, 1>(
        sh, build, nk,
        [&](int, int k) {
            const int64_t p = pidx(b, i, jc, k);
            const double d0 = dr[p], d1 = dr[v + p], d2 = dr[2 * v + p];
            const double e = build ? 0.0 : E[p];
            const double L = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
            const double invL = 1.0 / L;
            return PolePush{{d0 * invL, d1 * invL, d2 * invL}, e * invL, !(L < 1.0e-14)};
        },
        acc, cnt);
    if (pole_finish<32>(sh, acc, cnt, build, cache, false, true))
    {
        for (int k = tid; k <= nk; k += 32)
        {
            const int64_t p = pidx(b, i, jc, k);
            const double d0 = dr[p], d1 = dr[v + p], d2 = dr[2 * v + p];
            const double L = sqrt(d0 * d0 + d1 * d1 + d2 * d2);
            E[p] = (L < 1.0e-14) ? 0.0 : sh.x[0] * d0 + sh.x[1] * d1 + sh.x[2] * d2;
        }
        return;
    }
    if (*sh.status == 1) // no usable edge
    {
        for (int k = tid; k <= nk; k += 32)
            E[pidx(b, i, jc, k)] = 0.0;
        return;
    }
    if (*sh.status != 2)
        return; // build
    // singular system: the ring average, summed in k order by one thread
    if (tid == 0)
    {
        double avg = 0.0;
        for (int k = 0; k <= nk; ++k)
            avg += E[pidx(b, i, jc, k)];
        sh.x[0] = avg / double(nk + 1);
    }
    __syncwarp();
    for (int k = tid; k <= nk; k += 32)
        E[pidx(b, i, jc, k)] = sh.x[0];
}

// calc_Jcell of one cell (LunarSolver_Tools.cpp:837-892), with the weights the
// derived pass uses
__device__ void jcell_plain(const BlockView &b, int i, int j, int k)
{
    const double *Jx = b.f[F_Jxi], *Je = b.f[F_Jeta], *Jz = b.f[F_Jzeta];
    const double s[12] = {Jx[pidx(b, i, j, k)],         Jx[pidx(b, i, j + 1, k)],     Jx[pidx(b, i, j, k + 1)],
                          Jx[pidx(b, i, j + 1, k + 1)], Je[pidx(b, i, j, k)],         Je[pidx(b, i + 1, j, k)],
                          Je[pidx(b, i, j, k + 1)],     Je[pidx(b, i + 1, j, k + 1)], Jz[pidx(b, i, j, k)],
                          Jz[pidx(b, i + 1, j, k)],     Jz[pidx(b, i, j + 1, k)],     Jz[pidx(b, i + 1, j + 1, k)]};
    const int64_t p = pidx(b, i, j, k), v = b.vol;
    const int64_t w0 = weight_tile(weight_cell(b, i, j, k), 36);
    for (int c = 0; c < 3; ++c)
    {
        double J = 0.0;
        for (int q = 0; q < 12; ++q)
        {
            const int64_t w = w0 + (12 * c + q) * kWTile;
            J += (b.w32 ? double(b.w32[W32_J * v + w]) : b.f[F_WJ][w]) * s[q];
        }
        b.f[F_Jcell][c * v + p] = J;
    }
}

// first: the derived pass leaves the ring out, so a ring without a solution
// takes calc_Jcell's values here (else it holds them already)
__device__ void pole_jcell(const BlockView &b, int side, int64_t t, const PoleChunk &sh, double *cache, bool build,
                           bool first)
{
    const int nj = b.nj, nk = b.nk;
    const int64_t v = b.vol;
    const int i = int(t);
    const int jc = side < 0 ? 0 : nj - 1;
    const int jt = side < 0 ? jc + 1 : jc; // node plane one layer away from the Pole
    double acc = 0.0;
    int cnt = 0;
    // the 8 pushes of each k, in the order of the reference's loop: the four
    // eta edges of the ring's cell, then two xi and two zeta edges at jt
    pole_sum<kPoleThreads, 8>(
        sh, build, nk,
        [&](int q, int k) {
            const int fa = q < 4 ? 1 : q < 6 ? 0 : 2;
            const int di = q < 4 ? (q & 1) : q == 7, dk = q < 4 ? (q >> 1) : q == 5;
            const int64_t p = pidx(b, i + di, fa == 1 ? jc : jt, k + dk);
            const double *dr = b.f[F_drxi + fa];
            const double dx = dr[p], dy = dr[v + p], dz = dr[2 * v + p];
            const double J = build ? 0.0 : b.f[F_Jxi + fa][p];
            const double L = sqrt(dx * dx + dy * dy + dz * dz);
            return PolePush{{dx / L, dy / L, dz / L}, J / L, !(L < 1.0e-14)};
        },
        acc, cnt);
    const bool solved = pole_finish<kPoleThreads>(sh, acc, cnt, build, cache, false, true);
    if (build || (!solved && !first))
        return;
    double *Jc = b.f[F_Jcell];
    for (int k = threadIdx.x; k < nk; k += kPoleThreads)
    {
        if (!solved)
        {
            jcell_plain(b, i, jc, k);
            continue;
        }
        const int64_t p = pidx(b, i, jc, k);
        Jc[p] = sh.x[0];
        Jc[v + p] = sh.x[1];
        Jc[2 * v + p] = sh.x[2];
    }
}

// which of the three least-squares operations (cache slot), -1 otherwise
__host__ __device__ inline int pole_lsq_slot(int op)
{
    return op == POLE_BCELL                                  ? 0
           : (op == POLE_EETA_REG || op == POLE_ERES_REG)    ? 1
           : (op == POLE_JCELL || op == POLE_JCELL_FIRST)    ? 2
                                                             : -1;
}

// work items of an operation per CTA: rings by a CTA, rings by a warp, items by a thread
__host__ __device__ inline int pole_per_cta(int op)
{
    return pole_lsq_slot(op) == 2                                                      ? 1
           : (op == POLE_RING_U || op == POLE_RING_BXI || pole_lsq_slot(op) >= 0) ? kPoleThreads / 32
                                                                                  : kPoleThreads;
}

// up to four operations on every Pole (grid row).  cache: per Pole, per
// least-squares operation, per ring i (stride rings): A (9 values) and the
// push count
__global__ void __launch_bounds__(kPoleThreads) k_pole(const BlockView *__restrict__ bvs, const int *__restrict__ poles,
                                                       PoleOps ops, double *__restrict__ cache, int stride, int build)
{
    extern __shared__ __align__(16) unsigned char pole_smem[];
    int q = 0;
    while (q + 1 < ops.n && int(blockIdx.x) >= ops.cta0[q + 1])
        ++q;
    const int op = ops.op[q], per = pole_per_cta(op);
    const int64_t cta = int(blockIdx.x) - ops.cta0[q];
    const BlockView &b = bvs[poles[2 * blockIdx.y]];
    const int side = poles[2 * blockIdx.y + 1] > 0 ? 1 : -1;
    pdl_wait();
    if (per == kPoleThreads)
    {
        const int64_t t = cta * kPoleThreads + threadIdx.x;
        if (op == POLE_JEDGE)
            pole_jedge_one(b, side, t, ops.jeta_ring);
        else
            pole_one(b, side, op, t);
        return;
    }
    const int warp = threadIdx.x >> 5;
    const int64_t t = per == 1 ? cta : cta * per + warp;
    if (t >= pole_items(op, b.ni, b.nk))
        return; // the whole group leaves together
    // the group's chunk: products, solution and status, use flags
    unsigned char *mine = pole_smem + (per == 1 ? 0 : warp * PoleGroup<32>::bytes(build != 0));
    const int rows = build ? 9 : 3, row = per == 1 ? PoleGroup<kPoleThreads>::ROW : PoleGroup<32>::ROW;
    double *sp = reinterpret_cast<double *>(mine) + rows * row;
    const PoleChunk sh{reinterpret_cast<double *>(mine), reinterpret_cast<int *>(sp + 4), sp,
                       reinterpret_cast<int *>(sp + 3)};
    if (pole_lsq_slot(op) < 0)
    {
        pole_ring(b, side, op, t, sh);
        return;
    }
    const int ring = op == POLE_BCELL ? int(t >> 1) : int(t);
    double *c = cache + ((int64_t(blockIdx.y) * 3 + pole_lsq_slot(op)) * stride + ring) * 10;
    if (op == POLE_BCELL)
        pole_bcell(b, side, t, sh, c, build != 0);
    else if (op == POLE_EETA_REG || op == POLE_ERES_REG)
        pole_eeta(b, side, t, sh, c, build != 0, op == POLE_ERES_REG ? F_Ereseta : F_Eeta);
    else
        pole_jcell(b, side, t, sh, c, build != 0, op == POLE_JCELL_FIRST);
}

static void pole_launch(PoleOps ops, int ni, int nk, int npoles, cudaStream_t st, const BlockView *bvs,
                        const int *poles, double *cache, int stride, int build)
{
    int x = 0;
    size_t smem = 0;
    for (int q = 0; q < ops.n; ++q)
    {
        const int per = pole_per_cta(ops.op[q]);
        ops.cta0[q] = x;
        x += int((pole_items(ops.op[q], ni, nk) + per - 1) / per);
        smem = std::max(smem, per == 1              ? PoleGroup<kPoleThreads>::bytes(build != 0)
                              : per < kPoleThreads ? per * PoleGroup<32>::bytes(build != 0)
                                                   : size_t(0));
    }
    ops.cta0[ops.n] = x;
    pdl_launch(k_pole, dim3(unsigned(x), unsigned(npoles)), kPoleThreads, smem, st, bvs, poles, ops, cache, stride,
               build);
}

void launch_pole_ops(PoleOps ops, int ni, int nk, int npoles, cudaStream_t st, const BlockView *bvs, const int *poles,
                     double *cache, int stride)
{
    pole_launch(ops, ni, nk, npoles, st, bvs, poles, cache, stride, 0);
}

void launch_pole_build(int op, int ni, int nk, int npoles, cudaStream_t st, const BlockView *bvs, const int *poles,
                       double *cache, int stride)
{
    PoleOps ops{};
    ops.n = 1;
    ops.op[0] = op;
    pole_launch(ops, ni, nk, npoles, st, bvs, poles, cache, stride, 1);
}

} // namespace mhd
