// Kernel declarations shared by the C-ABI implementation.
#pragma once

#include "mhd_layout.cuh"
#include "mhd_hot.cuh"
#include "mhd_pole.cuh"
#include "mhd_geom.cuh"
#include "mhd_output.cuh"
#include "../../include/beta1_mhd.h"

namespace mhd
{

// Nondimensional constants passed by value to the kernels.
struct Consts
{
    double gamma;
    double cfl;
    double inver_MA2;
    double mom_hall;
    double state_coeff;
    double M_H, M_ref;
    double ne_floor;
};

// The runs' clocks (dt_key null: nothing to do)
struct RunClock
{
    unsigned long long *dt_key; // CFL minima in their order-preserving form
    double *dt, *time;
    long long *step;
    int *err;
    double dt_abort;
    int nruns;
    // the host's copy of error word, dt and time (mapped host memory): read
    // after a stream synchronisation, so a step needs no copies back
    volatile int *h_err;
    volatile double *h_dt, *h_time;
};
#ifdef __CUDACC__
__device__ __forceinline__ void begin_run(const RunClock &rc, int r)
{
    const double d = __longlong_as_double((long long)rc.dt_key[r]);
    rc.dt[r] = d;
    rc.h_dt[r] = d;
    // the first error of a span stays: a solve that gave up in an earlier step
    // must not lose its mark, by which later solves leave the barrier alone (no
    // other CTA or kernel touches the word meanwhile, the runs of a batch write
    // one value; an atomic here costs the mixed flux pass 200 bytes of spills)
    if ((!isfinite(d) || d < rc.dt_abort) && rc.err[0] == MHD_OK)
    {
        rc.err[0] = MHD_EDT;
        *rc.h_err = MHD_EDT;
    }
}
__device__ __forceinline__ void end_run(const RunClock &rc, int r)
{
    const double t = rc.time[r] + rc.dt[r];
    rc.time[r] = t;
    rc.h_time[r] = t;
    rc.step[r] += 1;
    rc.dt_key[r] = (unsigned long long)__double_as_longlong(1e100); // dt_local's initial bound
}
#endif

__global__ void k_ucontra(const BlockView *bvs);
__global__ void k_face_normals(const BlockView *bvs);
__global__ void k_divb(const BlockView *bvs);
// mixed precision (mhd_kernels_mixed.cu)
__global__ void k_geom32(const BlockView *bvs);
// Pole operations (mhd_pole.cuh) over every Pole in one launch: up to four
// that touch different points; POLE_JEDGE: Calc_J_Edge again on the J_xi /
// J_eta edges that read the B_zeta faces POLE_BZETA rewrote (staggered layers
// jc, jc + 1 of each Pole; jeta_ring = 0: the ring POLE_JETA writes left out).
// POLE_JCELL_FIRST: POLE_JCELL beside a derived pass that leaves the rings'
// J_cell out.  The ring sums run a warp or a CTA per ring; the least squares' geometry-only normal
// matrices are in `cache` (per Pole, per least-squares operation, `stride`
// rings, 10 values each), which launch_pole_build fills after every geometry
// change.  ni, nk: the largest of the Poles' blocks.
constexpr int POLE_JEDGE = NPOLE_OP, POLE_JCELL_FIRST = NPOLE_OP + 1;
struct PoleOps
{
    int n;
    int op[4];
    int cta0[5]; // first CTA of each operation; the grid's size last
    int jeta_ring;
};
void launch_pole_ops(PoleOps ops, int ni, int nk, int npoles, cudaStream_t st, const BlockView *bvs, const int *poles,
                     double *cache, int stride);
void launch_pole_build(int op, int ni, int nk, int npoles, cudaStream_t st, const BlockView *bvs, const int *poles,
                       double *cache, int stride);
__global__ void k_geometry(const BlockView *bvs, int blk, NodeMesh m, int G, int group0, double b0, double b1,
                           double b2);
// output-step minima / maxima over the inner cells of a run's blocks (run < 0:
// every block); keys[0..DIAG_NMIN) minima, keys[DIAG_NMIN..DIAG_NMIN + DIAG_NQ) maxima
__global__ void k_diag_init(unsigned long long *keys);
__global__ void k_diag(const BlockView *bvs, int run, unsigned long long *keys);
__global__ void k_begin_step(RunClock rc);
__global__ void k_arm_dt(unsigned long long *dt_key, int nruns);
__global__ void k_gather(double *pool, const uint64_t *dst, const uint64_t *src, int64_t n);
// copies and fixed values of one or more Syncs, independent of one another,
// with 64-bit or (pools of fewer than 2^32 points) 32-bit pool offsets
void launch_k_sync(cudaStream_t st, double *pool, const uint64_t *dst, const uint64_t *src, int64_t n,
                   const uint64_t *cdst, const double *cval, int64_t nconst);
void launch_k_sync(cudaStream_t st, double *pool, const uint32_t *dst, const uint32_t *src, int64_t n,
                   const uint32_t *cdst, const double *cval, int64_t nconst);
__global__ void k_set_consts(double *pool, const uint64_t *dst, const double *val, int64_t n);
void launch_k_wall_u(dim3 grid, cudaStream_t st, const BlockView *bvs, const int *walls, double gamma);
__global__ void k_gather_stage(double *tmp, const double *pool, const uint64_t *src, int64_t n);
__global__ void k_scatter_stage(double *pool, const double *tmp, const uint64_t *dst, int64_t n);
__global__ void k_aos_to_soa(const BlockView *bvs, int blk, int fid, int ncomp, int lo0, int lo1, int lo2, int n0,
                             int n1, int n2, const double *aos);
__global__ void k_soa_to_aos(const BlockView *bvs, int blk, int fid, int ncomp, int lo0, int lo1, int lo2, int n0,
                             int n1, int n2, double *aos);

// Krylov (mhd_krylov.cu).  GMRES state kept on the device, including the
// loop control, so that a whole solve runs inside one CUDA graph (conditional
// while nodes) or, eagerly, with the host reading the two loop flags.
// Restart length at most kMaxRestart.
constexpr int kMaxRestart = 30;
struct GmresState
{
    double H[31 * 31]; // H[i * 31 + j]: row i, column j (upper Hessenberg, rotated in place)
    double cs[31], sn[31], g[32];
    double hcol[32]; // h of the current column, then ||w|| at hcol[j + 1]
    double resid;    // |g[j + 1]|
    double beta;     // initial residual norm of the cycle
    double y[31];
    int breakdown;
    // control
    int j;                  // columns built in the current cycle
    int its;                // iterations of the current solve
    int m, maxit;           // restart length, iteration limit
    double ttol, atol;      // max(rtol ||b||, atol), atol
    double bnorm;
    int reason;             // 0 running, 2 rtol, 3 atol, -3 iteration limit
    int inner, outer;       // loop conditions (mirrors of the graph conditionals)
    long long total_its;    // cumulative over all solves
    long long total_cycles; // cumulative over all solves
    unsigned int dot_done[32]; // CTAs finished per dot product (the last one sums the partials)
};
// The implicit resistive solve as one persistent (cooperative) kernel:
// GMRES(m) with the operator, the orthogonalisation and the control flow
// all on the device, CTAs meeting at grid barriers between phases.
struct DevCopy // fixed values then copies of a point list (apply_list)
{
    const uint64_t *cdst;
    const double *cval;
    int64_t nconst;
    const uint64_t *dst, *src;
    double *tmp; // staging when a source is also a destination
    int64_t n;
};
// One point-wise write list of the fused resistive operator: pool[dst[q]] =
// kind 0: x[idx] / div (an unknown), 1: val * (x[idx] / div) (an alias),
// 2: val (a fixed value), 3: pool[idx] (a point no phase writes),
// 4: -dt * (discrete curl of Eres at the face packed in idx, block blk)
struct FusedList
{
    const uint64_t *dst;
    const int *kind;
    const int64_t *idx;
    const double *val;
    const int *blk;
    int64_t n;
    int64_t dyn; // the first dyn depend on the basis vector; the rest stay for the whole solve
};
// The region's faces the curl writes, per staggered point block, offset within
// a plane, face mask (n < 0: the whole region boxes); dyn as above
struct RegionList
{
    const uint32_t *pt;
    int64_t n, dyn;
};
enum : int
{
    FUSE_UNKNOWN = 0,
    FUSE_ALIAS = 1,
    FUSE_CONST = 2,
    FUSE_POOL = 3,
    FUSE_CURL = 4
};
// face packed as ((fa * 4096 + i + 64) * 4096 + j + 64) * 4096 + k + 64
__host__ __device__ inline int64_t fuse_pack(int fa, int i, int j, int k)
{
    return ((int64_t(fa) * 4096 + (i + 64)) * 4096 + (j + 64)) * 4096 + (k + 64);
}

constexpr int kResistBlocks = 24; // blocks the solve keeps in shared memory
struct ResistSolve
{
    const HotBlock *hb; // every block (in shared memory up to kResistBlocks)
    double *pool;
    int nblocks;
    const uint64_t *e, *dj, *j; // unknowns' offsets in Eres, dJ and J
    const double *eta;
    int64_t n;
    const uint64_t *alias; // aliases of unknown owners ...
    const int64_t *alias_of; // ... and the owner's unknown index
    const double *sign;
    int64_t nalias;
    DevCopy eres1form, db;
    const int *uloc; // per unknown: block, edge axis, i, j, k
    int merge1;      // Sync("Eres1form")'s fixed values may go with the unknowns' writes
    int merge2;      // Sync("dB")'s fixed values may go with the curl
    const int *rng; // per block region box
    int64_t nreg;   // points of the largest region box
    const double *dtp;
    double *V, *w, *x, *b, *r;
    double *partial; // 2 x 32 x gridDim.x
    GmresState *st;
    int m, maxit;
    double rtol, atol;
    unsigned *bar; // arrival count, count at the start, polling limit
    int *err;      // set to MHD_EKRYLOV when a barrier wait gives up
    volatile int *h_err; // ... and its copy in host memory
    // fused operator phases (n < 0: not fused, the copy-list phases run):
    // A: every Eres point the unknowns' writes and Sync("Eres1form") set,
    // each as one expression of the basis vector; B: the Sync("dB") copies,
    // each as the curl at its source (or a fixed or unchanged value)
    FusedList fa, fb;
    RegionList reg;
};
__global__ void k_gmres_resist(ResistSolve a);

// dot products out[c] = V_c . w for c < nvec (nvec = *jdev + 1 when jdev is
// given); V == nullptr computes w . w.  Each CTA stores its partial sum; the
// last CTA of each product adds the partials in a fixed order.
__global__ void k_dots(const double *V, int64_t ldv, int nvec, const double *w, int64_t n, double *partial,
                       const int *jdev, double *out, unsigned int *done);
__global__ void k_sub_proj(const double *V, int64_t ldv, int nvec, const double *h, double *w, int64_t n,
                           const int *jdev);
__global__ void k_add_small(double *a, const double *b, const int *jdev);
__global__ void k_div_guard(double *y, const double *x, const double *a, int64_t n, const int *guard);
__global__ void k_div_next(double *V, int64_t ldv, const double *w, const GmresState *st, int64_t n);
__global__ void k_gmres_init(GmresState *st, const double *b2, double rtol, double atol, int maxit, int m);
__global__ void k_cycle_start(GmresState *st, const double *beta2, cudaGraphConditionalHandle h, int use_handle);
__global__ void k_gmres_column(GmresState *st, const double *wnorm2);
__global__ void k_inner_check(GmresState *st, cudaGraphConditionalHandle h, int use_handle);
__global__ void k_gmres_solve_y(GmresState *st);
__global__ void k_add_basis(const double *V, int64_t ldv, const GmresState *st, double *x, int64_t n);
__global__ void k_outer_check(GmresState *st, cudaGraphConditionalHandle h, int use_handle);
__global__ void k_zero(double *x, int64_t n);
__global__ void k_residual(const double *b, const double *y, double *r, int64_t n);
// pool[dst[t]] = x[t] with x = x0 + (*jdev) * ldx when jdev is given
__global__ void k_scatter_vec(double *pool, const uint64_t *dst, const double *x0, int64_t ldx, const int *jdev,
                              int64_t n);
__global__ void k_resist_out(const double *pool, const uint64_t *e, const uint64_t *dj, const double *eta, double *y,
                             int64_t n);
__global__ void k_resist_rhs(const double *pool, const uint64_t *j, const double *eta, double *b, int64_t n);
__global__ void k_alias_copy(double *pool, const uint64_t *alias, const uint64_t *owner, const double *sign,
                             int64_t n);
__global__ void k_pack_vec(const double *pool, const uint64_t *src, double *x, int64_t n);

// Control state of the implicit Hall solve on the device: Newton with a
// backtracking line search around GMRES on finite-difference products.
// One-thread kernels update it and set the loop conditions (the graph's
// conditional handles inside a graph; the mirror flags, read by the host,
// when run eagerly).
struct HallCtl
{
    double f, f0, ft; // ||F|| of the iterate, of the initial guess, of the line-search trial
    double xnorm;     // ||X|| at the start of the Newton step
    double h;         // difference step of a product with a unit basis vector
    double hdx;       // ... with the correction dx (restart residual)
    double lambda;    // line-search step
    double rtol, atol;
    int it, maxit;    // Newton steps taken / allowed
    int cut;          // line-search halvings in this step
    int reason;       // 2 ||F|| <= atol, 3 ||F|| <= rtol ||F0||, -5 step limit
    int first;        // the first GMRES cycle of the Newton step (r = b, dx = 0, no product)
    int r_is_b;       // ... the cycle under way
    int newton, ls, restart; // loop conditions
    long long lin0;          // cumulative GMRES iterations before this solve
    long long pass[3];       // cumulative: Newton steps, restart products, line-search trials
};
// products per multi-dot pass: up to kMaxRestart + 1 basis vectors and one norm
constexpr int kMdMax = 32;
__global__ void k_hall_begin(HallCtl *c, const double *f2, const GmresState *st, double rtol, double atol, int maxit,
                             cudaGraphConditionalHandle h, int use);
__global__ void k_hall_step_begin(HallCtl *c, GmresState *st, const double *bx2, double rtol, double atol, int maxit,
                                  int m, cudaGraphConditionalHandle hout, int use);
__global__ void k_hall_cycle_prep(HallCtl *c, const double *dx2, cudaGraphConditionalHandle h, int use);
__global__ void k_hall_ls_begin(HallCtl *c, cudaGraphConditionalHandle h, int use);
__global__ void k_hall_ls_check(HallCtl *c, const double *ft2, cudaGraphConditionalHandle h, int use);
__global__ void k_hall_accept(HallCtl *c, cudaGraphConditionalHandle h, int use);
// what the points beside the unknowns take at a trial: n1 times sign x
// unknown idx, n2 copies of points no trial writes, n3 fixed values
struct HallList
{
    const uint64_t *d1;
    const int64_t *idx;
    const double *sign;
    int64_t n1;
    const uint64_t *d2, *s2;
    int64_t n2;
    const uint64_t *d3;
    const double *val;
    int64_t n3;
};
// Xt = X + (*a) v (v = v0 + (*jdev) ldv; Xt = X when a is null), written into the pool's unknowns
__global__ void k_hall_trial(double *pool, const uint64_t *e, const double *X, const double *a, const double *v0,
                             int64_t ldv, const int *jdev, double *Xt, int64_t n, HallList l);
// w = ((Xt - pool[e]) - F) / *h and out[c] = V_c . w for c <= j
__global__ void k_hall_jv_dots(const double *pool, const uint64_t *e, const double *Xt, const double *F,
                               const double *h, double *w, const double *V, int64_t ldv, const GmresState *st,
                               int64_t n, double *partial, double *out, unsigned *done);
// w -= sum_c hcol[c] V_c; out[c] = V_c . w (c <= j), out[j + 1] = w . w; then,
// in the last CTA, the Hessenberg column, the counters and the loop condition
__global__ void k_hall_proj_dots(const double *V, int64_t ldv, GmresState *st, double *w, int64_t n, double *partial,
                                 double *out, unsigned *done, cudaGraphConditionalHandle h, int use);
// V_{j+1} = (w - sum_c d[c] V_c) / hcol[j + 1], j the column just counted
__global__ void k_hall_next(double *V, int64_t ldv, const double *w, const GmresState *st, const double *d,
                            int64_t n);
// Ft = Xt - pool[e]; out[0] = Ft . Ft
__global__ void k_hall_res_dots(const double *pool, const uint64_t *e, const double *Xt, double *Ft, int64_t n,
                                double *partial, double *out, unsigned *done);
// r = b - ((Xt - pool[e]) - F) / *h
__global__ void k_hall_restart_r(const double *pool, const uint64_t *e, const double *Xt, const double *F,
                                 const double *h, const double *b, double *r, int64_t n);
// b = -F, r = b, dx = 0; out[0] = b . b, out[1] = X . X
__global__ void k_hall_gmres_prologue(const double *F, double *b, double *r, double *dx, const double *X, int64_t n,
                                      double *partial, double *out, unsigned *done);
// out[0] = x . x; where *known is set the value is *val already (val null: nobody asks for it)
__global__ void k_norm2(const double *x, int64_t n, double *partial, double *out, unsigned *done, const int *known,
                        const double *val);
// X = Xt, F = Ft
__global__ void k_hall_take(double *X, const double *Xt, double *F, const double *Ft, int64_t n);
// dst = src over nseg segments (seg: dst offset, src offset, length)
__global__ void k_copy_segments(double *dst, const double *src, const int64_t *seg, int nseg);


// Hot stencil kernels of a step (mhd_kernels_step.cu, mhd_kernels_mixed.cu).
// Each launcher returns its number of launches (one per chunk of blocks, see
// HotGrid) or -1 for an unknown variant; variants are register / occupancy
// forms of the same code (minimum CTAs per SM of the launch bounds) with the
// same bits, variant 0 the default.
// k_pv_uplus_dt (KIND_CELL1): minimum CTAs per SM 4, 1, 5, and variant 3: at 4
// without J_cell, which launch_k_jcell computes in a pass of its own before
// it; w32: J_cell from the FP32 weight copies (mixed form)
int launch_k_pv_uplus_dt(int variant, bool w32, const HotGrid &h, cudaStream_t st, Consts c, unsigned long long *dt_key);
// PV_H, U_plus and the face states on the whole array
int launch_k_pv_all(const HotGrid &h, cudaStream_t st, Consts c);
// fluid RHS and contravariant velocities: minimum CTAs per SM 2, 3
// (rc: the start of the step's run clocks, in the same launch)
int launch_k_fluid_ucontra(int variant, const HotGrid &h, cudaStream_t st, Consts c, RunClock rc);
// B_cell with the J edges: minimum CTAs per SM 2, 6; w32 as above
// (ind = false: without Bind_cell, FP64 weights; the Hall solve's trials)
int launch_k_bcell_jedge(int variant, bool w32, const HotGrid &h, cudaStream_t st, bool ind = true);
// B_cell alone, the J edges of (fB0, fJ0) alone (rng: per block a region box
// lo[3], hi[3] of at most nreg points; null: every inner edge), J_cell alone
int launch_k_bcell(const HotGrid &h, cudaStream_t st);
int launch_k_jedge(const HotGrid &h, cudaStream_t st, int fB0, int fJ0, const int *rng, int64_t nreg);
int launch_k_jcell(bool w32, const HotGrid &h, cudaStream_t st);
// the components of Eface that are zero; face EMF (the others): minimum CTAs per SM 2, 6; edge EMF: 3, 8
int launch_k_eface_zero(const HotGrid &h, cudaStream_t st);
int launch_k_eface(int variant, const HotGrid &h, cudaStream_t st);
int launch_k_eedge(int variant, const HotGrid &h, cudaStream_t st);
// RHS = mult curl E and B += dt / dtdiv RHS on the inner faces (fR0, fB0 < 0:
// not written; rng, nreg as above): minimum CTAs per SM 4, 6.  bs (may be
// null): B = B* + dt RHS with B* from a snapshot (bs[3 block + axis]: the
// snapshot's B arrays of each block, pool layout)
int launch_k_curl_e2f(int variant, const HotGrid &h, cudaStream_t st, int fE0, int fR0, int fB0, double mult,
                      const double *dtp, double dtdiv, int mult_is_neg_dt, const int *rng, int64_t nreg,
                      const double *const *bs = nullptr);
// the Euler update of the inner cells and faces in one pass, U += dt RHS_H and
// RHS_B = -curl E (stored in fR0 when >= 0), B += dt RHS_B; rc: the end of the
// step's run clocks.  Variants of k_curl_e2f.
int launch_k_update(int variant, const HotGrid &h, cudaStream_t st, int fR0, const double *dtp, RunClock rc);
int launch_k_rk2(const HotGrid &h, cudaStream_t st, int save);
int launch_k_eres_explicit(const HotGrid &h, cudaStream_t st, double inver_Rem);
// Hall cell EMF on every ghost layer, or (all = false) one, as deep as the edge EMF reads
int launch_k_hall_cell(const HotGrid &h, cudaStream_t st, Consts c, double hall_coef, bool all);
// Hall edge EMF (zb: boxes of zeroed edges): minimum CTAs per SM 4, 2
int launch_k_hall_edge(int variant, const HotGrid &h, cudaStream_t st, const int *zb, int nzb);
// k_fluid_mixed: minimum CTAs per SM 4, 1, 2; variants 3 and 4 are the
// face-tiled kernels (on `tiles`, the KIND_TILE1 grid of bvs)
int launch_k_fluid_mixed(int variant, const HotGrid &h, dim3 tiles, cudaStream_t st, const BlockView *bvs, Consts c,
                         RunClock rc);

} // namespace mhd
