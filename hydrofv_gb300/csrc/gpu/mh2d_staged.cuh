/*
 * mh2d_staged.cuh -- the FP64 2D step in three kernels per time step.
 *
 *   recon    per cell and direction: limited slopes and the Hancock half
 *            step, the states at the cell's two faces
 *            (src/integrator_muscl_hancock.c:682-755, :967-1041);
 *   flux     per face: the HLLC flux and its update term (F dt) A
 *            (src/riemann_solver_hllc.c:202-376);
 *   update   per cell: the gather in the reference's order, gravity, U -> W,
 *            the next step's CFL maxima; the last block advances the clock
 *            and forms the next step's dt.
 *
 * The pointwise arithmetic is that of numerics.cuh, so the results are the
 * bits of the reference's step (and of the fused kernel of mh2d_kernel.cuh).
 *
 * Why three kernels.  The fused kernel marches rows: a work item's rows are a
 * serial chain of divides, square roots and pow with four barriers each, so a
 * step costs at least one item (about 270 us) however small the grid is, and
 * 16 warps per SM (128 registers) cannot hide those chains.  One thread per
 * face or cell makes the step as long as three short chains and fills the
 * chip from a few thousand cells on; each kernel takes only the registers of
 * its own part, so more warps are resident.  The price is the workspace:
 * about 530 bytes per cell-update pass through L2 or HBM, 17% of the HBM rate
 * at 2.2 G cell-updates/s, under the arithmetic.  Time per step, fused ->
 * staged with the fused kernel's arithmetic: 64^2 276 -> 47 us, 122^2 with
 * gravity 282 -> 58, 401 x 250 van Leer 308 -> 113, 1024^2 blast 0.86 -> 0.65
 * ms, 2048^2 3.25 -> 3.07 ms.
 *
 * Blocks per SM: flux 4 / 5 / 6 / 7 takes 1.99 / 1.89 / 1.90 / 1.88 ms a step
 * on the 2048^2 shear layer and 0.356 / 0.338 / 0.347 / 0.348 on the 1024^2
 * blast; recon is the same with 5 to 8, update with 4 to 6.
 */
#ifndef HYDRO_GPU_MH2D_STAGED_CUH
#define HYDRO_GPU_MH2D_STAGED_CUH

#include "gpu_internal.h"
#include "staged_math.cuh"
#include "step_loop.cuh"

#ifndef MH2D_RECON_CTAS
#define MH2D_RECON_CTAS 6
#endif
#ifndef MH2D_FLUX_CTAS
#define MH2D_FLUX_CTAS 5
#endif
#ifndef MH2D_UPDATE_CTAS
#define MH2D_UPDATE_CTAS 5
#endif
#ifndef MH2D_LOOP_CTAS
#define MH2D_LOOP_CTAS 4
#endif

namespace hydro {

constexpr int kStagedThreads = 128;

/* Largest number of recon items (about two per cell) that steps in the
 * many-step kernel.  Time per step, three launches replayed from a graph
 * against the many-step kernel: 64^2 25.7 / 20.1 us, 128^2 29.9 / 26.1, 192^2
 * 38.2 / 34.2, 256^2 55.2 / 50.0, 320^2 71.5 / 71.1, 384^2 89.0 / 88.8, 512^2
 * 139 / 139; without a graph (short runs) the three launches take at least 34
 * us of host time. */
#ifndef MH2D_LOOP_ITEMS
#define MH2D_LOOP_ITEMS 200000
#endif
constexpr unsigned kStagedLoopItems = MH2D_LOOP_ITEMS;

/* Largest number of faces that the many-step kernel solves with their states
 * in one phase (staged_recon_flux): a grid barrier and a pass through the
 * workspace less, two threads a face, as long as that is one round of the
 * resident blocks (608 of 64 faces).  Time per step, two phases / one: 32^2
 * 22.1 / 20.0 us, 64^2 22.1 / 20.1, 96^2 23.3 / 22.8, 128^2 27.1 / 26.1, 160^2
 * 29.8 / 37.3. */
#ifndef MH2D_FUSED_FACES
#define MH2D_FUSED_FACES 35000
#endif
constexpr unsigned kStagedFusedFaces = MH2D_FUSED_FACES;
/* Blocks of the update kernel: the chip's 152 SMs full (on fewer, they take
 * turns). */
constexpr unsigned kStagedUpdateGrid = 152 * MH2D_UPDATE_CTAS;

/* Fields of the workspace: the low and high face states of each cell in x
 * and y.  The flux kernel leaves a face's update term where its left (lower)
 * state was. */
enum : int { WS_XLO = 0, WS_XHI = 4, WS_YLO = 8, WS_YHI = 12, WS_FIELDS = 16 };

inline __host__ __device__ unsigned staged_recon_items(int nx, int rows) { return (unsigned) rows * (nx + 2) + (unsigned) (rows + 2) * nx; }
inline __host__ __device__ unsigned staged_face_items(int nx, int rows) { return (unsigned) rows * (nx + 1) + (unsigned) (rows + 1) * nx; }

/* Face states of item k of the band: first the x items (rows r0 .. r1-1,
 * columns g-1 .. g+nx), then the y items (rows r0-1 .. r1, columns g ..
 * g+nx-1). */
template <int LIM, int FIRST_ORDER>
__device__ __forceinline__ void staged_recon(const Mh2dArgs<double> &a, const Mh2dBand &b, unsigned k, int buf, bool raw,
                                             const double dtA[2])
{
    const unsigned nx = (unsigned) a.nx, nX = (unsigned) (b.r1 - b.r0) * (nx + 2);
    const bool y = k >= nX;
    int r, c;
    if (!y) {
        const unsigned q = k / (nx + 2);
        r = b.r0 + (int) q;
        c = a.g - 1 + (int) (k - q * (nx + 2));
    } else {
        const unsigned j = k - nX, q = j / nx;
        r = b.r0 - 1 + (int) q;
        c = a.g + (int) (j - q * nx);
    }
    const double *const *W = a.W[buf];
    const double *const *U = a.U[buf];
    double w[5];
    fetch_w(a, W, U, raw, r, c, w);
    const double n = y ? w[2] : w[1], t = y ? w[1] : w[2];
    double lo[4], hi[4];
    if (FIRST_ORDER) {
        lo[0] = hi[0] = w[0]; lo[1] = hi[1] = n; lo[2] = hi[2] = t; lo[3] = hi[3] = w[3];
    } else {
        double wm[5], wp[5];
        fetch_w(a, W, U, raw, y ? r - 1 : r, y ? c : c - 1, wm);
        fetch_w(a, W, U, raw, y ? r + 1 : r, y ? c : c + 1, wp);
        const Fm f = make_fm();
        double s[4];
#pragma unroll
        for (int q = 0; q < 4; q++) s[q] = slope_of<LIM>(f, wm[q], w[q], wp[q]);
        const double h = y ? dtA[1] : dtA[0];
        if (flat(s, w[0], n, t, w[3]) && fx::moderate(h)) {
            lo[0] = hi[0] = w[0]; lo[1] = hi[1] = n; lo[2] = hi[2] = t; lo[3] = hi[3] = w[3];
        } else {
            const double d[4] = { s[0], y ? s[2] : s[1], y ? s[1] : s[2], s[3] };
            predict(f, h, dvi(h, w[0]), w[0], n, t, w[3], w[4], d, s[1], lo, hi);
        }
    }
    double *o = b.ws + (long long) (r - b.r0 + 1) * a.pitch + c + (y ? WS_YLO : WS_XLO) * b.plane;
#pragma unroll
    for (int q = 0; q < 4; q++) {
        o[q * b.plane] = lo[q];
        o[(4 + q) * b.plane] = hi[q];
    }
}

/* The state at the high or low face of cell (r, c) in y or x (staged_recon). */
template <int LIM, int FIRST_ORDER>
__device__ __forceinline__ void face_side(const Fm &f, const Mh2dArgs<double> &a, bool y, int r, int c, bool high, int buf, bool raw,
                                          const double dtA[2], double o[4])
{
    const double *const *W = a.W[buf];
    const double *const *U = a.U[buf];
    double w[5];
    fetch_w(a, W, U, raw, r, c, w);
    const double n = y ? w[2] : w[1], t = y ? w[1] : w[2];
    o[0] = w[0]; o[1] = n; o[2] = t; o[3] = w[3];
    if (FIRST_ORDER) return;
    double wm[5], wp[5], s[4];
    fetch_w(a, W, U, raw, y ? r - 1 : r, y ? c : c - 1, wm);
    fetch_w(a, W, U, raw, y ? r + 1 : r, y ? c : c + 1, wp);
#pragma unroll
    for (int q = 0; q < 4; q++) s[q] = slope_of<LIM>(f, wm[q], w[q], wp[q]);
    const double h = y ? dtA[1] : dtA[0];
    if (flat(s, w[0], n, t, w[3]) && fx::moderate(h)) return;
    const double d[4] = { s[0], y ? s[2] : s[1], y ? s[1] : s[2], s[3] };
    predict_side(f, high, h, dvi(h, w[0]), w[0], n, t, w[3], w[4], d, s[1], o);
}

struct FluxShared {
    static constexpr int NT = kStagedThreads;
    double rho[2][NT], u[2][NT], p[2][NT], a[2][NT];   /* both states of each face */
    double pg[NT];                                     /* star-pressure guess */
    short listT[NT], listS[NT];
    int nT, nS;
};

/* Where face k of the band lies: x faces first (row-major, nx + 1 a row), then
 * y faces; (r, c) is its left or lower cell. */
__device__ __forceinline__ bool face_at(const Mh2dArgs<double> &a, const Mh2dBand &b, unsigned k, int &r, int &c)
{
    const unsigned nx = (unsigned) a.nx, nX = (unsigned) (b.r1 - b.r0) * (nx + 1);
    const bool y = k >= nX;
    if (!y) {
        const unsigned q = k / (nx + 1);
        r = b.r0 + (int) q;
        c = a.g - 1 + (int) (k - q * (nx + 1));
    } else {
        const unsigned j = k - nX, q = j / nx;
        r = b.r0 - 1 + (int) q;
        c = a.g + (int) (j - q * nx);
    }
    return y;
}

/* The flux of one block's faces, one per thread with `on`: at (r, c), in y or
 * x, with the states L and R.  Faces are classified, the expensive guesses run
 * on compacted lists, and each thread finishes its own face from registers.
 * INL: the finish's quotients in line (staged_math.cuh). */
template <bool TAPE, bool INL>
__device__ __forceinline__ void face_flux(const Fm &fm, const Mh2dArgs<double> &a, const Mh2dBand &b, FluxShared &sm, bool on, bool y,
                                          int r, int c, const double L[4], const double R[4], double dt)
{
    const int tid = threadIdx.x;
    bool plain = true;
    const long long at = (long long) (r - b.r0 + 1) * a.pitch + c, tape_at = (long long) r * a.pitch + c;
    double aL = 0, aR = 0, pg = 0;
    int reg = PREG_PVRS;
    bool guessed = false;
    if (tid == 0) { sm.nT = 0; sm.nS = 0; }
    __syncthreads();
    if (on) {
        reg = face_classify(fm, a.gas, L[0], L[1], L[3], R[0], R[1], R[3], aL, aR, pg, plain);
        double p_min;
        if (reg == PREG_TRRS && plain && both_rarefactions(fm, a.gas, L[1], L[3], aL, R[1], R[3], aR, p_min)) pg = p_min;
        else guessed = reg == PREG_TRRS || reg == PREG_TSRS;
        if (guessed) {
            sm.rho[0][tid] = L[0]; sm.u[0][tid] = L[1]; sm.p[0][tid] = L[3]; sm.a[0][tid] = aL;
            sm.rho[1][tid] = R[0]; sm.u[1][tid] = R[1]; sm.p[1][tid] = R[3]; sm.a[1][tid] = aR;
            sm.pg[tid] = pg;
            if (reg == PREG_TRRS) sm.listT[atomicAdd(&sm.nT, 1)] = (short) tid;
            else sm.listS[atomicAdd(&sm.nS, 1)] = (short) tid;
        }
    }
    __syncthreads();
    double z0 = 0, z1 = 0;
    const int nT = sm.nT, nS = sm.nS;
    for (int i = tid; i < nT + nS; i += kStagedThreads) {
        if (i < nT) {
            const int f = sm.listT[i];
            sm.pg[f] = face_trrs(fm, a.gas, sm.u[0][f], sm.p[0][f], sm.a[0][f], sm.u[1][f], sm.p[1][f], sm.a[1][f], z0, z1);
            if constexpr (TAPE) { sm.rho[0][f] = z0; sm.rho[1][f] = z1; }
        } else {
            const int f = sm.listS[i - nT];
            sm.pg[f] = face_tsrs<INL>(fm, a.gas, sm.rho[0][f], sm.u[0][f], sm.p[0][f], sm.rho[1][f], sm.u[1][f], sm.p[1][f],
                                      sm.pg[f], z0, z1);
            if constexpr (TAPE) { sm.rho[0][f] = z0; sm.rho[1][f] = z1; }
        }
    }
    __syncthreads();
    if (!on) return;
    double F[4];
    double wave[3] = { 0.0, 0.0, 0.0 };
    if (guessed) pg = sm.pg[tid];
    if (reg == PREG_VACUUM) {
        vacuum_flux_dev(a.gas, L[0], L[1], L[2], L[3], aL, R[0], R[1], R[2], R[3], aR, F);
    } else {
        const int rc = face_finish<INL>(fm, a.gas, plain, L[0], L[1], L[2], L[3], aL, R[0], R[1], R[2], R[3], aR, pg, F, wave);
        if (rc) record_error(a.ctrl, rc, (int) blockIdx.x);
    }
    if constexpr (TAPE) {
        double *t = a.tape + (y ? MH2D_TAPE_FIELDS : 0) * a.tape_plane + tape_at;
        const double v[MH2D_TAPE_FIELDS] = { L[0], L[1], L[2], L[3], R[0], R[1], R[2], R[3], aL, aR, pg,
                                             guessed ? sm.rho[0][tid] : 0.0, guessed ? sm.rho[1][tid] : 0.0,
                                             (double) reg, wave[0], wave[1], wave[2] };
#pragma unroll
        for (int q = 0; q < MH2D_TAPE_FIELDS; q++) t[q * a.tape_plane] = v[q];
    }
    const double A = y ? a.area_y : a.area_x;
    double *o = b.ws + (y ? WS_YHI : WS_XHI) * b.plane + at;
#pragma unroll
    for (int q = 0; q < 4; q++) o[q * b.plane] = fm.mul(fm.mul(F[q], dt), A);
}

/* Faces k0 .. of one block from the workspace's states. */
template <bool TAPE, bool INL>
__device__ __forceinline__ void staged_flux(const Mh2dArgs<double> &a, const Mh2dBand &b, FluxShared &sm, unsigned k,
                                            unsigned total, double dt)
{
    const Fm fm = make_fm();
    const bool on = k < total;
    bool y = false;
    int r = b.r0, c = a.g;
    double L[4], R[4];
    if (on) {
        y = face_at(a, b, k, r, c);
        const long long at = (long long) (r - b.r0 + 1) * a.pitch + c;
        const double *l = b.ws + (y ? WS_YHI : WS_XHI) * b.plane + at;
        const double *h = b.ws + (y ? WS_YLO : WS_XLO) * b.plane + at + (y ? a.pitch : 1);
#pragma unroll
        for (int q = 0; q < 4; q++) { L[q] = l[q * b.plane]; R[q] = h[q * b.plane]; }
    }
    face_flux<TAPE, INL>(fm, a, b, sm, on, y, r, c, L, R, dt);
}

/* Faces k0 .. of one block, half as many as threads: each thread forms one
 * side's state, then the first half solves the faces.  Every cell's slopes are
 * formed by both of its faces, but the states pass through shared memory
 * instead of the workspace and a grid barrier. */
template <int LIM, int FIRST_ORDER>
__device__ __forceinline__ void staged_recon_flux(const Mh2dArgs<double> &a, const Mh2dBand &b, FluxShared &sm, double (*v)[kStagedThreads / 2],
                                                  unsigned k0, unsigned total, double dt, int buf, bool raw, const double dtA[2])
{
    constexpr int half = kStagedThreads / 2;
    const Fm fm = make_fm();
    const int right = threadIdx.x >= half, f = threadIdx.x - right * half;
    const bool on = k0 + f < total;
    bool y = false;
    int r = b.r0, c = a.g;
    double L[4], R[4];
    if (on) {
        y = face_at(a, b, k0 + f, r, c);
        face_side<LIM, FIRST_ORDER>(fm, a, y, y ? r + right : r, y ? c : c + right, !right, buf, raw, dtA, L);
        if (right) { sm.rho[1][f] = L[0]; sm.u[1][f] = L[1]; v[0][f] = L[2]; sm.p[1][f] = L[3]; }
    }
    __syncthreads();
    if (on && !right) { R[0] = sm.rho[1][f]; R[1] = sm.u[1][f]; R[2] = v[0][f]; R[3] = sm.p[1][f]; }
    face_flux<false, true>(fm, a, b, sm, on && !right, y, r, c, L, R, dt);
}

/* Cell k of the band: update, gravity, U -> W; mx receives a + |u|, a + |v|. */
template <bool GRAV>
__device__ __forceinline__ void staged_update(const Fm &f, const Mh2dArgs<double> &a, const Mh2dBand &b, unsigned k, int buf, double dt,
                                              double &mx_x, double &mx_y)
{
    const int ymap[4] = { 0, 2, 1, 3 };   /* y fluxes come back as (mass, mom_y, mom_x, energy) */
    const unsigned nx = (unsigned) a.nx, q0 = k / nx;
    const int r = b.r0 + (int) q0, c = a.g + (int) (k - q0 * nx);
    const long long idx = (long long) r * a.pitch + c;
    const double *fx = b.ws + WS_XHI * b.plane + (long long) (r - b.r0 + 1) * a.pitch + c;
    const double *fy = b.ws + WS_YHI * b.plane + (long long) (r - b.r0 + 1) * a.pitch + c;
    const double *const *Uin = a.U[buf];
    double *const *Uout = a.U[buf ^ 1];
    double *const *Wout = a.W[buf ^ 1];
    double Un[4], fl[4], fh[4], gl[4], gh[4];
#pragma unroll
    for (int q = 0; q < 4; q++) {
        fl[q] = fx[q * b.plane - 1];
        fh[q] = fx[q * b.plane];
        gl[q] = fy[ymap[q] * b.plane - a.pitch];
        gh[q] = fy[ymap[q] * b.plane];
        Un[q] = Uin[q][idx];
    }
    /* the first ghost layer receives its one-sided update (here, so that its
     * loads are in flight with the others) */
    if (c == a.g) {
#pragma unroll
        for (int q = 0; q < 4; q++) Uout[q][idx - 1] = f.sub(Uin[q][idx - 1], fl[q]);
    }
    if (c == a.g + a.nx - 1) {
#pragma unroll
        for (int q = 0; q < 4; q++) Uout[q][idx + 1] = f.add(Uin[q][idx + 1], fh[q]);
    }
    if (r == a.g) {
#pragma unroll
        for (int q = 0; q < 4; q++) Uout[q][idx - a.pitch] = f.sub(Uin[q][idx - a.pitch], gl[q]);
    }
    if (r == a.g + a.ny - 1) {
#pragma unroll
        for (int q = 0; q < 4; q++) Uout[q][idx + a.pitch] = f.add(Uin[q][idx + a.pitch], gh[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; q++) {
        Un[q] = f.sub(f.add(f.sub(f.add(Un[q], fl[q]), fh[q]), gl[q]), gh[q]);
    }
    if constexpr (GRAV) gravity_kick(-dt * a.gravity, Un[0], Un[2], Un[3]);
#pragma unroll
    for (int q = 0; q < 4; q++) Uout[q][idx] = Un[q];
    double w[4];
    to_primitive(f, a.gas, a.vol, Un[0], Un[1], Un[2], Un[3], w);
    const double as = sqi(dvi(f.mul(a.gas.gamma, w[3]), w[0]));
#pragma unroll
    for (int q = 0; q < 4; q++) Wout[q][idx] = w[q];
    Wout[4][idx] = as;
    const double sx = f.add(as, fabs(w[1])), sy = f.add(as, fabs(w[2]));
    if (lt(mx_x, sx)) mx_x = sx;
    if (lt(mx_y, sy)) mx_y = sy;
}

struct UpdateShared {
    unsigned long long red[2][kStagedThreads / 32];
    int am_last;
};

/* End of an update block: fold its maxima into the next step's words; the
 * last block of the grid advances the clock (src/integrator_muscl_hancock.c:
 * 1143-1154) and forms the next dt. */
__device__ __forceinline__ void staged_finish(const Mh2dArgs<double> &a, UpdateShared &sm, unsigned blocks, long long n,
                                              double dt, double mx_x, double mx_y)
{
    const int tid = threadIdx.x;
    HydroStepControl *ctrl = a.ctrl;
    block_maxima<kStagedThreads>(ctrl, sm.red, n, mx_x, mx_y);
    if (tid == 0) {
        __threadfence();
        sm.am_last = atomicAdd(&ctrl->blocks_done, 1u) == blocks - 1;
    }
    __syncthreads();
    if (!sm.am_last || tid >= 32) return;
    __threadfence();
    advance_clock(a, ctrl, n, ((volatile HydroStepControl *) ctrl)->t, ((volatile HydroStepControl *) ctrl)->tf, dt);
}

/* The step's n and dt, or false when nothing is to be done (not active, or
 * dt is zero, which the recon kernel records). */
__device__ __forceinline__ bool staged_step(HydroStepControl *ctrl, long long &n, double &dt)
{
    const int active = ctrl->active;
    n = ctrl->num_steps;
    dt = ctrl->step_dt;
    return active && dt != 0.0;
}

/* A step that was due but has a zero dt. */
__device__ __forceinline__ void record_zero_dt(HydroStepControl *ctrl)
{
    if (!ctrl->active || ctrl->error_code != 0) return;
    ctrl->dt = 0.0;
    record_error(ctrl, DEV_ERR_DT_ZERO, -1);
    ctrl->active = 0;
}

/* ------------------------------------------------------- one grid, one band */

template <int LIM, int FIRST_ORDER>
__global__ void __launch_bounds__(kStagedThreads, MH2D_RECON_CTAS)
staged_recon_kernel(const Mh2dArgs<double> a, const Mh2dBand b)
{
    pdl_wait();
    long long n;
    double dt;
    HydroStepControl *ctrl = a.ctrl;
    const double dtA[2] = { ctrl->step_dtA[0], ctrl->step_dtA[1] };
    if (!staged_step(ctrl, n, dt)) {
        if (blockIdx.x == 0 && threadIdx.x == 0) record_zero_dt(ctrl);
        return;
    }
    const unsigned k = blockIdx.x * kStagedThreads + threadIdx.x;
    if (k >= staged_recon_items(a.nx, b.r1 - b.r0)) return;
    staged_recon<LIM, FIRST_ORDER>(a, b, k, (int) (n & 1), n == 0, dtA);
}

template <bool TAPE>
__global__ void __launch_bounds__(kStagedThreads, MH2D_FLUX_CTAS)
staged_flux_kernel(const Mh2dArgs<double> a, const Mh2dBand b)
{
    __shared__ FluxShared sm;
    pdl_wait();
    long long n;
    double dt;
    if (!staged_step(a.ctrl, n, dt)) return;
    staged_flux<TAPE, false>(a, b, sm, blockIdx.x * kStagedThreads + threadIdx.x, staged_face_items(a.nx, b.r1 - b.r0), dt);
}

template <bool GRAV>
__global__ void __launch_bounds__(kStagedThreads, MH2D_UPDATE_CTAS)
staged_update_kernel(const Mh2dArgs<double> a, const Mh2dBand b)
{
    __shared__ UpdateShared sm;
    pdl_wait();
    long long n;
    double dt;
    if (!staged_step(a.ctrl, n, dt)) return;
    const Fm f = make_fm();
    double mx_x = -CUDART_INF, mx_y = -CUDART_INF;
    const unsigned cells = (unsigned) (b.r1 - b.r0) * a.nx;
    for (unsigned k = blockIdx.x * kStagedThreads + threadIdx.x; k < cells; k += gridDim.x * kStagedThreads)
        staged_update<GRAV>(f, a, b, k, (int) (n & 1), dt, mx_x, mx_y);
    staged_finish(a, sm, b.update_blocks, n, dt, mx_x, mx_y);
}

/* ------------------------------------------------------------- many grids */

/*
 * The stages of a batch: one launch per stage over the blocks of all
 * instances (bands) of a group.  A block finds its band in a map, copies the
 * instance's arguments to shared memory and runs the single grid's code, so
 * each instance has the single grid's bits.  Instances keep their own clock;
 * one that has stopped leaves at once.
 */
struct BatchBlock {
    Mh2dArgs<double> a;
    StagedBatchBand b;
    long long n;
    double dt, dtA[2];
    int go;
};

__device__ __forceinline__ bool batch_block(const StagedBatchArgs &g, const int *map, BatchBlock &sm)
{
    pdl_wait();
    const StagedBatchBand *band = g.bands + map[blockIdx.x];
    const Mh2dArgs<double> *inst = g.inst + band->inst;
    const int tid = threadIdx.x;
    static_assert(sizeof(Mh2dArgs<double>) % 8 == 0 && sizeof(StagedBatchBand) % 8 == 0, "copied as 8-byte words");
    for (int k = tid; k < (int) (sizeof(Mh2dArgs<double>) / 8); k += kStagedThreads)
        ((unsigned long long *) &sm.a)[k] = ((const unsigned long long *) inst)[k];
    for (int k = tid; k < (int) (sizeof(StagedBatchBand) / 8); k += kStagedThreads)
        ((unsigned long long *) &sm.b)[k] = ((const unsigned long long *) band)[k];
    if (tid == 0) {
        HydroStepControl *ctrl = inst->ctrl;
        sm.go = staged_step(ctrl, sm.n, sm.dt);
        sm.dtA[0] = ctrl->step_dtA[0];
        sm.dtA[1] = ctrl->step_dtA[1];
    }
    __syncthreads();
    return sm.go != 0;
}

template <int LIM, int FIRST_ORDER>
__global__ void __launch_bounds__(kStagedThreads, MH2D_RECON_CTAS)
staged_batch_recon_kernel(const StagedBatchArgs g, const int *map)
{
    __shared__ BatchBlock sm;
    if (!batch_block(g, map, sm)) {
        if (threadIdx.x == 0 && blockIdx.x == sm.b.first[0] && sm.b.band.r0 == sm.a.g) record_zero_dt(sm.a.ctrl);
        return;
    }
    const unsigned k = (blockIdx.x - sm.b.first[0]) * kStagedThreads + threadIdx.x;
    if (k >= staged_recon_items(sm.a.nx, sm.b.band.r1 - sm.b.band.r0)) return;
    staged_recon<LIM, FIRST_ORDER>(sm.a, sm.b.band, k, (int) (sm.n & 1), sm.n == 0, sm.dtA);
}

static __global__ void __launch_bounds__(kStagedThreads, MH2D_FLUX_CTAS)
staged_batch_flux_kernel(const StagedBatchArgs g, const int *map)
{
    __shared__ BatchBlock sm;
    __shared__ FluxShared fs;
    if (!batch_block(g, map, sm)) return;
    staged_flux<false, false>(sm.a, sm.b.band, fs, (blockIdx.x - sm.b.first[1]) * kStagedThreads + threadIdx.x,
                       staged_face_items(sm.a.nx, sm.b.band.r1 - sm.b.band.r0), sm.dt);
}

static __global__ void __launch_bounds__(kStagedThreads, MH2D_UPDATE_CTAS)
staged_batch_update_kernel(const StagedBatchArgs g, const int *map)
{
    __shared__ BatchBlock sm;
    __shared__ UpdateShared us;
    if (!batch_block(g, map, sm)) return;
    const Fm f = make_fm();
    double mx_x = -CUDART_INF, mx_y = -CUDART_INF;
    const unsigned cells = (unsigned) (sm.b.band.r1 - sm.b.band.r0) * sm.a.nx;
    for (unsigned k = (blockIdx.x - sm.b.first[2]) * kStagedThreads + threadIdx.x; k < cells;
         k += sm.b.update_grid * kStagedThreads)
        staged_update<false>(f, sm.a, sm.b.band, k, (int) (sm.n & 1), sm.dt, mx_x, mx_y);
    staged_finish(sm.a, us, sm.b.band.update_blocks, sm.n, sm.dt, mx_x, mx_y);
}

/* ------------------------------------------------ small grids: many steps */

/*
 * The same three stages, many steps in one cooperative launch, for grids
 * whose step is a few microseconds of work: grid barriers between the stages
 * instead of kernel boundaries.  A step has two or three barriers (about 1.5
 * us each); the three launches it replaces cost about 4 us each in gaps, ramps
 * and control-block reads, and 11 us of host time where no graph is
 * recorded.  Every block forms the next dt itself after the last barrier.
 *
 * The order of the phases and barriers is step_loop's (step_loop.cuh).  All
 * blocks are resident (cooperative launch), so every wait ends; a limit on the
 * polls guards against an error in that, after which the block records
 * DEV_ERR_SPIN_LIMIT, marks the run as stopped (launches behind this one leave
 * at once) and leaves, and so do the others.
 */
constexpr int kBarrierPolls = 1 << 22;

struct BarrierCount {
    unsigned *word;
    __device__ __forceinline__ unsigned arrive() { return atomicAdd(word, 1u); }
    __device__ __forceinline__ unsigned count() { return *(volatile unsigned *) word; }
};

__device__ __forceinline__ bool grid_barrier(HydroStepControl *ctrl, unsigned &target, int *ok)
{
    target += gridDim.x;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        BarrierCount c{ &ctrl->barrier_count };
        const bool in = arrive_and_wait(c, target, kBarrierPolls);
        __threadfence();
        if (!in) {
            record_error(ctrl, DEV_ERR_SPIN_LIMIT, -1);
            ctrl->active = 0;
        }
        *ok = in;
    }
    __syncthreads();
    return *ok != 0;
}

template <int LIM, int FIRST_ORDER, bool GRAV, bool FUSED>
__global__ void __launch_bounds__(kStagedThreads, MH2D_LOOP_CTAS)
staged_loop_kernel(const Mh2dArgs<double> a, const Mh2dBand b, int most)
{
    constexpr int NT = kStagedThreads;
    __shared__ FluxShared sm;
    __shared__ unsigned long long red[2][NT / 32];
    __shared__ double s_dt, s_dtA[2];
    __shared__ int ok, failed;
    __shared__ double v[1][NT / 2];
    HydroStepControl *ctrl = a.ctrl;
    volatile HydroStepControl *vc = ctrl;
    const int tid = threadIdx.x;
    const bool leader = blockIdx.x == 0 && tid == 0;
    if (!vc->active) return;
    long long n = vc->num_steps;
    double t = vc->t, dt = vc->step_dt, dtA[2] = { vc->step_dtA[0], vc->step_dtA[1] };
    const double tf = vc->tf;
    const long long last = vc->max_steps;
    const int stored = vc->store_count;
    const int rows = b.r1 - b.r0;
    const unsigned recon = staged_recon_items(a.nx, rows), faces = staged_face_items(a.nx, rows);
    const unsigned cells = (unsigned) rows * a.nx;
    const Fm f = make_fm();
    /* where the counter stood when the launch began: the leader moves the
     * base on its way out, past the launch's last barrier */
    unsigned target = vc->barrier_base;

    step_loop(
        most,
        [&]() {   /* a step without a dt */
            if (dt != 0.0) return true;
            if (leader) {
                ctrl->dt = dt;
                record_error(ctrl, DEV_ERR_DT_ZERO, -1);
                ctrl->active = 0;
            }
            return false;
        },
        [&]() {
            const int buf = (int) (n & 1);
            if constexpr (FUSED) {
                for (unsigned k = blockIdx.x * (NT / 2); k < faces; k += gridDim.x * (NT / 2))
                    staged_recon_flux<LIM, FIRST_ORDER>(a, b, sm, v, k, faces, dt, buf, n == 0, dtA);
            } else {
                for (unsigned k = blockIdx.x * NT + tid; k < recon; k += gridDim.x * NT)
                    staged_recon<LIM, FIRST_ORDER>(a, b, k, buf, n == 0, dtA);
                if (!grid_barrier(ctrl, target, &ok)) return false;
                for (unsigned k = blockIdx.x * NT; k < faces; k += gridDim.x * NT)
                    staged_flux<false, true>(a, b, sm, k + tid, faces, dt);
            }
            return true;
        },
        [&]() { return grid_barrier(ctrl, target, &ok); },
        [&]() { if (tid == 0) failed = vc->error_code != 0; },
        [&]() {
            const int buf = (int) (n & 1);
            double mx_x = -CUDART_INF, mx_y = -CUDART_INF;
            for (unsigned k = blockIdx.x * NT + tid; k < cells; k += gridDim.x * NT)
                staged_update<GRAV>(f, a, b, k, buf, dt, mx_x, mx_y);
            block_maxima<NT>(ctrl, red, n, mx_x, mx_y);
        },
        [&]() {
            if (!failed) return false;
            if (leader) {
                ctrl->barrier_base = target;
                ctrl->dt = dt;
                ctrl->active = 0;
            }
            return true;
        },
        [&]() {   /* every block: the next dt; block 0 publishes the clock */
            if (tid < 32) {
                const double tn = t + dt;
                double next, w;
                next_dt(a, ctrl, n + 1, tn, tf, next, w);
                if (tid == 0) s_dt = next;
                if (tid < 2) s_dtA[tid] = w;
            }
            __syncthreads();
            n += 1;
            t = t + dt;
            bool act = (t < tf) && (last < 0 || n < last), due = false;
            if (a.sp.is_storing && t >= a.sp.storing_interval * (double) (stored - a.sp.store_initial_offset + 1)) {
                due = true;
                act = false;
            }
            if (leader) {
                if (a.dt_log) a.dt_log[n - 1] = dt;
                ctrl->dt = dt;
                ctrl->t = t;
                ctrl->num_steps = n;
                ctrl->step_dt = s_dt;
                ctrl->step_dtA[0] = s_dtA[0];
                ctrl->step_dtA[1] = s_dtA[1];
                ctrl->barrier_base = target;
                ctrl->smax[(n + 1) % 3][0] = ordered_bits(-CUDART_INF);
                ctrl->smax[(n + 1) % 3][1] = ordered_bits(-CUDART_INF);
                if (due) ctrl->snapshot_due = 1;
                if (!act) ctrl->active = 0;
            }
            if (!act) return false;
            dt = s_dt;
            dtA[0] = s_dtA[0];
            dtA[1] = s_dtA[1];
            return true;
        });
}

}  // namespace hydro

#endif
