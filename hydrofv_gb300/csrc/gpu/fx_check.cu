/*
 * fx_check.cu -- evaluation entry points used by the tests:
 *  - the integer-pipe FP64 division, square root and power (fp64_int.cuh,
 *    pow_int.cuh) over arrays: the host build (checked on the CPU against
 *    the host's IEEE operations and libm) and the device build next to the
 *    hardware operations on the GPU;
 *  - the device build of the exported pointwise numerics (HLLC fluxes,
 *    guess_p, the exact solver) over arrays of states, so that the kernels'
 *    arithmetic is checked against the reference's known answers branch by
 *    branch (vacuum generation, TRRS, TSRS, rarefaction and shock sampling),
 *    including branches that whole simulations rarely reach.
 */
#include <cuda_runtime.h>

#include "fp64_int.cuh"
#include "pow_int.cuh"
#include "numerics.cuh"
#include "quad_exact.cuh"
#include "staged_math.cuh"
#include "step_control.h"
#include "step_loop.cuh"
#include "hydro_gpu.h"
#include <atomic>
#include <chrono>
#include <thread>
#include <vector>

using namespace hydro;

namespace {

/* op 0: a / b, op 1: sqrt(a), op 2: pow(a, b).  fast = the integer form where it applies
 * (else the hardware result), hw = the hardware operation, ok = 1 where the
 * integer form applied.  op 3, 4, 5: the minmod, van Leer and MC slope
 * limiters L(a, b) as the kernels evaluate them (fast = hw; ok = 1 where the
 * sign test was decided on the bits). */
__global__ void fx_eval_kernel(int op, long long n, const double *a, const double *b,
                               double *fast, double *hw, unsigned char *ok)
{
    const long long stride = (long long) gridDim.x * blockDim.x;
    for (long long i = (long long) blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
        bool k;
        double f;
        if (op == 0) {
            f = fx::div_fast(a[i], b[i], k);
            hw[i] = fx::div_hw(a[i], b[i]);
            fast[i] = k ? f : dv(a[i], b[i]);
        } else if (op == 1) {
            f = fx::sqrt_fast(a[i], k);
            hw[i] = fx::sqrt_hw(a[i]);
            fast[i] = k ? f : sq(a[i]);
        } else if (op == 2) {
            f = fx::pow_fast(a[i], b[i], k);
            hw[i] = fx::pow_hw(a[i], b[i]);
            fast[i] = k ? f : pw(a[i], b[i]);
        } else {
            k = fx::product_nonpositive(fx::bits(a[i]), fx::bits(b[i])) >= 0;
            f = (op == 3) ? limit_slope<LIM_MINMOD>(a[i], b[i])
              : (op == 4) ? limit_slope<LIM_VAN_LEER>(a[i], b[i]) : limit_slope<LIM_MC>(a[i], b[i]);
            fast[i] = f;
            hw[i] = f;
        }
        ok[i] = k ? 1 : 0;
    }
}

/* The exported pointwise numerics, device build (one state pair per thread;
 * the gas constants are formed per element because gamma varies). */
__global__ void pointwise_kernel(int op, long long n, const double *gamma, double tol,
                                 const double *L, const double *R, const double *aux, double *out,
                                 int *rc)
{
    const long long stride = (long long) gridDim.x * blockDim.x;
    for (long long k = (long long) blockIdx.x * blockDim.x + threadIdx.x; k < n; k += stride) {
        const GasConst<double> c = make_gas_const<double>(gamma[k], tol);
        const double *l = L + 4 * k, *r = R + 4 * k;
        int code = DEV_OK;
        if (op == 0) {
            double F[4];
            code = hllc_flux_2d(c, l[0], l[1], l[2], l[3], r[0], r[1], r[2], r[3], F);
            for (int q = 0; q < 4; q++) out[4 * k + q] = F[q];
        } else if (op == 1) {
            out[k] = guess_p(c, l[0], l[1], l[3], aux[2 * k], r[0], r[1], r[3], aux[2 * k + 1]);
        } else if (op == 2) {
            double F[3];
            code = exact_flux_1d(c, l[0], l[1], l[3], r[0], r[1], r[3], aux[k], F);
            for (int q = 0; q < 3; q++) out[3 * k + q] = F[q];
        } else if (op == 3) {
            double F[3];
            code = hllc_flux_1d(c, l[0], l[1], l[3], r[0], r[1], r[3], F);
            for (int q = 0; q < 3; q++) out[3 * k + q] = F[q];
        } else {
            double o[3];
            code = exact_solve_1d(c, l[0], l[1], l[3], r[0], r[1], r[3], aux[k], o);
            for (int q = 0; q < 3; q++) out[3 * k + q] = o[q];
        }
        rc[k] = code;
    }
}

/* The 1D kernel's four-lane exact solver: four consecutive threads per state
 * pair (op 5: the flux at x/t = aux[k], op 6: the sampled state). */
__global__ void pointwise_quad_kernel(int op, long long n, const double *gamma, double tol,
                                      const double *L, const double *R, const double *aux, double *out,
                                      int *rc)
{
    const Quad Q = make_quad();
    const long long quads = ((long long) gridDim.x * blockDim.x) >> 2;
    for (long long k = ((long long) blockIdx.x * blockDim.x + threadIdx.x) >> 2; k < n; k += quads) {
        const GasConst<double> c = make_gas_const<double>(gamma[k], tol);
        const double *l = L + 4 * k, *r = R + 4 * k;
        double o[3];
        int code;
        if (op == 5) {
            double s[3];
            code = quad_exact_solve(Q, c, l[0], l[1], l[3], r[0], r[1], r[3], aux[k], s);
            o[0] = s[0] * s[1];
            o[1] = s[0] * s[1] * s[1] + s[2];
            o[2] = (s[2] * c.g_gm1 + 0.5 * s[0] * s[1] * s[1]) * s[1];
        } else {
            code = quad_exact_solve(Q, c, l[0], l[1], l[3], r[0], r[1], r[3], aux[k], o);
        }
        if (Q.q == 0) {
            for (int q = 0; q < 3; q++) out[3 * k + q] = o[q];
            rc[k] = code;
        }
    }
}

}  // namespace

extern "C" {

void hydro_fx_eval_host(int op, long long n, const double *a, const double *b, double *out,
                        unsigned char *ok)
{
    for (long long i = 0; i < n; i++) {
        bool k = true;
        if (op <= 2) {
            out[i] = (op == 0) ? fx::div_fast(a[i], b[i], k)
                   : (op == 1) ? fx::sqrt_fast(a[i], k) : fx::pow_fast(a[i], b[i], k);
        } else if (op == 6) {
            /* the bit-level sign test itself: out = 1, 0 or -1 */
            out[i] = (double) fx::product_nonpositive(fx::bits(a[i]), fx::bits(b[i]));
        } else {
            /* host builds evaluate the limiters' FP64 expressions */
            out[i] = (op == 3) ? limit_slope<LIM_MINMOD>(a[i], b[i])
                   : (op == 4) ? limit_slope<LIM_VAN_LEER>(a[i], b[i]) : limit_slope<LIM_MC>(a[i], b[i]);
        }
        ok[i] = k ? 1 : 0;
    }
}

void hydro_fx_div_seeded_host(long long n, const double *a, const double *b, const float *seed_scale,
                              double *out, unsigned char *ok)
{
    for (long long i = 0; i < n; i++) {
        bool k;
        out[i] = fx::div_fast(a[i], b[i], k, seed_scale[i]);
        ok[i] = k ? 1 : 0;
    }
}

void hydro_fx_ratio_below_host(long long n, const double *x, const double *y, const double *tol,
                               unsigned char *out, unsigned char *decided)
{
    for (long long i = 0; i < n; i++) {
        bool d;
        out[i] = ratio_below_fast(x[i], y[i], tol[i], d) ? 1 : 0;
        decided[i] = d ? 1 : 0;
    }
}

void hydro_fx_quot_le_host(long long n, const double *x, const double *y, const double *z,
                           unsigned char *out, unsigned char *decided)
{
    for (long long i = 0; i < n; i++) {
        bool d;
        out[i] = quot_le_fast(x[i], y[i], z[i], d) ? 1 : 0;
        decided[i] = d ? 1 : 0;
    }
}

int hydro_gpu_fx_eval(int device, int op, long long n, const double *a, const double *b,
                      double *fast, double *hw, unsigned char *ok)
{
    if (n <= 0) return 0;
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return (int) e;
    const size_t nb = (size_t) n * sizeof(double);
    char *slab = nullptr;
    e = cudaMalloc(&slab, 4 * nb + (size_t) n);
    if (e != cudaSuccess) return (int) e;
    double *da = (double *) slab, *db = da + n, *df = db + n, *dh = df + n;
    unsigned char *dk = (unsigned char *) (dh + n);
    e = cudaMemcpy(da, a, nb, cudaMemcpyHostToDevice);
    if (op < 0 || op > 5) e = cudaErrorInvalidValue;
    if (e == cudaSuccess) e = cudaMemcpy(db, op == 1 ? a : b, nb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        fx_eval_kernel<<<4 * 152, 256>>>(op, n, da, db, df, dh, dk);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(fast, df, nb, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(hw, dh, nb, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(ok, dk, (size_t) n, cudaMemcpyDeviceToHost);
    cudaFree(slab);
    return (int) e;
}

int hydro_gpu_pointwise_eval(int device, int op, long long n, const double *gamma, double tol,
                             const double *L, const double *R, const double *aux, double *out,
                             int *rc)
{
    if (n <= 0) return 0;
    if (op < 0 || op > 6) return (int) cudaErrorInvalidValue;
    cudaError_t e = cudaSetDevice(device);
    if (e != cudaSuccess) return (int) e;
    const int width = (op == 0) ? 4 : (op == 1) ? 1 : 3;
    const int naux = (op == 1) ? 2 : (op == 2 || op >= 4) ? 1 : 0;
    const size_t nb = (size_t) n * sizeof(double);
    char *slab = nullptr;
    e = cudaMalloc(&slab, (9 + naux + width) * nb + (size_t) n * sizeof(int));
    if (e != cudaSuccess) return (int) e;
    double *dg = (double *) slab, *dl = dg + n, *dr = dl + 4 * n, *da = dr + 4 * n;
    double *dout = da + naux * n;
    int *drc = (int *) (dout + width * n);
    e = cudaMemcpy(dg, gamma, nb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dl, L, 4 * nb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(dr, R, 4 * nb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess && naux) e = cudaMemcpy(da, aux, naux * nb, cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        if (op >= 5) pointwise_quad_kernel<<<152, 128>>>(op, n, dg, tol, dl, dr, da, dout, drc);
        else pointwise_kernel<<<152, 128>>>(op, n, dg, tol, dl, dr, da, dout, drc);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(out, dout, width * nb, cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(rc, drc, (size_t) n * sizeof(int), cudaMemcpyDeviceToHost);
    cudaFree(slab);
    return (int) e;
}

}  // extern "C"

/* The staged step's face (staged_math.cuh) and the template of numerics.cuh
 * on the same state pairs: five values each, the flux and the guess regime. */
extern "C" void hydro_fx_staged_face_host(double gamma, double tol, long long n, const double *L, const double *R,
                                          double *out, int *rc, double *ref, int *rc_ref)
{
    const GasConst<double> c = make_gas_const<double>(gamma, tol);
    const Fm f = make_fm();
    for (long long k = 0; k < n; k++) {
        const double *l = L + 4 * k, *r = R + 4 * k;
        double a_L, a_R, pg, z0, z1, wave[3], *F = out + 5 * k;
        bool plain;
        const int reg = face_classify(f, c, l[0], l[1], l[3], r[0], r[1], r[3], a_L, a_R, pg, plain);
        rc[k] = DEV_OK;
        for (int q = 0; q < 4; q++) F[q] = ref[5 * k + q] = 0.0;
        F[4] = reg;
        if (reg == PREG_VACUUM) {
            hllc_vacuum_flux(c, l[0], l[1], l[2], l[3], a_L, r[0], r[1], r[2], r[3], a_R, F);
        } else {
            double p_min;
            if (reg == PREG_TRRS && plain && both_rarefactions(f, c, l[1], l[3], a_L, r[1], r[3], a_R, p_min)) pg = p_min;
            else if (reg == PREG_TRRS) pg = face_trrs(f, c, l[1], l[3], a_L, r[1], r[3], a_R, z0, z1);
            else if (reg == PREG_TSRS) pg = face_tsrs(f, c, l[0], l[1], l[3], r[0], r[1], r[3], pg, z0, z1);
            rc[k] = face_finish(f, c, plain, l[0], l[1], l[2], l[3], a_L, r[0], r[1], r[2], r[3], a_R, pg, F, wave);
        }
        ref[5 * k + 4] = hllc_classify(c, l[0], l[1], l[3], r[0], r[1], r[3], a_L, a_R, pg);
        rc_ref[k] = hllc_flux_2d(c, l[0], l[1], l[2], l[3], r[0], r[1], r[2], r[3], ref + 5 * k);
    }
}

/* The staged step's slopes, predictor and conversion beside the templates:
 * per cell 12 values each: low and high face states, then U -> W of
 * (w0, with w0[0] as the mass and w0[3] as the energy). */
extern "C" void hydro_fx_staged_cell_host(int limiter, double gamma, double dtA, long long n, const double *wm,
                                          const double *w0, const double *wp, double *out, double *ref)
{
    const GasConst<double> c = make_gas_const<double>(gamma, 1e-6);
    const Fm f = make_fm();
    for (long long k = 0; k < n; k++) {
        const double *a = wm + 4 * k, *b = w0 + 4 * k, *e = wp + 4 * k;
        double d[4], g[4], *o = out + 12 * k, *r = ref + 12 * k;
        for (int q = 0; q < 4; q++) {
            d[q] = limiter == LIM_MINMOD ? slope_of<LIM_MINMOD>(f, a[q], b[q], e[q])
                 : limiter == LIM_VAN_LEER ? slope_of<LIM_VAN_LEER>(f, a[q], b[q], e[q])
                                           : slope_of<LIM_MC>(f, a[q], b[q], e[q]);
            g[q] = limit_slope_rt(limiter, b[q] - a[q], e[q] - b[q]);
        }
        const double s = sound_speed(c, b[0], b[3]);
        if (flat(d, b[0], b[1], b[2], b[3]) && fx::moderate(dtA)) {
            for (int q = 0; q < 4; q++) o[q] = o[4 + q] = b[q];
        } else {
            predict(f, dtA, dv(dtA, b[0]), b[0], b[1], b[2], b[3], s, d, d[1], o, o + 4);
        }
        hancock_2d(dtA, dv(dtA, b[0]), b[0], b[1], b[2], b[3], s, g, g[1], r, r + 4);
        to_primitive(f, c, 0.37, b[0], b[1], b[2], b[3], o + 8);
        cons_to_prim_2d(c, 0.37, b[0], b[1], b[2], b[3], r + 8);
    }
}

/* The many-step launch's order (step_loop) and its barrier with host threads
 * as blocks.  One block lags behind whenever it looks at the error word, one
 * records an error in the faces of a step, one never arrives. */
namespace {

struct HostGrid {
    std::atomic<unsigned> count{ 0 };
    std::atomic<int> error{ 0 }, active{ 1 };
    std::atomic<long long> steps{ 0 };
    int blocks, polls, slow, bad, bad_step;
};

struct HostCount {
    HostGrid &g;
    unsigned arrive() { return g.count.fetch_add(1); }
    unsigned count()
    {
        std::this_thread::sleep_for(std::chrono::microseconds(50));
        return g.count.load();
    }
};

void host_record(HostGrid &g, int code)
{
    int none = 0;
    g.error.compare_exchange_strong(none, code);
}

/* One block; `left`: 1 out of steps, 2 a failed step, 3 a wait gave up. */
void host_block(HostGrid &g, int id, int steps, int &left, long long &n)
{
    unsigned target = 0;
    int error = 0;
    left = 1;
    step_loop(
        steps, [] { return true; },
        [&] {
            if (id == g.bad && n == g.bad_step) host_record(g, DEV_ERR_HLLC_WAVE_SPEED);
            return true;
        },
        [&] {
            target += (unsigned) g.blocks;
            HostCount c{ g };
            if (arrive_and_wait(c, target, g.polls)) return true;
            host_record(g, DEV_ERR_SPIN_LIMIT);
            g.active = 0;
            left = 3;
            return false;
        },
        [&] {
            if (id == g.slow) std::this_thread::sleep_for(std::chrono::milliseconds(30));
            error = g.error.load();
        },
        [] {},
        [&] {
            if (error == 0) return false;
            left = 2;
            if (id == 0) g.active = 0;
            return true;
        },
        [&] {
            n++;
            if (id == 0) g.steps = n;
            return true;
        });
}

}  // namespace

extern "C" void hydro_fx_step_loop_host(int blocks, int steps, int slow, int bad, int bad_step, int absent, int polls,
                                        int *left, long long *done, long long out[3])
{
    HostGrid g;
    g.blocks = blocks;
    g.polls = polls;
    g.slow = slow;
    g.bad = bad;
    g.bad_step = bad_step;
    std::vector<std::thread> threads;
    for (int id = 0; id < blocks; id++) {
        left[id] = 0;
        done[id] = 0;
        if (id == absent) continue;
        threads.emplace_back([&g, id, steps, left, done] { host_block(g, id, steps, left[id], done[id]); });
    }
    for (auto &t : threads) t.join();
    out[0] = g.steps;
    out[1] = g.error;
    out[2] = g.active;
}
