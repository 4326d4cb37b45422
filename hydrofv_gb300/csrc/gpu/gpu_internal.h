/*
 * gpu_internal.h -- declarations shared by the CUDA translation units.
 */
#ifndef HYDRO_GPU_INTERNAL_H
#define HYDRO_GPU_INTERNAL_H

#include <cuda_runtime.h>

#include <algorithm>
#include <functional>
#include <map>
#include <mutex>
#include <tuple>
#include <vector>

#include "mh2d_kernel.cuh"


namespace hydro {

/*
 * Rows per work item of the FP32 step when the caller sets none.  The step's
 * CTAs are persistent (one per resident slot) and take (strip, row chunk)
 * items from a queue.  An item of c rows also reconstructs the rows below it
 * (0.95 of a row's work: 2048^2 takes 317 / 244 / 179 us a step with 1 / 2 /
 * 12 rows), and the last items run while other slots are already idle.  In
 * units of a row's work with all slots busy (5.0 us) a step is modelled as
 *     items (c + 0.95) / slots + 1.2 + 0.24 c,
 * and as no less than an item alone, 2.1 + 0.48 c.  `items` gives the number
 * of items for a height.
 * Measured on 1064 slots, this choice / the best of 1 .. 64 rows / 32 rows, us
 * a step: 64^2 11.0 (1 row) / 11.0 / 86, 301 x 200 13.2 (1) / 13.2 / 94, 512^2
 * 23.8 (3) / 23.7 / 94, 700 x 900 42.9 (4) / 37.8 / 102, 1024^2 61.7 (6) / 61.7
 * / 103, 2048^2 179 (12) / 179 / 216, 4096^2 601 (24) / 600 / 600; 28 grids of
 * side 128 to 640 256 (12) / 256 / 300, 60 of side 500 to 900 1251 (24) / 1251
 * / 1253 (with the power in two instructions; a call of __powf makes 2048^2 183
 * and 4096^2 612).
 */
template <class Items>
int mh2d_fp32_chunk(int slots, Items items)
{
    static const int cand[] = { 1, 2, 3, 4, 6, 8, 12, 16, 20, 24, 32, 40, 48, 64 };
    if (slots <= 0) return 32;
    int best = 32;
    double best_t = 1e300;
    for (int c : cand) {
        const double full = (double) items(c) * (c + 0.95) / slots + 1.2 + 0.24 * c, one = 2.1 + 0.48 * c;
        const double t = full > one ? full : one;
        if (t < best_t) {
            best_t = t;
            best = c;
        }
    }
    return best;
}

/* Launch with programmatic stream serialization: the launch is processed
 * while the kernel before it in the stream runs; the step kernels wait for that
 * kernel's completion before they read or write (pdl_wait). */
template <class... P, class... A>
cudaError_t launch_after(void (*kernel)(P...), unsigned grid, unsigned threads, cudaStream_t s, const A &...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(threads);
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

/* Work items of c rows of an nx x ny grid. */
inline long long mh2d_item_count(int nx, int ny, int strip_w, int c)
{
    return (long long) ((nx + strip_w - 1) / strip_w) * ((ny + c - 1) / c);
}

/*
 * The single height that the guided plan below starts from: the same model
 * with the fused FP64 kernel's prologue (0.4 of a row).
 */
inline int mh2d_default_chunk(int nx, int ny, int strip_w, int slots)
{
    static const int cand[] = { 8, 12, 16, 20, 24, 32, 40, 48, 64 };
    if (slots <= 0 || strip_w <= 0) return 32;
    int best = 32;
    double best_eff = -1.0;
    for (int c : cand) {
        const long long items = mh2d_item_count(nx, ny, strip_w, c);
        const long long rounds = (items + slots - 1) / slots;
        const double eff = (double) items / (double) (rounds * slots) * (1.0 - 0.4 / c);
        if (eff > best_eff + 1e-9) {
            best_eff = eff;
            best = c;
        }
    }
    return best;
}

/*
 * Guided row chunks: tall items first, short items last.  The step's work
 * items go to the persistent CTAs in queue order, each CTA taking the next
 * item when it is done.  Tall items pay their per-item prologue (about half
 * a row: the rows below the chunk and its first y faces) less often; short
 * items at the end of the queue keep the last round full.  This models the
 * queue as greedy list scheduling of items costing (rows + 0.5) x (strip
 * width + 2 halo columns) on `slots` equal workers, and picks the heights
 * and the split with the smallest makespan (ties: fewer items).  tail_rows
 * = 0 is one of the candidates: a single height.
 */
inline double mh2d_queue_makespan(int nx, int ny, int strip_w, int slots, int h1, int h2, int tail)
{
    std::vector<double> free_at((size_t) slots, 0.0);
    std::make_heap(free_at.begin(), free_at.end(), std::greater<double>());
    const int strips = (nx + strip_w - 1) / strip_w;
    double makespan = 0.0;
    auto chunk = [&](int rows) {
        for (int s = 0; s < strips; s++) {
            const int sw = (s + 1) * strip_w <= nx ? strip_w : nx - s * strip_w;
            std::pop_heap(free_at.begin(), free_at.end(), std::greater<double>());
            double &t = free_at.back();
            t += (rows + 0.5) * (sw + 2) / (double) (strip_w + 2);
            if (t > makespan) makespan = t;
            std::push_heap(free_at.begin(), free_at.end(), std::greater<double>());
        }
    };
    const int big = ny - tail;
    for (int r = 0; r < big; r += h1) chunk(big - r < h1 ? big - r : h1);
    for (int r = big; r < ny; r += h2) chunk(ny - r < h2 ? ny - r : h2);
    return makespan;
}

inline void mh2d_guided_chunks(int nx, int ny, int strip_w, int slots, int &h1, int &h2, int &tail)
{
    /* 40 candidate queues besides the single height; one search per shape
     * (about 4 ms at 2048^2 on one host core), then cached */
    static const int tall[] = { 16, 24, 32, 48, 64 };
    static const int short_h[] = { 4, 8 };
    static const double waves[] = { 0.5, 1.0, 1.5, 2.0 };
    static std::mutex cache_mutex;
    static std::map<std::tuple<int, int, int, int>, std::tuple<int, int, int>> cache;
    const auto key = std::make_tuple(nx, ny, strip_w, slots);
    {
        std::lock_guard<std::mutex> lock(cache_mutex);
        const auto it = cache.find(key);
        if (it != cache.end()) {
            std::tie(h1, h2, tail) = it->second;
            return;
        }
    }
    h1 = mh2d_default_chunk(nx, ny, strip_w, slots);
    h2 = h1;
    tail = 0;
    if (slots <= 0 || strip_w <= 0 || nx <= 0 || ny <= 0) return;
    const int strips = (nx + strip_w - 1) / strip_w;
    double best = mh2d_queue_makespan(nx, ny, strip_w, slots, h1, h1, 0);
    for (int a : tall) {
        for (int b : short_h) {
            if (b >= a) continue;
            for (double w : waves) {
                /* enough short items for about w rounds of the persistent CTAs */
                int t = (int) (w * slots / strips) * b;
                t = ny - ((ny - t) / a) * a;                      /* tall part: whole chunks */
                if (t <= 0 || t >= ny) continue;
                const double m = mh2d_queue_makespan(nx, ny, strip_w, slots, a, b, t);
                if (m < best * (1.0 - 1e-9)) {
                    best = m;
                    h1 = a;
                    h2 = b;
                    tail = t;
                }
            }
        }
    }
    std::lock_guard<std::mutex> lock(cache_mutex);
    cache[key] = std::make_tuple(h1, h2, tail);
}

/* The rows of a step are processed in one band as long as its workspace stays
 * below a fixed size (kStagedWorkspaceBytes, 1 GiB).  Bands small enough for the L2
 * cache lost: 2048^2 3.07 ms with one band, 3.16 / 3.22 / 3.35 / 3.70 ms with
 * 160 / 96 / 48 / 24 MB (the launches' tails cost more than the traffic).
 *
 * Rows [r0, r1) (padded indices) of one grid and the workspace they use: a
 * plane holds rows r0 - 1 .. r1 with the grid's pitch. */
struct Mh2dBand {
    int r0, r1;
    unsigned update_blocks;   /* update blocks of the whole step of this grid (all bands) */
    long long plane;          /* doubles per workspace field */
    double *ws;
};

/* Most bytes of the staged FP64 step's workspace (16 fields of a band's rows). */
#ifndef MH2D_WORKSPACE_MB
#define MH2D_WORKSPACE_MB 1024
#endif
constexpr size_t kStagedWorkspaceBytes = (size_t) MH2D_WORKSPACE_MB << 20;

/* The staged FP64 step (mh2d_staged.cuh).  staged_plan splits the grid's rows
 * into bands whose workspace takes at most `budget` bytes (one row at least;
 * `bytes` receives what it takes); the caller points every band's `ws` at
 * that workspace. */
void staged_plan(const Mh2dArgs<double> &a, size_t budget, std::vector<Mh2dBand> &bands, size_t &bytes);
/* The same with the workspace: `alloc(&p, bytes)` is asked for
 * kStagedWorkspaceBytes at most, and for less where the device has no room
 * (more and shorter bands, down to single rows). */
template <class Alloc>
cudaError_t staged_alloc(const Mh2dArgs<double> &a, std::vector<Mh2dBand> &bands, Alloc alloc)
{
    size_t budget = kStagedWorkspaceBytes;
    for (;;) {
        size_t bytes = 0;
        void *p = nullptr;
        staged_plan(a, budget, bands, bytes);
        const cudaError_t e = alloc(&p, bytes);
        if (e == cudaSuccess) {
            for (auto &b : bands) b.ws = static_cast<double *>(p);
            return e;
        }
        if (e != cudaErrorMemoryAllocation || bands[0].r1 - bands[0].r0 == 1) return e;
        cudaGetLastError();
        budget = bytes / 2;
    }
}

/*
 * Memory that a session takes after the workspace (a solver's initial state, the
 * adjoint's tape): where the device has no room for it, the workspace gives
 * way.  `release()` gives it back, `alloc(p, bytes)` is asked again, and
 * `workspace(&p, bytes)` for a workspace in what is left, in more and shorter
 * bands.  A failure leaves no bands when not even single rows fit.
 */
template <class Alloc, class Release, class Workspace>
cudaError_t alloc_beside_workspace(const Mh2dArgs<double> &a, std::vector<Mh2dBand> &bands, void **p, size_t bytes, Alloc alloc,
                                   Release release, Workspace workspace)
{
    cudaError_t e = alloc(p, bytes);
    if (e != cudaErrorMemoryAllocation || bands.empty()) return e;
    cudaGetLastError();
    release();
    e = alloc(p, bytes);
    if (e != cudaSuccess) cudaGetLastError();
    const cudaError_t w = staged_alloc(a, bands, workspace);
    if (w != cudaSuccess) bands.clear();
    return e != cudaSuccess ? e : w;
}

cudaError_t staged_launch_step(const Mh2dArgs<double> &a, int limiter, const std::vector<Mh2dBand> &bands, cudaStream_t s);
/* Batches: band `band` of instance `inst`; its blocks of the recon, flux and
 * update launches start at first[0], first[1], first[2] of the group's. */
struct StagedBatchBand {
    Mh2dBand band;
    int inst;
    unsigned first[3], update_grid;
};

/* Bands that share the workspace: one launch per stage.  map[s][k] is the
 * band (index into `bands`) of block k of stage s (device memory). */
struct StagedBatchGroup {
    const int *map[3];
    unsigned blocks[3];
};

struct StagedBatchArgs {
    const Mh2dArgs<double> *inst;     /* device memory, one per instance */
    const StagedBatchBand *bands;     /* device memory */
};

/* Blocks of a band's stages. */
void staged_band_blocks(const Mh2dArgs<double> &a, const Mh2dBand &b, unsigned blocks[3]);
cudaError_t staged_launch_batch(const StagedBatchArgs &b, const std::vector<StagedBatchGroup> &groups, int limiter,
                                int first_order, cudaStream_t s);

/* Small grids: blocks of the many-step kernel (0: the grid steps with three
 * launches), and up to `steps` steps in one launch of it. */
unsigned staged_loop_grid(const Mh2dArgs<double> &a, int limiter, const std::vector<Mh2dBand> &bands, int device);
cudaError_t staged_launch_steps(const Mh2dArgs<double> &a, int limiter, const Mh2dBand &band, unsigned grid, int steps,
                                cudaStream_t s);

/*
 * Of `k` steps as many as the many-step kernel takes, in launches of at most
 * `most` steps by `loop(steps)`.  A launch that the driver refuses because the
 * process may use fewer of the SMs than the device has (its blocks would not be
 * resident together), or because it grants no cooperative launches, has done
 * nothing: `grid` comes back 0 and the steps left in `k` go in three launches
 * each, as on larger grids.
 */
template <class Loop>
cudaError_t staged_loop_steps(unsigned &grid, long long &k, int most, Loop loop)
{
    while (grid && k > 0) {
        const int steps = (int) (k < most ? k : most);
        const cudaError_t e = loop(steps);
        if (e == cudaErrorCooperativeLaunchTooLarge || e == cudaErrorNotSupported || e == cudaErrorNotPermitted) {
            cudaGetLastError();
            grid = 0;
        } else if (e != cudaSuccess) {
            return e;
        } else {
            k -= steps;
        }
    }
    return cudaSuccess;
}

template <class R>
cudaError_t mh2d_launch_step(const Mh2dArgs<R> &a, int limiter, cudaStream_t s);
template <class R>
int mh2d_resident_ctas(int limiter, int first_order, int device);
template <class R>
cudaError_t mh2d_launch_batch_step(const Mh2dBatchArgs<R> &b, int limiter, int first_order, int grid,
                                   cudaStream_t s);
template <class R>
cudaError_t mh2d_launch_prepare(const Mh2dArgs<R> &a, cudaStream_t s);
/* The first dt after the maxima of the state are known (prepare), and again
 * when the stopping time moves: one grid, and n instances in device memory. */
template <class R>
cudaError_t mh2d_launch_arm(const Mh2dArgs<R> &a, cudaStream_t s);
template <class R>
cudaError_t mh2d_launch_batch_arm(const Mh2dArgs<R> *inst, int n, cudaStream_t s);
template <class R>
cudaError_t mh2d_launch_materialize(const Mh2dArgs<R> &a, int buf, R *const out[4], cudaStream_t s);
template <class R>
cudaError_t mh2d_launch_totals(const Mh2dArgs<R> &a, int buf, double *out4, cudaStream_t s);
template <class R>
cudaError_t mh2d_launch_convert_all(const Mh2dArgs<R> &a, int buf, R *const out[4], cudaStream_t s);
template <class R>
cudaError_t mh2d_launch_ghost_sound_speed(const Mh2dArgs<R> &a, int buf, int mask, cudaStream_t s);
cudaError_t convert_f64_to_f32(const double *src, float *dst, long long n, cudaStream_t s);
cudaError_t convert_f32_to_f64(const float *src, double *dst, long long n, cudaStream_t s);

}  // namespace hydro

#endif
