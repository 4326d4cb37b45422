/*
 * mh2d.cu -- FP64 instantiations of the 2D step and its helper kernels.
 *
 * Compiled with --fmad=false: the FP64 path must issue the same IEEE
 * operations as the reference CPU code, which never contracts a*b+c.
 */
#include "mh2d_launch.cuh"
#include "mh2d_staged_launch.cuh"

namespace hydro {

template cudaError_t mh2d_launch_step<double>(const Mh2dArgs<double> &, int, cudaStream_t);
template cudaError_t mh2d_launch_prepare<double>(const Mh2dArgs<double> &, cudaStream_t);
template cudaError_t mh2d_launch_arm<double>(const Mh2dArgs<double> &, cudaStream_t);
template cudaError_t mh2d_launch_batch_arm<double>(const Mh2dArgs<double> *, int, cudaStream_t);
template cudaError_t mh2d_launch_materialize<double>(const Mh2dArgs<double> &, int,
                                                     double *const[4], cudaStream_t);
template cudaError_t mh2d_launch_totals<double>(const Mh2dArgs<double> &, int, double *, cudaStream_t);
template cudaError_t mh2d_launch_convert_all<double>(const Mh2dArgs<double> &, int, double *const[4], cudaStream_t);
template cudaError_t mh2d_launch_ghost_sound_speed<double>(const Mh2dArgs<double> &, int, int, cudaStream_t);

/* ------------------------------------------------------ the staged step */

#define HYDRO_STAGED_EXTERN(LIM, FO)                                                                                      \
    extern template cudaError_t staged_launch_recon<LIM, FO>(const Mh2dArgs<double> &, const Mh2dBand &, cudaStream_t); \
    extern template cudaError_t staged_launch_batch_recon<LIM, FO>(const StagedBatchArgs &, const StagedBatchGroup &, cudaStream_t); \
    extern template unsigned staged_loop_blocks<LIM, FO>(const Mh2dArgs<double> &, const Mh2dBand &, int);              \
    extern template cudaError_t staged_launch_loop<LIM, FO>(const Mh2dArgs<double> &, const Mh2dBand &, unsigned, int, cudaStream_t);
HYDRO_STAGED_EXTERN(LIM_MINMOD, 0)
HYDRO_STAGED_EXTERN(LIM_MINMOD, 1)
HYDRO_STAGED_EXTERN(LIM_VAN_LEER, 0)
HYDRO_STAGED_EXTERN(LIM_MC, 0)

/* f<LIM, FIRST_ORDER>(...) for `limiter` and `first_order`. */
#define STAGED_DISPATCH(f, ...)                                          \
    (first_order               ? f<LIM_MINMOD, 1>(__VA_ARGS__)           \
     : limiter == LIM_MINMOD   ? f<LIM_MINMOD, 0>(__VA_ARGS__)           \
     : limiter == LIM_VAN_LEER ? f<LIM_VAN_LEER, 0>(__VA_ARGS__)         \
                               : f<LIM_MC, 0>(__VA_ARGS__))

static unsigned update_grid(const Mh2dArgs<double> &a, const Mh2dBand &b)
{
    const unsigned n = staged_blocks((unsigned) (b.r1 - b.r0) * a.nx);
    return n < kStagedUpdateGrid ? n : kStagedUpdateGrid;
}

void staged_plan(const Mh2dArgs<double> &a, size_t budget, std::vector<Mh2dBand> &bands, size_t &bytes)
{
    const size_t row = (size_t) WS_FIELDS * a.pitch * sizeof(double);
    long long rows = (long long) (budget / row) - 2;
    /* item counts stay below 2^31 */
    const long long most = (1ll << 30) / (a.nx + 2) - 2;
    rows = rows < most ? rows : most;
    rows = rows < 1 ? 1 : (rows > a.ny ? a.ny : rows);
    const int n = (int) ((a.ny + rows - 1) / rows);
    const int h = (a.ny + n - 1) / n;             /* equal bands */
    bands.clear();
    for (int lo = 0; lo < a.ny; lo += h) {
        Mh2dBand b{};
        b.r0 = a.g + lo;
        b.r1 = a.g + (lo + h < a.ny ? lo + h : a.ny);
        b.plane = (long long) (h + 2) * a.pitch;
        bands.push_back(b);
    }
    unsigned blocks = 0;
    for (const auto &b : bands) blocks += update_grid(a, b);
    for (auto &b : bands) b.update_blocks = blocks;
    bytes = (size_t) (h + 2) * row;
}

cudaError_t staged_launch_step(const Mh2dArgs<double> &a, int limiter, const std::vector<Mh2dBand> &bands, cudaStream_t s)
{
    const int first_order = a.first_order;
    if (bands.empty()) return cudaErrorMemoryAllocation;
    for (const Mh2dBand &b : bands) {
        cudaError_t e = STAGED_DISPATCH(staged_launch_recon, a, b, s);
        if (e != cudaSuccess) return e;
        const unsigned faces = staged_blocks(staged_face_items(a.nx, b.r1 - b.r0));
        e = a.tape ? launch_pdl(staged_flux_kernel<true>, faces, s, a, b) : launch_pdl(staged_flux_kernel<false>, faces, s, a, b);
        if (e != cudaSuccess) return e;
        e = a.gravity != 0.0 ? launch_pdl(staged_update_kernel<true>, update_grid(a, b), s, a, b)
                             : launch_pdl(staged_update_kernel<false>, update_grid(a, b), s, a, b);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

void staged_band_blocks(const Mh2dArgs<double> &a, const Mh2dBand &b, unsigned blocks[3])
{
    blocks[0] = staged_blocks(staged_recon_items(a.nx, b.r1 - b.r0));
    blocks[1] = staged_blocks(staged_face_items(a.nx, b.r1 - b.r0));
    blocks[2] = update_grid(a, b);
}

cudaError_t staged_launch_batch(const StagedBatchArgs &b, const std::vector<StagedBatchGroup> &groups, int limiter,
                                int first_order, cudaStream_t s)
{
    for (const StagedBatchGroup &g : groups) {
        cudaError_t e = STAGED_DISPATCH(staged_launch_batch_recon, b, g, s);
        if (e != cudaSuccess) return e;
        e = launch_pdl(staged_batch_flux_kernel, g.blocks[1], s, b, g.map[1]);
        if (e != cudaSuccess) return e;
        e = launch_pdl(staged_batch_update_kernel, g.blocks[2], s, b, g.map[2]);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

unsigned staged_loop_grid(const Mh2dArgs<double> &a, int limiter, const std::vector<Mh2dBand> &bands, int device)
{
    const int first_order = a.first_order;
    if (bands.size() != 1) return 0;
    if (staged_recon_items(a.nx, a.ny) > kStagedLoopItems) return 0;
    return STAGED_DISPATCH(staged_loop_blocks, a, bands[0], device);
}

cudaError_t staged_launch_steps(const Mh2dArgs<double> &a, int limiter, const Mh2dBand &band, unsigned grid, int steps,
                                cudaStream_t s)
{
    const int first_order = a.first_order;
    return STAGED_DISPATCH(staged_launch_loop, a, band, grid, steps, s);
}

}  // namespace hydro
