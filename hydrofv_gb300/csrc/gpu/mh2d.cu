/*
 * mh2d.cu -- FP64 instantiations of the 2D step and its helper kernels.
 *
 * Compiled with --fmad=false: the FP64 path must issue the same IEEE
 * operations as the reference CPU code, which never contracts a*b+c.
 */
#include "mh2d_launch.cuh"
#include "mh2d_staged_launch.cuh"

namespace hydro {

template int mh2d_resident_ctas<double>(int, int, int);
template cudaError_t mh2d_launch_batch_step<double>(const Mh2dBatchArgs<double> &, int, int, int, cudaStream_t);
template cudaError_t mh2d_launch_step<double>(const Mh2dArgs<double> &, int, cudaStream_t);
template cudaError_t mh2d_launch_step_tape<double>(const Mh2dArgs<double> &, int, cudaStream_t);
template cudaError_t mh2d_launch_prepare<double>(const Mh2dArgs<double> &, cudaStream_t);
template cudaError_t mh2d_launch_materialize<double>(const Mh2dArgs<double> &, int,
                                                     double *const[4], cudaStream_t);
template cudaError_t mh2d_launch_totals<double>(const Mh2dArgs<double> &, int, double *, cudaStream_t);
template cudaError_t mh2d_launch_convert_all<double>(const Mh2dArgs<double> &, int, double *const[4], cudaStream_t);
template cudaError_t mh2d_launch_ghost_sound_speed<double>(const Mh2dArgs<double> &, int, int, cudaStream_t);

/* ------------------------------------------------------ the staged step */

extern template cudaError_t staged_launch_recon<LIM_MINMOD, 0>(const Mh2dArgs<double> &, const Mh2dBand &, bool, cudaStream_t);
extern template cudaError_t staged_launch_recon<LIM_MINMOD, 1>(const Mh2dArgs<double> &, const Mh2dBand &, bool, cudaStream_t);
extern template cudaError_t staged_launch_recon<LIM_VAN_LEER, 0>(const Mh2dArgs<double> &, const Mh2dBand &, bool, cudaStream_t);
extern template cudaError_t staged_launch_recon<LIM_MC, 0>(const Mh2dArgs<double> &, const Mh2dBand &, bool, cudaStream_t);

/* Whether a band's kernels run as one-warp blocks: with fewer items than
 * this the 128-thread blocks would leave schedulers without a warp. */
static bool staged_small(const Mh2dArgs<double> &a, const Mh2dBand &b)
{
    return staged_recon_items(a.nx, b.r1 - b.r0) <= kStagedSmallItems;
}

static unsigned update_grid(const Mh2dArgs<double> &a, const Mh2dBand &b)
{
    const unsigned cells = (unsigned) (b.r1 - b.r0) * a.nx;
    if (staged_small(a, b)) return staged_blocks(cells, kStagedSmall);
    const unsigned n = staged_blocks(cells, kStagedThreads);
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

cudaError_t staged_launch_arm(const Mh2dArgs<double> &a, cudaStream_t s)
{
    staged_arm_kernel<<<1, 32, 0, s>>>(a);
    return cudaGetLastError();
}

template <int NT, bool TAPE>
static cudaError_t launch_flux(const Mh2dArgs<double> &a, const Mh2dBand &b, cudaStream_t s)
{
    return launch_pdl(staged_flux_kernel<NT, TAPE>, staged_blocks(staged_face_items(a.nx, b.r1 - b.r0), NT), NT, s, a, b);
}

template <int NT>
static cudaError_t launch_update(const Mh2dArgs<double> &a, const Mh2dBand &b, cudaStream_t s)
{
    if (a.gravity != 0.0) return launch_pdl(staged_update_kernel<NT, true>, update_grid(a, b), NT, s, a, b);
    return launch_pdl(staged_update_kernel<NT, false>, update_grid(a, b), NT, s, a, b);
}

cudaError_t staged_launch_step(const Mh2dArgs<double> &a, int limiter, const std::vector<Mh2dBand> &bands, cudaStream_t s)
{
    for (const Mh2dBand &b : bands) {
        const bool small = staged_small(a, b);
        cudaError_t e = a.first_order             ? staged_launch_recon<LIM_MINMOD, 1>(a, b, small, s)
                        : limiter == LIM_MINMOD   ? staged_launch_recon<LIM_MINMOD, 0>(a, b, small, s)
                        : limiter == LIM_VAN_LEER ? staged_launch_recon<LIM_VAN_LEER, 0>(a, b, small, s)
                                                  : staged_launch_recon<LIM_MC, 0>(a, b, small, s);
        if (e != cudaSuccess) return e;
        if (a.tape) e = small ? launch_flux<kStagedSmall, true>(a, b, s) : launch_flux<kStagedThreads, true>(a, b, s);
        else e = small ? launch_flux<kStagedSmall, false>(a, b, s) : launch_flux<kStagedThreads, false>(a, b, s);
        if (e != cudaSuccess) return e;
        e = small ? launch_update<kStagedSmall>(a, b, s) : launch_update<kStagedThreads>(a, b, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace hydro
