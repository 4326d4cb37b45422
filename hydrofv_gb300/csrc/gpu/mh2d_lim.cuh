/*
 * mh2d_lim.cuh -- definitions of the per-limiter launchers declared in
 * mh2d_launch.cuh, and the macro that instantiates them for one
 * (precision, limiter).  Included only by the translation units that
 * instantiate step kernels.
 */
#ifndef HYDRO_GPU_MH2D_LIM_CUH
#define HYDRO_GPU_MH2D_LIM_CUH

#include "gpu_internal.h"
#include "mh2d_launch.cuh"

namespace hydro {

template <class R, int LIM, int FIRST_ORDER>
cudaError_t mh2d_launch_step_lim(const Mh2dArgs<R> &a, int grid, cudaStream_t s)
{
    constexpr int nt = mh2d_threads<R>();
    if (a.gravity == 0.0) return launch_after(mh2d_step_kernel<R, LIM, nt, FIRST_ORDER, false>, grid, nt, s, a);
    if constexpr (sizeof(R) == 4) return launch_after(mh2d_step_kernel<R, LIM, nt, FIRST_ORDER, true>, grid, nt, s, a);
    return cudaErrorNotSupported;
}

template <class R, int LIM, int FIRST_ORDER>
cudaError_t mh2d_launch_batch_lim(const Mh2dBatchArgs<R> &b, int grid, cudaStream_t s)
{
    constexpr int nt = mh2d_threads<R>();
    return launch_after(mh2d_batch_step_kernel<R, LIM, nt, FIRST_ORDER>, grid, nt, s, b);
}

template <class R, int LIM, int FIRST_ORDER>
cudaError_t mh2d_step_occupancy(int *per_sm)
{
    return cudaOccupancyMaxActiveBlocksPerMultiprocessor(per_sm, mh2d_step_kernel<R, LIM, mh2d_threads<R>(), FIRST_ORDER>,
                                                         mh2d_threads<R>(), 0);
}

}  // namespace hydro

/* Everything one (precision, limiter, first-order) combination launches: FP64
 * (the allocation-free run: no gravity, MUSCL-Hancock) the single grid's step,
 * FP32 the batch's and the resident blocks besides. */
#define HYDRO_MH2D_INSTANTIATE_STEP(R, LIM, FO)                                                            \
    template cudaError_t mh2d_launch_step_lim<R, LIM, FO>(const Mh2dArgs<R> &, int, cudaStream_t);
#define HYDRO_MH2D_INSTANTIATE(R, LIM, FO)                                                                 \
    HYDRO_MH2D_INSTANTIATE_STEP(R, LIM, FO)                                                               \
    template cudaError_t mh2d_step_occupancy<R, LIM, FO>(int *);                                          \
    template cudaError_t mh2d_launch_batch_lim<R, LIM, FO>(const Mh2dBatchArgs<R> &, int, cudaStream_t);

#endif
