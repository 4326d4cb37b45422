/*
 * mh2d_staged_launch.cuh -- launchers of the staged FP64 step
 * (mh2d_staged.cuh).  The recon kernels are instantiated per limiter
 * (mh2d_lim_*.cu), the flux and update kernels in mh2d.cu.
 */
#ifndef HYDRO_GPU_MH2D_STAGED_LAUNCH_CUH
#define HYDRO_GPU_MH2D_STAGED_LAUNCH_CUH

#include "gpu_internal.h"
#include "mh2d_staged.cuh"

namespace hydro {

/* Launch with programmatic stream serialization: the launch is processed
 * while the kernel before it in the stream runs; every staged kernel waits
 * for that kernel's completion before it reads or writes (pdl_wait). */
template <class... P, class... A>
cudaError_t launch_pdl(void (*kernel)(P...), unsigned grid, cudaStream_t s, const A &...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kStagedThreads);
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

inline unsigned staged_blocks(unsigned items) { return (items + kStagedThreads - 1) / kStagedThreads; }

template <int LIM, int FIRST_ORDER>
cudaError_t staged_launch_recon(const Mh2dArgs<double> &a, const Mh2dBand &b, cudaStream_t s)
{
    return launch_pdl(staged_recon_kernel<LIM, FIRST_ORDER>, staged_blocks(staged_recon_items(a.nx, b.r1 - b.r0)), s, a, b);
}

template <int LIM, int FIRST_ORDER>
cudaError_t staged_launch_batch_recon(const StagedBatchArgs &b, const StagedBatchGroup &g, cudaStream_t s)
{
    return launch_pdl(staged_batch_recon_kernel<LIM, FIRST_ORDER>, g.blocks[0], s, b, g.map[0]);
}

/* Blocks of the many-step kernel that are resident at once (0: it cannot be
 * launched), and its cooperative launch. */
template <int LIM, int FIRST_ORDER>
int staged_loop_resident(bool gravity, int device)
{
    int per_sm = 0, sms = 0, coop = 0;
    const cudaError_t e = gravity
        ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, staged_loop_kernel<LIM, FIRST_ORDER, true>, kStagedThreads, 0)
        : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, staged_loop_kernel<LIM, FIRST_ORDER, false>, kStagedThreads, 0);
    if (e != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return coop ? per_sm * sms : 0;
}

template <int LIM, int FIRST_ORDER>
cudaError_t staged_launch_loop(const Mh2dArgs<double> &a, const Mh2dBand &b, unsigned grid, int steps, cudaStream_t s)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kStagedThreads);
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeCooperative;
    at.val.cooperative = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return a.gravity != 0.0 ? cudaLaunchKernelEx(&cfg, staged_loop_kernel<LIM, FIRST_ORDER, true>, a, b, steps)
                            : cudaLaunchKernelEx(&cfg, staged_loop_kernel<LIM, FIRST_ORDER, false>, a, b, steps);
}

}  // namespace hydro

#define HYDRO_STAGED_INSTANTIATE(LIM, FO) \
    template cudaError_t staged_launch_recon<LIM, FO>(const Mh2dArgs<double> &, const Mh2dBand &, cudaStream_t); \
    template cudaError_t staged_launch_batch_recon<LIM, FO>(const StagedBatchArgs &, const StagedBatchGroup &, cudaStream_t); \
    template int staged_loop_resident<LIM, FO>(bool, int);                                                           \
    template cudaError_t staged_launch_loop<LIM, FO>(const Mh2dArgs<double> &, const Mh2dBand &, unsigned, int, cudaStream_t);

#endif
