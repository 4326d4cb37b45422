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

template <class... P, class... A>
cudaError_t launch_pdl(void (*kernel)(P...), unsigned grid, cudaStream_t s, const A &...args)
{
    return launch_after(kernel, grid, kStagedThreads, s, args...);
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

/* The many-step kernel for a grid: with gravity or without, faces and their
 * states in one phase or in two. */
typedef void (*StagedLoop)(Mh2dArgs<double>, Mh2dBand, int);

template <int LIM, int FIRST_ORDER>
StagedLoop staged_loop(bool gravity, bool fused)
{
    if (gravity) return fused ? staged_loop_kernel<LIM, FIRST_ORDER, true, true> : staged_loop_kernel<LIM, FIRST_ORDER, true, false>;
    return fused ? staged_loop_kernel<LIM, FIRST_ORDER, false, true> : staged_loop_kernel<LIM, FIRST_ORDER, false, false>;
}

inline bool staged_fused(const Mh2dArgs<double> &a, const Mh2dBand &b) { return staged_face_items(a.nx, b.r1 - b.r0) <= kStagedFusedFaces; }

/* Blocks of the many-step kernel (0: it cannot be launched): as many as it has
 * work for or as are resident at once; and its cooperative launch. */
template <int LIM, int FIRST_ORDER>
unsigned staged_loop_blocks(const Mh2dArgs<double> &a, const Mh2dBand &b, int device)
{
    const bool fused = staged_fused(a, b);
    const int rows = b.r1 - b.r0;
    const unsigned blocks = fused ? staged_blocks(2 * staged_face_items(a.nx, rows)) : staged_blocks(staged_recon_items(a.nx, rows));
    int per_sm = 0, sms = 0, coop = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, staged_loop<LIM, FIRST_ORDER>(a.gravity != 0.0, fused), kStagedThreads,
                                                      0) != cudaSuccess ||
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess ||
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, device) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    const unsigned resident = coop ? (unsigned) (per_sm * sms) : 0u;
    return blocks < resident ? blocks : resident;
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
    return cudaLaunchKernelEx(&cfg, staged_loop<LIM, FIRST_ORDER>(a.gravity != 0.0, staged_fused(a, b)), a, b, steps);
}

}  // namespace hydro

#define HYDRO_STAGED_INSTANTIATE(LIM, FO) \
    template cudaError_t staged_launch_recon<LIM, FO>(const Mh2dArgs<double> &, const Mh2dBand &, cudaStream_t); \
    template cudaError_t staged_launch_batch_recon<LIM, FO>(const StagedBatchArgs &, const StagedBatchGroup &, cudaStream_t); \
    template unsigned staged_loop_blocks<LIM, FO>(const Mh2dArgs<double> &, const Mh2dBand &, int);                  \
    template cudaError_t staged_launch_loop<LIM, FO>(const Mh2dArgs<double> &, const Mh2dBand &, unsigned, int, cudaStream_t);

#endif
