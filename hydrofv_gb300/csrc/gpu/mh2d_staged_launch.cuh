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
cudaError_t launch_pdl(void (*kernel)(P...), unsigned grid, unsigned block, cudaStream_t s, const A &...args)
{
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(block);
    cfg.stream = s;
    cudaLaunchAttribute at;
    at.id = cudaLaunchAttributeProgrammaticStreamSerialization;
    at.val.programmaticStreamSerializationAllowed = 1;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    return cudaLaunchKernelEx(&cfg, kernel, args...);
}

inline unsigned staged_blocks(unsigned items, unsigned nt) { return (items + nt - 1) / nt; }

template <int LIM, int FIRST_ORDER>
cudaError_t staged_launch_recon(const Mh2dArgs<double> &a, const Mh2dBand &b, bool small, cudaStream_t s)
{
    const unsigned items = staged_recon_items(a.nx, b.r1 - b.r0);
    if (small)
        return launch_pdl(staged_recon_kernel<LIM, FIRST_ORDER, kStagedSmall>, staged_blocks(items, kStagedSmall),
                          kStagedSmall, s, a, b);
    return launch_pdl(staged_recon_kernel<LIM, FIRST_ORDER, kStagedThreads>, staged_blocks(items, kStagedThreads),
                      kStagedThreads, s, a, b);
}

}  // namespace hydro

#define HYDRO_STAGED_INSTANTIATE(LIM, FO) \
    template cudaError_t staged_launch_recon<LIM, FO>(const Mh2dArgs<double> &, const Mh2dBand &, bool, cudaStream_t);

#endif
