/*
 * mh2d_lim_mc.cu -- FP64 step kernels with the monotonized-central limiter: single grid
 * (with and without gravity), adjoint tape and batched forms.
 *
 * Compiled with --fmad=false: the FP64 path must issue the same IEEE
 * operations as the reference CPU code, which never contracts a*b+c.
 */
#include "mh2d_lim.cuh"
#include "mh2d_staged_launch.cuh"

namespace hydro {

HYDRO_MH2D_INSTANTIATE_STEP(double, LIM_MC, 0)
HYDRO_STAGED_INSTANTIATE(LIM_MC, 0)

}  // namespace hydro
