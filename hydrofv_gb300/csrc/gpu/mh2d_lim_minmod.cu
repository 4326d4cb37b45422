/*
 * mh2d_lim_minmod.cu -- FP64 step kernels with the minmod limiter: single grid
 * (with and without gravity), adjoint tape and batched forms.
 *
 * Compiled with --fmad=false: the FP64 path must issue the same IEEE
 * operations as the reference CPU code, which never contracts a*b+c.
 */
#include "mh2d_lim.cuh"
#include "mh2d_staged_launch.cuh"

namespace hydro {

HYDRO_MH2D_INSTANTIATE_STEP(double, LIM_MINMOD, 0)
HYDRO_STAGED_INSTANTIATE(LIM_MINMOD, 0)

}  // namespace hydro
