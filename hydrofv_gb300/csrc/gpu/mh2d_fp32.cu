/*
 * mh2d_fp32.cu -- FP32-state instantiations of the 2D step (the precision
 * form) and its helper kernels, plus the FP64 <-> FP32 conversions used on
 * upload and download.
 *
 * State, fluxes and limiters run in FP32 (FMA contraction allowed); FP64 is
 * kept for the dt reduction (the maxima are FP64 ordered-bit words and dt is
 * computed in FP64), for pressure recovery where kinetic energy exceeds half
 * of the total energy (cons_to_prim_2d_guarded) and for the compensated
 * conserved totals.
 */
#include "mh2d_lim.cuh"
#include "hydro_gpu.h"

namespace hydro {

HYDRO_MH2D_INSTANTIATE(float, LIM_MINMOD, 0)
HYDRO_MH2D_INSTANTIATE(float, LIM_MINMOD, 1)
HYDRO_MH2D_INSTANTIATE(float, LIM_VAN_LEER, 0)
HYDRO_MH2D_INSTANTIATE(float, LIM_MC, 0)
template int mh2d_resident_ctas<float>(int, int, int);
template cudaError_t mh2d_launch_batch_step<float>(const Mh2dBatchArgs<float> &, int, int, int, cudaStream_t);
template cudaError_t mh2d_launch_step<float>(const Mh2dArgs<float> &, int, cudaStream_t);
template cudaError_t mh2d_launch_prepare<float>(const Mh2dArgs<float> &, cudaStream_t);
template cudaError_t mh2d_launch_arm<float>(const Mh2dArgs<float> &, cudaStream_t);
template cudaError_t mh2d_launch_batch_arm<float>(const Mh2dArgs<float> *, int, cudaStream_t);
template cudaError_t mh2d_launch_materialize<float>(const Mh2dArgs<float> &, int,
                                                    float *const[4], cudaStream_t);
template cudaError_t mh2d_launch_totals<float>(const Mh2dArgs<float> &, int, double *, cudaStream_t);

cudaError_t convert_f64_to_f32(const double *src, float *dst, long long n, cudaStream_t s)
{
    convert_kernel<double, float><<<1024, 256, 0, s>>>(src, dst, n);
    return cudaGetLastError();
}

cudaError_t convert_f32_to_f64(const float *src, double *dst, long long n, cudaStream_t s)
{
    convert_kernel<float, double><<<1024, 256, 0, s>>>(src, dst, n);
    return cudaGetLastError();
}

/* The short forms of fast32.cuh beside the general ones (hydro_gpu_fp32_eval). */
__global__ void fp32_forms_kernel(int op, long long n, const GasConst<float> gas, float vol, const float *a, const float *b,
                                  float *fast, float *general)
{
    for (long long k = blockIdx.x * (long long) blockDim.x + threadIdx.x; k < n; k += (long long) gridDim.x * blockDim.x) {
        if (op == 0) {
            const float L[4] = { a[4 * k], a[4 * k + 1], a[4 * k + 2], a[4 * k + 3] };
            const float R[4] = { b[4 * k], b[4 * k + 1], b[4 * k + 2], b[4 * k + 3] };
            float F[4] = { 0.0f, 0.0f, 0.0f, 0.0f };
            const int rc = fast_flux(gas, L, R, F);
            const FluxOut o = flux_general(gas, make_float4(L[0], L[1], L[2], L[3]), make_float4(R[0], R[1], R[2], R[3]));
            const float G[4] = { o.F.x, o.F.y, o.F.z, o.F.w };
            for (int q = 0; q < 4; q++) {
                fast[5 * k + q] = F[q];
                general[5 * k + q] = G[q];
            }
            fast[5 * k + 4] = (float) rc;
            general[5 * k + 4] = (float) o.rc;
        } else if (op == 1) {
            float w[5];
            fast_primitive(gas, vol, a[4 * k], a[4 * k + 1], a[4 * k + 2], a[4 * k + 3], w);
            const PrimOut o = primitive_general(gas, vol, a[4 * k], a[4 * k + 1], a[4 * k + 2], a[4 * k + 3]);
            const float g[5] = { o.w.x, o.w.y, o.w.z, o.w.w, o.a };
            for (int q = 0; q < 5; q++) {
                fast[5 * k + q] = w[q];
                general[5 * k + q] = g[q];
            }
        } else if (op <= 4) {
            fast[k] = op == 2 ? fast_slope<LIM_MINMOD>(a[k], b[k])
                    : op == 3 ? fast_slope<LIM_VAN_LEER>(a[k], b[k]) : fast_slope<LIM_MC>(a[k], b[k]);
            general[k] = op == 2 ? limit_slope<LIM_MINMOD>(a[k], b[k])
                       : op == 3 ? limit_slope<LIM_VAN_LEER>(a[k], b[k]) : limit_slope<LIM_MC>(a[k], b[k]);
        } else {
            fast[k] = op == 5 ? fast_div(a[k], b[k]) : fast_sqrt(a[k]);
            general[k] = op == 5 ? a[k] / b[k] : sqrtf(a[k]);
        }
    }
}

}  // namespace hydro

extern "C" int hydro_gpu_fp32_eval(int device, int op, long long n, double gamma, double tol, double vol, const float *a,
                                   const float *b, float *fast, float *general)
{
    using namespace hydro;
    if (n <= 0) return 0;
    if (op < 0 || op > 6) return (int) cudaErrorInvalidValue;
    const size_t in = (op <= 1 ? 4 : 1) * (size_t) n, out = (op <= 1 ? 5 : 1) * (size_t) n;
    cudaError_t e = cudaSetDevice(device);
    float *slab = nullptr;
    if (e == cudaSuccess) e = cudaMalloc(&slab, 2 * (in + out) * sizeof(float));
    if (e != cudaSuccess) return (int) e;
    float *da = slab, *db = da + in, *df = db + in, *dg = df + out;
    e = cudaMemcpy(da, a, in * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) e = cudaMemcpy(db, b, in * sizeof(float), cudaMemcpyHostToDevice);
    if (e == cudaSuccess) {
        fp32_forms_kernel<<<152, 128>>>(op, n, make_gas_const<float>(gamma, tol), (float) vol, da, db, df, dg);
        e = cudaGetLastError();
    }
    if (e == cudaSuccess) e = cudaMemcpy(fast, df, out * sizeof(float), cudaMemcpyDeviceToHost);
    if (e == cudaSuccess) e = cudaMemcpy(general, dg, out * sizeof(float), cudaMemcpyDeviceToHost);
    cudaFree(slab);
    return (int) e;
}
