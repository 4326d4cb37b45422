/*
 * fast32.cuh -- the FP32 state form's quotients, square roots and powers for
 * ordinary operands.
 *
 * The FP32 step is bound by instruction issue.  Its unit is compiled with
 * approximate division and square root (at most 2 ulp over the whole range of
 * float); most of its operands are ordinary numbers, for which a quotient is
 * two instructions and a root one.  Fast wraps a float whose quotient is
 * a * (1 / b) with the hardware's reciprocal (the definition that the PTX ISA
 * gives for div.approx: at most 2 ulp for a divisor of 2^-126 to 2^126), whose
 * root is PTX's sqrt.approx.ftz and whose power is CUDA's __powf, so the
 * templates of numerics.cuh can be instantiated with it.  A face or cell is
 * checked once, for bounds under which every divisor and root is a normal
 * number, and takes the general instantiation, out of line, where the check
 * fails or the face opens a vacuum.  tests/test_gpu_fp32_forms.py holds the
 * quotient and the root to those bounds and the faces, cells and slopes to the
 * general forms' bits.
 *
 * Shear 2048^2, 100 steps: 0.237 ms a step with the general forms, 0.227 with
 * the slopes alone, 0.182 with slopes, faces and primitives, vacuum faces in
 * the out-of-line form.
 */
#ifndef HYDRO_GPU_FAST32_CUH
#define HYDRO_GPU_FAST32_CUH

#include "numerics.cuh"

namespace hydro {

struct Fast {
    float v;
    Fast() = default;
    __device__ __forceinline__ Fast(float x) : v(x) {}
    __device__ __forceinline__ Fast(double x) : v((float) x) {}
    __device__ __forceinline__ Fast(int x) : v((float) x) {}
    __device__ __forceinline__ explicit operator double() const { return (double) v; }
};

__device__ __forceinline__ Fast operator+(Fast a, Fast b) { return Fast(a.v + b.v); }
__device__ __forceinline__ Fast operator-(Fast a, Fast b) { return Fast(a.v - b.v); }
__device__ __forceinline__ Fast operator*(Fast a, Fast b) { return Fast(a.v * b.v); }
__device__ __forceinline__ Fast operator-(Fast a) { return Fast(-a.v); }
__device__ __forceinline__ bool operator<(Fast a, Fast b) { return a.v < b.v; }
__device__ __forceinline__ bool operator<=(Fast a, Fast b) { return a.v <= b.v; }
__device__ __forceinline__ bool operator>(Fast a, Fast b) { return a.v > b.v; }
__device__ __forceinline__ bool operator>=(Fast a, Fast b) { return a.v >= b.v; }

/* a / b as a * (1 / b), and the root: PTX instructions with subnormals taken
 * as zero. */
__device__ __forceinline__ float fast_div(float a, float b)
{
    float q;
    asm("{\n\t.reg .f32 r;\n\trcp.approx.ftz.f32 r, %2;\n\tmul.f32 %0, %1, r;\n\t}" : "=f"(q) : "f"(a), "f"(b));
    return q;
}

__device__ __forceinline__ float fast_sqrt(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__device__ __forceinline__ Fast dv(Fast a, Fast b) { return Fast(fast_div(a.v, b.v)); }
__device__ __forceinline__ Fast sq(Fast x) { return Fast(fast_sqrt(x.v)); }
__device__ __forceinline__ Fast pw(Fast x, Fast y) { return Fast(__powf(x.v, y.v)); }
__device__ __forceinline__ Fast prod(Fast a, Fast b) { return Fast(prod(a.v, b.v)); }
__device__ __forceinline__ Fast operator/(Fast a, Fast b) { return dv(a, b); }

/* Densities and pressures in 1e-12 .. 1e8 and |u| < 1e8: a star pressure is
 * below 4e24, p* / p below 4e36, a wave speed below 5e28, and a difference of
 * speeds is zero or above 1e-27 (one rounding of a speed of at least 1e-12).
 * The divisors are then normal numbers below 2^126, or zero or infinite, where
 * both forms agree. */
__device__ __forceinline__ bool ordinary(float x) { return x > 1e-12f && x < 1e8f; }

static_assert(sizeof(GasConst<Fast>) == sizeof(GasConst<float>), "the same constants");
__device__ __forceinline__ const GasConst<Fast> &fast_gas(const GasConst<float> &c)
{
    return reinterpret_cast<const GasConst<Fast> &>(c);
}

/* The general forms, out of line (by value: the fast path's states stay in
 * registers). */
struct FluxOut {
    float4 F;
    int rc;
};

static __device__ __noinline__ FluxOut flux_general(const GasConst<float> &c, float4 L, float4 R)
{
    float F[4] = { 0.0f, 0.0f, 0.0f, 0.0f };
    FluxOut o;
    o.rc = hllc_flux_2d(c, L.x, L.y, L.z, L.w, R.x, R.y, R.z, R.w, F);
    o.F = make_float4(F[0], F[1], F[2], F[3]);
    return o;
}

struct PrimOut {
    float4 w;
    float a;
};

static __device__ __noinline__ PrimOut primitive_general(const GasConst<float> &c, float vol, float m, float mx, float my,
                                                         float E)
{
    float w[4];
    cons_to_prim_2d_guarded(c, vol, m, mx, my, E, w);
    PrimOut o;
    o.w = make_float4(w[0], w[1], w[2], w[3]);
    o.a = sound_speed(c, w[0], w[3]);
    return o;
}

/* hllc_flux_2d of states (rho, u_normal, u_tangential, p). */
__device__ __forceinline__ int fast_flux(const GasConst<float> &c, const float L[4], const float R[4], float F[4])
{
    const GasConst<Fast> &g = fast_gas(c);
    const Fast l[4] = { L[0], L[1], L[2], L[3] }, r[4] = { R[0], R[1], R[2], R[3] };
    Fast a_L, a_R, pg, f[4];
    const bool plain = ordinary(L[0]) && ordinary(R[0]) && ordinary(L[3]) && ordinary(R[3]) &&
                       fabsf(L[1]) < 1e8f && fabsf(R[1]) < 1e8f && ordinary(c.gm1) && c.tol > 1e-30f;
    const int reg = plain ? hllc_classify(g, l[0], l[1], l[3], r[0], r[1], r[3], a_L, a_R, pg) : PREG_VACUUM;
    if (reg == PREG_VACUUM) {
        const FluxOut o = flux_general(c, make_float4(L[0], L[1], L[2], L[3]), make_float4(R[0], R[1], R[2], R[3]));
        F[0] = o.F.x;
        F[1] = o.F.y;
        F[2] = o.F.z;
        F[3] = o.F.w;
        return o.rc;
    }
    if (reg == PREG_TRRS) pg = guess_p_trrs(g, l[1], l[3], a_L, r[1], r[3], a_R);
    else if (reg == PREG_TSRS) pg = guess_p_tsrs(g, l[0], l[1], l[3], r[0], r[1], r[3], pg);
    const int rc = hllc_finish(g, l[0], l[1], l[2], l[3], a_L, r[0], r[1], r[2], r[3], a_R, pg, f);
#pragma unroll
    for (int q = 0; q < 4; q++) F[q] = f[q].v;
    return rc;
}

/* cons_to_prim_2d_guarded and the sound speed: w = (rho, u, v, p, a). */
__device__ __forceinline__ void fast_primitive(const GasConst<float> &c, float vol, float m, float mx, float my, float E,
                                               float w[5])
{
    if (!(m > 1e-25f && m < 1e12f && vol > 1e-20f && vol < 1e10f)) {
        const PrimOut q = primitive_general(c, vol, m, mx, my, E);
        w[0] = q.w.x;
        w[1] = q.w.y;
        w[2] = q.w.z;
        w[3] = q.w.w;
        w[4] = q.a;
        return;
    }
    const GasConst<Fast> &g = fast_gas(c);
    Fast o[4];
    cons_to_prim_2d_guarded(g, Fast(vol), Fast(m), Fast(mx), Fast(my), Fast(E), o);
#pragma unroll
    for (int q = 0; q < 4; q++) w[q] = o[q].v;
    const float a2 = fast_div(c.gamma * w[3], w[0]);
    w[4] = fabsf(a2) < 1e-37f ? sqrtf(a2) : fast_sqrt(a2);
}

/* limit_slope, without branches on the signs: the same values for finite
 * operands.  (MC beside a NaN or an infinity may differ in sign; the faces of
 * such a cell have no wave speeds and end the run either way.) */
template <int LIM>
__device__ __forceinline__ float fast_slope(float a, float b)
{
    float s;
    if (LIM == LIM_MINMOD) s = (fabsf(a) < fabsf(b)) ? a : b;
    else if (LIM == LIM_VAN_LEER) s = 2.0f * a * b / (a + b + 1e-10f);
    else s = copysignf(fminf(0.5f * fabsf(a + b), 2.0f * fminf(fabsf(a), fabsf(b))), a);
    return a * b <= 0.0f ? 0.0f : s;
}

}  // namespace hydro

#endif
