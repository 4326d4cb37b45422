/*
 * fp64_int.cuh -- correctly rounded FP64 division and square root on the
 * integer pipes.
 *
 * GB300 retires FP64 at 2 lanes/clk/SM against 128 for FP32 and INT32, and
 * the FP64 MUSCL-Hancock step is bound by its FP64 pipe, which in turn is
 * mostly busy with the FMA sequences behind '/' and sqrt.  The functions
 * here compute the same IEEE-754 round-to-nearest-even results with 32/64-bit
 * integer multiplies (IMAD) and one FP32 MUFU seed, leaving the FP64 pipe to
 * the additions and multiplications of the scheme.
 *
 * Division a / b of normal operands (mantissas ma, mb in [2^52, 2^53)), with
 * B = mb 2^8 and A = ma 2^(7 + s) (s = [ma < mb], so A / B is in [1/2, 1)):
 *   1. Y ~ 2^92 / B to 32 bits: the FP32 reciprocal of mb's leading 24 bits
 *      (relative error ~2^-22) and one integer Newton step Y0 (1 + e) with
 *      the residual e = 1 - B Y0 2^-92, kept below the exact value;
 *   2. the quotient in two digits, each a 32-bit high product with Y and the
 *      exact remainder modulo 2^64: 31 bits, then 22 bits that come out exact
 *      or one too large;
 *   3. the rounding from the signed remainder: up above B / 2, down below
 *      -B / 2 (a quotient of two 53-bit integers is never a midpoint).
 * This is long division with a reciprocal of one digit (Knuth, TAOCP vol. 2,
 * 4.3.1; Moller & Granlund, "Improved division by invariant integers", IEEE
 * TC 2011).  The bounds beside the code hold for every seed with |e| < 2^-21,
 * which is checked.
 *
 * Square root of a normal positive x (mantissa M = m 2^52, m in [1, 4), the
 * exponent left over even):
 *   1. Y ~ 2^32 / sqrt(m): the FP32 reciprocal square root and one integer
 *      Newton step (checked like the divide's);
 *   2. 31 bits of the root, s1 = m Y; the exact remainder M 2^8 - s1^2 and Y
 *      give 22 more;
 *   3. the exact remainder R of that root S decides the rounding: up where
 *      R > S, down where R <= -S (a square root is never a midpoint).
 *
 * Cost on one SM with 24 resident warps: an inlined divide 27.4 cycles per
 * warp (33.8 with 53-bit quotients from a 64 x 64 high product), out of line
 * 36.8 (46.7), a square root out of line 29.9 (50.1, which checked its result
 * with a 128-bit product); latency out of line 282 (448) and 298 (496) cycles.
 *
 * Correctness does not rest on the seed's accuracy: both check the seed's
 * residual, and every operand or result outside the fast path
 * (zero, subnormal, infinite, NaN, negative for sqrt, quotients that
 * overflow the normal range before rounding or underflow) or a failed check
 * takes the hardware operation.  The results are therefore bit-identical to
 * '/' and sqrt.  Host builds keep the plain operators; the integer forms are
 * also compiled for the host (with host seeds) so that they can be checked
 * against the host's IEEE operations on the CPU.
 *
 * The same file holds the other FP64-pipe savings of the step kernel, each
 * exact: the slope limiter's sign test on the bits (product_nonpositive),
 * ordered comparisons (lt, le), and the reference's "+ 0.0" terms
 * (add_zero, zero_minus).  All of them read a double's bits through an
 * opaque move (bits): with a plain bitcast the compiler recognises zero,
 * sign and exponent tests as floating-point class tests and emits FP64
 * compares again.  The divide and square root run out of line on the device
 * (div_dev, sqrt_dev), one copy per kernel: inlined at the step kernel's ~40
 * call sites they overflow the instruction cache.
 */
#ifndef HYDRO_GPU_FP64_INT_CUH
#define HYDRO_GPU_FP64_INT_CUH

#include <math.h>
#include <string.h>

#ifdef __CUDACC__
#define FXHD __host__ __device__ __forceinline__
#else
#define FXHD static inline
#endif

namespace hydro {
namespace fx {

typedef unsigned long long u64;
typedef long long i64;

/* The bits of a double.  On the device through an opaque move: a plain
 * bitcast lets the compiler recognise the bit tests below (zero, exponent
 * range, sign) as floating-point class tests and emit them as FP64 compares
 * on the FP64 pipe, which is what these forms exist to avoid. */
FXHD u64 bits(double x)
{
#if defined(__CUDA_ARCH__)
    u64 u;
    asm("mov.b64 %0, %1;" : "=l"(u) : "d"(x));
    return u;
#else
    u64 b;
    memcpy(&b, &x, sizeof b);
    return b;
#endif
}

FXHD double from_bits(u64 b)
{
#if defined(__CUDA_ARCH__)
    return __longlong_as_double((i64) b);
#else
    double x;
    memcpy(&x, &b, sizeof x);
    return x;
#endif
}

FXHD unsigned fbits(float x)
{
#if defined(__CUDA_ARCH__)
    return (unsigned) __float_as_uint(x);
#else
    unsigned b;
    memcpy(&b, &x, sizeof b);
    return b;
#endif
}

FXHD float from_fbits(unsigned b)
{
#if defined(__CUDA_ARCH__)
    return __uint_as_float(b);
#else
    float x;
    memcpy(&x, &b, sizeof x);
    return x;
#endif
}

/* FP32 seeds: reciprocal and reciprocal square root of x in [1, 4). */
FXHD float rcp_seed(float x)
{
#if defined(__CUDA_ARCH__)
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return 1.0f / x;
#endif
}

FXHD float rsqrt_seed(float x)
{
#if defined(__CUDA_ARCH__)
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return y;
#else
    return 1.0f / sqrtf(x);
#endif
}

static const u64 FRAC = 0x000fffffffffffffull;
static const u64 HIDDEN = 0x0010000000000000ull;
static const u64 SIGN = 0x8000000000000000ull;

/* 32-bit high products. */
FXHD unsigned mulhi32(unsigned a, unsigned b)
{
#if defined(__CUDA_ARCH__)
    return __umulhi(a, b);
#else
    return (unsigned) (((u64) a * b) >> 32);
#endif
}

FXHD int mulhi32s(int a, int b)
{
#if defined(__CUDA_ARCH__)
    return __mulhi(a, b);
#else
    return (int) (((i64) a * b) >> 32);
#endif
}

/* A divisor's reciprocal, for one or several quotients: B = mb 2^8 (61
 * bits), Y = 2^92 / B - d with 1 <= d < 3.2 (32 bits), and its sign and
 * exponent word. */
struct Recip {
    u64 B;
    unsigned Y, hb;
    bool ok;      /* normal divisor, seed within its bound */
};

/* seed_scale multiplies the FP32 seed: 1 in the kernels; the tests perturb
 * it to exercise the check. */
FXHD Recip recip(double b, float seed_scale = 1.0f)
{
    const u64 ub = bits(b);
    Recip r;
    r.hb = (unsigned) (ub >> 32);
    r.B = ((ub & FRAC) | HIDDEN) << 8;
    /* the seed, kept below 1 so that its fixed-point form is a shift */
    const float y = fminf(rcp_seed(from_fbits(0x3f800000u | ((unsigned) (ub >> 29) & 0x7fffffu))) * seed_scale, 0x1.fffffep-1f);
    const unsigned Y0 = (fbits(y) << 8) | 0x80000000u;
    /* e = 1 - B Y0 2^-92 to 60 bits; one Newton step Y0 (1 + e) needs
     * |e| < 2^-21 (then e^2 is below the last place of Y) */
    const u64 p = (r.B >> 32) * Y0 + mulhi32((unsigned) r.B, Y0);
    const i64 e = (i64) ((1ull << 60) - p);
    const unsigned eh = (unsigned) ((u64) e >> 32);
    r.ok = eh + 0x80u < 0x100u && ((r.hb >> 20) & 0x7ffu) - 1u < 2046u;
    r.Y = Y0 + (unsigned) (mulhi32s((int) (unsigned) ((u64) e >> 8), (int) (Y0 >> 1)) >> 19) - 1u;
    return r;
}

/* RN(a / b) with b's reciprocal when `ok` comes back true (see the header
 * comment). */
FXHD double div_recip(double a, const Recip &r, bool &ok)
{
    const u64 ua = bits(a);
    const unsigned ha = (unsigned) (ua >> 32);
    const u64 ma = (ua & FRAC) | HIDDEN;
    const int s = (ma << 8) < r.B ? 1 : 0;
    /* 31 quotient bits, at most 5.2 low; the remainder is below 6.2 B < 2^64 */
    const unsigned q1 = mulhi32((unsigned) ((ma << (10 + s)) >> 32), r.Y);
    const u64 R1 = ((u64) ((unsigned) ma << (6 + s)) << 32) - (u64) q1 * r.B;
    /* 22 more: the product is at most 4.7 / 64 low, so with 5 / 64 added they
     * are exact or one too large and the remainder lies in (-B, B) */
    const unsigned q2 = (mulhi32((unsigned) (R1 >> 32), r.Y) + 5u) >> 6;
    const i64 R2 = (i64) ((R1 << 22) - (u64) q2 * r.B);
    const i64 half = (i64) (r.B >> 1);
    u64 Q = (u64) q1 * (1u << 22) + q2;
    /* nearest: a quotient of two 53-bit integers is never a midpoint */
    Q += (R2 > half) ? 1ull : 0ull;
    Q -= (R2 < -half) ? 1ull : 0ull;
    const unsigned ea = (ha >> 20) & 0x7ffu, eb = (r.hb >> 20) & 0x7ffu;
    const unsigned e = ea - eb + 1022u - (unsigned) s;       /* biased exponent of the quotient - 1 */
    const unsigned sign = (ha ^ r.hb) & 0x80000000u;
    const bool a_zero = (ua << 1) == 0ull;
    ok = r.ok && (a_zero || (ea - 1u < 2046u && e < 2046u));
    const u64 res = Q + ((u64) (sign + (e << 20)) << 32);
    return from_bits(a_zero ? (u64) sign << 32 : res);
}

/* RN(a / b) when `ok` comes back true. */
FXHD double div_fast(double a, double b, bool &ok, float seed_scale = 1.0f)
{
    return div_recip(a, recip(b, seed_scale), ok);
}

/* RN(sqrt(x)) when `ok` comes back true. */
FXHD double sqrt_fast(double x, bool &ok)
{
    const u64 ux = bits(x);
    const unsigned ex = (unsigned) (ux >> 52);                /* sign bit included */
    const unsigned odd = (ex & 1u) ^ 1u;                      /* unbiased exponent - 52 is odd */
    const u64 M = ((ux & FRAC) | HIDDEN) << odd;              /* m 2^52, m in [1, 4) */
    const unsigned M30 = (unsigned) (M >> 22);                /* m 2^30 */

    const float fm = from_fbits(((127u + odd) << 23) | ((unsigned) (ux >> 29) & 0x7fffffu));
    const float y = fminf(rsqrt_seed(fm), 0x1.fffffep-1f);
    const unsigned Y0 = (fbits(y) << 8) | 0x80000000u;        /* y 2^32, y in (1/2, 1) */
    /* e = 1 - m y^2 to 2^-29; the Newton step Y0 (1 + e / 2) needs |e| < 2^-20 */
    const i64 e = (i64) ((1ull << 62) - (u64) M30 * mulhi32(Y0, Y0));
    const unsigned eh = (unsigned) ((u64) e >> 32);
    const bool seed_ok = eh + 0x400u < 0x800u;
    const unsigned Y = Y0 + (unsigned) (mulhi32s((int) (unsigned) ((u64) e >> 11), (int) (Y0 >> 1)) >> 19);
    /* 31 bits of the root S = sqrt(m) 2^52, then 22 more from the remainder
     * of either sign; S comes out within one of the rounded root */
    const unsigned s1 = mulhi32(M30, Y);
    const i64 r1 = (i64) ((M << 8) - (u64) s1 * s1);
    const int s2 = mulhi32s((int) (r1 >> 6), (int) (Y >> 1)) >> 2;
    const u64 T = ((u64) s1 << 23) + (u64) (i64) s2;          /* 2 S - s2 */
    i64 S = (i64) ((u64) s1 << 22) + s2;
    const i64 R2 = (i64) (((u64) r1 << 44) - T * (u64) (i64) s2);   /* S_exact^2 - S^2 */
    /* nearest: (S +- 1/2)^2 = S^2 +- S + 1/4 */
    const i64 d = (R2 > S ? 1 : 0) - (R2 <= -S ? 1 : 0);
    S += d;
    const int t = ((int) ex - 1075 - (int) odd) >> 1;         /* exponent left over, halved */
    ok = ex - 1u < 2046u && seed_ok;
    return from_bits(((u64) (unsigned) (t + 1048) << 52) + (u64) S);
}

/*
 * The limiter's sign test a * b <= 0 decided on the bits where that is exact
 * without the multiply: 1 (true), 0 (false), or -1 when it is not decided
 * here (a NaN or infinite operand, a subnormal one, or a product of normal
 * operands small enough to underflow to zero: the caller evaluates the FP64
 * expression).  A zero times a finite operand is a signed zero (true);
 * otherwise the product's sign is the XOR of the signs, and for
 * ea + eb >= 973 the product is at least 2^-1074 in magnitude.
 */
FXHD int product_nonpositive(u64 ua, u64 ub)
{
    const u64 aa = ua & ~SIGN, ab = ub & ~SIGN;
    const unsigned ea = (unsigned) (aa >> 52), eb = (unsigned) (ab >> 52);
    if (ea == 0x7ffu || eb == 0x7ffu) return -1;
    if (aa == 0ull || ab == 0ull) return 1;
    if (ea == 0u || eb == 0u || ea + eb < 973u) return -1;
    return (int) ((ua ^ ub) >> 63);
}

/* Ordered key of a non-NaN double's bits: monotone in the value, with +0
 * and -0 equal. */
FXHD i64 okey(u64 b) { return (i64) b >= 0 ? (i64) b : -(i64) (b & ~SIGN); }
FXHD bool nan_bits(u64 b) { return (b & ~SIGN) > 0x7ff0000000000000ull; }

#if defined(__CUDACC__)
/* Hardware operations for the cases the fast paths leave out; kept out of
 * line so that the fast path's call sites stay small. */
static __device__ __noinline__ double div_hw(double a, double b) { return a / b; }
static __device__ __noinline__ double sqrt_hw(double x) { return sqrt(x); }

/* The device forms, out of line: one copy per kernel instead of one per
 * call site.  The step kernel has ~40 divide / square-root sites; inlined,
 * their integer sequences overflow the instruction cache (measured on the
 * 2048^2 shear layer: 744 M cell-updates/s inlined, 819 M out of line). */
static __device__ __noinline__ double div_dev(double a, double b)
{
    bool ok;
    const double q = div_fast(a, b, ok);
    return ok ? q : div_hw(a, b);
}

/* 1 / x: the divide with a known numerator, which the compiler folds into
 * the integer sequence (the quotient step becomes a shift of Y1). */
static __device__ __noinline__ double rcp_dev(double x)
{
    bool ok;
    const double q = div_fast(1.0, x, ok);
    return ok ? q : div_hw(1.0, x);
}

static __device__ __noinline__ double sqrt_dev(double x)
{
    bool ok;
    const double r = sqrt_fast(x, ok);
    return ok ? r : sqrt_hw(x);
}
#endif

}  // namespace fx

/* a / b and sqrt(x) as the kernels use them: the integer forms on the
 * device for double (the non-template overloads), the operators for every
 * other type and on the host. */
template <class R>
FXHD R dv(R a, R b) { return a / b; }

template <class R>
FXHD R sq(R x) { return sqrt(x); }

/* 1 / x as the kernels evaluate it (the value of dv(1, x)). */
template <class R>
FXHD R rv(R x) { return R(1) / x; }

FXHD double rv(double x)
{
#if defined(__CUDA_ARCH__)
    return fx::rcp_dev(x);
#else
    return 1.0 / x;
#endif
}

FXHD double dv(double a, double b)
{
#if defined(__CUDA_ARCH__)
    return fx::div_dev(a, b);
#else
    return a / b;
#endif
}

/* The same with the integer form inlined, for kernels with few divides: the
 * staged step's recon and update kernels and the flux kernel's classification
 * (2048^2 2.274 -> 2.243 ms per step; with the flux kernel's finish inlined
 * too it is 2.31 - 2.34). */
FXHD double dvi(double a, double b)
{
#if defined(__CUDA_ARCH__)
    bool ok;
    const double q = fx::div_fast(a, b, ok);
    return ok ? q : fx::div_hw(a, b);
#else
    return a / b;
#endif
}

FXHD double sqi(double x)
{
#if defined(__CUDA_ARCH__)
    bool ok;
    const double r = fx::sqrt_fast(x, ok);
    return ok ? r : fx::sqrt_hw(x);
#else
    return sqrt(x);
#endif
}

FXHD double sq(double x)
{
#if defined(__CUDA_ARCH__)
    return fx::sqrt_dev(x);
#else
    return sqrt(x);
#endif
}

/* x + 0.0 and 0.0 - x as the kernels evaluate them (the reference's literal
 * "+ 0.0" terms, which only turn -0.0 into +0.0).  On the device, for
 * double, a compare and select on the bits: x + 0.0 is x except that -0.0
 * becomes +0.0, and 0.0 - x is -x except that both zeros give +0.0.  A NaN
 * stays a NaN (its payload bits are not canonicalised as an FP64 add would). */
template <class R>
FXHD R add_zero(R x) { return x + R(0); }

template <class R>
FXHD R zero_minus(R x) { return R(0) - x; }

FXHD double add_zero(double x)
{
#if defined(__CUDA_ARCH__)
    const fx::u64 u = fx::bits(x);
    return fx::from_bits(u == fx::SIGN ? 0ull : u);
#else
    return x + 0.0;
#endif
}

FXHD double zero_minus(double x)
{
#if defined(__CUDA_ARCH__)
    const fx::u64 u = fx::bits(x);
    return fx::from_bits((u << 1) == 0ull ? 0ull : (u ^ fx::SIGN));
#else
    return 0.0 - x;
#endif
}

/* x == 0.0 (either zero; false for NaN), on the bits for double on the device. */
template <class R>
FXHD bool eq_zero(R x) { return x == R(0); }

FXHD bool eq_zero(double x)
{
#if defined(__CUDA_ARCH__)
    return (fx::bits(x) << 1) == 0ull;
#else
    return x == 0.0;
#endif
}

/* Ordered comparisons as the kernels evaluate them: IEEE semantics (false
 * when either operand is NaN, +0 == -0), on the integer pipes for double on
 * the device. */
template <class R>
FXHD bool lt(R a, R b) { return a < b; }

template <class R>
FXHD bool le(R a, R b) { return a <= b; }

FXHD bool lt(double a, double b)
{
#if defined(__CUDA_ARCH__)
    const fx::u64 ua = fx::bits(a), ub = fx::bits(b);
    return !fx::nan_bits(ua) && !fx::nan_bits(ub) && fx::okey(ua) < fx::okey(ub);
#else
    return a < b;
#endif
}

FXHD bool le(double a, double b)
{
#if defined(__CUDA_ARCH__)
    const fx::u64 ua = fx::bits(a), ub = fx::bits(b);
    return !fx::nan_bits(ua) && !fx::nan_bits(ub) && fx::okey(ua) <= fx::okey(ub);
#else
    return a <= b;
#endif
}

}  // namespace hydro

#endif
