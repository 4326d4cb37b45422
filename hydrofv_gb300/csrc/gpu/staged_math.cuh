/*
 * staged_math.cuh -- the pointwise arithmetic of the staged FP64 step.
 *
 * The same IEEE results as the templates of numerics.cuh, for fewer cycles of
 * the FP64 pipe, which bounds the step:
 *
 *  - Sums and products are issued as fma(a, 1, b) and fma(a, b, -0) with the
 *    1 and the -0 in registers (Fm).  The product a * 1 is exact, and adding
 *    -0 changes no value and no sign of zero, so the one rounding is that of
 *    a + b and a * b.  A GB300 SM retires a DFMA with three register operands
 *    every 16 cycles per warp, but a DADD, a DMUL or a DFMA with a constant
 *    or immediate operand every 19 (measured with 4 to 24 warps on one SM).
 *    The two constants are read from memory so that the compiler cannot turn
 *    the fma back into an add or a multiply.
 *  - Scalings by powers of two go into an fma (x - 0.5 s as fma(-0.5, s, x):
 *    0.5 s is exact, so the one rounding is the sum's) or become an exponent
 *    step on the integer pipe.
 *  - Products that the formulas repeat (rho u, S - u, rho (S - u)) are formed
 *    once and selected with the side.
 *  - Comparisons of positive numbers compare the bit patterns as integers.
 *
 * Per cell-update of the 2048^2 shear layer this leaves 285 FP64 instructions
 * of 16 cycles where there were 335 of 19 (divides excluded): recon 248 -> 161
 * us, flux 487 -> 440 us per million cells, the step 3.07 -> 2.51 ms.
 *
 * Each shortcut holds for operands in a stated range; whatever lies outside
 * (zero or negative densities, exponents near the ends, infinities, NaN)
 * takes the templates of numerics.cuh, out of line.
 *
 * Compiled with --fmad=false; the host build (tests) uses the same code with
 * the C library's fma.
 */
#ifndef HYDRO_GPU_STAGED_MATH_CUH
#define HYDRO_GPU_STAGED_MATH_CUH

#include "numerics.cuh"

#ifdef __CUDACC__
#define SLOW_PATH [[maybe_unused]] static __host__ __device__ __noinline__
#else
#define SLOW_PATH static
#endif

namespace hydro {

#if defined(__CUDACC__)
static __device__ double d_fma_const[3] = { 1.0, -0.0, -0.5 };
#endif

/* a + b, a - b and a * b as fused multiply-adds (see the header comment). */
struct Fm {
    double one, mz, mh;   /* 1, -0, -0.5 */
    FXHD double add(double a, double b) const { return fma(a, one, b); }
    FXHD double sub(double a, double b) const { return fma(-b, one, a); }
    FXHD double mul(double a, double b) const { return fma(a, b, mz); }
};

FXHD Fm make_fm()
{
    Fm f;
#if defined(__CUDA_ARCH__)
    f.one = *(volatile double *) &d_fma_const[0];
    f.mz = *(volatile double *) &d_fma_const[1];
    f.mh = *(volatile double *) &d_fma_const[2];
#else
    f.one = 1.0;
    f.mz = -0.0;
    f.mh = -0.5;
#endif
    return f;
}

namespace fx {

FXHD unsigned hi(double x) { return (unsigned) (bits(x) >> 32); }

/* Positive and between 2^-250 and 2^250. */
FXHD bool moderate(double x) { return hi(x) - (773u << 20) < (500u << 20); }

FXHD bool finite(double x) { return (hi(x) & 0x7ff00000u) != 0x7ff00000u; }

/* x / 2 and 2 x of a normal x that stays normal. */
FXHD double halve(double x) { return from_bits(bits(x) - HIDDEN); }
FXHD double twice(double x) { return from_bits(bits(x) + HIDDEN); }

/* x >= 0 of a finite x (-0 too). */
FXHD bool not_below_zero(double x) { const u64 b = bits(x); return (i64) b >= 0 || b == SIGN; }

/* 0 < |x| < 2^-962. */
FXHD bool tiny(double x)
{
    const u64 b = bits(x);
    const unsigned h = (unsigned) (b >> 32) & 0x7fffffffu;
    return h < (61u << 20) && (h | (unsigned) b) != 0u;
}

}  // namespace fx

/* ---------------------------------------------------------------- limiter */

template <int LIM>
SLOW_PATH double slope_slow(double a, double b) { return limit_slope<LIM>(a, b); }

/* limit_slope for a = w - w_minus, b = w_plus - w.  The shortcut needs both
 * magnitudes in [2^-1021, 2^1021) and their product above 2^-1074, so that
 * 2 m, (a + b) / 2 and the sign of a b are exact on the bits; a zero operand
 * beside a finite one gives zero. */
template <int LIM>
FXHD double slope(const Fm &f, double a, double b)
{
    const fx::u64 ua = fx::bits(a), ub = fx::bits(b);
    const fx::u64 aa = ua & ~fx::SIGN, ab = ub & ~fx::SIGN;
    const unsigned ha = (unsigned) (aa >> 32), hb = (unsigned) (ab >> 32);
    const unsigned lo = 2u << 20, span = 2042u << 20;
    if (ha - lo < span && hb - lo < span && ha + hb >= (975u << 20)) {
        if ((ua ^ ub) >> 63) return 0.0;
        if (LIM == LIM_MINMOD) return (aa < ab) ? a : b;
        if (LIM == LIM_VAN_LEER)
            return dv(f.mul(fx::twice(a), b), f.add(f.add(a, b), 1e-10));
        const fx::u64 m = (aa < ab ? aa : ab) + fx::HIDDEN;                       /* 2 min(|a|, |b|) */
        const fx::u64 avg = (fx::bits(f.add(a, b)) & ~fx::SIGN) - fx::HIDDEN;     /* |a + b| / 2 */
        return fx::from_bits((avg < m ? avg : m) | (ua & fx::SIGN));
    }
    if ((aa == 0ull && hb < 0x7ff00000u) || (ab == 0ull && ha < 0x7ff00000u)) return 0.0;
    return slope_slow<LIM>(a, b);
}

/* -------------------------------------------------------------- predictor */

SLOW_PATH double half_step_slow(double x, double s, double h) { return x + h * s; }

/* x + h s for h = -0.5 or 0.5: h s is exact unless s is subnormal or nearly
 * so, and then only a zero or tiny x lets the difference show. */
FXHD double half_step(double x, double s, double h)
{
    if ((fx::hi(x) & 0x7fffffffu) < (61u << 20) && fx::tiny(s)) return half_step_slow(x, s, h);
    return fma(h, s, x);
}

/* hancock_2d (numerics.cuh). */
FXHD void predict(const Fm &f, double dtA, double dtA_rho, double rho, double n, double t, double p, double a,
                  const double d[4], double d_rho_vel, double lo[4], double hi[4])
{
    const double cn = f.mul(dtA, n);
    const double up = f.add(f.one, cn), um = f.sub(f.one, cn);
    const double dr = f.mul(dtA, rho);
    const double draa = f.mul(f.mul(f.mul(dr, a), a), d[1]);
    const double drv = f.mul(dr, d_rho_vel), drp = f.mul(dtA_rho, d[3]);
    const double mh = f.mh, ph = -f.mh;
    lo[0] = half_step(rho, add_zero(f.add(f.mul(up, d[0]), drv)), mh);
    lo[1] = half_step(n, f.add(add_zero(f.mul(up, d[1])), drp), mh);
    lo[2] = half_step(t, add_zero(f.mul(up, d[2])), mh);
    lo[3] = half_step(p, f.add(add_zero(draa), f.mul(up, d[3])), mh);
    hi[0] = half_step(rho, add_zero(f.sub(f.mul(um, d[0]), drv)), ph);
    hi[1] = half_step(n, f.sub(add_zero(f.mul(um, d[1])), drp), ph);
    hi[2] = half_step(t, add_zero(f.mul(um, d[2])), ph);
    hi[3] = half_step(p, f.add(zero_minus(draa), f.mul(um, d[3])), ph);
}

/* ------------------------------------------------------------------- HLLC */

SLOW_PATH int classify_slow(const GasConst<double> &c, double rho_L, double u_L, double p_L, double rho_R, double u_R,
                            double p_R, double &a_L, double &a_R, double &ppv)
{
    return hllc_classify(c, rho_L, u_L, p_L, rho_R, u_R, p_R, a_L, a_R, ppv);
}

SLOW_PATH int finish_slow(const GasConst<double> &c, double rho_L, double u_L, double v_L, double p_L, double a_L,
                          double rho_R, double u_R, double v_R, double p_R, double a_R, double pg, double F[4],
                          double wave[3])
{
    return hllc_finish(c, rho_L, u_L, v_L, p_L, a_L, rho_R, u_R, v_R, p_R, a_R, pg, F, wave);
}

SLOW_PATH bool vacuum_slow(const GasConst<double> &c, double as, double du) { return le(dv(as * 2.0, c.gp1), du); }

SLOW_PATH double pvrs_slow(double sp, double du, double rs, double as) { return 0.5 * sp - 0.125 * du * rs * as; }

/* hllc_classify (numerics.cuh); `plain` comes back false where the operands
 * lie outside the shortcuts' range. */
FXHD int face_classify(const Fm &f, const GasConst<double> &c, double rho_L, double u_L, double p_L, double rho_R,
                       double u_R, double p_R, double &a_L, double &a_R, double &ppv, bool &plain)
{
    plain = fx::moderate(rho_L) && fx::moderate(rho_R) && fx::moderate(p_L) && fx::moderate(p_R);
    if (!plain) return classify_slow(c, rho_L, u_L, p_L, rho_R, u_R, p_R, a_L, a_R, ppv);
    a_L = sqi(dvi(f.mul(c.gamma, p_L), rho_L));
    a_R = sqi(dvi(f.mul(c.gamma, p_R), rho_R));
    const double as = f.add(a_L, a_R), du = f.sub(u_R, u_L);
    /* 2 (a_L + a_R) / (gamma + 1) lies in [2^(d-1), 2^(d+1)] (quot_le_fast):
     * a negative u_R - u_L, or one below 2^(d-1), is not above it */
    const unsigned hd = fx::hi(du);
    const int d = (int) (fx::hi(as) >> 20) + 1 - (int) (fx::hi(c.gp1) >> 20);
    ppv = 0.0;
    if ((int) hd >= 0 && (int) (hd >> 20) - 1023 > d - 2 && vacuum_slow(c, as, du)) return PREG_VACUUM;
    const double sp = f.add(p_L, p_R), rs = f.add(rho_L, rho_R);
    const unsigned ed = (hd >> 20) & 0x7ffu;
    /* (0.125 du) rs as = 0.125 (du rs as) where no product leaves the normal range */
    if (ed - 573u < 900u || (fx::bits(du) << 1) == 0ull) ppv = fma(-0.125, f.mul(f.mul(du, rs), as), fx::halve(sp));
    else ppv = pvrs_slow(sp, du, rs, as);
    const fx::i64 bl = (fx::i64) fx::bits(p_L), br = (fx::i64) fx::bits(p_R), bp = (fx::i64) fx::bits(ppv);
    const fx::i64 lo = bl < br ? bl : br, up = bl < br ? br : bl;
    if (!fx::finite(ppv)) return classify_slow(c, rho_L, u_L, p_L, rho_R, u_R, p_R, a_L, a_R, ppv);
    if (bp < lo) return PREG_TRRS;
    return (bp <= up && up <= lo + (fx::i64) fx::HIDDEN) ? PREG_PVRS : PREG_TSRS;
}

/* guess_p_trrs and guess_p_tsrs (numerics.cuh); they also hand back their
 * factors (p^((g-1)/2g) and g_K of each side), which the adjoint's tape keeps. */
FXHD double face_trrs(const Fm &f, const GasConst<double> &c, double u_L, double p_L, double a_L, double u_R, double p_R,
                      double a_R, double &zL, double &zR)
{
    zL = pw(p_L, c.half_gm1_g);
    zR = pw(p_R, c.half_gm1_g);
    const double pg = dv(f.sub(f.add(a_L, a_R), f.mul(c.half_gm1, f.sub(u_R, u_L))), f.add(dv(a_L, zL), dv(a_R, zR)));
    return pw(pg, c.g_half_gm1);
}

FXHD double face_tsrs(const Fm &f, const GasConst<double> &c, double rho_L, double u_L, double p_L, double rho_R,
                      double u_R, double p_R, double ppv, double &gL, double &gR)
{
    gL = sq(dv(dv(2.0, f.mul(c.gp1, rho_L)), f.add(ppv, f.mul(p_L, c.gm1_gp1))));
    gR = sq(dv(dv(2.0, f.mul(c.gp1, rho_R)), f.add(ppv, f.mul(p_R, c.gm1_gp1))));
    return dv(f.sub(f.add(f.mul(gL, p_L), f.mul(gR, p_R)), f.sub(u_R, u_L)), f.add(gL, gR));
}

/* hllc_finish (numerics.cuh); `plain` from face_classify. */
FXHD int face_finish(const Fm &f, const GasConst<double> &c, bool plain, double rho_L, double u_L, double v_L, double p_L,
                     double a_L, double rho_R, double u_R, double v_R, double p_R, double a_R, double pg, double F[4],
                     double wave[3])
{
    const double ps = lt(pg, c.tol) ? c.tol : pg;
    if (!plain || !fx::moderate(ps))
        return finish_slow(c, rho_L, u_L, v_L, p_L, a_L, rho_R, u_R, v_R, p_R, a_R, pg, F, wave);
    double q_L = 1.0, q_R = 1.0, aq_L = a_L, aq_R = a_R;
    const fx::i64 bs = (fx::i64) fx::bits(ps);
    if (bs > (fx::i64) fx::bits(p_L)) {
        q_L = sq(f.add(f.one, f.mul(c.q_coef, f.sub(dv(ps, p_L), f.one))));
        aq_L = f.mul(a_L, q_L);
    }
    if (bs > (fx::i64) fx::bits(p_R)) {
        q_R = sq(f.add(f.one, f.mul(c.q_coef, f.sub(dv(ps, p_R), f.one))));
        aq_R = f.mul(a_R, q_R);
    }
    const double S_L = f.sub(u_L, aq_L), S_R = f.add(u_R, aq_R);
    const double d_L = f.sub(S_L, u_L), d_R = f.sub(S_R, u_R);
    const double m_L = f.mul(rho_L, u_L), m_R = f.mul(rho_R, u_R);
    const double rd_L = f.mul(rho_L, d_L), rd_R = f.mul(rho_R, d_R);
    const double S_s = dv(f.sub(f.add(f.sub(p_R, p_L), f.mul(m_L, d_L)), f.mul(m_R, d_R)), f.sub(rd_L, rd_R));
    if (!fx::finite(S_L) || !fx::finite(S_R) || !fx::finite(S_s))
        return finish_slow(c, rho_L, u_L, v_L, p_L, a_L, rho_R, u_R, v_R, p_R, a_R, pg, F, wave);
    wave[0] = q_L;
    wave[1] = q_R;
    wave[2] = S_s;
    const bool beyond_L = fx::not_below_zero(S_L);
    const bool left = beyond_L || fx::not_below_zero(S_s);
    const bool star = left ? !beyond_L : fx::not_below_zero(S_R);
    const double rho = left ? rho_L : rho_R, u = left ? u_L : u_R, v = left ? v_L : v_R, p = left ? p_L : p_R;
    const double m = left ? m_L : m_R, S = left ? S_L : S_R, rd = left ? rd_L : rd_R;
    const double E = f.mul(rho, fma(-f.mh, f.add(f.mul(u, u), f.mul(v, v)), dv(p, f.mul(rho, c.gm1))));
    F[0] = m;
    F[1] = f.add(f.mul(m, u), p);
    F[2] = f.mul(m, v);
    F[3] = f.mul(u, f.add(E, p));
    if (star) {
        const double rs = dv(rd, f.sub(S, S_s));
        const double es = f.mul(rs, f.add(dv(E, rho), f.mul(f.sub(S_s, u), f.add(S_s, dv(p, rd)))));
        F[0] = f.add(m, f.mul(S, f.sub(rs, rho)));
        F[1] = f.add(F[1], f.mul(S, f.sub(f.mul(rs, S_s), m)));
        F[2] = f.add(F[2], f.mul(S, f.sub(f.mul(rs, v), f.mul(rho, v))));
        F[3] = f.add(F[3], f.mul(S, f.sub(es, E)));
    }
    return DEV_OK;
}

/* ------------------------------------------------------------- conversion */

SLOW_PATH void to_primitive_slow(const GasConst<double> &c, double vol, double m, double mx, double my, double E, double w[4])
{
    cons_to_prim_2d(c, vol, m, mx, my, E, w);
}

/* cons_to_prim_2d (numerics.cuh). */
FXHD void to_primitive(const Fm &f, const GasConst<double> &c, double vol, double m, double mx, double my, double E,
                       double w[4])
{
    if (!fx::moderate(m)) {
        to_primitive_slow(c, vol, m, mx, my, E, w);
        return;
    }
    w[0] = dvi(m, vol);
    w[1] = dvi(mx, m);
    w[2] = dvi(my, m);
    const double ke = f.mul(fx::halve(m), f.add(f.mul(w[1], w[1]), f.mul(w[2], w[2])));
    w[3] = dvi(f.mul(c.gm1, f.sub(E, ke)), vol);
}

}  // namespace hydro

#endif
