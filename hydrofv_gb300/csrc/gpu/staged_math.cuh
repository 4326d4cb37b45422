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
 *    The constants are read from memory so that the compiler cannot turn the
 *    fma back into an add or a multiply; through the read-only path, which
 *    keeps them in L1 (volatile loads, which go to L2, took 70.8 us a step of
 *    316^2 where these take 65.8).
 *  - Scalings by powers of two go into an fma (x - 0.5 s as fma(-0.5, s, x):
 *    0.5 s is exact, so the one rounding is the sum's) or become an exponent
 *    step on the integer pipe.
 *  - Products that the formulas repeat (rho u, S - u, rho (S - u)) are formed
 *    once and selected with the side.
 *  - Comparisons of positive numbers compare the bit patterns as integers.
 *
 *  - Differences and sums of nearly equal numbers, and the limiters, become
 *    integer arithmetic.
 *
 * FP64 instructions per cell-update of the shear layer: 335 of 19 cycles from
 * the plain expressions, 285 of 16 as fused multiply-adds (2048^2: 3.07 -> 2.51
 * ms a step), 250 with the integer forms (2.11 -> 1.85 ms).
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
    f.one = __ldg(&d_fma_const[0]);
    f.mz = __ldg(&d_fma_const[1]);
    f.mh = __ldg(&d_fma_const[2]);
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

FXHD int leading_zeros(u64 n)
{
#if defined(__CUDA_ARCH__)
    return __clzll((long long) n);
#else
    return __builtin_clzll(n);
#endif
}

/* n 2^(e-1075) for 0 < n < 2^53 and a normal result: the double with the bits
 * of `sign`. */
FXHD double scaled(u64 n, unsigned e, u64 sign)
{
    const int lz = leading_zeros(n);
    return from_bits(((u64) (e + 10 - lz) << 52) + (n << (lz - 11)) + sign);
}

FXHD unsigned least(unsigned a, unsigned b) { return a < b ? a : b; }
FXHD unsigned most(unsigned a, unsigned b) { return a < b ? b : a; }

/* The 53 significant bits of a normal x, k < 10 places up. */
FXHD i64 fixed(double x, unsigned k)
{
    const u64 m = (bits(x) & (HIDDEN - 1)) | HIDDEN;
#if defined(__CUDA_ARCH__)
    const unsigned lo = (unsigned) m, h = (unsigned) (m >> 32);
    return (i64) (((u64) __funnelshift_l(lo, h, k) << 32) | (lo << k));
#else
    return (i64) (m << k);
#endif
}

/* Both of one sign and one binade, magnitudes between 2^-250 and 2^250: their
 * difference is that of their bit patterns in units of the last place. */
FXHD bool one_binade(double x, double y)
{
    const unsigned h = hi(x);
    return ((h ^ hi(y)) >> 20) == 0u && (h & 0x7fffffffu) - (773u << 20) < (500u << 20);
}

/* x - y and x + y of numbers of one binade, without the FP64 pipe. */
FXHD double near_diff(double x, double y)
{
    const i64 d = (i64) (bits(x) - bits(y));
    if (d == 0) return 0.0;
    return scaled((u64) (d < 0 ? -d : d), (hi(x) >> 20) & 0x7ffu, (bits(x) ^ (u64) d) & SIGN);
}

FXHD double near_sum(double x, double y)
{
    const u64 t = (bits(x) & (HIDDEN - 1)) + (bits(y) & (HIDDEN - 1));            /* (2^53 + t) / 2, to even */
    return from_bits((bits(x) & ~(HIDDEN - 1)) + HIDDEN + (t >> 1) + (t & (t >> 1) & 1));
}

/* 0 < |x| < 2^-962. */
FXHD bool tiny(double x)
{
    const u64 b = bits(x);
    const unsigned h = (unsigned) (b >> 32) & 0x7fffffffu;
    return h < (61u << 20) && (h | (unsigned) b) != 0u;
}

}  // namespace fx

/* a - b and a + b where the operands are mostly of one binade: about 20 integer
 * instructions, whose issue slots are free where an FP64 instruction takes the
 * FP64 pipe for 64 of them.  The shear layer of 2048^2 takes 1.98 ms a step
 * without them, 1.85 with the eight below.  Not worth it: sums of operands
 * whose exponents may differ (45 instructions, 1.95 ms). */
FXHD double diff(const Fm &f, double a, double b) { return fx::one_binade(a, b) ? fx::near_diff(a, b) : f.sub(a, b); }
FXHD double sum(const Fm &f, double a, double b) { return fx::one_binade(a, b) ? fx::near_sum(a, b) : f.add(a, b); }

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

/*
 * The limited slope of three neighbours and the limiter's branch (code, as
 * limit_slope_partials numbers them).  Where they share a sign and their
 * magnitudes are close (nearly all of a smooth flow) the two differences are
 * integers in units of the smallest one's last place.  Below 2^52 they, their
 * sum and the limited value (in half units) are exact as integers and as
 * doubles, so minmod and MC take no FP64 instruction.  recon of the 1024^2
 * shear layer, MC: 66 FP64 instructions a cell where there were 88, 160 -> 128
 * us.  Van Leer keeps the product, the 1e-10 and the quotient (1024^2, a whole
 * step: 516 us, 530 with the quotient called and a + b on the FP64 pipe).
 */
template <int LIM>
FXHD bool near_slope(const Fm &f, double wm, double w, double wp, double &s, int &code)
{
    const unsigned em = fx::hi(wm) >> 20, ec = fx::hi(w) >> 20, ep = fx::hi(wp) >> 20;      /* with the sign */
    const unsigned e = fx::least(fx::least(em, ec), ep), up = fx::most(fx::most(em, ec), ep);
    if (up - e > 9u || (e & 0x7ffu) - 773u >= 500u) return false;
    const fx::i64 c = fx::fixed(w, ec - e);
    fx::i64 x = c - fx::fixed(wm, em - e), y = fx::fixed(wp, ep - e) - c;
    s = 0.0;
    code = 0;
    if (x == 0 || y == 0 || (x ^ y) < 0) return true;
    const fx::u64 sign = (fx::bits(w) ^ (fx::u64) x) & fx::SIGN;
    if (x < 0) { x = -x; y = -y; }
    if ((unsigned) ((fx::u64) (x | y) >> 52) != 0u) return false;
    code = 1;
    if (LIM == LIM_VAN_LEER) {
        const unsigned q = e & 0x7ffu;
        const double a = fx::scaled((fx::u64) x, q, sign), b = fx::scaled((fx::u64) y, q, sign);
        s = dvi(f.mul(fx::twice(a), b), f.add(fx::scaled((fx::u64) (x + y), q, sign), 1e-10));
        return true;
    }
    const fx::i64 m = x < y ? x : y;
    if (LIM == LIM_MINMOD) {
        code = x < y ? 1 : 2;
        s = fx::scaled((fx::u64) m, e & 0x7ffu, sign);
        return true;
    }
    const fx::i64 two = m << 2, avg = x + y;                                           /* in half units */
    if (two < avg) code = y < x ? 3 : 2;
    s = fx::scaled((fx::u64) (avg < two ? avg : two), (e & 0x7ffu) - 1u, sign);
    return true;
}

template <int LIM>
FXHD double slope_of(const Fm &f, double wm, double w, double wp)
{
    double s;
    int code;
    if (near_slope<LIM>(f, wm, w, wp, s, code)) return s;
    /* gas at rest beside gas at rest */
    if ((fx::bits(w) == fx::bits(wm) || fx::bits(w) == fx::bits(wp)) && fx::finite(wm) && fx::finite(wp)) return 0.0;
    return slope<LIM>(f, f.sub(w, wm), f.sub(wp, w));
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

/* All four slopes are +0 and the predictor leaves the state as it is, to the
 * sign of a zero (x + 0.5 (+0) is x for every finite x but -0). */
FXHD bool flat(const double s[4], double rho, double n, double t, double p)
{
    return (fx::bits(s[0]) | fx::bits(s[1]) | fx::bits(s[2]) | fx::bits(s[3])) == 0ull && fx::moderate(rho) && fx::moderate(p) &&
           fx::finite(n) && fx::finite(t) && fx::bits(n) != fx::SIGN && fx::bits(t) != fx::SIGN;
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

/* One side of predict: the state at the cell's high face or at its low one. */
FXHD void predict_side(const Fm &f, bool high, double dtA, double dtA_rho, double rho, double n, double t, double p, double a,
                       const double d[4], double d_rho_vel, double o[4])
{
    const double cn = f.mul(dtA, n);
    const double u = f.add(f.one, high ? -cn : cn);
    const double dr = f.mul(dtA, rho);
    const double draa = f.mul(f.mul(f.mul(dr, a), a), d[1]);
    const double drv = f.mul(dr, d_rho_vel), drp = f.mul(dtA_rho, d[3]);
    const double h = high ? -f.mh : f.mh;
    o[0] = half_step(rho, add_zero(f.add(f.mul(u, d[0]), high ? -drv : drv)), h);
    o[1] = half_step(n, f.add(add_zero(f.mul(u, d[1])), high ? -drp : drp), h);
    o[2] = half_step(t, add_zero(f.mul(u, d[2])), h);
    o[3] = half_step(p, f.add(high ? zero_minus(draa) : add_zero(draa), f.mul(u, d[3])), h);
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
    const double as = sum(f, a_L, a_R), du = f.sub(u_R, u_L);
    /* 2 (a_L + a_R) / (gamma + 1) lies in [2^(d-1), 2^(d+1)] (quot_le_fast):
     * a negative u_R - u_L, or one below 2^(d-1), is not above it */
    const unsigned hd = fx::hi(du);
    const int d = (int) (fx::hi(as) >> 20) + 1 - (int) (fx::hi(c.gp1) >> 20);
    ppv = 0.0;
    if ((int) hd >= 0 && (int) (hd >> 20) - 1023 > d - 2 && vacuum_slow(c, as, du)) return PREG_VACUUM;
    const double sp = sum(f, p_L, p_R), rs = sum(f, rho_L, rho_R);
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

/*
 * A two-rarefaction face whose star pressure is surely not above min(p_L,
 * p_R): both q are then 1 and the flux does not depend on it, so the three
 * powers need not be formed.  With p' <= p the two pressures, a the sound
 * speed beside p, z = (g-1)/2g and x = p'/p, the guess
 *     p*^z = (a_L + a_R - (g-1)/2 du) / (a_L p_L^-z + a_R p_R^-z)
 * is at most p'^z if du (g-1)/2 >= a (1 - x^z), and 1 - x^z <= z (1/x - 1),
 * so g p' du >= a (p - p') is enough.  1e-9 (a_L + a_R) of du is kept as a
 * margin for the roundings of the guess, which grow with 1/z (no shortcut
 * above 1e5, or for gamma below 1).  c.tol, the guess's floor, must not be
 * above p' either.
 *
 * With the powers of the remaining faces only, the shear layer takes 2.11 ms a
 * step at 2048^2 (2.27 with all powers), 155 us at 512^2 (168) and 54 us at
 * 256^2 (60).
 */
FXHD bool both_rarefactions(const Fm &f, const GasConst<double> &c, double u_L, double p_L, double a_L, double u_R,
                            double p_R, double a_R, double &p_min)
{
    const fx::i64 bl = (fx::i64) fx::bits(p_L), br = (fx::i64) fx::bits(p_R);
    const bool l_above = br < bl;
    p_min = l_above ? p_R : p_L;
    if ((fx::i64) fx::bits(c.tol) > (l_above ? br : bl) || fx::bits(c.g_half_gm1) > fx::bits(1e5)) return false;
    const double p = l_above ? p_L : p_R, a = l_above ? a_L : a_R;
    const double du = fma(c.gamma, f.sub(u_R, u_L), f.mul(-1e-9, f.add(a_L, a_R)));
    const fx::i64 have = (fx::i64) fx::bits(f.mul(p_min, du)), need = (fx::i64) fx::bits(f.mul(a, f.sub(p, p_min)));
    return have >= need && fx::finite(du);
}

template <bool INL>
FXHD double dvx(double a, double b) { return INL ? dvi(a, b) : dv(a, b); }
template <bool INL>
FXHD double sqx(double x) { return INL ? sqi(x) : sq(x); }

template <bool INL = false>
FXHD double face_tsrs(const Fm &f, const GasConst<double> &c, double rho_L, double u_L, double p_L, double rho_R,
                      double u_R, double p_R, double ppv, double &gL, double &gR)
{
    gL = sqx<INL>(dvx<INL>(dvx<INL>(2.0, f.mul(c.gp1, rho_L)), f.add(ppv, f.mul(p_L, c.gm1_gp1))));
    gR = sqx<INL>(dvx<INL>(dvx<INL>(2.0, f.mul(c.gp1, rho_R)), f.add(ppv, f.mul(p_R, c.gm1_gp1))));
    return dvx<INL>(f.sub(f.add(f.mul(gL, p_L), f.mul(gR, p_R)), f.sub(u_R, u_L)), f.add(gL, gR));
}

/* hllc_finish (numerics.cuh); `plain` from face_classify.  INL puts the
 * quotients and roots in line, so that independent ones overlap: faster where
 * a warp is alone on its scheduler (the many-step kernel: 64^2 23.7 -> 22.4 us a step, 256^2
 * 52.7 -> 50.6, with the maxima on the integer pipe), slower where
 * the code no longer fits the instruction cache (2048^2: 2.31 ms a step
 * against 2.24). */
template <bool INL = false>
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
        q_L = sqx<INL>(f.add(f.one, f.mul(c.q_coef, diff(f, dvx<INL>(ps, p_L), 1.0))));
        aq_L = f.mul(a_L, q_L);
    }
    if (bs > (fx::i64) fx::bits(p_R)) {
        q_R = sqx<INL>(f.add(f.one, f.mul(c.q_coef, diff(f, dvx<INL>(ps, p_R), 1.0))));
        aq_R = f.mul(a_R, q_R);
    }
    const double S_L = f.sub(u_L, aq_L), S_R = f.add(u_R, aq_R);
    const double d_L = f.sub(S_L, u_L), d_R = f.sub(S_R, u_R);
    const double m_L = f.mul(rho_L, u_L), m_R = f.mul(rho_R, u_R);
    const double rd_L = f.mul(rho_L, d_L), rd_R = f.mul(rho_R, d_R);
    const double S_s = dvx<INL>(f.sub(f.add(diff(f, p_R, p_L), f.mul(m_L, d_L)), f.mul(m_R, d_R)), f.sub(rd_L, rd_R));
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
    const double E = f.mul(rho, fma(-f.mh, f.add(f.mul(u, u), f.mul(v, v)), dvx<INL>(p, f.mul(rho, c.gm1))));
    F[0] = m;
    F[1] = f.add(f.mul(m, u), p);
    F[2] = f.mul(m, v);
    F[3] = f.mul(u, f.add(E, p));
    if (star) {
        const double rs = dvx<INL>(rd, f.sub(S, S_s));
        const double es = f.mul(rs, f.add(dvx<INL>(E, rho), f.mul(f.sub(S_s, u), f.add(S_s, dvx<INL>(p, rd)))));
        F[0] = f.add(m, f.mul(S, diff(f, rs, rho)));
        F[1] = f.add(F[1], f.mul(S, f.sub(f.mul(rs, S_s), m)));
        F[2] = f.add(F[2], f.mul(S, diff(f, f.mul(rs, v), f.mul(rho, v))));
        F[3] = f.add(F[3], f.mul(S, diff(f, es, E)));
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
