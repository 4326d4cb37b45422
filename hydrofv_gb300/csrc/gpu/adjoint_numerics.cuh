/*
 * adjoint_numerics.cuh -- hand-written reverse mode (vector-Jacobian
 * products) of the pointwise pieces of one MUSCL-Hancock + HLLC step, and
 * the branch codes that identify which piece of a piecewise-smooth function
 * an evaluation took.
 *
 * Each *_vjp function recomputes the primal intermediates it needs with the
 * same expressions as numerics.cuh (so its branch decisions are the
 * forward pass's, bit for bit) and then applies the transposed chain rule.
 * The tie conventions at kinks are the ones Dual uses in dual.cuh, so the
 * reverse code here is the exact transpose of the tangent-linear model run
 * through numerics.cuh:
 *
 *   limiters          src/slope_limiter.c:49-91
 *   Hancock predictor src/integrator_muscl_hancock.c:682-755, :967-1041
 *   sound speed       src/utils.c:23-26
 *   HLLC 2D           src/riemann_solver_hllc.c:202-376, guesses
 *                     src/riemann_solver.c:154-224, vacuum
 *                     src/riemann_solver.c:230-733
 *   U <-> W           src/system.c:763-802, :884-905
 */
#ifndef HYDRO_GPU_ADJOINT_NUMERICS_CUH
#define HYDRO_GPU_ADJOINT_NUMERICS_CUH

#include "staged_math.cuh"

/* `#pragma unroll` for the device compiler only (the host compiler builds
 * these functions too, and does not know the pragma) */
#if defined(__CUDA_ARCH__)
#define HYDRO_UNROLL _Pragma("unroll")
#else
#define HYDRO_UNROLL
#endif

namespace hydro {

/* ------------------------------------------------------ contracted reals */

/*
 * A double whose sums with products contract into fused multiply-adds.  The
 * reverse sweep is bound by the FP64 pipe and its arithmetic is derivatives
 * only (nothing of it decides a branch of the forward pass), so
 * x y + z is one instruction and one rounding instead of two.  The
 * contraction is written here, not left to the compiler: every kernel (and
 * the host build) forms the same values, so the gradient does not depend on
 * the tape or on the checkpoints.
 */
struct Fd;
struct FdProd {
    double a, b;                              /* a b, not yet rounded */
};

/* Plain sums and products as register-only FMAs (staged_math.cuh); the
 * constants are read from memory once per thread. */
HD double fd_add(double x, double y)
{
#if defined(__CUDA_ARCH__)
    return fma(x, d_fma_const[0], y);
#else
    return x + y;
#endif
}

HD double fd_mul(double x, double y)
{
#if defined(__CUDA_ARCH__)
    return fma(x, y, d_fma_const[1]);
#else
    return x * y;
#endif
}

struct Fd {
    double v;
    Fd() = default;
    HD Fd(double x) : v(x) {}
    HD Fd(const FdProd &p) : v(fd_mul(p.a, p.b)) {}
    HD Fd &operator+=(const Fd &x) { v = fd_add(v, x.v); return *this; }
    HD Fd &operator-=(const Fd &x) { v = fd_add(-x.v, v); return *this; }
    HD Fd &operator+=(const FdProd &p) { v = fma(p.a, p.b, v); return *this; }
    HD Fd &operator-=(const FdProd &p) { v = fma(-p.a, p.b, v); return *this; }
};
HD FdProd operator*(const Fd &x, const Fd &y) { return FdProd{ x.v, y.v }; }
HD FdProd operator*(const FdProd &p, const Fd &y) { return FdProd{ fd_mul(p.a, p.b), y.v }; }
HD FdProd operator*(const Fd &x, const FdProd &p) { return FdProd{ x.v, fd_mul(p.a, p.b) }; }
HD FdProd operator*(const FdProd &p, const FdProd &q) { return FdProd{ fd_mul(p.a, p.b), fd_mul(q.a, q.b) }; }
HD Fd operator+(const Fd &x, const Fd &y) { return Fd(fd_add(x.v, y.v)); }
HD Fd operator-(const Fd &x, const Fd &y) { return Fd(fd_add(-y.v, x.v)); }
HD Fd operator+(const FdProd &p, const Fd &y) { return Fd(fma(p.a, p.b, y.v)); }
HD Fd operator+(const Fd &x, const FdProd &p) { return Fd(fma(p.a, p.b, x.v)); }
HD Fd operator-(const FdProd &p, const Fd &y) { return Fd(fma(p.a, p.b, -y.v)); }
HD Fd operator-(const Fd &x, const FdProd &p) { return Fd(fma(-p.a, p.b, x.v)); }
HD Fd operator+(const FdProd &p, const FdProd &q) { return Fd(fma(p.a, p.b, fd_mul(q.a, q.b))); }
HD Fd operator-(const FdProd &p, const FdProd &q) { return Fd(fma(p.a, p.b, -fd_mul(q.a, q.b))); }
HD Fd operator-(const Fd &x) { return Fd(-x.v); }
HD FdProd operator-(const FdProd &p) { return FdProd{ -p.a, p.b }; }

/* ---------------------------------------------------------------- limiter */

/* Slope d = L(a, b) with its partial derivatives and a branch code:
 * 0  a*b <= 0 (d = 0);
 * 1  minmod a / van Leer / MC centred 0.5(a+b);
 * 2  minmod b / MC 2|a| branch;  3  MC 2|b| branch. */
template <int LIM>
HD double limit_slope_partials(double a, double b, double &da, double &db, int &code)
{
#if defined(__CUDA_ARCH__)
    /* the branch decided on the bits, with the forward limiter's ranges and
     * exact scalings (slope, staged_math.cuh); other operands take the code
     * below */
    if (LIM != LIM_VAN_LEER) {
        const fx::u64 ua = fx::bits(a), ub = fx::bits(b);
        const fx::u64 aa = ua & ~fx::SIGN, ab = ub & ~fx::SIGN;
        const unsigned ha = (unsigned) (aa >> 32), hb = (unsigned) (ab >> 32);
        const unsigned lo = 2u << 20, span = 2042u << 20;
        const bool in = ha - lo < span && hb - lo < span && ha + hb >= (975u << 20);
        const bool zero = (aa == 0ull && hb < 0x7ff00000u) || (ab == 0ull && ha < 0x7ff00000u);
        if (zero || (in && ((ua ^ ub) >> 63))) { da = 0.0; db = 0.0; code = 0; return 0.0; }
        if (in) {
            const bool take_b = ab < aa;
            if (LIM == LIM_MINMOD) {
                if (aa < ab) { da = 1.0; db = 0.0; code = 1; return a; }
                da = 0.0; db = 1.0; code = 2; return b;
            }
            const fx::u64 two = (take_b ? ab : aa) + fx::HIDDEN;
            const fx::u64 avg = (fx::bits(fd_add(a, b)) & ~fx::SIGN) - fx::HIDDEN;
            if (two < avg) {
                da = take_b ? 0.0 : 2.0;
                db = take_b ? 2.0 : 0.0;
                code = take_b ? 3 : 2;
                return fx::from_bits(two | (ua & fx::SIGN));
            }
            da = 0.5; db = 0.5; code = 1;
            return fx::from_bits(avg | (ua & fx::SIGN));
        }
    }
#endif
    const double d = limit_slope<LIM>(a, b);
    if (a * b <= 0.0) { da = 0.0; db = 0.0; code = 0; return d; }
    if (LIM == LIM_MINMOD) {
        if (fabs(a) < fabs(b)) { da = 1.0; db = 0.0; code = 1; }
        else { da = 0.0; db = 1.0; code = 2; }
        return d;
    }
    if (LIM == LIM_VAN_LEER) {
        const double s = a + b + 1e-10;
        da = dv(2.0 * b - d, s);
        db = dv(2.0 * a - d, s);
        code = 1;
        return d;
    }
    /* MC: fmin(avg, 2 fmin(|a|, |b|)) (signs mirrored for a < 0); ties take
     * the first argument of each fmin. */
    const double fa = fabs(a), fb = fabs(b);
    const bool take_b = fb < fa;
    const double two = 2.0 * (take_b ? fb : fa);
    const double avg = (a > 0.0) ? 0.5 * (a + b) : -0.5 * (a + b);
    if (two < avg) {
        if (take_b) { da = 0.0; db = 2.0; code = 3; }
        else { da = 2.0; db = 0.0; code = 2; }
    } else {
        da = 0.5; db = 0.5; code = 1;
    }
    return d;
}

/* The same for a = w0 - wm, b = wp - w0; minmod and MC of close neighbours on
 * the integer pipes (near_slope). */
template <int LIM>
HD double slope_partials(double wm, double w0, double wp, double &da, double &db, int &code)
{
#if defined(__CUDA_ARCH__)
    double s;
    if (LIM != LIM_VAN_LEER && near_slope<LIM>(Fm(), wm, w0, wp, s, code)) {
        const double one = LIM == LIM_MINMOD ? 1.0 : code == 1 ? 0.5 : 2.0;
        da = (LIM == LIM_MINMOD ? code == 1 : code == 1 || code == 2) ? one : 0.0;
        db = (LIM == LIM_MINMOD ? code == 2 : code == 1 || code == 3) ? one : 0.0;
        return s;
    }
#endif
    return limit_slope_partials<LIM>(fd_add(-wm, w0), fd_add(-w0, wp), da, db, code);
}

/* ------------------------------------------------------------ sound speed */

/* a = sqrt(gamma p / rho): rho_b += -a/(2 rho) a_b, p_b += a/(2 p) a_b. */
HD void sound_speed_vjp(double rho, double p, double a, double ab, double &rhob, double &pb)
{
    if (ab == 0.0) return;
    rhob -= ab * dv(0.5 * a, rho);
    pb += ab * dv(0.5 * a, p);
}

/* ------------------------------------------------------------- predictor */

/*
 * Reverse of hancock_2d.  Inputs are those of the forward call (with
 * dtA_rho = dtA / rho); lob / hib are the adjoints of the extrapolated
 * states.  Writes rhob, nb, tb, pb, ab, the slope adjoints db[4] and
 * d_rho_velb (the slope that feeds the density row).
 */
HD void hancock_2d_vjp(double dtA_, double dtA_rho_, double rho_, double inv_rho_, double n_, double a_,
                       const double d_[4], double d_rho_vel_, const double lob_[4],
                       const double hib_[4], Fd &rhob, Fd &nb, Fd &tb, Fd &pb,
                       Fd &ab, Fd db[4], Fd &d_rho_velb)
{
    const Fd dtA = dtA_, dtA_rho = dtA_rho_, rho = rho_, inv_rho = inv_rho_, n = n_, a = a_, d_rho_vel = d_rho_vel_;
    Fd d[4], lob[4], hib[4], s[4];
HYDRO_UNROLL
    for (int q = 0; q < 4; q++) {
        d[q] = d_[q];
        lob[q] = lob_[q];
        hib[q] = hib_[q];
        s[q] = lob[q] + hib[q];
    }
    const Fd hn = Fd(0.5) * (dtA * n);
    const Fd up = Fd(-0.5) - hn, um = Fd(0.5) - hn;        /* -(1 + dtA n) / 2, (1 - dtA n) / 2 */
    const Fd dr = dtA * rho;
    tb = s[2];
    pb = s[3];
    /* nb = s1 + dtA (up_bar - um_bar), up_bar = -lob . d / 2, um_bar = hib . d / 2 */
    nb = s[1] + (dtA * Fd(-0.5)) * (s[0] * d[0] + (s[1] * d[1] + (s[2] * d[2] + s[3] * d[3])));
    const Fd h0 = Fd(-0.5) * s[0], h3 = Fd(-0.5) * s[3];   /* h3: adjoint of dr a a d[1] */
    d_rho_velb = dr * h0;
    const Fd aa = a * a, h3d = h3 * d[1];
    const Fd drb = h0 * d_rho_vel + h3d * aa;
    ab = (Fd(2.0) * h3d) * (dr * a);
    const Fd h1 = Fd(-0.5) * s[1];
    const Fd dtA_rhob = h1 * d[3];
    rhob = s[0] - dtA_rhob * (dtA_rho * inv_rho);          /* d(dtA/rho)/drho */
    rhob += drb * dtA;
HYDRO_UNROLL
    for (int q = 0; q < 4; q++) db[q] = up * lob[q] + um * hib[q];
    db[1] += h3 * (dr * aa);
    db[3] += h1 * dtA_rho;
}

/* ------------------------------------------------------------------ HLLC */

/* Primal intermediates of one HLLC face (same expressions as
 * hllc_classify / guess_p_* / hllc_finish). */
struct HllcFwd {
    double aL, aR, ppv, pg, ps, qL, qR, SL, SR, Ss;
    int reg;       /* PREG_* */
    int region;    /* 0 left, 1 left star, 2 right star, 3 right; -1 vacuum */
};

HD int hllc_fwd(const GasConst<double> &c, double rl, double ul, double pl, double rr, double ur,
                double pr, HllcFwd &s)
{
    s.reg = hllc_classify(c, rl, ul, pl, rr, ur, pr, s.aL, s.aR, s.ppv);
    s.region = -1;
    s.pg = s.ps = s.qL = s.qR = s.SL = s.SR = s.Ss = 0.0;
    if (s.reg == PREG_VACUUM) return DEV_OK;
    s.pg = s.ppv;
    if (s.reg == PREG_TRRS) s.pg = guess_p_trrs(c, ul, pl, s.aL, ur, pr, s.aR);
    else if (s.reg == PREG_TSRS) s.pg = guess_p_tsrs(c, rl, ul, pl, rr, ur, pr, s.ppv);
    s.ps = lt(s.pg, c.tol) ? c.tol : s.pg;
    s.qL = hllc_q(c, pl, s.ps);
    s.qR = hllc_q(c, pr, s.ps);
    s.SL = ul - s.aL * s.qL;
    s.SR = ur + s.aR * s.qR;
    s.Ss = dv(pr - pl + rl * ul * (s.SL - ul) - rr * ur * (s.SR - ur),
              rl * (s.SL - ul) - rr * (s.SR - ur));
    if (le(0.0, s.SL)) s.region = 0;
    else if (le(s.SL, 0.0) && le(0.0, s.Ss)) s.region = 1;
    else if (le(s.Ss, 0.0) && le(0.0, s.SR)) s.region = 2;
    else if (le(s.SR, 0.0)) s.region = 3;
    else return DEV_ERR_HLLC_WAVE_SPEED;
    return DEV_OK;
}

/* The intermediates of a non-vacuum face from the tape: sound speeds,
 * unfloored guess, regime and the finish's q_L, q_R and S* as the forward
 * pass computed them. */
HD int hllc_fwd_from_tape(const GasConst<double> &c, double rl, double ul, double pl, double rr, double ur,
                          double pr, double aL, double aR, double pg, int reg, double qL, double qR, double Ss,
                          HllcFwd &s)
{
    s.aL = aL;
    s.aR = aR;
    s.reg = reg;
    s.region = -1;
    s.ppv = reg == PREG_TSRS ? 0.5 * (pl + pr) - 0.125 * (ur - ul) * (rl + rr) * (aL + aR) : 0.0;   /* used there alone */
    s.pg = pg;
    s.ps = s.qL = s.qR = s.SL = s.SR = s.Ss = 0.0;
    if (reg == PREG_VACUUM) return DEV_OK;
    s.ps = lt(s.pg, c.tol) ? c.tol : s.pg;
    s.qL = qL;
    s.qR = qR;
    s.SL = fd_add(ul, -fd_mul(s.aL, s.qL));
    s.SR = fd_add(ur, fd_mul(s.aR, s.qR));
    s.Ss = Ss;
    if (le(0.0, s.SL)) s.region = 0;
    else if (le(s.SL, 0.0) && le(0.0, s.Ss)) s.region = 1;
    else if (le(s.Ss, 0.0) && le(0.0, s.SR)) s.region = 2;
    else if (le(s.SR, 0.0)) s.region = 3;
    else return DEV_ERR_HLLC_WAVE_SPEED;
    return DEV_OK;
}

/* Which sampler branch the vacuum flux takes (S = 0):
 * 0 zero state, 1 right-vacuum sampler on the left state, 2 left-vacuum
 * sampler on the right state; *sub: 0 data state, 1 fan, 2 vacuum. */
HD int vacuum_case(const GasConst<double> &c, double rl, double ul, double al, double rr,
                   double ur, double ar, int &sub)
{
    int which;
    if (rl <= 0.0 && rr <= 0.0) { sub = 0; return 0; }
    if (rl <= 0.0) which = 1;
    else if (rr <= 0.0) which = 2;
    else if (0.0 <= 2.0 * al / c.gm1) which = 1;
    else if (2.0 * ar / c.gm1 <= 0.0) which = 2;
    else { sub = 0; return 0; }
    if (which == 1) {
        if (0.0 <= ul - al) sub = 0;
        else sub = (0.0 < ul + 2.0 * al / c.gm1) ? 1 : 2;
    } else {
        if (0.0 >= ur + ar) sub = 0;
        else sub = (0.0 > ur - 2.0 * ar / c.gm1) ? 1 : 2;
    }
    return which;
}

/* Branch code of one face: regime, guess floor, shock/rarefaction side of
 * each wave speed, region; for vacuum faces the sampler branch. */
HD int hllc_code(const GasConst<double> &c, const HllcFwd &s, double rl, double ul, double pl,
                 double rr, double ur, double pr)
{
    if (s.reg == PREG_VACUUM) {
        int sub;
        const int which = vacuum_case(c, rl, ul, s.aL, rr, ur, s.aR, sub);
        return 0x100 | (which << 2) | sub;
    }
    return s.reg | ((s.pg < c.tol) << 2) | ((s.ps > pl) << 3) | ((s.ps > pr) << 4)
         | ((s.region & 3) << 5);
}

/* Reverse of a vacuum-sampler fan: o = (rho t, (+-a + h u)*2/(g+1), v, p t^gamma),
 * t = (2/(g+1) +- (u/((g+1) a)) (g-1))^(2/(g-1)) at S = 0. */
HD void vacuum_fan_vjp(const GasConst<double> &c, bool right, double rho, double u, double p,
                       double a, const double ob[4], double &rhob, double &ub, double &vb,
                       double &pb, double &ab)
{
    const double k = (u - 0.0) * c.gm1 / (c.gp1 * a);
    const double t0 = right ? (c.two_gp1 + k) : (c.two_gp1 - k);
    const double t = pw(t0, c.two_gm1);
    const double tg = pw(t, c.gamma);
    rhob += ob[0] * t;
    const double tb = ob[0] * rho + ob[3] * p * c.gamma * tg / t;
    pb += ob[3] * tg;
    ab += (right ? 1.0 : -1.0) * ob[1] * 2.0 / c.gp1;
    ub += ob[1] * c.half_gm1 * 2.0 / c.gp1;
    vb += ob[2];
    const double t0b = tb * c.two_gm1 * t / t0;
    const double kb = right ? t0b : -t0b;
    ub += kb * c.gm1 / (c.gp1 * a);
    ab += -kb * k / a;
}

/* Reverse of the vacuum / vacuum-generation flux (kept out of line: rare,
 * and its pow-heavy samplers would otherwise raise the register count of
 * every face). */
#ifdef __CUDACC__
static __host__ __device__ __noinline__
#else
static
#endif
void hllc_vacuum_vjp(const GasConst<double> &c, const double L[4], const double Rs[4], double aL, double aR,
                     const double Fb[4], double Lb[4], double Rb[4])
{
    const double rl = L[0], ul = L[1], vl = L[2], pl = L[3];
    const double rr = Rs[0], ur = Rs[1], vr = Rs[2], pr = Rs[3];
    double rLb = 0, uLb = 0, vLb = 0, pLb = 0, rRb = 0, uRb = 0, vRb = 0, pRb = 0, aLb = 0, aRb = 0;
    int sub;
    const int which = vacuum_case(c, rl, ul, aL, rr, ur, aR, sub);
    double o[4];
    solve_vacuum(c, rl, ul, vl, pl, aL, rr, ur, vr, pr, aR, 0.0, o);
    const double E = o[0] * (0.5 * (o[1] * o[1] + o[2] * o[2]) + o[3] / (o[0] * c.gm1));
    const double Eb = Fb[3] * o[1];
    double ob[4];
    ob[0] = Fb[0] * o[1] + Fb[1] * o[1] * o[1] + Fb[2] * o[1] * o[2] + Eb * 0.5 * (o[1] * o[1] + o[2] * o[2]);
    ob[1] = Fb[0] * o[0] + Fb[1] * 2.0 * o[0] * o[1] + Fb[2] * o[0] * o[2] + Fb[3] * (E + o[3])
          + Eb * o[0] * o[1];
    ob[2] = Fb[2] * o[0] * o[1] + Eb * o[0] * o[2];
    ob[3] = Fb[1] + Fb[3] * o[1] + Eb / c.gm1;
    if (which == 1) {
        if (sub == 0) { rLb += ob[0]; uLb += ob[1]; vLb += ob[2]; pLb += ob[3]; }
        else if (sub == 1) vacuum_fan_vjp(c, true, rl, ul, pl, aL, ob, rLb, uLb, vLb, pLb, aLb);
    } else if (which == 2) {
        if (sub == 0) { rRb += ob[0]; uRb += ob[1]; vRb += ob[2]; pRb += ob[3]; }
        else if (sub == 1) vacuum_fan_vjp(c, false, rr, ur, pr, aR, ob, rRb, uRb, vRb, pRb, aRb);
    }
    if (rl > 0.0) sound_speed_vjp(rl, pl, aL, aLb, rLb, pLb);
    if (rr > 0.0) sound_speed_vjp(rr, pr, aR, aRb, rRb, pRb);
    Lb[0] = rLb; Lb[1] = uLb; Lb[2] = vLb; Lb[3] = pLb;
    Rb[0] = rRb; Rb[1] = uRb; Rb[2] = vRb; Rb[3] = pRb;
}

/*
 * Reverse of hllc_flux_2d given the face's forward intermediates s.  L, Rs
 * = (rho, u_normal, u_tangential, p) of the left / right face states, Fb =
 * adjoint of the flux (mass, normal momentum, tangential momentum, energy).
 * With have_z the guess factors (z0, z1) are taken as given (from the tape)
 * instead of recomputed.  Writes Lb, Rb.
 */
HD void hllc_vjp_core(const GasConst<double> &c, const double L[4], const double Rs[4], const HllcFwd &s,
                      bool have_z, double z0, double z1, const double Fb_[4], double Lb[4], double Rb[4])
{
    if (s.reg == PREG_VACUUM) {
        hllc_vacuum_vjp(c, L, Rs, s.aL, s.aR, Fb_, Lb, Rb);
        return;
    }
    /* Only the forward intermediates in s decide branches; the reverse below
     * is derivatives only, so a quotient that appears several times is
     * formed once as a reciprocal (a derivative, not a bit-parity value). */
    const Fd rl = L[0], ul = L[1], pl = L[3], rr = Rs[0], ur = Rs[1], pr = Rs[3];
    const Fd F0 = Fb_[0], F1 = Fb_[1], F2 = Fb_[2], F3 = Fb_[3];
    const Fd inv_rl = rv(L[0]), inv_rr = rv(Rs[0]), inv_pl = rv(L[3]), inv_pr = rv(Rs[3]);
    const Fd inv_gm1 = c.inv_gm1;
    Fd rLb = 0.0, uLb = 0.0, pLb = 0.0, rRb = 0.0, uRb = 0.0, pRb = 0.0;
    /* ---- region flux of the selected side K ---- */
    const bool left = s.region <= 1;
    const Fd rho = left ? rl : rr, u = left ? ul : ur, v = left ? L[2] : Rs[2], p = left ? pl : pr;
    const Fd inv_rho = left ? inv_rl : inv_rr;
    const Fd K2 = Fd(0.5) * (u * u + v * v);
    const Fd E = rho * K2 + p * inv_gm1;
    const Fd fm = rho * u;
    const Fd fmb = F0 + (F1 * u + F2 * v);
    Fd ub = F1 * fm + F3 * (E + p), vb = F2 * fm, pb = F3 * u + F1, Eb = F3 * u;
    Fd rhob = fmb * u;
    ub += fmb * rho;
    Fd SLb = 0.0, SRb = 0.0, Ssb = 0.0;
    if (s.region == 1 || s.region == 2) {
        const Fd S = left ? s.SL : s.SR, Ss = s.Ss;
        const Fd Smu = S - u, D = rho * Smu;
        const Fd inv_SmS = rv((S - Ss).v), inv_D = rv(D.v);
        const Fd rs = D * inv_SmS;
        const Fd pD = p * inv_D;
        const Fd Z = Ss + pD, dS = Ss - u;
        const Fd Er = E * inv_rho;
        const Fd Y = dS * Z + Er;
        const Fd drs = rs - rho;
        /* F += S (rs - rho, rs Ss - rho u, (rs - rho) v, es - E), es = rs Y */
        Fd Sb = (F0 + F2 * v) * drs + (F1 * (rs * Ss - fm) + F3 * (rs * Y - E));
        const Fd SF1 = S * F1, SF3 = S * F3, SF02 = S * (F0 + F2 * v);
        Ssb += SF1 * rs;
        const Fd rsb = SF02 + (SF1 * Ss + SF3 * Y);
        rhob -= SF02 + SF1 * u;
        ub -= SF1 * rho;
        vb += (S * F2) * drs;
        const Fd Yb = SF3 * rs;
        Eb += Yb * inv_rho - SF3;
        rhob -= Yb * (Er * inv_rho);
        const Fd YZ = Yb * Z, Zb = Yb * dS;
        Ssb += YZ + Zb;
        ub -= YZ;
        const Fd ZD = Zb * inv_D;
        pb += ZD;
        /* rs = N / M, N = D = rho (S - u), M = S - Ss */
        const Fd rM = rsb * inv_SmS;
        const Fd Nb = rM - ZD * pD;
        const Fd Mb = -(rM * rs);
        rhob += Nb * Smu;
        const Fd Nr = Nb * rho;
        ub -= Nr;
        Sb += Nr + Mb;
        Ssb -= Mb;
        if (left) SLb = Sb;
        else SRb = Sb;
    }
    rhob += Eb * K2;
    const Fd Er_ = Eb * rho;
    ub += Er_ * u;
    vb += Er_ * v;
    pb += Eb * inv_gm1;
    if (left) { rLb = rhob; uLb = ub; pLb = pb; }
    else { rRb = rhob; uRb = ub; pRb = pb; }

    /* ---- S* ---- */
    if (!eq_zero(Ssb.v)) {
        const Fd dL = Fd(s.SL) - ul, dR = Fd(s.SR) - ur;
        const Fd Dd = rl * dL - rr * dR;
        const Fd Nnb = dv(Ssb.v, Dd.v);
        const Fd Ddb = -(Nnb * s.Ss);
        pRb += Nnb;
        pLb -= Nnb;
        const Fd kL = Nnb * ul + Ddb, kR = Nnb * ur + Ddb;
        rLb += kL * dL;
        uLb += rl * (Nnb * (dL - ul) - Ddb);
        SLb += kL * rl;
        rRb -= kR * dR;
        uRb -= rr * (Nnb * (dR - ur) - Ddb);
        SRb -= kR * rr;
    }

    /* ---- wave speeds ---- */
    const Fd aL = s.aL, aR = s.aR, ps = s.ps;
    uLb += SLb;
    Fd aLb = -(SLb * s.qL);
    uRb += SRb;
    Fd aRb = SRb * s.qR;
    Fd psb = 0.0;
    const double hq = 0.5 * c.q_coef;
    if (lt(L[3], s.ps)) {
        const Fd qb = (SLb * aL) * Fd(-hq);
        const Fd t = Fd(dv(qb.v, s.qL)) * inv_pl;
        psb += t;
        pLb -= t * (ps * inv_pl);
    }
    if (lt(Rs[3], s.ps)) {
        const Fd qb = (SRb * aR) * Fd(hq);
        const Fd t = Fd(dv(qb.v, s.qR)) * inv_pr;
        psb += t;
        pRb -= t * (ps * inv_pr);
    }
    const Fd pgb = lt(s.pg, c.tol) ? Fd(0.0) : psb;

    /* ---- star-pressure guess (both q are 1 up to the smaller pressure) ---- */
    Fd ppvb = 0.0;
    if (!lt(L[3], s.ps) && !lt(Rs[3], s.ps)) {
        ppvb = 0.0;
    } else if (s.reg == PREG_PVRS) {
        ppvb = pgb;
    } else if (s.reg == PREG_TRRS) {
        const Fd izL = rv(have_z ? z0 : pw(L[3], c.half_gm1_g)), izR = rv(have_z ? z1 : pw(Rs[3], c.half_gm1_g));
        const Fd hg = c.half_gm1;
        const Fd num = (aL + aR) - hg * (ur - ul);
        const Fd wL = aL * izL, wR = aR * izR;
        const Fd den = wL + wR;
        /* pg = (num / den)^(1/hg): d pg = (pg / hg) (d num / num - d den / den) */
        const Fd k = pgb * (Fd(c.g_half_gm1) * s.pg);
        const Fd numb = dv(k.v, num.v), denb = dv(-k.v, den.v);
        aLb += denb * izL + numb;
        aRb += denb * izR + numb;
        uRb -= numb * hg;
        uLb += numb * hg;
        /* den = aL zL^-1 + aR zR^-1, zK = pK^hg: d den / d pK = -aK hg zK^-1 / pK */
        const Fd dh = denb * c.half_gm1_g;
        pLb -= dh * (wL * inv_pl);
        pRb -= dh * (wR * inv_pr);
    } else {
        /* not contracted: g_K is the forward pass's, as the tape keeps it */
        const double BL = s.ppv + L[3] * c.gm1_gp1, BR = s.ppv + Rs[3] * c.gm1_gp1;
        const Fd gL = have_z ? z0 : sq(dv(dv(2.0, c.gp1 * L[0]), BL));
        const Fd gR = have_z ? z1 : sq(dv(dv(2.0, c.gp1 * Rs[0]), BR));
        const Fd Nnb = dv(pgb.v, (gL + gR).v);
        const Fd Ddb = -(Nnb * s.pg);
        const Fd gLb = Nnb * pl + Ddb, gRb = Nnb * pr + Ddb;
        pLb += Nnb * gL;
        pRb += Nnb * gR;
        uRb -= Nnb;
        uLb += Nnb;
        const Fd hL = (Fd(0.5) * gLb) * gL, hR = (Fd(0.5) * gRb) * gR;
        rLb -= hL * inv_rl;
        rRb -= hR * inv_rr;
        const Fd BLb = dv(-hL.v, BL), BRb = dv(-hR.v, BR);
        ppvb = BLb + BRb;
        pLb += BLb * c.gm1_gp1;
        pRb += BRb * c.gm1_gp1;
    }
    if (!eq_zero(ppvb.v)) {
        pLb += Fd(0.5) * ppvb;
        pRb += Fd(0.5) * ppvb;
        const Fd du = ur - ul, sr = rl + rr, sa = aL + aR;
        const Fd w = Fd(-0.125) * ppvb;
        const Fd wd = w * du, dub = (w * sr) * sa;
        const Fd srb = wd * sa, sab = wd * sr;
        uRb += dub;
        uLb -= dub;
        rLb += srb;
        rRb += srb;
        aLb += sab;
        aRb += sab;
    }
    /* a = sqrt(gamma p / rho): da = a/2 (dp/p - drho/rho) */
    const Fd hL = (Fd(0.5) * aLb) * aL, hR = (Fd(0.5) * aRb) * aR;
    rLb -= hL * inv_rl;
    pLb += hL * inv_pl;
    rRb -= hR * inv_rr;
    pRb += hR * inv_pr;
    Lb[0] = rLb.v; Lb[1] = uLb.v; Lb[2] = left ? vb.v : 0.0; Lb[3] = pLb.v;
    Rb[0] = rRb.v; Rb[1] = uRb.v; Rb[2] = left ? 0.0 : vb.v; Rb[3] = pRb.v;
}

/* Reverse of hllc_flux_2d from the face states alone (forward intermediates
 * recomputed).  Returns DEV_OK or DEV_ERR_HLLC_WAVE_SPEED; *code (may be
 * NULL) receives the face's branch code. */
HD int hllc_vjp(const GasConst<double> &c, const double L[4], const double Rs[4], const double Fb[4],
                double Lb[4], double Rb[4], int *code)
{
    HllcFwd s;
    const int rc = hllc_fwd(c, L[0], L[1], L[3], Rs[0], Rs[1], Rs[3], s);
    if (code) *code = hllc_code(c, s, L[0], L[1], L[3], Rs[0], Rs[1], Rs[3]);
    if (rc != DEV_OK) {
        for (int q = 0; q < 4; q++) { Lb[q] = 0.0; Rb[q] = 0.0; }
        return rc;
    }
    hllc_vjp_core(c, L, Rs, s, false, 0.0, 0.0, Fb, Lb, Rb);
    return DEV_OK;
}

/* ------------------------------------------------------- cell recon */

/*
 * MUSCL-Hancock reconstruction of one cell along one direction, as the step
 * kernel does it: wm, w0, wp = (rho, vx, vy, p) of the cells below, at and
 * above along the sweep, a0 = sound speed of w0.  dir 0 (x): states in
 * (rho, vx, vy, p) order; dir 1 (y): (rho, vy, vx, p), and the density row
 * takes the x-velocity slope (src/integrator_muscl_hancock.c:988-993).
 * lo / hi = states at the cell's low / high face.
 */
template <int LIM, class R>
HD void recon_cell(int dir, R dtA, const R wm[4], const R w0[4], const R wp[4], R a0, R lo[4], R hi[4])
{
    R d[4];
    if (dir == 0) {
HYDRO_UNROLL
        for (int q = 0; q < 4; q++) d[q] = limit_slope<LIM>(w0[q] - wm[q], wp[q] - w0[q]);
        hancock_2d(dtA, dv(dtA, w0[0]), w0[0], w0[1], w0[2], w0[3], a0, d, d[1], lo, hi);
    } else {
        d[0] = limit_slope<LIM>(w0[0] - wm[0], wp[0] - w0[0]);
        const R dvx = limit_slope<LIM>(w0[1] - wm[1], wp[1] - w0[1]);
        d[1] = limit_slope<LIM>(w0[2] - wm[2], wp[2] - w0[2]);
        d[2] = dvx;
        d[3] = limit_slope<LIM>(w0[3] - wm[3], wp[3] - w0[3]);
        hancock_2d(dtA, dv(dtA, w0[0]), w0[0], w0[2], w0[1], w0[3], a0, d, dvx, lo, hi);
    }
}

/* Branch code of recon_cell: 2 bits per limiter call. */
template <int LIM>
HD int recon_code(const double wm[4], const double w0[4], const double wp[4])
{
    int code = 0;
HYDRO_UNROLL
    for (int q = 0; q < 4; q++) {
        double da, db;
        int c;
        limit_slope_partials<LIM>(w0[q] - wm[q], wp[q] - w0[q], da, db, c);
        code |= c << (2 * q);
    }
    return code;
}

/*
 * Reverse of recon_cell (a0 = sound speed of w0, folded back into w0;
 * inv_rho, inv_p = 1/rho, 1/p of w0).
 * Given lob / hib (sweep order), writes in storage order (rho, vx, vy, p):
 *   own  adjoint reaching w0 itself, including its share of the slopes;
 *   A    adjoint of the backward differences w0 - wm (wm receives -A);
 *   B    adjoint of the forward differences wp - w0 (wp receives +B).
 */
template <int LIM>
HD void recon_cell_vjp(int dir, double dtA, const double wm[4], const double w0[4], const double wp[4],
                       double a0, double inv_rho, double inv_p, const double lob[4], const double hib[4],
                       double own[4], double A[4], double B[4])
{
    double pa[4], pb[4], d[4];
    int code;
HYDRO_UNROLL
    for (int q = 0; q < 4; q++) d[q] = slope_partials<LIM>(wm[q], w0[q], wp[q], pa[q], pb[q], code);
    const int in_ = (dir == 0) ? 1 : 2;    /* storage index of the normal velocity */
    const int it_ = (dir == 0) ? 2 : 1;    /* storage index of the tangential velocity */
    double ds[4];                          /* slopes in sweep order */
    ds[0] = d[0];
    ds[1] = d[in_];
    ds[2] = d[it_];
    ds[3] = d[3];
    Fd rhob, nb, tb, pbb, ab, dvxb, dsb[4];
    hancock_2d_vjp(dtA, dtA * inv_rho, w0[0], inv_rho, w0[in_], a0, ds, d[1], lob, hib, rhob, nb, tb, pbb,
                   ab, dsb, dvxb);
    Fd db[4], ow[4];                       /* slope adjoints, storage order */
    db[0] = dsb[0];
    db[in_] = dsb[1];
    db[it_] = dsb[2];
    db[3] = dsb[3];
    db[1] += dvxb;
    /* a = sqrt(gamma p / rho): da = a/2 (dp/p - drho/rho) */
    const Fd h = (Fd(0.5) * ab) * Fd(a0);
    ow[0] = rhob - h * Fd(inv_rho);
    ow[in_] = nb;
    ow[it_] = tb;
    ow[3] = pbb + h * Fd(inv_p);
HYDRO_UNROLL
    for (int q = 0; q < 4; q++) {
        if (LIM == LIM_VAN_LEER) {
            const Fd x = db[q] * Fd(pa[q]), y = db[q] * Fd(pb[q]);
            A[q] = x.v;
            B[q] = y.v;
            own[q] = (ow[q] + db[q] * Fd(pa[q] - pb[q])).v;
        } else {
            /* pa and pb are equal, or one of them is zero */
            const bool a = fx::bits(pa[q]) != 0ull, b = fx::bits(pb[q]) != 0ull;
            const Fd t = db[q] * Fd(a ? pa[q] : pb[q]);
            A[q] = a ? t.v : 0.0;
            B[q] = b ? t.v : 0.0;
            own[q] = (ow[q] + t * Fd(a == b ? 0.0 : a ? 1.0 : -1.0)).v;
        }
    }
}

/* ------------------------------------------------ forced-branch forward */

/*
 * The forward pieces with every branch decision given (a code recorded from
 * another evaluation) instead of taken: the map whose derivative the
 * adjoint computes, as a function that stays on one smooth piece.  With the
 * evaluation's own codes the values are bit for bit those of numerics.cuh.
 */
template <int LIM>
HD double limit_slope_forced(double a, double b, int code)
{
    if (code == 0) return 0.0;
    if (LIM == LIM_MINMOD) return (code == 1) ? a : b;
    if (LIM == LIM_VAN_LEER) return dv(2.0 * a * b, a + b + 1e-10);
    if (code == 1) return (a > 0.0) ? 0.5 * (a + b) : -(-0.5 * (a + b));
    return 2.0 * ((code == 2) ? a : b);
}

template <int LIM>
HD void recon_cell_forced(int dir, double dtA, const double wm[4], const double w0[4], const double wp[4],
                          double a0, int code, double lo[4], double hi[4])
{
    double d[4];
HYDRO_UNROLL
    for (int q = 0; q < 4; q++) d[q] = limit_slope_forced<LIM>(w0[q] - wm[q], wp[q] - w0[q], (code >> (2 * q)) & 3);
    if (dir == 0) {
        hancock_2d(dtA, dv(dtA, w0[0]), w0[0], w0[1], w0[2], w0[3], a0, d, d[1], lo, hi);
    } else {
        const double ds[4] = { d[0], d[2], d[1], d[3] };
        hancock_2d(dtA, dv(dtA, w0[0]), w0[0], w0[2], w0[1], w0[3], a0, ds, d[1], lo, hi);
    }
}

/* Vacuum flux (S = 0) with the sampler branch given. */
HD void vacuum_flux_forced(const GasConst<double> &c, double rl, double ul, double vl, double pl, double al,
                           double rr, double ur, double vr, double pr, double ar, int which, int sub,
                           double F[4])
{
    double s[4] = { 0.0, 0.0, 0.0, 0.0 };
    if (which != 0 && sub != 2) {
        const bool right = (which == 1);
        const double rho = right ? rl : rr, u = right ? ul : ur, v = right ? vl : vr, p = right ? pl : pr;
        const double a = right ? al : ar;
        if (sub == 0) {
            s[0] = rho; s[1] = u; s[2] = v; s[3] = p;
        } else if (right) {
            double tmp = c.two_gp1 + (u - 0.0) * c.gm1 / (c.gp1 * a);
            tmp = pw(tmp, c.two_gm1);
            s[0] = rho * tmp;
            s[1] = (a + c.half_gm1 * u + 0.0) * 2.0 / c.gp1;
            s[2] = v;
            s[3] = p * pw(tmp, c.gamma);
        } else {
            double tmp = c.two_gp1 - (u - 0.0) * c.gm1 / (c.gp1 * a);
            tmp = pw(tmp, c.two_gm1);
            s[0] = rho * tmp;
            s[1] = (-a + c.half_gm1 * u + 0.0) * 2.0 / c.gp1;
            s[2] = v;
            s[3] = p * pw(tmp, c.gamma);
        }
    }
    const double E = s[0] * (0.5 * (s[1] * s[1] + s[2] * s[2]) + s[3] / (s[0] * c.gm1));
    F[0] = s[0] * s[1];
    F[1] = s[0] * s[1] * s[1] + s[3];
    F[2] = s[0] * s[1] * s[2];
    F[3] = s[1] * (E + s[3]);
}

/* HLLC 2D flux with the branch code of hllc_code given. */
HD void hllc_flux_2d_forced(const GasConst<double> &c, double rl, double ul, double vl, double pl, double rr,
                            double ur, double vr, double pr, int code, double F[4])
{
    const double aL = (rl > 0.0) ? sound_speed(c, rl, pl) : 0.0;
    const double aR = (rr > 0.0) ? sound_speed(c, rr, pr) : 0.0;
    if (code & 0x100) {
        vacuum_flux_forced(c, rl, ul, vl, pl, aL, rr, ur, vr, pr, aR, (code >> 2) & 3, code & 3, F);
        return;
    }
    const int reg = code & 3;
    const double ppv = 0.5 * (pl + pr) - 0.125 * (ur - ul) * (rl + rr) * (aL + aR);
    double pg = ppv;
    if (reg == PREG_TRRS) pg = guess_p_trrs(c, ul, pl, aL, ur, pr, aR);
    else if (reg == PREG_TSRS) pg = guess_p_tsrs(c, rl, ul, pl, rr, ur, pr, ppv);
    const double ps = (code & 4) ? c.tol : pg;
    const double qL = (code & 8) ? sq(1.0 + c.q_coef * (dv(ps, pl) - 1.0)) : 1.0;
    const double qR = (code & 16) ? sq(1.0 + c.q_coef * (dv(ps, pr) - 1.0)) : 1.0;
    const double SL = ul - aL * qL;
    const double SR = ur + aR * qR;
    const double Ss = dv(pr - pl + rl * ul * (SL - ul) - rr * ur * (SR - ur), rl * (SL - ul) - rr * (SR - ur));
    const int region = (code >> 5) & 3;
    const bool left = region <= 1;
    const double rho = left ? rl : rr, u = left ? ul : ur, v = left ? vl : vr, p = left ? pl : pr;
    const double E = rho * (0.5 * (u * u + v * v) + dv(p, rho * c.gm1));
    const double fm = rho * u;
    F[0] = fm;
    F[1] = fm * u + p;
    F[2] = fm * v;
    F[3] = u * (E + p);
    if (region == 1 || region == 2) {
        const double S = left ? SL : SR;
        const double rs = dv(rho * (S - u), S - Ss);
        const double es = rs * (dv(E, rho) + (Ss - u) * (Ss + dv(p, rho * (S - u))));
        F[0] = fm + S * (rs - rho);
        F[1] = F[1] + S * (rs * Ss - rho * u);
        F[2] = F[2] + S * (rs * v - rho * v);
        F[3] = F[3] + S * (es - E);
    }
}

/* ------------------------------------------------------------ conversion */

/* Reverse of cons_to_prim_2d: wb (rho, u, v, p) -> Ub (m, mx, my, E), accumulated. */
HD void cons_to_prim_2d_vjp(const GasConst<double> &c, double vol, double m, double mx, double my,
                            const double wb[4], double Ub[4])
{
    const Fd im = rv(m), iv = rv(vol);
    const Fd w1 = Fd(mx) * im, w2 = Fd(my) * im;
    const Fd Pb = (Fd(wb[3]) * c.gm1) * iv, mP = Fd(m) * Pb;
    Fd U0 = Ub[0], U1 = Ub[1], U2 = Ub[2];
    const Fd w1b = Fd(wb[1]) - mP * w1, w2b = Fd(wb[2]) - mP * w2;
    U1 += w1b * im;
    U2 += w2b * im;
    U0 += Fd(wb[0]) * iv - (Fd(0.5) * Pb) * (w1 * w1 + w2 * w2);
    U0 -= (w1b * w1 + w2b * w2) * im;
    Ub[0] = U0.v;
    Ub[1] = U1.v;
    Ub[2] = U2.v;
    Ub[3] += Pb.v;
}

/* Reverse of the 2D primitive -> conserved conversion (src/system.c:884-905):
 * Ub -> wb, accumulated. */
HD void prim_to_cons_2d_vjp(const GasConst<double> &c, double vol, const double w[4],
                            const double Ub[4], double wb[4])
{
    const double rho = w[0], u = w[1], v = w[2];
    const double m = rho * vol;
    const double mb = Ub[0] + Ub[1] * u + Ub[2] * v;
    wb[0] += mb * vol + Ub[3] * vol * 0.5 * (u * u + v * v);
    wb[1] += Ub[1] * m + Ub[3] * vol * rho * u;
    wb[2] += Ub[2] * m + Ub[3] * vol * rho * v;
    wb[3] += dv(Ub[3] * vol, c.gm1);
}

/* The same conversion forward, templated for the tangent-linear state. */
template <class R>
HD void prim_to_cons_2d(const GasConst<R> &c, R vol, const R w[4], R U[4])
{
    const R m = w[0] * vol;
    U[0] = m;
    U[1] = m * w[1];
    U[2] = m * w[2];
    U[3] = vol * (R(0.5) * w[0] * (w[1] * w[1] + w[2] * w[2]) + dv(w[3], c.gm1));
}

}  // namespace hydro

#endif
