// godunov64.cuh - the exact Riemann solver's FP64 path with few FP64 operations.
//
// The same solver as physics.cuh's (kernel.cu:128-570, newton :635-680, devtwo
// :682-749): the same wave patterns, the same p* and the same sampled states,
// for faces inside the short forms' range (godunov_tame); other faces take
// physics.cuh's code.  GB300's FP64 pipe bounds this solver (one library pow
// holds it for 1,640 cycles per warp, a division or a square root for 150), so:
//   - x^gm and x^(1/gm), gm = (gamma-1)/(2 gamma), when 1/gm is a small whole
//     number (5 for gamma 5/3, 7 for 7/5): products and an n-th root by one
//     step of the binomial series from the FP32 value;
//   - the bisection's decisions (devtwo) without its residuals: see bisect_p64;
//   - Newton with FP32 derivatives: see newton_p64;
//   - the sampled interval selected before its state is formed.
// 1021x509 blast, 8 steps: 18.7 ms with physics.cuh's code, 2.25 ms here (with
// uniform tiles and 16x16 tiles 1.35).
#pragma once

#include "physics.cuh"

namespace ast {

// a double well inside FP32's range as FP32 (truncated; no FP64 conversion)
__device__ __forceinline__ float low_float(double a)
{
    const long long i = d64::bits(a);
    const int hi = (int)(i >> 32);
    const unsigned m = ((unsigned)(hi & 0x7fffffff) << 3) | ((unsigned)i >> 29);
    const unsigned v = m - ((1023u - 127u) << 23);
    // |a| < 2^-126: zero
    return __uint_as_float(((hi & 0x7fffffff) < ((1023 - 126) << 20)) ? 0u : (v | ((unsigned)hi & 0x80000000u)));
}

// positive with 2^-40 <= a < 2^40, and |a| < 2^40: FP32 holds these, their
// products in pairs and the quotients below
__device__ __forceinline__ bool tame_pos32(double a)
{
    return (unsigned)(__double2hiint(a) - ((1023 - 40) << 20)) < (80u << 20);
}
__device__ __forceinline__ bool tame32(double a) { return (__double2hiint(a) & 0x7fffffff) < ((1023 + 40) << 20); }
__device__ __forceinline__ bool godunov_tame(double rL, double pL, double unL, double utL, double rR, double pR,
                                             double unR, double utR)
{
    return tame_pos32(rL) && tame_pos32(pL) && tame_pos32(rR) && tame_pos32(pR) && tame32(unL) && tame32(unR) &&
           tame32(utL) && tame32(utR);
}
__device__ __forceinline__ bool godunov_tame(const RPre<double>& q)
{
    return godunov_tame(q.rI, q.pI, q.enI, q.teI, q.rII, q.pII, q.enII, q.teII);
}

// y^n, n = 2 .. 16
__device__ __forceinline__ double ipow(const d64::Pipe& o, double y, int n)
{
    double r = (n & 1) ? y : 1.0, b = y;
    bool one = !(n & 1);
    for (int k = n >> 1; k; k >>= 1) {
        b = o.mul(b, b);
        if (k & 1) {
            r = one ? b : o.mul(r, b);
            one = false;
        }
    }
    return r;
}

// x^gm for 1/gm = n: with w = x^(-1/n) from FP32 and e = 1 - x w^n,
// x^(-1/n) = w (1 - e)^(-1/n) = w (1 + e/n + (n+1) e^2/(2 n^2) + ...), |e| of
// some 1e-6; its reciprocal.  Other gm: the library's pow.
__device__ __forceinline__ double pow_gm(const Gas<double>& g, double x)
{
    using namespace d64;
    const Pipe o(g);
    if (g.n == 0) return pow(x, g.gm);
    const double w = (double)exp2f(-(float)g.gm * log2f(low_float(x)));
    const double e = fma(flip(x), ipow(o, w, g.n), o.one);
    return o.rcp(fma(w, o.mul(e, fma(e, o.mul(o.mul(o.half, g.gm), o.add(g.gm, 1.0)), g.gm)), w));
}
// x^(1/gm)
__device__ __forceinline__ double pow_inv_gm(const Gas<double>& g, double x)
{
    return g.n ? ipow(d64::Pipe(g), x, g.n) : pow(x, 1.0 / g.gm);
}
// rare_coef (physics.cuh) from y = (p/p_K)^gm: (1 - y^n)/(1 - y) = 1 + y + ...
// + y^(n-1), and its limit rho c within the same absolute distance of p_K
__device__ __forceinline__ double rare_coef_y(const Gas<double>& g, double rc, double y, double p, double pK)
{
    using namespace d64;
    const Pipe o(g);
    double s = o.add(1.0, y);
    for (int k = 2; k < g.n; k++) s = fma(s, y, 1.0);
    return sel(bits(abs(o.sub(p, pK))) < bits(g.eps), rc, o.mul(o.mul(g.gm, rc), s));
}

// godunov_sides and godunov_pre (physics.cuh) of a tame face
__device__ __forceinline__ RPre<double> godunov_sides64(const Gas<double>& g, double rL, double pL, double unL,
                                                        double utL, double rR, double pR, double unR, double utR)
{
    using namespace d64;
    const Pipe o(g);
    RPre<double> q;
    q.swap = bits(pL) > bits(pR);
    q.enI = sel(q.swap, flip(unR), unL);
    q.teI = sel(q.swap, utR, utL);
    q.pI = sel(q.swap, pR, pL);
    q.rI = sel(q.swap, rR, rL);
    q.enII = sel(q.swap, flip(unL), unR);
    q.teII = sel(q.swap, utL, utR);
    q.pII = sel(q.swap, pL, pR);
    q.rII = sel(q.swap, rL, rR);
    q.cI = o.sqrt_ratio(o.mul(g.ga, q.pI), q.rI);
    q.cII = o.sqrt_ratio(o.mul(g.ga, q.pII), q.rII);
    q.Udf = o.sub(q.enI, q.enII);
    q.Urz = q.Uvk = 0.0;
    q.pattern = 4;
    return q;
}

__device__ __forceinline__ RPre<double> godunov_pre64(const Gas<double>& g, double rL, double pL, double unL,
                                                      double utL, double rR, double pR, double unR, double utR)
{
    using namespace d64;
    const Pipe o(g);
    RPre<double> q = godunov_sides64(g, rL, pL, unL, utL, rR, pR, unR, utR);
    const double dp = o.sub(q.pII, q.pI);
    const double Uud = o.mul(dp, o.rsqrt(o.mul(q.rI, fma(g.hg2, q.pII, o.mul(g.hg1, q.pI)))));
    if (bits(q.Udf) > 0) {
        q.pattern = bits(q.Udf) <= bits(Uud) ? 2 : 3;
        return q;
    }
    // Udf <= 0 <= Uud: vacuum, two rarefactions or pattern 2
    const double k2 = o.mul(2.0, g.inv_g1);
    q.Uvk = o.mul(-k2, o.add(q.cII, q.cI));
    if (key(q.Udf) < key(q.Uvk)) {
        q.pattern = 0;
        return q;
    }
    // equal pressures (a contact, or two equal rarefactions): Urz = 0 >= Udf
    if (bits(dp) == 0) {
        q.pattern = 1;
        return q;
    }
    // Urz = -2 cII/(gamma-1) (1 - x^gm), x = pI/pII: FP32 decides unless Udf
    // lies within 1e-4 of it.  ln x to FP32 precision over all of x: from x
    // itself, near 1 (where FP32 no longer tells x from 1) from 1 - x (which
    // in turn loses a small x)
    const double x = o.mul(q.pI, o.rcp(q.pII));
    const float xf = low_float(x), lx = xf < 0.5f ? logf(xf) : log1pf(-low_float(o.sub(1.0, x)));
    const float y = -expm1f((float)g.gm * lx);
    const float zf = -low_float(k2) * low_float(q.cII) * y, uf = low_float(q.Udf);
    const bool sure = fabsf(uf - zf) > 1e-4f * fabsf(zf) && y < 1.0f;
    if (sure && uf > zf) {
        q.pattern = 2;
        return q;
    }
    q.Urz = o.mul(o.mul(k2, q.cII), o.sub(pow_gm(g, x), 1.0));   // a zero is +0, as key() needs it
    q.pattern = (sure || key(q.Udf) <= key(q.Urz)) ? 1 : 2;
    return q;
}

// The residual of devtwo as physics.cuh forms it (out of line: seldom needed)
static __device__ __noinline__ double lev_exact(const Gas<double>& g, double enI, double pI, double rI, double cI,
                                                double enII, double pII, double cII, double x)
{
    return lev_res(g, enI, pI, rI, cI, enII, pII, cII, x);
}
// physics.cuh's solver, sampler and side states, out of line, for the faces
// and tolerances that the short forms leave to them
struct WildSolve {
    double p;
    int iters;
    unsigned status;
};
static __device__ __noinline__ WildSolve solve_wild(const Gas<double>& g, RPre<double> q)
{
    RiemannCount rc;
    rc.clear();
    WildSolve w;
    w.p = solve_p_reference(g, q, rc);
    w.iters = q.pattern == 2 ? rc.bisect_iters : rc.newton_iters;
    w.status = rc.status;
    return w;
}
__device__ __forceinline__ double solve_exact(const Gas<double>& g, const RPre<double>& q, RiemannCount& rc)
{
    const WildSolve w = solve_wild(g, q);
    rc.status |= w.status;
    if (q.pattern == 2) {
        rc.bisect_calls++;
        rc.bisect_iters += w.iters;
    } else {
        rc.newton_calls++;
        rc.newton_iters += w.iters;
        if (w.iters > rc.newton_max) rc.newton_max = w.iters;
    }
    return w.p;
}
struct WildSample {
    WildFlux f;
    unsigned status;
};
static __device__ __noinline__ WildSample sample_wild(const Gas<double>& g, RPre<double> q, double p)
{
    RiemannCount rc;
    rc.clear();
    WildSample w;
    w.f.S = godunov_sample(g, q, p, w.f.F, rc);
    w.status = rc.status;
    return w;
}
static __device__ __noinline__ RPre<double> pre_wild(const Gas<double>& g, double rL, double pL, double unL, double utL,
                                                     double rR, double pR, double unR, double utR)
{
    return godunov_pre(g, rL, pL, unL, utL, rR, pR, unR, utR);
}
static __device__ __noinline__ RPre<double> sides_wild(const Gas<double>& g, double rL, double pL, double unL,
                                                       double utL, double rR, double pR, double unR, double utR)
{
    return godunov_sides(g, rL, pL, unL, utL, rR, pR, unR, utR);
}

// The bisection of devtwo (kernel.cu:682-749) on [pI, pII], its iterates and
// its result, without evaluating its residual at every iterate.  The residual
// f rises and is concave, so f(x) has the sign of x - p*, and near p* it is
// f'(p*) (x - p*): with p* known, every decision is a comparison, and the
// stopping test |f(x)| <= tol is made on that product.  p* comes from an FP32
// Newton iteration and a Newton step with the FP64 residual (its error then
// some 1e-14 p).  Where the product lies within `band` (above the rounding of
// f and the error of p*) of tol, the residual itself decides; a tolerance
// near the rounding of f takes the plain bisection.  27 iterations of about
// 130 FP64 operations become one evaluation and an addition per iteration.
__device__ __forceinline__ double bisect_p64(const Gas<double>& g, const RPre<double>& q, RiemannCount& rc)
{
    using namespace d64;
    const Pipe o(g);
    const float pIf = low_float(q.pI), pIIf = low_float(q.pII), cIf = low_float(q.cI), cIIf = low_float(q.cII);
    const float dUf = low_float(q.Udf), tolf = (float)g.tol;
    const float band = 2.3e-13f * (cIf + cIIf + fabsf(low_float(q.enI)) + fabsf(low_float(q.enII)));
    const float kIf = 1.0f / (low_float(q.rI) * cIf), kIIf = 1.0f / (low_float(q.rII) * cIIf);
    const float gaf = (float)g.ga, gpf = (float)g.gp, gmf = (float)g.gm, k2f = 2.0f * (float)g.inv_g1, ga4 = 0.25f / gaf;
    // f and f' in FP32 (f' also serves the FP64 steps)
    auto eval = [&](float p, float& f, float& df) {
        const float ri = p / pIf, qq = gpf * ri + gmf, is = rsqrtf(qq);
        const float t = exp2f(gmf * log2f(p / pIIf));
        f = (p - pIf) * kIf * is + k2f * cIIf * (t - 1.0f) - dUf;
        df = ((gaf + 1.0f) * ri + 3.0f * gaf - 1.0f) * is * is * is * kIf * ga4 + t * kIIf * (pIIf / p);
    };
    // a derivative the FP32 range does not hold
    auto bad = [](float df) { return !(df > 1e-30f && df < 1e30f); };
    bool ok = band < 0.125f * tolf;
    float pf = (pIf * kIf + pIIf * kIIf + dUf) / (kIf + kIIf), df = 1.0f;   // the acoustic value
    pf = fminf(fmaxf(pf, pIf), pIIf);
    for (int k = 0; ok && k < 16; k++) {
        float f;
        eval(pf, f, df);
        const float pn = fminf(fmaxf(pf - f / df, pIf), pIIf);
        const bool done = fabsf(pn - pf) <= 1e-6f * pf;
        pf = pn;
        if (done) break;
    }
    // FP64 Newton steps until one is below 3e-7 p (usually the first)
    double p = (double)pf;
    if (ok) {
        const double ipI = o.rcp(q.pI), ipII = o.rcp(q.pII), kI = o.rcp(o.mul(q.rI, q.cI));
        const double gpI = o.mul(g.gp, ipI), c2 = o.mul(o.mul(2.0, g.inv_g1), q.cII);
        ok = false;
        for (int k = 0; k < 4; k++) {
            const double fI = o.mul(o.mul(o.sub(p, q.pI), kI), o.rsqrt(fma(gpI, p, g.gm)));
            const double f = fma(c2, o.sub(pow_gm(g, o.mul(p, ipII)), 1.0), o.sub(fI, q.Udf));
            float dummy;
            eval(low_float(p), dummy, df);
            if (bad(df)) break;
            const float step = (float)f / df;
            p = o.sub(p, (double)step);
            if (fabsf(step) <= 3e-7f * pf) {
                ok = bits(p) >= bits(q.pI) && bits(p) <= bits(q.pII);
                break;
            }
            if (!(bits(p) >= bits(q.pI) && bits(p) <= bits(q.pII))) break;
        }
    }
    if (!ok) return solve_exact(g, q, rc);
    // iterates outside (lo, hi) are far from the stopping test
    const double far = (double)(8.0f * (tolf + band) / df);
    const long long lo = key(o.sub(p, far)), hi = key(o.add(p, far));
    auto near = [&](double x) { return bits(x) > lo && bits(x) < hi; };
    auto residual = [&](double x) {
        return lev_exact(g, q.enI, q.pI, q.rI, q.cI, q.enII, q.pII, q.cII, x);
    };
    rc.bisect_calls++;
    if (near(q.pI) && fabs(residual(q.pI)) <= g.tol) return q.pI;
    if (near(q.pII) && fabs(residual(q.pII)) <= g.tol) return q.pII;
    double kl = q.pI, kp = q.pII, kc;
    int it = 0;
    for (;;) {
        it++;
        // (kl + kp)/2: the sum's exponent less one
        kc = from(bits(o.add(kl, kp)) - (1ll << 52));
        bool above = bits(kc) > bits(p);
        if (near(kc)) {
            const float d = fabsf((float)o.sub(kc, p)), est = d * df, err = band + 2.0f * est * (d / pf) + 4e-6f * est;
            if (est + err <= tolf) break;
            if (!(est - err > tolf)) {
                const double f = residual(kc);
                if (fabs(f) <= g.tol) break;
                above = f >= 0.0;
            }
        }
        if (it >= g.max_iter) { rc.status |= 0x08u; break; }
        if (above) kp = kc;
        else kl = kc;
    }
    rc.bisect_iters += it;
    return kc;
}

// The two-shock Newton iteration (newton, kernel.cu:635-680) from the acoustic
// start value with the residual in FP64 and the derivative in FP32: an
// iterate's step is good to 1e-7 of itself, so the iteration converges as
// fast and stops at the same iterate, whose last step is below tol: the result
// agrees to 1e-7 tol.  Tolerances above 1e-7, and caps that may end the
// iteration before it converges, take the plain iteration.
__device__ __forceinline__ double newton_p64(const Gas<double>& g, const RPre<double>& q, RiemannCount& rc)
{
    using namespace d64;
    const Pipe o(g);
    if (g.max_iter < 16 || g.tol > 1e-7) return solve_exact(g, q, rc);
    const double kI = o.rcp(o.mul(q.rI, q.cI)), kII = o.rcp(o.mul(q.rII, q.cII));
    const double gI = o.mul(g.gp, o.rcp(q.pI)), gII = o.mul(g.gp, o.rcp(q.pII));
    double pn = o.mul(fma(q.pI, kI, fma(q.pII, kII, q.Udf)), o.rcp(o.add(kI, kII)));
    // (p_I/(rho_I c_I) + p_II/(rho_II c_II) + Udf)/(1/(rho_I c_I) + 1/(rho_II c_II)), the reference's with both
    // terms divided by the impedances' product
    const float kIf = low_float(kI), kIIf = low_float(kII), tolp = fmaxf((float)g.tol * low_float(pn), 1.2e-38f);
    const float ga4 = 0.25f / (float)g.ga, b = 3.0f * (float)g.ga - 1.0f, gg = ((float)g.ga + 1.0f) / (float)g.gp;
    const float gmf = (float)g.gm;
    int k = 0;
    for (;;) {
        const double p = pn;
        k++;
        const double qI = fma(gI, p, g.gm), qII = fma(gII, p, g.gm);
        // p far above both pressures (qII <= qI): FP32 does not hold the derivative's terms
        if (__double2hiint(qI) >= ((1023 + 100) << 20)) return solve_exact(g, q, rc);
        const double sI = o.rsqrt(qI), sII = o.rsqrt(qII);
        const double f = fma(o.mul(o.sub(p, q.pI), kI), sI, fma(o.mul(o.sub(p, q.pII), kII), sII, flip(q.Udf)));
        const float uI = low_float(sI), uII = low_float(sII);
        // (gamma + 1) p/p_K + b from q_K = gp p/p_K + gm
        const float dI = (gg * (low_float(qI) - gmf) + b) * ga4 * uI * uI * uI * kIf;
        const float dII = (gg * (low_float(qII) - gmf) + b) * ga4 * uII * uII * uII * kIIf;
        const float df = dI + dII;
        if (!(df > 1e-30f && df < 1e30f)) return solve_exact(g, q, rc);   // FP32 does not hold it
        const float step = (float)f / df;
        pn = o.sub(p, (double)step);
        if (!(fabsf(step) >= tolp)) break;
        if (k >= g.max_iter) { rc.status |= 0x04u; break; }
    }
    rc.newton_calls++;
    rc.newton_iters += k;
    if (k > rc.newton_max) rc.newton_max = k;
    return pn;
}

// rho a/(a - rho du): the density behind a shock of mass flux a; its flux from
// (rho, p, en, te), en in the swapped frame
__device__ __forceinline__ void godunov_flux64(const Gas<double>& g, bool swap, double r, double p, double en,
                                               double te, double F[4])
{
    using namespace d64;
    const Pipe o(g);
    en = sel(swap, flip(en), en);
    const double m = o.mul(r, en);
    F[0] = m;
    F[1] = fma(m, en, p);
    F[2] = o.mul(m, te);
    // en (e + p), e + p = ga p/(ga - 1) + r (en^2 + te^2)/2
    F[3] = fma(o.mul(o.half, m), fma(en, en, o.mul(te, te)), o.mul(o.mul(o.mul(g.ga, g.inv_g1), p), en));
}

// godunov_sample (physics.cuh) of patterns 1, 2 and 3 at w = 0
__device__ __forceinline__ double godunov_sample64(const Gas<double>& g, const RPre<double>& q, double p, double F[4])
{
    using namespace d64;
    const Pipe o(g);
    const bool two_raref = q.pattern == 1, shockII = q.pattern == 3;
    // mass-flux coefficients of the two waves
    double aI, aII;
    if (two_raref) {
        // p* in closed form: (p*/pI)^gm = B, (p*/pII)^gm = B (pI/pII)^gm
        const double B = o.mul(o.sub(q.Udf, q.Uvk), o.rcp(o.sub(q.Urz, q.Uvk)));
        p = o.mul(q.pI, ipow(o, B, g.n));
        aI = rare_coef_y(g, o.mul(q.rI, q.cI), B, p, q.pI);
        // (pI/pII)^gm = 1 + Urz (gamma - 1)/(2 cII)
        aII = rare_coef_y(g, o.mul(q.rII, q.cII), o.mul(B, fma(o.mul(q.Urz, g.hg1), o.rcp(q.cII), 1.0)), p, q.pII);
    } else {
        const double x = o.mul(q.rI, fma(g.hg2, p, o.mul(g.hg1, q.pI)));
        aI = o.mul(x, o.rsqrt(x));
        if (shockII) {
            const double z = o.mul(q.rII, fma(g.hg2, p, o.mul(g.hg1, q.pII)));
            aII = o.mul(z, o.rsqrt(z));
        } else {
            const double z = o.mul(p, o.rcp(q.pII));
            if (g.n) aII = rare_coef_y(g, o.mul(q.rII, q.cII), pow_gm(g, z), p, q.pII);
            else aII = rare_coef(g, q.rII, q.cII, p, q.pII);
        }
    }
    const double u = o.mul(fma(aI, q.enI, fma(aII, q.enII, o.sub(q.pI, q.pII))), o.rcp(o.add(aI, aII)));
    // heads (d) and tails (dd) of the two waves; a shock is both
    const double wI = o.sub(q.enI, u), wII = o.sub(q.enII, u);
    double dI, ddI, dII, ddII;
    if (two_raref) {
        dI = o.sub(q.enI, q.cI);
        ddI = fma(flip(wI), g.hg1, o.sub(u, q.cI));
    } else {
        dI = ddI = fma(flip(aI), o.rcp(q.rI), q.enI);
    }
    if (shockII) {
        dII = ddII = fma(aII, o.rcp(q.rII), q.enII);
    } else {
        dII = o.add(q.enII, q.cII);
        ddII = fma(flip(wII), g.hg1, o.add(u, q.cII));
    }
    const double UU = max_pos(max_abs(dI, dII), max_abs(ddI, ddII));
    // the interval that holds w = 0
    const bool left = key(u) >= key(-0.0);   // 0 <= u: the contact's side I
    const double en0 = sel(left, q.enI, q.enII), p0 = sel(left, q.pI, q.pII), r0 = sel(left, q.rI, q.rII);
    const double te = sel(left, q.teI, q.teII), c0 = sel(left, q.cI, q.cII);
    const double d = sel(left, dI, flip(dII)), dd = sel(left, ddI, flip(ddII));   // side II mirrored
    double r, en, ps;
    if (key(d) >= key(-0.0)) {
        // outside the wave: the side's own state
        r = r0; en = en0; ps = p0;
    } else if (key(dd) > key(0.0)) {
        // inside a rarefaction fan
        const double e = sel(left, en0, flip(en0));
        const double ce = o.mul(fma(g.g1, e, o.mul(2.0, c0)), o.rcp(g.g2));
        ps = o.mul(p0, pow_inv_gm(g, o.mul(ce, o.rcp(c0))));
        const double ic = o.rcp(ce);
        r = o.mul(o.mul(o.mul(g.ga, ps), ic), ic);
        en = sel(left, ce, flip(ce));
    } else {
        // between the wave and the contact
        const double a = sel(left, aI, aII), w = sel(left, wI, flip(wII));
        ps = p;
        en = u;
        if (left ? !two_raref : shockII) {
            r = o.mul(o.mul(r0, a), o.rcp(fma(flip(r0), w, a)));
        } else {
            const double ic = o.rcp(fma(g.hg1, w, c0));
            r = o.mul(o.mul(o.mul(g.ga, p), ic), ic);
        }
    }
    godunov_flux64(g, q.swap, r, ps, en, te, F);
    return max_pos(UU, g.eps8);
}

// ------------------------------------------------------------------ by precision
// The step's entry points: FP32 takes physics.cuh's code; FP64 the short forms
// where the face allows them.
__device__ __forceinline__ RPre<float> face_pre(const Gas<float>& g, float rL, float pL, float unL, float utL,
                                                float rR, float pR, float unR, float utR)
{
    return godunov_pre(g, rL, pL, unL, utL, rR, pR, unR, utR);
}
__device__ __forceinline__ RPre<double> face_pre(const Gas<double>& g, double rL, double pL, double unL, double utL,
                                                 double rR, double pR, double unR, double utR)
{
    if (godunov_tame(rL, pL, unL, utL, rR, pR, unR, utR))
        return godunov_pre64(g, rL, pL, unL, utL, rR, pR, unR, utR);
    return pre_wild(g, rL, pL, unL, utL, rR, pR, unR, utR);
}
__device__ __forceinline__ RPre<float> face_sides_of(const Gas<float>& g, float rL, float pL, float unL, float utL,
                                                     float rR, float pR, float unR, float utR)
{
    return godunov_sides(g, rL, pL, unL, utL, rR, pR, unR, utR);
}
__device__ __forceinline__ RPre<double> face_sides_of(const Gas<double>& g, double rL, double pL, double unL,
                                                      double utL, double rR, double pR, double unR, double utR)
{
    if (godunov_tame(rL, pL, unL, utL, rR, pR, unR, utR))
        return godunov_sides64(g, rL, pL, unL, utL, rR, pR, unR, utR);
    return sides_wild(g, rL, pL, unL, utL, rR, pR, unR, utR);
}
// p* of a queued face by the reference's iteration
__device__ __forceinline__ double face_solve(const Gas<double>& g, const RPre<double>& q, RiemannCount& rc)
{
    if (!godunov_tame(q)) return solve_exact(g, q, rc);
    return q.pattern == 2 ? bisect_p64(g, q, rc) : newton_p64(g, q, rc);
}
// the sampled flux: MODE as in godunov_sample
template <int MODE>
__device__ __forceinline__ float face_sample(const Gas<float>& g, const RPre<float>& q, float p, float F[4],
                                             RiemannCount& rc)
{
    return godunov_sample<float, MODE>(g, q, p, F, rc);
}
template <int MODE>
__device__ __forceinline__ double face_sample(const Gas<double>& g, const RPre<double>& q, double p, double F[4],
                                              RiemannCount& rc)
{
    const bool fits = MODE == kSampleClosed ? q.pattern == 1 && g.n != 0 : tame_pos32(p);
    if (fits && godunov_tame(q)) return godunov_sample64(g, q, p, F);
    const WildSample w = sample_wild(g, q, p);
    rc.status |= w.status;
    return w.f.get(F);
}

}  // namespace ast
