// The x component of a visible Beckmann slope (alpha = 1): the reference inverts the marginal CDF by a fixed
// number of FP64 bisections (CLARITAS/CLARITAS.py:1925-2038), each an exp and an erfc (or erfcx and log) on a
// pipe that issues one FP64 warp instruction per 16 cycles per SM. That made the rough microsurface walk the
// whole cost of rough scenes: of ~50 evaluations per slope only the last few decide anything.
//
// Here the same bisection runs, with the same midpoints, and a midpoint's comparison is evaluated only where
// it could go either way. A root estimate (FP32 search, one FP64 Halley step with closed-form derivatives) and a
// bound on how far it and an evaluated midpoint can be off give a radius; outside it the sign of the
// comparison follows from monotonicity (131072 rough photons with records 176 -> 44 ms; 47 with up to four Newton
// steps in place of the Halley step). The result is therefore the reference's bit for bit (checked over the
// declared range of both branches against the plain bisection). Where the estimate is not trusted (no
// convergence, a root next to the switch of formulas at 5) the radius is infinite: every midpoint is evaluated.
//
// Host-compilable: the CPU test builds this file with the host's exp, erfc and log.
#pragma once
#include <math.h>

#ifdef __CUDACC__
#define CLR_SLOPE_FN __device__
#else
#define CLR_SLOPE_FN static inline
#endif

namespace clr {
namespace {

enum { SF_NONE = 0, SF_PROJECTED_AREA = 10, SF_CDF = 11, SF_INVERSE_CDF = 12 };

/* B(x) = 1 - x sqrt(pi) erfcx(x) (:1925-1939) */
CLR_SLOPE_FN double o_tail_B(double x) {
    if (!(x >= 0.0) || !isfinite(x)) return -1.0;
    const double SQRT_PI = 1.77245385090551602729816748334114518;
    if (x < 5.0) {
        double e = exp(x * x) * erfc(x);
        double b = 1.0 - x * SQRT_PI * e;
        return (isfinite(b) && b > 0.0) ? b : -1.0;
    }
    double y = 1.0 / (x * x);
    double b = 0.5 * y - 0.75 * y * y + 1.875 * y * y * y - 6.5625 * y * y * y * y + 29.53125 * y * y * y * y * y -
               162.421875 * y * y * y * y * y * y + 1055.7421875 * y * y * y * y * y * y * y;
    return (isfinite(b) && b > 0.0) ? b : -1.0;
}

/* denominator of the alpha=1 visible-slope marginal CDF, the same for every slope (:1949) */
CLR_SLOPE_FN double o_visible_q(double slope_i) {
    const double K = 0.28209479177387814347403972578038629;
    return K * exp(-slope_i * slope_i) + 0.5 * slope_i * erfc(-slope_i);
}
/* alpha=1 visible-slope marginal CDF, ordinary branch (:1944-1957), with q = o_visible_q(slope_i) */
CLR_SLOPE_FN int o_visible_cdf(double slope, double slope_i, double q, double* out) {
    if (!isfinite(slope) || !isfinite(slope_i)) return 0;
    if (slope >= slope_i) { *out = 1.0; return 1; }
    const double K = 0.28209479177387814347403972578038629;
    if (!(q > 0.0) || !isfinite(q)) return 0;
    double n = K * exp(-slope * slope) + 0.5 * slope_i * erfc(-slope);
    double f = n / q;
    if (!isfinite(f)) return 0;
    if (f < 0.0 && f > -1.0e-13) f = 0.0;
    if (f > 1.0 && f < 1.0 + 1.0e-13) f = 1.0;
    if (f < 0.0 || f > 1.0) return 0;
    *out = f;
    return 1;
}

/* Estimate of the root of F(s) = u on the ordinary branch and the radius outside which the sign of the
 * computed F(mid) - u is that of mid - root. F' = exp(-s^2) (slope_i - s) / (sqrt(pi) q) > 0 below slope_i and
 * F''/F' = -2 s - 1/(slope_i - s). The two terms of n are good to a few ulps each (exp 1, erfc 5) and no larger than
 * those of q, whose absolute sum over q is `spread` (1 for slope_i >= 0, under 8 down to -1): the computed F is off
 * by less than 1e-15 spread. F(root +- r) differs from u by more than the errors of both evaluations when
 * r = 8e-15 spread / F', with the curvature over r negligible by the checks. */
CLR_SLOPE_FN void o_visible_root(double slope_i, double q, double u, double* root, double* radius) {
    *root = 0.0;
    *radius = HUGE_VAL;
    const float si = (float)fmin(slope_i, 1.0e6), qf = (float)fmin(q, 1.0e6), uf = (float)u;
    if (!(qf > 0.0f)) return;
    float lo = -6.5f, hi = fminf(si, 6.0f), s = fminf(-0.2f, 0.5f * (lo + hi));
    for (int it = 0; it < 14; ++it) {  // safeguarded Newton on the CDF
        const float e = expf(-s * s);
        const float f = (0.28209479f * e + 0.5f * si * erfcf(-s)) / qf - uf;
        if (f > 0.0f) hi = s; else lo = s;
        float nx = s - f * 1.77245385f * qf / (e * (si - s));
        if (fabsf(nx - s) <= 4.0e-6f) break;
        if (!(nx > lo && nx < hi)) nx = 0.5f * (lo + hi);
        s = nx;
    }
    const double K = 0.28209479177387814347403972578038629, SQRT_PI = 1.77245385090551602729816748334114518;
    double t = (double)s, step = 1.0, p = 0.0, bend = 0.0;
    for (int it = 0; it < 4; ++it) {  // one step, more only where FP32 left a poor start
        if (!(t < slope_i)) return;
        const double e = exp(-t * t), room = slope_i - t;
        p = e * room / (SQRT_PI * q);
        if (!(p > 0.0)) return;
        const double newton = ((K * e + 0.5 * slope_i * erfc(-t)) / q - u) / p;
        bend = fabs(t) + 1.0 / room;
        step = newton / (1.0 + newton * (t + 0.5 / room));
        t -= step;
        // third order: what is left is below (step bend)^2 step
        if (fabs(step) * bend <= 1.0e-5) break;
    }
    const double room = slope_i - t, spread = slope_i >= 0.0 ? 1.0 : 8.0;
    if (!(room > 0.0) || !(fabs(step) * bend <= 1.0e-5) || !(fabs(t) < 8.0)) return;
    const double r = 8.0e-15 * spread / p + 4.0 * (step * bend) * (step * bend) * fabs(step) + 1.0e-15;
    if (!(r <= 1.0e-3 * room) || !(r <= 1.0e-4)) return;
    *root = t;
    *radius = r;
}

/* The same on the tail branch (x = -slope_i > 1): the root of lr(t) = log(u), lr' = -2 t / C(t), decreasing, and
 * lr''/lr' = 1/t - 2 y + 2 t / C with y = x + t.
 * The computed lr is noisy through 1 - y sqrt(pi) erfcx(y): exp(y^2) carries y^2 ulps and the difference is as
 * small as 0.019 at y = 5. Above 5 the asymptotic series is smooth (its own truncation error moves the root
 * but not the order of the values), so only the two sides of 5 may not be compared through one estimate. */
CLR_SLOPE_FN void o_tail_root(double x, double Bx, double target, double hi0, double* root, double* radius) {
    *root = 0.0;
    *radius = HUGE_VAL;
    if (!(x < 1.0e6) || !(target > -30.0)) return;
    // start: lr ~ -(2 x t + t^2) bends below by the log term; a few safeguarded steps in FP64 arithmetic with the
    // FP32 erfcx-free form of C keep the expensive evaluations to two
    const float xf = (float)x, tf = (float)target, bf = (float)Bx;
    float lo = 0.0f, hi = (float)hi0 * 64.0f, t = fminf((float)hi0, sqrtf(-tf * bf) + 1.0e-6f);
    for (int it = 0; it < 24; ++it) {
        const float y = xf + t;
        float B;
        if (y < 4.0f) {
            B = 1.0f - y * 1.77245385f * expf(y * y) * erfcf(y);
        } else {
            const float w = 1.0f / (y * y);
            B = w * (0.5f + w * (-0.75f + w * (1.875f + w * (-6.5625f + w * 29.53125f))));
        }
        const float C = t / y + (xf / y) * B;
        const float f = -(2.0f * xf * t + t * t) + logf(C / bf) - tf;  // decreasing in t
        if (f > 0.0f) lo = t; else hi = t;
        float nx = t + f * C / (2.0f * t);
        if (fabsf(nx - t) <= 4.0e-6f * t) break;
        if (!(nx > lo && nx < hi)) nx = 0.5f * (lo + hi);
        t = nx;
    }
    double s = (double)t, step = 1.0, C = 1.0, bend = 0.0;
    bool enough = false;
    for (int it = 0; it < 4; ++it) {
        if (!(s > 0.0)) return;
        const double y = x + s, By = o_tail_B(y);
        if (!(By > 0.0)) return;
        C = s / y + (x / y) * By;
        const double newton = (-(2.0 * x * s + s * s) + log(C / Bx) - target) * C / (2.0 * s);  // added
        bend = 1.0 / s + 2.0 * y + 2.0 * s / C;
        step = newton / (1.0 + newton * (0.5 / s - y + s / C));
        s += step;
        // above 5 the derivatives are those of the whole function, 2e-6 off the cut series': a second step
        enough = fabs(step) * bend <= (x + s < 4.99 ? 1.0e-5 : 1.0e-9);
        if (enough) break;
    }
    if (!(s > 0.0) || !enough) return;
    const double y = x + s;
    if (fabs(y - 5.0) < 1.0e-2) return;
    // noise of lr through C (relative error of B's difference below 5, a few ulps above), and of the sum
    const double eps = (y < 5.0 ? (1.0e-15 * y * y + 4.0e-15) / C : 2.0e-14) + 2.0e-14;
    const double r = 4.0 * eps * C / (2.0 * s) + 4.0 * (step * bend) * (step * bend) * fabs(step) + 1.0e-15 * s;
    if (!(r <= 1.0e-4 * s)) return;
    *root = s;
    *radius = r;
}

/* x component of the visible slope for 0 < u1 < 1 and a finite slope_i <= cot(1e-4): the bracket and the
 * bisections of :1985-2027. Returns 0 with *fc set on a numerical failure. */
CLR_SLOPE_FN int o_visible_slope_x(double slope_i, double u1, double* slope_x, int* fc) {
    double root, radius;
    if (slope_i < -1.0) {
        double x = -slope_i, Bx = o_tail_B(x);
        if (!(Bx > 0.0) || !isfinite(Bx)) { *fc = SF_PROJECTED_AREA; return 0; }
        double target = log(u1), lo = 0.0, hi = fmax(1.0 / x, 1.0e-12);
        o_tail_root(x, Bx, target, hi, &root, &radius);
        // 1: lr(t) > target, 0: not, -1: a numerical failure. The values on the other side of the change of
        // formula at y = 5 may be off by 3e-6 of B: 1e-4 of lr covers them, a distance of 1e-2 from 5 is kept.
        auto above = [&](double t) -> int {
            const double d = t - root;
            if (fabs(d) > radius) {
                const bool same = (x + t < 5.0) == (x + root < 5.0);
                if (same || fabs(d) > 1.0e-2) return d < 0.0 ? 1 : 0;
            }
            double y = x + t, By = o_tail_B(y);
            if (!(By > 0.0) || !isfinite(By)) return -1;
            double Cc = t / y + (x / y) * By;
            if (!(Cc > 0.0) || !isfinite(Cc)) return -1;
            double lr = -(2.0 * x * t + t * t) + log(Cc / Bx);
            if (!isfinite(lr)) return -1;
            return lr <= target ? 0 : 1;
        };
        int bracketed = 0;
        for (int it = 0; it < 64; ++it) {
            const int a = above(hi);
            if (a < 0) { *fc = SF_CDF; return 0; }
            if (a == 0) { bracketed = 1; break; }
            hi *= 2.0;
            if (!isfinite(hi)) { *fc = SF_INVERSE_CDF; return 0; }
        }
        if (!bracketed) { *fc = SF_INVERSE_CDF; return 0; }
        for (int it = 0; it < 52; ++it) {
            double mid = 0.5 * (lo + hi);
            if (mid == lo || mid == hi) break;  // every further step decides as before
            const int a = above(mid);
            if (a < 0) { *fc = SF_CDF; return 0; }
            if (a) lo = mid; else hi = mid;
        }
        *slope_x = -(x + 0.5 * (lo + hi));
        return 1;
    }
    const double q = o_visible_q(slope_i);
    double lo = fmin(-1.0, slope_i - 1.0), hi = slope_i, f = 1.0;
    o_visible_root(slope_i, q, u1, &root, &radius);
    int bracketed = 0;
    for (int it = 0; it < 64; ++it) {
        if (fabs(lo - root) > radius) f = lo < root ? 0.0 : 1.0;
        else if (!o_visible_cdf(lo, slope_i, q, &f)) { *fc = SF_CDF; return 0; }
        if (f <= u1) { bracketed = 1; break; }
        lo = (lo < 0.0) ? 2.0 * lo : lo - 1.0;
        if (!isfinite(lo)) { *fc = SF_INVERSE_CDF; return 0; }
    }
    if (!bracketed) { *fc = SF_INVERSE_CDF; return 0; }
    for (int it = 0; it < 48; ++it) {
        double mid = 0.5 * (lo + hi);
        if (fabs(mid - root) > radius) f = mid < root ? 0.0 : 1.0;
        else if (!o_visible_cdf(mid, slope_i, q, &f)) { *fc = SF_CDF; return 0; }
        if (f < u1) lo = mid; else hi = mid;
    }
    *slope_x = 0.5 * (lo + hi);
    return 1;
}

}  // namespace
}  // namespace clr
