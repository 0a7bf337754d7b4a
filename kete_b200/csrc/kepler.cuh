// kepler.cuh -- universal-variable two-body propagation on the device.
//
// Restates kete_core/propagation/kepler.rs:119-297 (g_1, g_2, solve_kepler_universal,
// analytic_2_body) and kete_core/fitting/newton.rs:18-65 (newton_raphson).  The
// reference's recursive interval halving (depth <= 10) becomes an explicit stack of
// pending half-intervals, processed in the same order.  Elliptic steps are solved by a faster
// iteration first (kepler_elliptic); what it does not solve goes the reference's way.
#pragma once
#include "common.cuh"

namespace kb {

constexpr double PARABOLIC_BETA = 1e-10;

// f(x) and f'(x) of the universal Kepler equation as the reference iterates them
// (kepler.rs:189-199, 217-227; its derivative takes g1 without the division by sqrt(|beta|),
// which leaves a linearly converging iteration).
struct KepEq {
    double r0, rv0, beta, b_sqrt, dt;
    bool hyperbolic;
    double mu;  // GM of the central body (GMS in kete)
    // what f and f' need of x: sine (sinh) and cosine (cosh) of b x, and sin(b x / 2)
    struct At {
        double sn, cs, half;
    };
    __device__ __forceinline__ At at(double x) const {
        At o;
        if (!hyperbolic) {
            sincos(b_sqrt * x, &o.sn, &o.cs);
            o.half = sin(b_sqrt * x / 2.0);
        } else {
            o.sn = sinh(b_sqrt * x);
            o.cs = cosh(b_sqrt * x);
            o.half = 0.0;
        }
        return o;
    }
    __device__ __forceinline__ double g1(const At& k) const { return k.sn / b_sqrt; }
    __device__ __forceinline__ double g2(const At& k) const {
        return hyperbolic ? (1.0 - k.cs) / beta : 2.0 * (k.half * k.half) / beta;
    }
    __device__ __forceinline__ double f(double x, const At& k) const {
        const double g1x = g1(k);
        const double g3 = (x - g1x) / beta;
        return r0 * g1x + rv0 * g2(k) + mu * g3 - dt;
    }
    __device__ __forceinline__ double d(const At& k) const {
        const double g3d = (1.0 - k.cs) / beta;
        return r0 * k.cs + rv0 * k.sn + mu * g3d;
    }
};

// newton_raphson (fitting/newton.rs:18-65): two damped half steps per iteration,
// the second reusing f unless |f'| < 1e-3.  At most 100 iterations.  One evaluation of the
// functions at x serves f and f'; g1, g2: at the solution.
__device__ __forceinline__ int newton_steps(const KepEq& q, double start, double atol, double& out,
                                            double& g1, double& g2) {
    double x = start;
    KepEq::At k = q.at(x);
    if (fabs(q.d(k)) < 1e-12) {
        x += 0.1;
        k = q.at(x);
    }
    for (int it = 0; it < 100; ++it) {
        double f_eval = q.f(x, k);
        if (fabs(f_eval) < atol) {
            out = x;
            g1 = q.g1(k);
            g2 = q.g2(k);
            return ST_OK;
        }
        double d_eval = q.d(k);
        if (fabs(d_eval) < 1e-12) return ST_CONVERGENCE;
        if (!isfinite(d_eval) || !isfinite(f_eval)) return ST_CONVERGENCE;
        x -= 0.5 * f_eval / d_eval;
        k = q.at(x);
        d_eval = q.d(k);
        if (fabs(d_eval) < 1e-3) f_eval = q.f(x, k);
        x -= 0.5 * f_eval / d_eval;
        k = q.at(x);
    }
    return ST_CONVERGENCE;
}

static __device__ __noinline__ int newton(const KepEq& q, double start, double atol, double& out,
                                          double& g1, double& g2) {
    return newton_steps(q, start, atol, out, g1, g2);
}

// The elliptic equation by its true derivatives, all of which one sine and cosine give (with
// w = b x: f' = r, f'' = dr/dx, and each further pair is -beta times the one before): a step is
// the fifth-order reversion of the series when it is short, otherwise Laguerre's of degree 5
// (Conway 1986), which converges from anywhere in practice.  Belt orbits over +-1000 days take
// two evaluations, where the reference's iteration takes 8 of three on average and up to 28 (a
// warp waits for its longest); 100,000 of them 55 -> 29 us a call, then bound by the host.
// Ends when |f| < atol or when the step left is so short (its remainder below 1e-17) that the
// new sine and cosine follow from it.  ST_CONVERGENCE: left to the reference's iteration, as
// are near-parabolic orbits whose x mu / beta is so large that the rounding of f reaches atol
// (which values of f pass there, and which intervals are halved, decides the result).
__device__ __forceinline__ int kepler_elliptic(const KepEq& q, double start, double atol,
                                               double& out, double& s, double& c) {
    double x = start;
    const double b = q.b_sqrt, ib = 1.0 / b, ibeta = 1.0 / q.beta;
    if (!(q.mu * fabs(x) * ibeta < 5e3)) return ST_CONVERGENCE;
#pragma unroll 1
    for (int it = 0; it < 12; ++it) {
        sincos(0.5 * (b * x), &s, &c);
        const double sn = 2.0 * s * c, omc = 2.0 * (s * s), cs = 1.0 - omc;
        const double g1 = sn * ib, g2 = omc * ibeta, g3 = (x - g1) * ibeta;
        const double f = q.r0 * g1 + q.rv0 * g2 + q.mu * g3 - q.dt;
        if (fabs(f) < atol) {
            out = x;
            return ST_OK;
        }
        const double f1 = q.r0 * cs + q.rv0 * g1 + q.mu * g2;
        const double f2 = (q.mu - q.r0 * q.beta) * g1 + q.rv0 * cs;
        const double i1 = 1.0 / f1, d1 = f * i1;
        const double k2 = f2 * i1, k3 = ((q.mu - q.r0 * q.beta) * cs - q.rv0 * b * sn) * i1;
        // how far f bends over the step, against its slope
        const double bend = fmax(fmax(fabs(d1 * b), fabs(d1 * k2)), sqrt(fabs(k3)) * fabs(d1));
        double dx;
        if (bend < 0.3) {
            // y = f / f' = x - k2 x^2 / 2 + k3 x^3 / 6 - k4 x^4 / 24 reverted
            const double e2 = 0.5 * k2, e3 = k3 * (1.0 / 6.0), e4 = -q.beta * k2 * (1.0 / 24.0);
            dx = d1 * (1.0 + d1 * (e2 + d1 * (2.0 * e2 * e2 - e3 +
                                              d1 * (5.0 * e2 * (e2 * e2 - e3) + e4))));
        } else {
            const double disc = fabs(16.0 * f1 * f1 - 20.0 * f * f2);
            dx = 5.0 * f / (f1 + copysign(sqrt(disc), f1));
        }
        x -= dx;
        const double w = b * dx;
        if (bend < 5e-4) {
            // rotate by -w / 2: the series' next terms lie below 1e-24
            const double h = -0.5 * w, h2 = h * h;
            const double sh = h * (1.0 - h2 * (1.0 / 6.0) * (1.0 - h2 * 0.05));
            const double ch = 1.0 - 0.5 * h2 * (1.0 - h2 * (1.0 / 12.0));
            const double s0 = s;
            s = s * ch + c * sh;
            c = c * ch - s0 * sh;
            out = x;
            return ST_OK;
        }
        if (!(fabs(w) < 1e3)) break;
    }
    return ST_CONVERGENCE;
}

// dt modulo the period, with fmod's value: the quotient's product is subtracted exactly, so
// only a quotient rounded across an integer needs mending.
__device__ __forceinline__ double fmod_period(double dt, double period) {
    const double n = trunc(dt / period);
    if (!(fabs(n) < 1e9)) return fmod(dt, period);
    double r = fma(-n, period, dt);
    if (r != 0.0 && (r < 0.0) != (dt < 0.0)) r += copysign(period, dt);
    if (fabs(r) >= period) r -= copysign(period, dt);
    return r;
}

// The universal anomaly s of a step and its g1, g2 (g_1, g_2 of kepler.rs:119-150).
struct KeplerStep {
    double s, beta, b_sqrt, g1, g2;
};

// FAST: kepler_elliptic first.  Without, the reference's iteration alone and inline: fewer
// registers, for the force kernels that call it around a step loop (the faster form there cost
// the pooled kernel at 128 registers 156 bytes of spills and 4%).
template <bool FAST = true>
__device__ __forceinline__ int solve_kepler_universal(double dt, double r0, double v0, double rv0,
                                                      KeplerStep& o, double mu = GMS) {
    auto reference = [&](const KepEq& q, double guess) {
        return FAST ? newton(q, guess, 1e-11, o.s, o.g1, o.g2)
                    : newton_steps(q, guess, 1e-11, o.s, o.g1, o.g2);
    };
    const double beta = 2.0 * mu / r0 - powi<2>(v0);
    const double b_sqrt = sqrt(fabs(beta));
    o.beta = beta;
    o.b_sqrt = b_sqrt;
    double s, c;
    if (beta >= PARABOLIC_BETA) {
        const double period = mu * powi<-3>(b_sqrt);
        const double dtm = fmod_period(dt, period * TAU);
        const KepEq q{r0, rv0, beta, b_sqrt, dtm, false, mu};
        const double guess = (1.0 / b_sqrt) * dtm / period;
        if (FAST && kepler_elliptic(q, guess, 1e-11, o.s, s, c) == ST_OK) {
            o.g1 = 2.0 * s * c / b_sqrt;
            o.g2 = 2.0 * (s * s) / beta;
        } else if (reference(q, guess) != ST_OK) {
            return ST_CONVERGENCE;
        }
    } else if (fabs(beta) < PARABOLIC_BETA) {
        const double a0 = -6.0 * dt / mu;
        const double a1 = 6.0 * r0 / mu;
        const double a2 = 3.0 * rv0 / mu;
        const double p = (3.0 * a1 - powi<2>(a2)) / 3.0;
        const double qq = (9.0 * a1 * a2 - 27.0 * a0 - 2.0 * powi<3>(a2)) / 27.0;
        const double w = pow(qq / 2.0 + sqrt(powi<2>(qq) / 4.0 + powi<3>(p) / 27.0), 1.0 / 3.0);
        o.s = w - p / (3.0 * w) - a2 / 3.0;
        o.g1 = o.s;
        o.g2 = powi<2>(o.s) / 2.0;
    } else {
        const KepEq q{r0, rv0, beta, b_sqrt, dt, true, mu};
        // kete's starting point uses its GMS_SQRT literal (kepler.rs:228)
        const double mu_sqrt = mu == GMS ? GMS_SQRT : sqrt(mu);
        if (reference(q, mu_sqrt * fabs(beta) * dt) != ST_OK) return ST_CONVERGENCE;
    }
    return ST_OK;
}

// The f and g update of one closed-form step from its solution (kepler.rs:270-288).
__device__ __forceinline__ void two_body_apply(const KeplerStep& k, double r0, double rv0,
                                               double p[3], double v[3], double mu = GMS) {
    const double g1 = k.g1, g2 = k.g2;
    const double f = 1.0 - mu / r0 * g2;
    const double g = r0 * g1 + rv0 * g2;
    double np[3];
#pragma unroll
    for (int i = 0; i < 3; ++i) np[i] = p[i] * f + v[i] * g;
    const double nr0 = norm3(np[0], np[1], np[2]);
    const double f_dot = -mu / (nr0 * r0) * g1;
    const double g_dot = 1.0 - (mu / nr0) * g2;
#pragma unroll
    for (int i = 0; i < 3; ++i) {
        v[i] = p[i] * f_dot + v[i] * g_dot;
        p[i] = np[i];
    }
}

// One closed-form step; returns ST_CONVERGENCE when the solver fails.
template <bool FAST = true>
__device__ __forceinline__ int two_body_leaf(double time, double p[3], double v[3]) {
    const double r0 = norm3(p[0], p[1], p[2]);
    const double v0 = norm3(v[0], v[1], v[2]);
    const double rv0 = p[0] * v[0] + p[1] * v[1] + p[2] * v[2];
    KeplerStep k;
    if (solve_kepler_universal<FAST>(time, r0, v0, rv0, k) != ST_OK) return ST_CONVERGENCE;
    two_body_apply(k, r0, rv0, p, v);
    return ST_OK;
}

// The reference's interval halving (kepler.rs:254-297), in place: a stack of the remaining
// half-intervals and the depth value their recursive call would receive; WHOLE: from the whole
// step, otherwise from its halves, once it has failed.  step(dt): one closed-form step of the
// caller's state; state_ok(): the state is a number.
template <bool WHOLE, class Step, class Check>
__device__ __forceinline__ int halved_intervals(double time, Step step, Check state_ok) {
    double st_dt[12];
    int st_depth[12];
    st_dt[0] = st_dt[1] = WHOLE ? time : time * 0.5;
    st_depth[0] = st_depth[1] = WHOLE ? 0 : 1;
    int top = WHOLE ? 1 : 2;
    int guard = 0;
    while (top > 0) {
        if (++guard > 4096) return ST_TIMEOUT;
        --top;
        const double dt = st_dt[top];
        int depth = st_depth[top];
        if (depth >= 10) return ST_CONVERGENCE;
        depth += 1;
        if (fabs(dt) < 1e-10) continue;
        if (!state_ok()) return ST_CONVERGENCE;
        if (step(dt) == ST_OK) continue;
        if (top + 2 > 12) return ST_CONVERGENCE;
        st_dt[top] = dt * 0.5;
        st_depth[top] = depth;
        st_dt[top + 1] = 0.5 * dt;
        st_depth[top + 1] = depth;
        top += 2;
    }
    return ST_OK;
}

__device__ __forceinline__ bool two_body_state_ok(const double p[3], const double v[3]) {
    return isfinite(p[0] * v[0] + p[1] * v[1] + p[2] * v[2]);
}

static __device__ __noinline__ int analytic_2_body_halved(double time, double p[3], double v[3]) {
    return halved_intervals<false>(time, [&](double dt) { return two_body_leaf(dt, p, v); },
                                   [&]() { return two_body_state_ok(p, v); });
}

// The same by the reference's iteration alone (solve_kepler_universal<false>).
static __device__ __noinline__ int analytic_2_body_reference(double time, double p[3], double v[3]) {
    return halved_intervals<true>(time, [&](double dt) { return two_body_leaf<false>(dt, p, v); },
                                  [&]() { return two_body_state_ok(p, v); });
}

// analytic_2_body (kepler.rs:254-297), in place: the whole interval at once, then halves.
static __device__ __noinline__ int analytic_2_body(double time, double p[3], double v[3]) {
    if (fabs(time) < 1e-10) return ST_OK;
    if (!two_body_state_ok(p, v)) return ST_CONVERGENCE;
    if (two_body_leaf(time, p, v) == ST_OK) return ST_OK;
    return analytic_2_body_halved(time, p, v);
}

}  // namespace kb
