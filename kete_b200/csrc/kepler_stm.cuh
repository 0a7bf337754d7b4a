// kepler_stm.cuh -- two-body state-transition matrices and covariance propagation.
//
// kete's compute_stm / propagate_covariance (src/kete/state_transition.py:8-59,
// kete_core/propagation/state_transition.rs:52-122) integrate the variational equations
// with RK4(5) and carry three defects: the acceleration Jacobian is off by a factor -1/2
// (acceleration.rs:267-290), the scaled-time equations use the unscaled GM
// (state_transition.rs:6-47 with acceleration.rs:66-80), and the matrix comes back
// transposed (state_transition.rs:86-121).  Here the matrix is d(p1, v1)/d(p0, v0) of the
// closed-form two-body solution itself: the final state is analytic_2_body's (kepler.rs:
// 254-297, the same interval halving), and each closed-form step is differentiated in
// closed form.  The universal anomaly's derivative comes from the implicit function
// theorem on the Kepler equation, ds = -dF / F'(s), at the anomaly of the unreduced
// equation (the elliptic solve reduces time modulo the period, which moves with the
// state).  Leaf Jacobians chain in the order the steps run.
#pragma once
#include "common.cuh"
#include "kepler.cuh"

namespace kb {

// g0 .. g5 of the universal functions at anomaly s (g_k = s^k c_k(z), z = beta s^2, Stumpff
// functions), given g1 and g2 of the same beta.  For |z| < 0.1 g3 .. g5 come from the
// alternating series, which stays accurate where (s - g1) / beta and its successors cancel, and
// g1 and g2 from those by g_k = s^k / k! - beta g_(k+2): the solver's hyperbolic (1 - cosh) / beta
// cancels too (at perihelion, beta = -3e-8, an eighth of a day: 3e-10 of a block of the matrix).
struct Universal {
    double g0, g1, g2, g3, g4, g5;
};
__device__ __forceinline__ Universal universal_functions(double s, double beta, double g1, double g2) {
    Universal u;
    u.g0 = 1.0 - beta * g2;
    u.g1 = g1;
    u.g2 = g2;
    const double z = beta * s * s, s2 = s * s;
    if (fabs(z) < 0.1) {
        // c_k(z) = sum_j (-z)^j / (2j + k)!, eight terms (next term below 1e-24)
        double c3 = 0.0, c4 = 0.0, c5 = 0.0, zp = 1.0;
        double f3 = 6.0, f4 = 24.0, f5 = 120.0;  // 3!, 4!, 5!
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            c3 += zp * (1.0 / f3);
            c4 += zp * (1.0 / f4);
            c5 += zp * (1.0 / f5);
            zp *= -z;
            f3 *= (double)((2 * j + 4) * (2 * j + 5));
            f4 *= (double)((2 * j + 5) * (2 * j + 6));
            f5 *= (double)((2 * j + 6) * (2 * j + 7));
        }
        u.g3 = s2 * s * c3;
        u.g4 = s2 * s2 * c4;
        u.g5 = s2 * s2 * s * c5;
        u.g2 = 0.5 * s2 - beta * u.g4;
        u.g1 = s - beta * u.g3;
        u.g0 = 1.0 - beta * u.g2;
        return u;
    }
    const double ib = 1.0 / beta;
    u.g3 = (s - g1) * ib;
    u.g4 = (0.5 * s2 - g2) * ib;
    u.g5 = (s2 * s * (1.0 / 6.0) - u.g3) * ib;
    return u;
}

// One closed-form step of dt from (p, v), in place, with its 6x6 Jacobian J (row-major,
// rows d(p1, v1), columns d(p0, v0)).  Values follow two_body_leaf exactly.
//
// p1 = f p + g v and v1 = f' p + g' v with scalars f, g, f', g' of r0, sigma = p . v and beta
// alone, so each block of J is a multiple of the identity plus outer products of p and v: three
// partial derivatives of four scalars give all 36 entries (dual numbers in six directions took
// some 1,500 operations and 166 registers).  With d g_k / ds = g_(k-1) and d g_k / dbeta =
// (k g_(k+2) - s g_(k+1)) / 2, and ds = -dF / F'(s) from the Kepler equation F = r0 g1 +
// sigma g2 + mu g3 = dt.
__device__ __forceinline__ int two_body_leaf_stm(double dt, double p[3], double v[3], double mu,
                                                 double J[36]) {
    const double r0 = norm3(p[0], p[1], p[2]);
    const double v0 = norm3(v[0], v[1], v[2]);
    const double rv0 = p[0] * v[0] + p[1] * v[1] + p[2] * v[2];
    KeplerStep k;
    if (solve_kepler_universal(dt, r0, v0, rv0, k, mu) != ST_OK) return ST_CONVERGENCE;
    const double beta = k.beta;
    // the anomaly of the unreduced equation: whole revolutions added back
    double s = k.s;
    if (beta >= PARABOLIC_BETA) {
        const double period = mu * powi<-3>(k.b_sqrt) * TAU;
        s += rint((dt - fmod_period(dt, period)) / period) * TAU / k.b_sqrt;
    }
    const Universal u = universal_functions(s, beta, k.g1, k.g2);
    const double g1b = 0.5 * (u.g3 - s * u.g2), g2b = u.g4 - 0.5 * s * u.g3,
                 g3b = 0.5 * (3.0 * u.g5 - s * u.g4), g0b = -0.5 * s * u.g1;
    const double r = r0 * u.g0 + rv0 * u.g1 + mu * u.g2;
    const double ir = 1.0 / r, ir0 = 1.0 / r0;
    // the anomaly's partials in (r0, sigma, beta)
    const double sp[3] = {-u.g1 * ir, -u.g2 * ir, -(r0 * g1b + rv0 * g2b + mu * g3b) * ir};
    const double gs = r0 * u.g0 + rv0 * u.g1;                             // dg / ds
    const double rs = (mu - r0 * beta) * u.g1 + rv0 * u.g0;               // dr / ds
    const double rd[3] = {u.g0, u.g1, r0 * g0b + rv0 * g1b + mu * g2b};   // dr at fixed s
    const double gd_[3] = {u.g1, u.g2, r0 * g1b + rv0 * g2b};             // dg at fixed s
    const double g1d[3] = {0.0, 0.0, g1b}, g2d[3] = {0.0, 0.0, g2b};
    const double f = 1.0 - mu * ir0 * u.g2, g = r0 * u.g1 + rv0 * u.g2;
    const double fd = -mu * ir * ir0 * u.g1, gd = 1.0 - mu * ir * u.g2;
    double df[3], dg[3], dfd[3], dgd[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double t1 = u.g0 * sp[q] + g1d[q], t2 = u.g1 * sp[q] + g2d[q];  // total dg1, dg2
        const double tr = rs * sp[q] + rd[q];                                 // total dr
        df[q] = -mu * ir0 * t2;
        dg[q] = gs * sp[q] + gd_[q];
        dfd[q] = -mu * ir * ir0 * t1 - fd * ir * tr;
        dgd[q] = -mu * ir * (t2 - u.g2 * ir * tr);
    }
    df[0] += mu * ir0 * ir0 * u.g2;
    dfd[0] -= fd * ir0;
    // to the columns: dr0 = p / r0 dp, dsigma = v dp + p dv, dbeta = -2 mu p / r0^3 dp - 2 v dv
    const double bp = -2.0 * mu * ir0 * ir0 * ir0;
#pragma unroll
    for (int blk = 0; blk < 2; ++blk) {  // rows of p1, then of v1
        const double* da = blk ? dfd : df;
        const double* db = blk ? dgd : dg;
        const double a = blk ? fd : f, b = blk ? gd : g;
        const double app = da[0] * ir0 + bp * da[2], bpp = db[0] * ir0 + bp * db[2];
#pragma unroll
        for (int i = 0; i < 3; ++i) {
            // d/dp: p (app p + da1 v) + v (bpp p + db1 v); d/dv: p (da1 p - 2 da2 v) + v (...)
            const double pp = p[i] * app + v[i] * bpp, pv = p[i] * da[1] + v[i] * db[1];
            const double vv = -2.0 * (p[i] * da[2] + v[i] * db[2]);
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                J[(3 * blk + i) * 6 + c] = (i == c ? a : 0.0) + pp * p[c] + pv * v[c];
                J[(3 * blk + i) * 6 + 3 + c] = (i == c ? b : 0.0) + pv * p[c] + vv * v[c];
            }
        }
    }
    two_body_apply(k, r0, rv0, p, v, mu);
    return ST_OK;
}

// The halved intervals of a step that failed as a whole, leaf Jacobians chained in the order
// they run.
static __device__ __noinline__ int analytic_2_body_stm_halved(double time, double p[3], double v[3],
                                                              double mu, double Phi[36]) {
#pragma unroll
    for (int k = 0; k < 36; ++k) Phi[k] = (k % 7 == 0) ? 1.0 : 0.0;
    return halved_intervals<false>(
        time,
        [&](double dt) {
            double J[36], tmp[36];
            if (two_body_leaf_stm(dt, p, v, mu, J) != ST_OK) return (int)ST_CONVERGENCE;
            for (int r = 0; r < 6; ++r)
                for (int c = 0; c < 6; ++c) {
                    double acc = 0.0;
#pragma unroll
                    for (int k = 0; k < 6; ++k) acc += J[r * 6 + k] * Phi[k * 6 + c];
                    tmp[r * 6 + c] = acc;
                }
            for (int k = 0; k < 36; ++k) Phi[k] = tmp[k];
            return (int)ST_OK;
        },
        [&]() { return two_body_state_ok(p, v); });
}

}  // namespace kb
