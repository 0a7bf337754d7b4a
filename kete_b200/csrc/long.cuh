// long.cuh -- system integration without SPK perturbers: propagate_n_body_vec
// (kete_core/propagation/mod.rs:142-237) with vec_accel (acceleration.rs:197-249).
//
// The nine massive bodies of SIMPLE_PLANETS (Sun, Mercury, Venus, Earth-Moon barycentre,
// Mars to Neptune; gravity.rs:137-153) are integrated together with a batch of test
// particles by ONE Radau integration over all their coordinates: the step size and the
// convergence test take the maximum over the whole system (radau.rs:317-346 on a DVector).
// A thread block integrates one batch, one thread per body; each force evaluation is
// block-collective (the massive bodies' predicted states go through shared memory), and the
// convergence and step-size maxima are block reductions, so every thread takes the same
// decisions.  Every body feels every massive body but itself; the comet / dust model acts
// relative to the Sun on the batch's test particles after the first, as the reference's
// `idx > n_massive` (acceleration.rs:239-240) has it.  Each corrector starts from the
// predicted b (predict_b_row) and the integration runs in the frame the massive states are
// given in (heliocentric at the start epoch); results are relative to the Sun's final state.
#pragma once
#include "common.cuh"
#include "forces.cuh"
#include "internal.h"
#include "radau.cuh"

namespace kb {

constexpr int LONG_MASSIVE = 9;

// The largest v of a warp's lanes.
__device__ __forceinline__ double warp_max(double v) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

__device__ __forceinline__ double long_block_max(double v, double* s_red) {
    v = warp_max(v);
    const int warp = threadIdx.x >> 5;
    __syncthreads();  // s_red free from the previous reduction
    if ((threadIdx.x & 31) == 0) s_red[warp] = v;
    __syncthreads();
    double m = s_red[0];
    for (int w = 1; w < (int)(blockDim.x >> 5); ++w) m = fmax(m, s_red[w]);
    return m;
}

// GravParams::add_acceleration (gravity.rs:171-216) of a massive body on a body at relative
// position rp / velocity rv, into w: the Newtonian part, and the relativistic and J2 terms that
// the Sun and Jupiter add to it.
__device__ __forceinline__ void long_newton(double mass, const double rp[3], double w[3], double& ir,
                                            double& ir3) {
    const double r2 = rp[0] * rp[0] + rp[1] * rp[1] + rp[2] * rp[2];
    ir = rsqrt(r2);
    ir3 = ir * ir * ir;
    const double kk = mass * ir3;
    w[0] -= rp[0] * kk;
    w[1] -= rp[1] * kk;
    w[2] -= rp[2] * kk;
}

__device__ __forceinline__ void long_sun_jupiter(double mass, double radius, bool jupiter,
                                                 const double rp[3], const double rv[3], double ir,
                                                 double ir3, double w[3]) {
    const double r_v = 4.0 * (rp[0] * rv[0] + rp[1] * rv[1] + rp[2] * rv[2]);
    const double rel_v2 = rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2];
    const double gr_const = mass * C_AU_PER_DAY_INV_SQUARED * ir3;
    const double c = 4. * mass * ir - rel_v2;
#pragma unroll
    for (int i = 0; i < 3; ++i) w[i] += gr_const * (c * rp[i] + r_v * rv[i]);
    const double rc = c_tab.rot_c, rs = c_tab.rot_s;
    const double ez = -rs * rp[1] + rc * rp[2];
    const double zr = ez * ir;
    const double z_squared = 5.0 * (zr * zr);
    const double rr = radius * ir;
    const double coef = 1.5 * (jupiter ? JUPITER_J2 : SUN_J2) * mass * (rr * rr) * ir3;
    const double ey = rc * rp[1] + rs * rp[2];
    const double jx = rp[0] * coef * (z_squared - 1.0);
    const double jy = ey * coef * (z_squared - 1.0);
    const double jz = ez * coef * (z_squared - 3.0);
    w[0] += jx;
    w[1] += rc * jy - rs * jz;
    w[2] += rs * jy + rc * jz;
}

__device__ __forceinline__ void long_pair(int k, const double rp[3], const double rv[3], double w[3]) {
    const int kind = c_tab.simple_kind[k];
    double ir, ir3;
    long_newton(c_tab.simple_mass[k], rp, w, ir, ir3);
    if (kind == FK_SUN || kind == FK_JUPITER)
        long_sun_jupiter(c_tab.simple_mass[k], c_tab.simple_radius[k], kind == FK_JUPITER, rp, rv, ir,
                         ir3, w);
}

// Block-collective vec_accel at one evaluation point: every thread passes its body's
// point; the acceleration of active bodies lands in out.  Returns ST_IMPACT for the whole
// block when an exact evaluation finds a body within a massive body's radius.
__device__ __forceinline__ int long_eval(bool exact, int body, int m, const double xe[3],
                                         const double ve[3], const NonGrav& ng, double* s_m,
                                         double out[3]) {
    __syncthreads();  // the previous evaluation's reads of s_m are done
    if (body < LONG_MASSIVE) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            s_m[6 * body + c] = xe[c];
            s_m[6 * body + 3 + c] = ve[c];
        }
    }
    __syncthreads();
    int hit = 0;
    double acc[3] = {0.0, 0.0, 0.0};
    if (body < m) {
        for (int k = 0; k < LONG_MASSIVE; ++k) {
            if (k == body) continue;
            const double rp[3] = {xe[0] - s_m[6 * k], xe[1] - s_m[6 * k + 1], xe[2] - s_m[6 * k + 2]};
            const double rv[3] = {ve[0] - s_m[6 * k + 3], ve[1] - s_m[6 * k + 4], ve[2] - s_m[6 * k + 5]};
            if (exact && norm3(rp[0], rp[1], rp[2]) <= c_tab.simple_radius[k]) hit = 1;
            double w[3] = {0.0, 0.0, 0.0};
            long_pair(k, rp, rv, w);
            if (c_tab.simple_naif[k] == 10 && body > LONG_MASSIVE && ng.kind != 0) {
                const double3 na = nongrav_accel(ng, make_double3(rp[0], rp[1], rp[2]),
                                                 make_double3(rv[0], rv[1], rv[2]));
                w[0] += na.x;
                w[1] += na.y;
                w[2] += na.z;
            }
            acc[0] += w[0];
            acc[1] += w[1];
            acc[2] += w[2];
        }
    }
    out[0] = acc[0];
    out[1] = acc[1];
    out[2] = acc[2];
    return __syncthreads_or(hit) ? ST_IMPACT : ST_OK;
}

__global__ void __launch_bounds__(64) nbody_long_kernel(LongArgs a) {
    __shared__ double s_m[6 * LONG_MASSIVE];
    __shared__ double s_red[2];
    const int body = threadIdx.x;
    const int64_t i0 = (int64_t)blockIdx.x * a.batch;
    const int64_t rem = a.n - i0;
    const int nb = (int)(rem < a.batch ? rem : a.batch);
    const int m = LONG_MASSIVE + nb;
    const bool active = body < m;
    const int64_t obj = body >= LONG_MASSIVE ? i0 + (body - LONG_MASSIVE) : -1;
    const int64_t n = a.n;

    double x[3] = {0, 0, 0}, v[3] = {0, 0, 0}, acc[3] = {0, 0, 0};
    NonGrav ng;
    ng.base = nullptr;
    ng.stride = n;
    ng.kind = 0;
    if (body < LONG_MASSIVE) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            x[c] = a.planets[6 * body + c];
            v[c] = a.planets[6 * body + 3 + c];
        }
    } else if (active) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            x[c] = a.pos[c * n + obj];
            v[c] = a.vel[c * n + obj];
        }
        if (a.nongrav) {
            ng.base = a.nongrav + obj;
            ng.kind = (int)a.nongrav[obj];
        }
    }
    double b[3][7], g[3][7];
#pragma unroll
    for (int c = 0; c < 3; ++c)
#pragma unroll
        for (int k = 0; k < 7; ++k) b[c][k] = g[c][k] = 0.0;

    int rc = ST_OK;
    if (a.planet_status) {  // massive states read from the SPK on the device
        int bad = 0;
        if (body < LONG_MASSIVE && a.planet_status[body] != ST_OK) bad = 1;
        if (__syncthreads_or(bad)) rc = ST_DAF_LIMITS;
    }
    const double tf = a.jd1;
    double t = a.jd0;
    if (rc == ST_OK) rc = long_eval(true, body, m, x, v, ng, s_m, acc);
    if (rc == ST_OK && !(fabs(tf - t) < 1e-10)) {
        double h = copysign(0.1, tf - t), h_prev = 0.0;
        bool predict = false;
        int failures = 0;
        rc = ST_TIMEOUT;
        for (int loop = 0; loop < a.max_loops; ++loop) {
            if (fabs(t - tf) <= fabs(h)) h = tf - t;
            if (predict) {
#pragma unroll
                for (int c = 0; c < 3; ++c) predict_b_row(b[c], h / h_prev);
            }
            bool converged = false;
            int erc = ST_OK;
            double next_h = h;
            const double h2 = h * h;
            for (int iter = 0; iter < 10 && !converged; ++iter) {
                double b6_old[3] = {b[0][6], b[1][6], b[2][6]};
                double ev[3] = {acc[0], acc[1], acc[2]};
#pragma unroll
                for (int j = 1; j < 8; ++j) {
                    const double f = c_tab.spacing[j];
                    double xs[3], vs[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        double bw = 0.0, bu = 0.0;
#pragma unroll
                        for (int k = 0; k < 7; ++k) {
                            bw += c_tab.w_pow[j][k] * b[c][k];
                            bu += c_tab.u_pow[j][k] * b[c][k];
                        }
                        xs[c] = x[c] + f * v[c] * h + c_tab.frac2[j] * h2 * (acc[c] / 2.0 + bw);
                        vs[c] = v[c] + f * h * (acc[c] + bu);
                    }
                    long_eval(false, body, m, xs, vs, ng, s_m, ev);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        double gk = (ev[c] - acc[c]) * c_tab.inv_frac[j];
#pragma unroll
                        for (int z = 1; z < 7; ++z)
                            if (z < j) gk = (gk - g[c][z - 1]) * c_tab.inv_diff[j][z];
#pragma unroll
                        for (int k = 0; k < 7; ++k)
                            if (k == j - 1) g[c][k] = gk;
                    }
                }
#pragma unroll
                for (int c = 0; c < 3; ++c)
#pragma unroll
                    for (int jj = 0; jj < 7; ++jj) {
                        double s2 = g[c][jj];
#pragma unroll
                        for (int k = jj + 1; k < 7; ++k) s2 += c_tab.c[k][jj] * g[c][k];
                        b[c][jj] = s2;
                    }
                double ratio = 0.0, fem = 0.0, mb6 = 0.0;
                if (active) {
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const double fe = fabs(ev[c]) + 1e-6;
                        ratio = fmax(ratio, fabs(b[c][6] - b6_old[c]) / fe);
                        fem = fmax(fem, fe);
                        mb6 = fmax(mb6, fabs(b[c][6]));
                    }
                }
                if (long_block_max(ratio, s_red) < 1e-14) {
                    const double fem_max = long_block_max(fem, s_red);
                    const double b6_max = long_block_max(mb6, s_red);
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        double dw = 0.0, du = 0.0;
#pragma unroll
                        for (int k = 0; k < 7; ++k) {
                            dw += b[c][k] * c_tab.w[k];
                            du += b[c][k] * c_tab.u[k];
                        }
                        x[c] += v[c] * h + h2 * (acc[c] * 0.5 + dw);
                        v[c] += h * (acc[c] + du);
                    }
                    t += h;
                    erc = long_eval(true, body, m, x, v, ng, s_m, acc);
                    next_h = h * clampd(pow(1e-6 * fem_max / b6_max, 1.0 / 7.0), 0.25, 4.0);
                    converged = true;
                }
            }
            if (erc != ST_OK) {
                rc = erc;
                break;
            }
            if (converged) {
                h_prev = h;
                predict = true;
                h = next_h;
                if (fabs(t - tf) < 1e-12) {
                    rc = ST_OK;
                    break;
                }
                failures = 0;
            } else {
                predict = false;
                failures += 1;
                h *= 0.7;
                if (failures > 10) {
                    rc = ST_CONVERGENCE;
                    break;
                }
            }
            if (fabs(h) < 0.005) h = copysign(0.005, h);
        }
    }
    // results relative to the Sun's final state
    __syncthreads();
    if (body == 0) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            s_m[c] = x[c];
            s_m[3 + c] = v[c];
        }
    }
    __syncthreads();
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    if (obj >= 0 && active) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            a.out_pos[c * n + obj] = rc == ST_OK ? x[c] - s_m[c] : nan;
            a.out_vel[c * n + obj] = rc == ST_OK ? v[c] - s_m[3 + c] : nan;
        }
        a.status[obj] = rc;
    }
    if (a.out_planets && blockIdx.x == gridDim.x - 1 && body < LONG_MASSIVE) {
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            a.out_planets[6 * body + c] = rc == ST_OK ? x[c] - s_m[c] : nan;
            a.out_planets[6 * body + 3 + c] = rc == ST_OK ? v[c] - s_m[3 + c] : nan;
        }
    }
}

// -------------------------------------------------------------------------------------------
// The same integration with the seven corrector nodes, the bodies and the massive bodies' terms
// in parallel (batches of up to 23 test particles, 32 bodies with the massive ones).
//
// What bounds it is the latency of one corrector iteration: a batch is one chain of steps, and
// every body waits for all.  The points (node, body) of an iteration lie densely over the lanes,
// and three warps share each 32 of them (three massive bodies each, their constants operands, the
// Sun's and Jupiter's longer terms in two different ones).  The terms go through shared memory to
// a thread per (point, coordinate) that adds them in the list's order: nbody_long_kernel's sums
// to the bit.  A thread per (coordinate, body) holds its state and b in registers and forms the
// divided differences, b and the next points; LP_SETS sets of warps do so for the same bodies,
// each for its share of the nodes' points, as a lone warp issues FP64 at half the rate that
// several reach.  The next step's length is formed by a warp of its own during the exact
// evaluation.
// 200 batches of 10 over ten years (1062 steps, 5574 iterations): 19.2 ms, on 52 of 148 SMs two
// blocks; 130 batches 13.3 ms, one batch 11.5 ms.  A warp per node whose lanes went through the
// nine pairs took 28.8 ms (13,900 instructions an iteration against 8,500, 23% of the FP64 pipe against 31%).
// NG: with the comet model, whose call costs the kernel 1.8 KB of spills, kept out of the build
// without (46.2 ms; 58.8 with the model's term in the Sun's warps, 50.6 for a warp per node).
// -------------------------------------------------------------------------------------------
constexpr int LP_BODIES = 32;
constexpr int LP_SUBS = 3;
constexpr int LP_SETS = 4;
constexpr int LP_NARROW = 480, LP_WIDE = 7 * LP_BODIES * LP_SUBS;  // threads of the two builds
constexpr int LP_TERMS = 7;     // the first three bodies' sum, then a term each
constexpr int LP_NG_TERMS = 3;  // with comets: the third body in its place; the Sun, Mercury, comet

// doubles of shared memory for m bodies: the points' states, terms and accelerations, |b6|
__host__ __device__ constexpr int long_points_doubles(int m, bool ng) {
    return 7 * m * (6 + 3 * (LP_TERMS + (ng ? LP_NG_TERMS : 0)) + 3) + 3 * m;
}
__host__ __device__ constexpr int long_points_threads(int m) {
    return LP_SUBS * 32 * ((7 * m + 31) / 32);
}

// Massive body K's term at point p (x in xe, body `body`, the node's massive bodies from column
// p0 of X).
template <int K, bool EXACT>
__device__ __forceinline__ void long_term(const double* X, int P, int p, int p0, int body,
                                          const double xe[3], int& hit, double w[3]) {
    double rp[3], ir, ir3;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        rp[c] = xe[c] - X[c * P + p0 + K];
        w[c] = 0.0;
    }
    const double mass = c_tab.simple_mass[K];
    long_newton(mass, rp, w, ir, ir3);
    if (K == 0 || K == 5) {  // the Sun and Jupiter (simple_kind)
        double rv[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) rv[c] = X[(3 + c) * P + p] - X[(3 + c) * P + p0 + K];
        long_sun_jupiter(mass, c_tab.simple_radius[K], K == 5, rp, rv, ir, ir3, w);
    }
    if (EXACT && K != body && norm3(rp[0], rp[1], rp[2]) <= c_tab.simple_radius[K]) hit = 1;
#pragma unroll
    for (int c = 0; c < 3; ++c) w[c] = K == body ? 0.0 : w[c];
}

template <bool EXACT, bool NG>
__device__ __forceinline__ int long_terms(int sub, const double* X, double* W, int P, int p, int p0,
                                          int body, const NonGrav& ng) {
    double xe[3], w[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) xe[c] = X[c * P + p];
    int hit = 0;
    auto store = [&](int slot) {
#pragma unroll
        for (int c = 0; c < 3; ++c) W[(3 * slot + c) * P + p] = w[c];
    };
    if (sub == 0) {
        double s[3];
        long_term<0, EXACT>(X, P, p, p0, body, xe, hit, s);
        if (NG) {  // the comet term comes in between
#pragma unroll
            for (int c = 0; c < 3; ++c) W[(3 * LP_TERMS + c) * P + p] = s[c];
#pragma unroll
            for (int c = 0; c < 3; ++c) s[c] = 0.0;
        }
        long_term<1, EXACT>(X, P, p, p0, body, xe, hit, w);
        if (NG) {
#pragma unroll
            for (int c = 0; c < 3; ++c) W[(3 * LP_TERMS + 3 + c) * P + p] = w[c];
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) s[c] += w[c];
        long_term<2, EXACT>(X, P, p, p0, body, xe, hit, w);
#pragma unroll
        for (int c = 0; c < 3; ++c) w[c] = NG ? w[c] : s[c] + w[c];
        store(0);
    } else if (sub == 1) {
        long_term<5, EXACT>(X, P, p, p0, body, xe, hit, w);
        store(3);
        long_term<3, EXACT>(X, P, p, p0, body, xe, hit, w);
        store(1);
        long_term<4, EXACT>(X, P, p, p0, body, xe, hit, w);
        store(2);
    } else {
        if (NG && ng.kind != 0) {
            const double3 rp = make_double3(xe[0] - X[p0], xe[1] - X[P + p0], xe[2] - X[2 * P + p0]);
            const double3 rv = make_double3(X[3 * P + p] - X[3 * P + p0], X[4 * P + p] - X[4 * P + p0],
                                            X[5 * P + p] - X[5 * P + p0]);
            const double3 na = ng.kind == 1 && ng.p(9) == 0.0 ? nongrav_terms<false>(ng, rp, rv)
                                                              : nongrav_accel(ng, rp, rv);
            W[(3 * LP_TERMS + 6) * P + p] = na.x;
            W[(3 * LP_TERMS + 7) * P + p] = na.y;
            W[(3 * LP_TERMS + 8) * P + p] = na.z;
        }
        long_term<6, EXACT>(X, P, p, p0, body, xe, hit, w);
        store(4);
        long_term<7, EXACT>(X, P, p, p0, body, xe, hit, w);
        store(5);
        long_term<8, EXACT>(X, P, p, p0, body, xe, hit, w);
        store(6);
    }
    return hit;
}

// Component c of the acceleration at point p (comet: the point's body has a comet term).
template <bool NG>
__device__ __forceinline__ double long_sum(const double* W, int P, int p, int c, bool comet) {
    double acc = W[c * P + p];
    if (NG) {
        double w = W[(3 * LP_TERMS + c) * P + p];
        if (comet) w += W[(3 * LP_TERMS + 6 + c) * P + p];
        acc = (w + W[(3 * LP_TERMS + 3 + c) * P + p]) + acc;
    }
#pragma unroll
    for (int k = 1; k < LP_TERMS; ++k) acc += W[(3 * k + c) * P + p];
    return acc;
}

// THREADS: the largest block; MINB blocks of it share an SM (64 registers a thread: batches of up
// to 13); NG: some particles have a non-gravitational model.
template <int THREADS, int MINB, bool NG>
__global__ void __launch_bounds__(THREADS, MINB) nbody_long_points_kernel(LongArgs a) {
    extern __shared__ __align__(16) double s_long[];
    __shared__ double s_sun[6], s_next;
    __shared__ int s_hit, s_bad;
    const int64_t i0 = (int64_t)blockIdx.x * a.batch, n = a.n;
    const int64_t rem = n - i0;
    const int m = LONG_MASSIVE + (int)(rem < a.batch ? rem : a.batch);
    const int P = 7 * m, C = 3 * m;
    double* X = s_long;
    double* W = X + 6 * P;
    double* E = W + 3 * (LP_TERMS + (NG ? LP_NG_TERMS : 0)) * P;
    double* s_b6 = E + 3 * P;
    const int t0 = threadIdx.x, warp = t0 >> 5, lane = t0 & 31;
    // this thread's point and share of its terms
    const int wp = blockDim.x / (32 * LP_SUBS);
    const int sub = warp / wp, p = t0 - sub * wp * 32;
    const bool point = p < P;
    const int node = p / m, body = p - node * m, p0 = node * m;
    // the (coordinate, body) this thread forms g, b and the state update for
    const int tw = (C + 31) / 32, set = warp / tw;
    const int ti = t0 - set * tw * 32;
    const bool task = set < LP_SETS && ti < C;
    const int tc = task ? ti / m : 0, tb = task ? ti - tc * m : 0;
    // the warps of the exact evaluation (points 0 .. m - 1 and the first set)
    const bool exact_warp = warp < tw || p < 32;
    const int exact_threads = 32 * (tw + LP_SUBS - 1);
    auto exact_sync = [&]() { asm volatile("bar.sync 1, %0;" ::"r"(exact_threads) : "memory"); };

    NonGrav ng;
    ng.base = nullptr;
    ng.stride = n;
    ng.kind = 0;
    if (NG && point && body > LONG_MASSIVE) {
        ng.base = a.nongrav + i0 + (body - LONG_MASSIVE);
        ng.kind = (int)*ng.base;
    }
    double x = 0.0, v = 0.0, ac = 0.0, b[7];
#pragma unroll
    for (int k = 0; k < 7; ++k) b[k] = 0.0;
    if (task) {
        if (tb < LONG_MASSIVE) {
            x = a.planets[6 * tb + tc];
            v = a.planets[6 * tb + 3 + tc];
        } else {
            x = a.pos[tc * n + i0 + (tb - LONG_MASSIVE)];
            v = a.vel[tc * n + i0 + (tb - LONG_MASSIVE)];
        }
    }
    if (t0 == 0) s_hit = s_bad = 0;
    __syncthreads();
    // massive states read from the SPK on the device
    if (a.planet_status && t0 < LONG_MASSIVE && a.planet_status[t0] != ST_OK) s_bad = 1;
    // exact evaluation of the current state into E's columns 0 .. m - 1, by exact_warp
    auto exact = [&]() {
        if (task && set == 0) {
            X[tc * P + tb] = x;
            X[(3 + tc) * P + tb] = v;
        }
        exact_sync();
        if (p < m && long_terms<true, NG>(sub, X, W, P, p, 0, body, ng)) s_hit = 1;
        exact_sync();
        if (p < m) E[sub * P + p] = long_sum<NG>(W, P, p, sub, ng.kind != 0);
    };
    if (exact_warp) exact();
    __syncthreads();
    ac = E[tc * P + tb];
    int rc = s_bad ? ST_DAF_LIMITS : (s_hit ? ST_IMPACT : ST_OK);
    const double tf = a.jd1;
    double t = a.jd0;
    if (rc == ST_OK && !(fabs(tf - t) < 1e-10)) {
        double h = copysign(0.1, tf - t), h_prev = 0.0;
        bool predict = false;
        int failures = 0;
        rc = ST_TIMEOUT;
        for (int loop = 0; loop < a.max_loops; ++loop) {
            if (fabs(t - tf) <= fabs(h)) h = tf - t;
            if (predict && task) predict_b_row(b, h / h_prev);
            bool converged = false;
            for (int iter = 0; iter < 10 && !converged; ++iter) {
                if (task) {
                    const double h2 = h * h;
                    auto next_point = [&](int j) {
                        const double f = c_tab.spacing[j];
                        double bw = 0.0, bu = 0.0;
#pragma unroll
                        for (int k = 0; k < 7; ++k) {
                            bw += c_tab.w_pow[j][k] * b[k];
                            bu += c_tab.u_pow[j][k] * b[k];
                        }
                        const int q = (j - 1) * m + tb;
                        X[tc * P + q] = x + f * v * h + c_tab.frac2[j] * h2 * (ac / 2.0 + bw);
                        X[(3 + tc) * P + q] = v + f * h * (ac + bu);
                    };
#pragma unroll
                    for (int j = 1; j < 8; ++j)
                        if (set == (j - 1) * LP_SETS / 7) next_point(j);
                }
                __syncthreads();
                if (point) long_terms<false, NG>(sub, X, W, P, p, p0, body, ng);
                __syncthreads();
                if (point) E[sub * P + p] = long_sum<NG>(W, P, p, sub, ng.kind != 0);
                __syncthreads();
                int above = 0;
                if (task) {
                    double g[7], fe = 0.0;
#pragma unroll
                    for (int jj = 1; jj < 8; ++jj) {
                        const double ev = E[tc * P + (jj - 1) * m + tb];
                        double gk = (ev - ac) * c_tab.inv_frac[jj];
#pragma unroll
                        for (int z = 1; z < 7; ++z)
                            if (z < jj) gk = (gk - g[z - 1]) * c_tab.inv_diff[jj][z];
                        g[jj - 1] = gk;
                        // the convergence test reads the last node's evaluation
                        if (jj == 7) fe = fabs(ev) + 1e-6;
                    }
                    const double b6_old = b[6];
#pragma unroll
                    for (int jj = 0; jj < 7; ++jj) {
                        double s2 = g[jj];
#pragma unroll
                        for (int k = jj + 1; k < 7; ++k) s2 += c_tab.c[k][jj] * g[k];
                        b[jj] = s2;
                    }
                    above = fabs(b[6] - b6_old) >= 1e-14 * fe;
                    if (set == 0) s_b6[ti] = fabs(b[6]);
                }
                if (!__syncthreads_or(above)) {
                    if (task) {
                        double dw = 0.0, du = 0.0;
#pragma unroll
                        for (int k = 0; k < 7; ++k) {
                            dw += b[k] * c_tab.w[k];
                            du += b[k] * c_tab.u[k];
                        }
                        x = x + (v * h + (h * h) * (ac * 0.5 + dw));
                        v = v + h * (ac + du);
                    }
                    t += h;
                    // the next step from max(|a| + 1e-6) at the last node and max|b6|
                    if (warp == LP_SUBS * wp - 1) {
                        double fem = 0.0, mb6 = 0.0;
                        for (int q = lane; q < C; q += 32) {
                            fem = fmax(fem, fabs(E[(q / m) * P + 6 * m + q % m]) + 1e-6);
                            mb6 = fmax(mb6, s_b6[q]);
                        }
                        fem = warp_max(fem);
                        mb6 = warp_max(mb6);
                        if (lane == 0)
                            s_next = h * clampd(pow(1e-6 * fem / mb6, 1.0 / 7.0), 0.25, 4.0);
                    }
                    if (exact_warp) exact();
                    __syncthreads();
                    ac = E[tc * P + tb];
                    converged = true;
                }
            }
            if (s_hit) {
                rc = ST_IMPACT;
                break;
            }
            if (converged) {
                h_prev = h;
                predict = true;
                h = s_next;
                if (fabs(t - tf) < 1e-12) {
                    rc = ST_OK;
                    break;
                }
                failures = 0;
            } else {
                predict = false;
                failures += 1;
                h *= 0.7;
                if (failures > 10) {
                    rc = ST_CONVERGENCE;
                    break;
                }
            }
            if (fabs(h) < 0.005) h = copysign(0.005, h);
        }
    }
    // results relative to the Sun's final state
    if (task && tb == 0) {
        s_sun[tc] = x;
        s_sun[3 + tc] = v;
    }
    __syncthreads();
    if (!task || set != 0) return;
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
    const double ox = rc == ST_OK ? x - s_sun[tc] : nan;
    const double ov = rc == ST_OK ? v - s_sun[3 + tc] : nan;
    if (tb >= LONG_MASSIVE) {
        const int64_t obj = i0 + (tb - LONG_MASSIVE);
        a.out_pos[tc * n + obj] = ox;
        a.out_vel[tc * n + obj] = ov;
        if (tc == 0) a.status[obj] = rc;
    } else if (a.out_planets && blockIdx.x == gridDim.x - 1) {
        a.out_planets[6 * tb + tc] = ox;
        a.out_planets[6 * tb + 3 + tc] = ov;
    }
}

}  // namespace kb
