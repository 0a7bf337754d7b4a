// radau_pool.cuh -- node-parallel Radau (8 lanes per object, as radau_nodes.cuh) whose
// ephemeris records are evaluated by the whole warp as one pool of work.
//
// Every corrector iteration of a step evaluates the force at the same eight times (the
// seven nodes and the step end), and about four fifths of an uncached evaluation is the
// Chebyshev records of the bodies, which depend on the time alone.  Each node therefore keeps
// the bodies' positions (and the Sun's and Jupiter's velocities) at its time in shared memory,
// and only the first iteration of a step needs records.  Those are evaluated by the whole
// warp: an object's eight times by four lanes each when one object of the warp starts a step,
// by two each when two do, every lane its own when more do -- three positions in lockstep, a
// velocity at a time, each result written to its node's column.  (Lanes that took single
// (time, body) pairs from one list, divisions by the body count included, needed 1.3 times the
// instructions of the whole kernel.)
//
// The integration of each object is the one of radau_nodes.cuh with the step-end lane
// (lane 7 evaluates the step end during each corrector iteration and supplies the exact
// evaluation of the accepted step), the predicted corrector start and the compensated state
// update, in the same arithmetic.  Every form in this file (variants 9 and 10 with and without the
// queue, a warp per object) gives an object the same results to the bit; with the planets,
// objects without a non-gravitational model get those of the cached variants 6 to 8
// (radau_nodes.cuh) to the bit but for one in two thousand.  That matters beyond tidiness: the
// corrector's 1e-14 test lies in the rounding noise of b6, so a different rounding anywhere changes
// which steps are retried, and close approaches amplify that from 1e-11 AU to 1e-6 and more.
//
// What bounds it (100,000 objects of the +-5 yr mix, ncu): the L1 data pipe, 72% of the active
// cycles -- about half of its wavefronts are the record loads (each lane reads its own
// coefficients: 4 wavefronts a 16-byte load at the least), the rest the columns and the b and
// node rows -- then fixed-latency FP64 dependencies (2.1 of 8.1 cycles an instruction); the
// FP64 pipe is 33% active.  Replacing the library's rsqrt and pow by shorter chains, merging
// the terms of Sun and Jupiter and scaling the coefficients on the host changed nothing
// (133.5 ms against 132.6 on the million), so the arithmetic stays as it was.  Per warp round
// the instructions fell from 2730 to 2180; a million objects of the mix take 122 ms (171.3
// before, 261 in the form that the library used without tuning), 10,000 of the main belt over a
// year 0.75 ms (1.0).
//
// The kernel carries no general ephemeris evaluation: the host orders the objects whose span
// leaves the fast plan's window after the others and integrates those with a form that has
// it (launch_nodes_ordered).  An out-of-line call makes the caller keep its live registers
// across it, so the centre changes at an object's start and end run in kernels of their own
// before and after (pool_prepare_kernel, pool_finish_kernel), and the non-gravitational term
// (relative to the Sun) is added after the bodies' terms are summed, where few values are
// live: inline for the JPL comet model without delay, and as the one call for the delayed
// model and dust.
#pragma once
#include "common.cuh"
#include "forces.cuh"
#include "internal.h"
#include "pool_plan.h"
#include "radau.cuh"
#include "radau_nodes.cuh"

namespace kb {

static __constant__ PoolPlans c_plans;

__device__ __forceinline__ void prefetch_l1(const void* p) {
    asm volatile("prefetch.global.L1 [%0];" ::"l"(p));
}

// The record of series S that holds TDB seconds jds (index clamped to the segment).
__device__ __forceinline__ const double2* pool_record(const PoolSeries& S, const double* pool,
                                                      double jds) {
    int idx = __double2int_rd((jds - S.start_s) * S.inv_intlen);
    idx = min(max(idx, 0), S.n_rec - 1);
    return reinterpret_cast<const double2*>(pool + S.offset + (int64_t)idx * S.rsize);
}

// The positions of three series at one time, in lockstep (nine sums and three recurrences in
// flight); the second and third may be shorter than the first.  The arithmetic of each is
// cheb_pos3's.
template <int S, bool KM>
__device__ __forceinline__ void pool_positions3(const PoolSeries& A, const PoolSeries& B,
                                                const PoolSeries& C, bool has_b, bool has_c,
                                                const double* __restrict__ pool, double jds,
                                                double* col, int stride) {
    const double2* r[3] = {pool_record(A, pool, jds), pool_record(B, pool, jds),
                           pool_record(C, pool, jds)};
    const int np[3] = {A.pairs, B.pairs, C.pairs};
    if (S > 1) {  // a warp to itself: fetch the rest of the records while the first lines load
#pragma unroll
        for (int q = 0; q < 3; ++q)
            for (int o = 8; o < 3 * np[q]; o += 8) prefetch_l1(r[q] + o);
    }
    double x2[3], t1[3], t2[3], acc[3][3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        const double2 h = __ldg(r[q]);
        const double xx = (jds - h.x) * h.y;
        x2[q] = 2.0 * xx;
        t2[q] = 1.0;
        t1[q] = xx;
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double2 a = __ldg(r[q] + 2 + c);
            acc[q][c] = a.x + a.y * xx;
        }
    }
    const double2 zero2 = make_double2(0.0, 0.0);
#pragma unroll 1
    for (int k = 1; k < np[0]; ++k) {
        double2 co[3][3];
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            r[q] += 3;
            const bool in = q == 0 || k < np[q];
#pragma unroll
            for (int c = 0; c < 3; ++c) co[q][c] = in ? __ldg(r[q] + 2 + c) : zero2;
        }
#pragma unroll
        for (int h = 0; h < 2; ++h)
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double nt = x2[q] * t1[q] - t2[q];
#pragma unroll
                for (int c = 0; c < 3; ++c) acc[q][c] += (h ? co[q][c].y : co[q][c].x) * nt;
                t2[q] = t1[q];
                t1[q] = nt;
            }
    }
    constexpr double INV_AU_KM = KM ? 1.0 : 1.0 / AU_KM;
    const int slot[3] = {A.slot, B.slot, C.slot};
#pragma unroll
    for (int q = 0; q < 3; ++q)
        if (q == 0 || (q == 1 && has_b) || (q == 2 && has_c)) {
            double* d = col + slot[q] * stride;
#pragma unroll
            for (int c = 0; c < 3; ++c) d[c * stride] = acc[q][c] * INV_AU_KM;
        }
}

// The velocity of one series (cheb_pair's arithmetic).
template <bool KM>
__device__ __forceinline__ void pool_velocity(const PoolSeries& A, const double* __restrict__ pool,
                                              double jds, double* col, int stride) {
    const double2* r = pool_record(A, pool, jds);
    const double2 h0 = __ldg(r);
    const double tss = __ldg(r + 1).x;
    const double x2 = 2.0 * ((jds - h0.x) * h0.y);
    double acc[3], u2 = 1.0, u1 = x2, fi = 2.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) acc[c] = __ldg(r + 2 + c).y;
    const int np = A.pairs;
#pragma unroll 1
    for (int k = 1; k < np; ++k) {
        r += 3;
        double2 co[3];
#pragma unroll
        for (int c = 0; c < 3; ++c) co[c] = __ldg(r + 2 + c);
#pragma unroll
        for (int h = 0; h < 2; ++h) {
            const double nu = x2 * u1 - u2;
            const double lu = u1 * fi;
#pragma unroll
            for (int c = 0; c < 3; ++c) acc[c] += (h ? co[c].y : co[c].x) * lu;
            u2 = u1;
            u1 = nu;
            fi += 1.0;
        }
    }
    double* d = col + A.slot * stride;
#pragma unroll
    for (int c = 0; c < 3; ++c) d[c * stride] = KM ? acc[c] : acc[c] * tss;
}

// What an exact evaluation reports besides the acceleration.
struct PoolExact {
    int32_t impact_id;  // the first body the point lies inside (0: none)
    double min_r2;      // smallest squared distance to a body other than the Sun
};

__device__ __forceinline__ void pool_checks(const PoolBody& B, double r2, bool exact, bool track,
                                            PoolExact& ex) {
    if (exact && r2 <= B.radius2 && ex.impact_id == 0) ex.impact_id = B.naif_id;
    if (track && exact && B.kind != FK_SUN && ex.impact_id == 0 && r2 < ex.min_r2) ex.min_r2 = r2;
}

// The scalars of one body's terms at relative position rp (and velocity rv): what the sums
// need besides rp and rv themselves.  The arithmetic is body_terms's.
struct PoolVel {  // the Sun and Jupiter: Newtonian, relativistic, J2 about the ecliptic's pole
    double kk, gr, c, r_v, jm, jk, j1, j2;  // J2's components: jm jk, j1, j2
};
__device__ __forceinline__ PoolVel pool_vel_terms(const PoolBody& B, const double rp[3],
                                                  const double rv[3], double r2) {
    PoolVel o;
    const double ir = rsqrt(r2);
    const double ir3 = ir * ir * ir;
    const double mass = B.mass;
    o.kk = mass * ir3;
    o.r_v = 4.0 * (rp[0] * rv[0] + rp[1] * rv[1] + rp[2] * rv[2]);
    const double rel_v2 = rv[0] * rv[0] + rv[1] * rv[1] + rv[2] * rv[2];
    o.gr = mass * C_AU_PER_DAY_INV_SQUARED * ir3;
    o.c = 4. * mass * ir - rel_v2;
    const double rc = c_tab.rot_c, rs = c_tab.rot_s;
    const double ez = -rs * rp[1] + rc * rp[2];
    const double zr = ez * ir;
    const double z_squared = 5.0 * (zr * zr);
    const double rr = B.radius * ir;
    const double coef = B.j2m * (rr * rr) * ir3;
    const double ey = rc * rp[1] + rs * rp[2];
    o.jm = rp[0] * coef;
    o.jk = z_squared - 1.0;
    const double jy = ey * coef * (z_squared - 1.0);
    const double jz = ez * coef * (z_squared - 3.0);
    o.j1 = rc * jy - rs * jz;
    o.j2 = rs * jy + rc * jz;
    return o;
}

// J2 of the Earth about the equator's pole: the common factor and z^2 of its components.
__device__ __forceinline__ void pool_earth_terms(const PoolBody& B, double rp2, double ir,
                                                 double ir3, double& coef, double& z_squared) {
    const double zr = rp2 * ir;
    z_squared = 5.0 * (zr * zr);
    const double rr = B.radius * ir;
    coef = B.j2m * (rr * rr) * ir3;
}

__device__ __forceinline__ double pool_r2(const double r[3]) {
    return r[0] * r[0] + r[1] * r[1] + r[2] * r[2];
}

__device__ __forceinline__ void pool_relative(const double x[3], const double* c, int stride,
                                              double r[3]) {
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = x[k] - c[k * stride];
}

// KM: the columns hold the series' sums unscaled (chained bodies: their positions), and the
// scaling is fused into the differences, as the general forms evaluate a plan that does not fit
// their per-lane cache (the asteroid masses): the results are then theirs to the bit but for one
// object in three hundred.  (Rounded positions differ from theirs in every object, which close
// approaches took to 9e-8 of the velocities' scale within two years; the time is the same.)
constexpr double POOL_INV_AU = 1.0 / AU_KM;
template <bool KM>
__device__ __forceinline__ void pool_body_position(const PoolBody& B, const double x[3],
                                                   const double* col, int stride, double r[3]) {
    const double* c = col + B.slot * stride;
    if (!KM) return pool_relative(x, c, stride, r);
    const double scale = B.chain >= 0 ? 1.0 : POOL_INV_AU;
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = fma(-c[k * stride], scale, x[k]);
}
template <bool KM>
__device__ __forceinline__ void pool_body_velocity(const PoolBody& B, const double v[3],
                                                   const double* col, int stride, double r[3]) {
    const double* c = col + B.vslot * stride;
    if (!KM) return pool_relative(v, c, stride, r);
#pragma unroll
    for (int k = 0; k < 3; ++k) r[k] = fma(-c[k * stride], B.vscale, v[k]);
}

// The force at (x, v) from a cache column, one lane summing every body in the plan's order
// (the non-gravitational term is not included; NG_SUN: it is na, added after the Sun's terms as
// the differentiation kernels sum it).  Bodies whose positions alone enter go two at a time,
// their chains interleaved.
template <bool NG_SUN = false, bool KM = false>
__device__ __forceinline__ void pool_forces(const PoolBody* body, int n_vel, int n_body,
                                            const double* col, int stride, bool exact, bool track,
                                            const double x[3], const double v[3], PoolExact& ex,
                                            double acc[3], const double* na = nullptr) {
    acc[0] = acc[1] = acc[2] = 0.0;
#pragma unroll 1
    for (int i = 0; i < n_vel; ++i) {
        const PoolBody& B = body[i];
        double rp[3], rv[3];
        pool_body_position<KM>(B, x, col, stride, rp);
        pool_body_velocity<KM>(B, v, col, stride, rv);
        const double r2 = pool_r2(rp);
        pool_checks(B, r2, exact, track, ex);
        const PoolVel t = pool_vel_terms(B, rp, rv, r2);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            acc[c] -= rp[c] * t.kk;
            acc[c] += t.gr * (t.c * rp[c] + t.r_v * rv[c]);
        }
        acc[0] += t.jm * t.jk;
        acc[1] += t.j1;
        acc[2] += t.j2;
        if (NG_SUN && i == 0) {
            acc[0] += na[0];
            acc[1] += na[1];
            acc[2] += na[2];
        }
    }
#pragma unroll 1
    for (int i = n_vel; i < n_body; i += 2) {
        const PoolBody &A = body[i], &B = body[i + 1];
        double ra[3], rb[3];
        pool_body_position<KM>(A, x, col, stride, ra);
        pool_body_position<KM>(B, x, col, stride, rb);
        const double r2a = pool_r2(ra), r2b = pool_r2(rb);
        const double ia = rsqrt(r2a), ib = rsqrt(r2b);
        const double ia3 = ia * ia * ia, ib3 = ib * ib * ib;
        pool_checks(A, r2a, exact, track, ex);
        pool_checks(B, r2b, exact, track, ex);
        const double ka = A.mass * ia3, kb_ = B.mass * ib3;
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] -= ra[c] * ka;
        if (A.kind == FK_EARTH) {
            double coef, z2;
            pool_earth_terms(A, ra[2], ia, ia3, coef, z2);
            acc[0] += ra[0] * coef * (z2 - 1.0);
            acc[1] += ra[1] * coef * (z2 - 1.0);
            acc[2] += ra[2] * coef * (z2 - 3.0);
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) acc[c] -= rb[c] * kb_;
    }
}

// A struck body ends the list of those that count, for the impact (the first of the plan) as for the
// closest approach.  The sub-lanes of a node, each of which saw its own bodies, go through all of
// them again here in the plan's order, as pool_forces does.
template <bool KM>
__device__ __forceinline__ PoolExact pool_impact(const PoolBody* body, int n_body, const double* col,
                                                     int stride, bool exact, bool track, double x0,
                                                     double x1, double x2, double min_before) {
    const double x[3] = {x0, x1, x2};
    PoolExact ex;
    ex.impact_id = 0;
    ex.min_r2 = min_before;
#pragma unroll 1
    for (int i = 0; i < n_body; ++i) {
        double rp[3];
        pool_body_position<KM>(body[i], x, col, stride, rp);
        pool_checks(body[i], pool_r2(rp), exact, track, ex);
    }
    return ex;
}

// Out of line for the planets (one object over a year 207 -> 202 us); with the asteroids' longer
// plan the call costs the pooled kernel spills (9,973 objects over two years 3.62 -> 3.64 ms).
static __device__ __noinline__ PoolExact pool_impact_planets(const PoolBody* body, int n_body,
                                                             const double* col, int stride, bool exact,
                                                             bool track, double x0, double x1, double x2,
                                                             double min_before) {
    return pool_impact<false>(body, n_body, col, stride, exact, track, x0, x1, x2, min_before);
}

// The same sum by the four sub-lanes of a node, to the bit: every sub-lane forms the scalars
// of its bodies (the Sun or Jupiter, and pairs of the others), then sub-lane c adds up
// component c in the plan's order.  term: the warp's scalars, slot k of a node at k * NODE_G.
// Returns component min(sub, 2).
constexpr int TERM_VEL = MAX_FORCE + 2;  // after the kk of every body: 7 a body with velocity
constexpr int TERM_EARTH = TERM_VEL + 14;
constexpr int TERM_SLOTS = TERM_EARTH + 2;
template <bool NG_SUN = false, bool KM = false>
__device__ __forceinline__ double pool_forces_wide(const PoolBody* body, int n_body, int sub,
                                                   const double* col, int stride, double* term,
                                                   bool exact, bool track, const double x[3],
                                                   const double v[3], PoolExact& ex,
                                                   double na = 0.0) {
    const int iv = sub & 1;
    const double min_before = ex.min_r2;
    {
        const PoolBody& B = body[iv];
        double rp[3], rv[3];
        pool_body_position<KM>(B, x, col, stride, rp);
        pool_body_velocity<KM>(B, v, col, stride, rv);
        const double r2 = pool_r2(rp);
        if (sub < 2) pool_checks(B, r2, exact, track, ex);
        const PoolVel t = pool_vel_terms(B, rp, rv, r2);
        // sub-lanes 2 and 3 repeat the terms (no branch) and write the same values
        term[iv * NODE_G] = t.kk;
        double* e = term + (TERM_VEL + 7 * iv) * NODE_G;
        e[0] = t.gr; e[NODE_G] = t.c; e[2 * NODE_G] = t.r_v; e[3 * NODE_G] = t.jm;
        e[4 * NODE_G] = t.jk; e[5 * NODE_G] = t.j1; e[6 * NODE_G] = t.j2;
    }
#pragma unroll 1
    for (int i0 = 2; i0 < n_body; i0 += 8) {
        const int i = min(i0 + 2 * sub, n_body), k = min(i0 + 2 * sub + 1, n_body);
        const PoolBody &A = body[i], &B = body[k];
        double ra[3], rb[3];
        pool_body_position<KM>(A, x, col, stride, ra);
        pool_body_position<KM>(B, x, col, stride, rb);
        const double r2a = pool_r2(ra), r2b = pool_r2(rb);
        const double ia = rsqrt(r2a), ib = rsqrt(r2b);
        const double ia3 = ia * ia * ia, ib3 = ib * ib * ib;
        pool_checks(A, r2a, exact, track, ex);
        pool_checks(B, r2b, exact, track, ex);
        term[i * NODE_G] = A.mass * ia3;
        term[k * NODE_G] = B.mass * ib3;
        if (A.kind == FK_EARTH) {
            double coef, z2;
            pool_earth_terms(A, ra[2], ia, ia3, coef, z2);
            term[TERM_EARTH * NODE_G] = coef;
            term[(TERM_EARTH + 1) * NODE_G] = z2;
        }
    }
    if (__any_sync(0xffffffffu, ex.impact_id != 0)) {
        if (NG_SUN)  // the differentiation passes ask whether, not which
#pragma unroll
            for (int o = NODE_G; o < 32; o <<= 1)
                ex.impact_id = max(ex.impact_id, __shfl_xor_sync(0xffffffffu, ex.impact_id, o));
        else if (KM)
            ex = pool_impact<true>(body, n_body, col, stride, exact, track, x[0], x[1], x[2], min_before);
        else
            ex = pool_impact_planets(body, n_body, col, stride, exact, track, x[0], x[1], x[2], min_before);
    }
    if (track)
#pragma unroll
        for (int o = NODE_G; o < 32; o <<= 1)
            ex.min_r2 = fmin(ex.min_r2, __shfl_xor_sync(0xffffffffu, ex.min_r2, o));
    __syncwarp();
    const int c = sub < 2 ? sub : 2;
    const double xc = c == 0 ? x[0] : (c == 1 ? x[1] : x[2]);
    const double vc = c == 0 ? v[0] : (c == 1 ? v[1] : v[2]);
    const double* cc = col + c * stride;
    double acc = 0.0;
#pragma unroll
    for (int i = 0; i < 2; ++i) {
        const double* e = term + (TERM_VEL + 7 * i) * NODE_G;
        const double bp = cc[body[i].slot * stride], bv = cc[body[i].vslot * stride];
        const double rp = KM ? fma(-bp, POOL_INV_AU, xc) : xc - bp;
        const double rv = KM ? fma(-bv, body[i].vscale, vc) : vc - bv;
        acc -= rp * term[i * NODE_G];
        acc += e[0] * (e[NODE_G] * rp + e[2 * NODE_G] * rv);
        const double jm = c == 0 ? e[3 * NODE_G] : (c == 1 ? e[5 * NODE_G] : e[6 * NODE_G]);
        const double jk = c == 0 ? e[4 * NODE_G] : 1.0;
        acc += jm * jk;
        if (NG_SUN && i == 0) acc += na;
    }
    const double coef = term[TERM_EARTH * NODE_G];
    const double z2 = term[(TERM_EARTH + 1) * NODE_G] - (c == 2 ? 3.0 : 1.0);
#pragma unroll 4
    for (int i = 2; i < n_body; ++i) {
        const double bp = cc[body[i].slot * stride];
        const double rp = KM ? fma(-bp, body[i].chain >= 0 ? 1.0 : POOL_INV_AU, xc) : xc - bp;
        acc -= rp * term[i * NODE_G];
        if (i == POOL_EARTH) acc += rp * coef * z2;
    }
    return acc;
}

// The centre and frame changes of the pooled kernel's objects, in kernels of their own (one
// thread per object of the part order[range[0] .. range[2])): their code (a general state
// query of the centre's chain) runs once per object, and inside the step loop's kernel it
// cost instruction-cache misses to every warp of the SM.
//
// Before the integration: the checks of the inputs and to_ssb_equatorial (mod.rs:79-80) at
// the epoch; the barycentric equatorial state goes to the output arrays, the outcome to
// status, where nbody_pool_kernel reads both.
static __global__ void pool_prepare_kernel(NBodyArgs a) {
    const int64_t first = a.range[0], end = a.range[2], n = a.n;
    for (int64_t k = first + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < end;
         k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t obj = a.order[k];
        const double t0 = a.jd0[obj];
        double p[3] = {a.pos[obj], a.pos[n + obj], a.pos[2 * n + obj]};
        double v[3] = {a.vel[obj], a.vel[n + obj], a.vel[2 * n + obj]};
        const bool finite = isfinite(p[0]) && isfinite(p[1]) && isfinite(p[2]) &&
                            isfinite(v[0]) && isfinite(v[1]) && isfinite(v[2]) && isfinite(t0);
        int rc = finite ? ST_OK : ST_VALUE_ERROR;
        if (rc == ST_OK && (a.chain.len > 0 || a.frame == FRAME_ECLIPTIC))
            rc = to_ssb_equatorial(t0, a.frame, a.chain, p, v);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            a.out_pos[c * n + obj] = p[c];
            a.out_vel[c * n + obj] = v[c];
        }
        a.status[obj] = rc;
    }
}

// After it: from_ssb_equatorial (mod.rs:107-116) at the target epoch for every object that
// arrived; a failure there gives NaN and its status, as in the other forms.
static __global__ void pool_finish_kernel(NBodyArgs a) {
    const int64_t first = a.range[0], end = a.range[2], n = a.n;
    if (!(a.chain.len > 0 || a.frame == FRAME_ECLIPTIC)) return;
    for (int64_t k = first + (int64_t)blockIdx.x * blockDim.x + threadIdx.x; k < end;
         k += (int64_t)gridDim.x * blockDim.x) {
        const int64_t obj = a.order[k];
        if (a.status[obj] != ST_OK) continue;
        double p[3] = {a.out_pos[obj], a.out_pos[n + obj], a.out_pos[2 * n + obj]};
        double v[3] = {a.out_vel[obj], a.out_vel[n + obj], a.out_vel[2 * n + obj]};
        const int rc = from_ssb_equatorial(a.jd1[obj], a.frame, a.chain, p, v);
        if (rc != ST_OK) {
            const double nan = __longlong_as_double(0x7ff8000000000000LL);
            p[0] = p[1] = p[2] = v[0] = v[1] = v[2] = nan;
            a.status[obj] = rc;
        }
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            a.out_pos[c * n + obj] = p[c];
            a.out_vel[c * n + obj] = v[c];
        }
    }
}

// The start of an object the wide form (S = 4) integrates: outside the fast window (as the
// ordering kernels test it) it is left to the general form (ST_PENDING); otherwise the checks and
// the centre change that pool_prepare_kernel makes.
__device__ __forceinline__ int pool_start(const NBodyArgs& a, double t0, double t1, double p[3],
                                          double v[3]) {
    if (!in_window(t0, t1, a.lo, a.hi)) return ST_PENDING;
    const bool finite = isfinite(p[0]) && isfinite(p[1]) && isfinite(p[2]) && isfinite(v[0]) &&
                        isfinite(v[1]) && isfinite(v[2]) && isfinite(t0);
    if (!finite) return ST_VALUE_ERROR;
    if (a.chain.len > 0 || a.frame == FRAME_ECLIPTIC)
        return to_ssb_equatorial(t0, a.frame, a.chain, p, v);
    return ST_OK;
}

__device__ __forceinline__ void pool_store(const NBodyArgs& a, int64_t i, int rc, const double x[3],
                                           const double v[3], int32_t impact_id, double t_impact,
                                           double min_r2, const RadauCounters& cnt) {
    const int64_t n = a.n;
    a.status[i] = rc;
    if (rc == ST_PENDING) return;
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        a.out_pos[c * n + i] = rc == ST_OK ? x[c] : nan;
        a.out_vel[c * n + i] = rc == ST_OK ? v[c] : nan;
    }
    if (a.impact_id) a.impact_id[i] = rc == ST_IMPACT ? impact_id : 0;
    if (a.impact_jd) a.impact_jd[i] = rc == ST_IMPACT ? t_impact : 0.0;
    if (a.min_dist) a.min_dist[i] = min_r2 < 1e300 ? sqrt(min_r2) : 1e300;
    if (a.counters) {
        a.counters[i] = cnt.steps;
        a.counters[n + i] = cnt.iterations;
        a.counters[2 * n + i] = cnt.exact;
    }
}

// Per-group state in shared memory (doubles): the object's epoch, target epoch, step, previous
// step, position, velocity and acceleration at the epoch.  Every lane of a group needs the
// same values; keeping them out of the lanes' registers leaves the registers to the hot loop.
constexpr int ST_T = 0, ST_TF = 1, ST_H = 2, ST_HP = 3, ST_X = 4, ST_V = 7, ST_A = 10;
constexpr int ST_ROW = 13;
// Rows read two doubles at a time: b (7 + 1 pad per component), the evaluations (8 nodes per
// component), the node table (W row, U row, spacing and its square).
constexpr int POOL_B = 8, POOL_NODE = 18;

// S = 1: eight lanes an object, four objects a warp.  S = 4: a warp an object, four sub-lanes
// a node, for the objects whose integration is waited for: a step then takes less than half the
// time, for about 1.6 times the work.  Both give the same results to the bit.
//
// Shared memory of a block of THREADS threads in either role (doubles): a column of `slots`
// cached values per node of every group (slot k of column i at k * COLS + i), then the rows of
// every group, then (S = 4) the warps' scalars.
template <int S, int THREADS>
struct PoolShared {
    static constexpr int GROUPS = THREADS / (NODE_G * S);
    static constexpr int COLS = GROUPS * NODE_G;
    static constexpr int ROWS = 3 * POOL_B + 3 * NODE_G + 6 + ST_ROW + 1 + NODE_G;  // even
    static constexpr int TERMS = S > 1 ? GROUPS * TERM_SLOTS * NODE_G : 0;
    __host__ __device__ static constexpr int doubles(int slots) {
        return slots * COLS + GROUPS * ROWS + TERMS;
    }
};

// What both roles of a block read: the node table (row 8 is the step end, f = 1), the series
// and the bodies.
struct PoolTables {
    const double* node;
    const PoolSeries* src;
    const PoolBody* body;  // shared memory (sub-lanes read different bodies)
    int n_pos, n_series, n_body, n_vel, n_slot;
    const PoolPlan* plan;
};

// One round's record evaluations: every series at the times of the groups whose first lane's bit is
// set in M (TDB seconds in ste, a row of ROWS doubles per group; this group's is gi), into the
// columns of s_cache.  The 32 lanes take one group's eight columns four lanes each, two groups'
// two lanes each, or (three or four groups) each lane its own; with S = 4 the warp is one group.
template <int S, int COLS, int ROWS, bool KM = false>
__device__ __forceinline__ void pool_records(const PoolTables& T, unsigned M, int gi,
                                             const double* ste, double* s_cache) {
    const int warp_lane = threadIdx.x & 31, lane = threadIdx.x & (NODE_G - 1);
    int share, shares, g;
    if (S > 1) {
        share = warp_lane / NODE_G;
        shares = S;
        g = gi;
    } else {
        const unsigned g4 = (M & 1u) | ((M >> 7) & 2u) | ((M >> 14) & 4u) | ((M >> 21) & 8u);
        const int count = __popc(g4);
        const int g_lo = __ffs(g4) - 1, g_hi = 31 - __clz(g4);
        const int own = warp_lane / NODE_G;
        share = count == 1 ? own : (count == 2 ? (own & 1) : 0);
        shares = count == 1 ? 4 : (count == 2 ? 2 : 1);
        g = count == 1 ? g_lo : (count == 2 ? (own < 2 ? g_lo : g_hi) : own);
        if (count > 2 && !((g4 >> own) & 1u)) share = MAX_SERIES;  // not at new times
        g += (threadIdx.x >> 5) * (32 / NODE_G);
    }
    const double jds = ste[(g - gi) * ROWS + lane];
    const double* pool = c_eph.pool;
    double* dst = s_cache + g * NODE_G + lane;
#pragma unroll 1
    for (int k = share; k < T.n_pos; k += 3 * shares) {
        const int kb_ = k + shares, kc = kb_ + shares;
        const bool has_b = kb_ < T.n_pos, has_c = kc < T.n_pos;
        pool_positions3<S, KM>(T.src[k], T.src[has_b ? kb_ : k], T.src[has_c ? kc : k], has_b, has_c,
                           pool, jds, dst, COLS);
    }
#pragma unroll 1
    for (int k = T.n_pos + share; k < T.n_series; k += shares)
        pool_velocity<KM>(T.src[k], pool, jds, dst, COLS);
    __syncwarp();
}

// Bodies given relative to a centre (the Earth and Moon), in a node's column after its records.
template <bool KM = false>
__device__ __forceinline__ void pool_chain(const PoolTables& T, double* col, int stride) {
#pragma unroll 1
    for (int i = 0; i < T.n_body; ++i) {
        const int ch = T.plan->b[i].chain, sl = T.plan->b[i].slot;
        if (ch < 0) continue;
#pragma unroll
        for (int q = 0; q < 3; ++q) {
            double& p = col[(sl + q) * stride];
            const double centre = col[(ch + q) * stride];
            p = KM ? fma(p, POOL_INV_AU, __dmul_rn(centre, POOL_INV_AU)) : p + centre;
        }
    }
}

// The predictor at a node (row nrow) from the group's b and state.
__device__ __forceinline__ void pool_predict(const double2* nrow, const double* sb,
                                             const double* st, double xe[3], double ve[3]) {
    const double2 fr = nrow[8];
    const double h = st[ST_H], f = fr.x;
    const double h2 = h * h;
    const double2* b2 = reinterpret_cast<const double2*>(sb);
    double bw[3] = {0.0, 0.0, 0.0}, bu[3] = {0.0, 0.0, 0.0};
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double2 w = nrow[k], u = nrow[4 + k];
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            const double2 b = b2[4 * c + k];
            bw[c] += w.x * b.x;
            bu[c] += u.x * b.x;
            if (k < 3) {
                bw[c] += w.y * b.y;
                bu[c] += u.y * b.y;
            }
        }
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        const double ac = st[ST_A + c], vc = st[ST_V + c];
        xe[c] = st[ST_X + c] + f * vc * h + fr.y * h2 * (ac / 2.0 + bw[c]);
        ve[c] = vc + f * h * (ac + bu[c]);
    }
}

// One component's corrector: divided differences g of its seven node evaluations (row se),
// then b = g C into out.
__device__ __forceinline__ void pool_divided(const double* se, double ac, double g[7], double& e7) {
    const double2* e2 = reinterpret_cast<const double2*>(se);
    const double2 e01 = e2[0], e23 = e2[1], e45 = e2[2];
    const double e[7] = {e01.x, e01.y, e23.x, e23.y, e45.x, e45.y, e2[3].x};
#pragma unroll
    for (int j = 1; j < 8; ++j) {
        double gk = (e[j - 1] - ac) * c_tab.inv_frac[j];
#pragma unroll
        for (int z = 1; z < j; ++z) gk = (gk - g[z - 1]) * c_tab.inv_diff[j][z];
        g[j - 1] = gk;
    }
    e7 = e[6];
}
__device__ __forceinline__ void pool_store_b(const double g[7], double* out) {
    double b[8];
#pragma unroll
    for (int jj = 0; jj < 7; ++jj) {
        double s2 = g[jj];
#pragma unroll
        for (int k = jj + 1; k < 7; ++k) s2 += c_tab.c[k][jj] * g[k];
        b[jj] = s2;
    }
    b[7] = 0.0;
    double2* o = reinterpret_cast<double2*>(out);
#pragma unroll
    for (int k = 0; k < 4; ++k) o[k] = make_double2(b[2 * k], b[2 * k + 1]);
}

// PREPARED: objects of the order, from queues (a.queue; S = 4: its heavy objects) or, without,
// one per group, with pool_prepare_kernel before and pool_finish_kernel after; otherwise one
// per group in the caller's order, centre and frame changed here.
template <int S, int THREADS, bool PREPARED, bool KM>
__device__ __forceinline__ void pool_run(const NBodyArgs& a, const PoolTables& T, double* smem) {
    using Sh = PoolShared<S, THREADS>;
    constexpr int GL = NODE_G * S, COLS = Sh::COLS;  // lanes of a group; cache columns
    const int warp_lane = threadIdx.x & 31;
    const int lane = threadIdx.x & (NODE_G - 1);                 // the node
    const int sub = S == 1 ? 0 : warp_lane / NODE_G;             // the sub-lane of the node
    const int gi = threadIdx.x / GL;                             // the group in the block
    const int lane0 = S == 1 ? (warp_lane & ~(NODE_G - 1)) : 0;  // the group's first lane
    const unsigned gmask = S == 1 ? 0xFFu << lane0 : 0xffffffffu;
    const int64_t group = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) / GL;
    double* s_cache = smem;
    double* rows = smem + T.n_slot * COLS + gi * Sh::ROWS;
    double* sb = rows;
    double* se = sb + 3 * POOL_B;
    double* scmp = se + 3 * NODE_G;
    double* st = scmp + 6;
    double* ste = st + ST_ROW + 1;
    double* term = smem + T.n_slot * COLS + Sh::GROUPS * Sh::ROWS + gi * TERM_SLOTS * NODE_G + lane;
    const bool leader = lane == 0 && sub == 0;
    const bool owner = lane < 3 && sub == 0;  // forms one component's g, b and state
    const int comp = lane < 3 ? lane : 0;
    const double2* nrow =
        reinterpret_cast<const double2*>(T.node + (lane < 7 ? lane + 1 : 8) * POOL_NODE);
    const bool se_lane = lane == 7;
    double* col = s_cache + gi * NODE_G + lane;
    const bool track = a.min_dist != nullptr;

    int64_t obj = -1;
    int phase = PH_DONE;
    bool fresh = false;  // the group's next evaluations are at new times
    int iter = 0, failures = 0, attempts = 0;
    RadauCounters cnt;
    NonGrav ng;
    ng.base = nullptr;
    ng.stride = a.n;
    ng.kind = 0;
    int32_t impact_id = 0;
    double min_r2 = 1e300;
    bool first = true;
    int outcome = ST_OK;  // outcome of a finished object, stored at the top of the next round

    auto fetch = [&]() -> bool {
        int64_t k;
        if (!PREPARED) {  // one object per group, in the caller's order
            k = first ? group : a.n;
            if (k >= a.n) return false;
            first = false;
            obj = k;
        } else {
            // the objects inside the fast window: order[range[0] .. range[2]), those with a
            // non-gravitational model from range[1] on (launch_nodes_ordered).  wide: how many
            // heavy objects lead each of the two parts, and the queue of them.
            int q = 0;
            if (S > 1) {
                if (leader) {
                    const int w0 = a.wide[0], w1 = a.wide[1];
                    const int t = atomicAdd(a.wide + 2, 1);
                    q = t < w0 ? a.range[0] + t
                               : (t - w0 < w1 ? a.range[1] + (t - w0) : a.range[2]);
                }
            } else if (a.queue) {
                // groups on the first SMs take the non-gravitational part first, the others
                // the rest; each turns to the other part when its own is used up.  Only a few
                // SMs then fetch the non-gravitational model's code, which evicts the step loop
                // from an SM's instruction cache.  (The queues start after the heavy objects.)
                if (leader) {
                    const int r0 = a.range[0], r1 = a.range[1], r2 = a.range[2];
                    unsigned smid, nsm;
                    asm("mov.u32 %0, %%smid;" : "=r"(smid));
                    asm("mov.u32 %0, %%nsmid;" : "=r"(nsm));
                    const bool ng_first =
                        r2 > r1 && (int64_t)smid * (r2 - r0) < (int64_t)nsm * (r2 - r1) + (r2 - r0);
                    q = r2;  // nothing left
                    for (int pass = 0; pass < 2; ++pass) {
                        const bool ng_part = (pass == 0) == ng_first;
                        const int lo = ng_part ? r1 : r0, hi = ng_part ? r2 : r1;
                        if (hi > lo) {
                            const int t = atomicAdd(ng_part ? a.queue_ng : a.queue, 1);
                            if (t < hi - lo) {
                                q = lo + t;
                                break;
                            }
                        }
                    }
                }
            } else {
                q = first ? (int)group + a.range[0] : a.range[2];  // one object per group
                first = false;
            }
            k = __shfl_sync(gmask, q, lane0);
            if (k >= a.range[2]) return false;
            obj = a.order ? a.order[k] : k;
        }
        int frc = ST_OK;
        if (leader) {
            const int64_t n = a.n;
            const double t0 = a.jd0[obj], t1 = a.jd1[obj];
            double p[3], v[3];
            if (!PREPARED) {
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    p[c] = a.pos[c * n + obj];
                    v[c] = a.vel[c * n + obj];
                }
                frc = pool_start(a, t0, t1, p, v);
            } else {
                // the state at the epoch as pool_prepare_kernel left it (barycentric
                // equatorial, in the output arrays) and the outcome of its checks
                frc = a.status[obj];
#pragma unroll
                for (int c = 0; c < 3; ++c) {
                    p[c] = a.out_pos[c * n + obj];
                    v[c] = a.out_vel[c * n + obj];
                }
            }
            st[ST_T] = t0;
            st[ST_TF] = t1;
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                st[ST_X + c] = p[c];
                st[ST_V + c] = v[c];
            }
        }
        if (sub == 0) {
            sb[lane] = sb[POOL_B + lane] = sb[2 * POOL_B + lane] = 0.0;
            if (lane < 6) scmp[lane] = 0.0;
        }
        ng.base = a.nongrav ? a.nongrav + obj : nullptr;
        ng.kind = a.nongrav ? (int)a.nongrav[obj] : 0;
        impact_id = 0;
        min_r2 = 1e300;
        cnt = RadauCounters();
        iter = 0;
        failures = 0;
        attempts = 0;
        outcome = __shfl_sync(gmask, frc, lane0);
        phase = outcome == ST_OK ? PH_EXACT_INIT : PH_STORE;
        fresh = outcome == ST_OK;
        __syncwarp(gmask);
        return true;
    };

    auto finish = [&](int code) {
        outcome = code;
        phase = PH_STORE;
        fresh = false;
    };

    // step start with step h (every lane computes the same): |h| >= MIN_STEP, then truncate
    // to the final time (radau.rs:187-190,214-216); after an accepted step the corrector
    // starts from the predicted b (predict_b_row).  The leader publishes the step.
    auto start_step = [&](double h, double t, double tf, bool predict, double h_prev) {
        if (fabs(h) < 0.005) h = copysign(0.005, h);
        if (fabs(t - tf) <= fabs(h)) h = tf - t;
        if (predict && owner) predict_b_row(sb + POOL_B * comp, h / h_prev);
        if (leader) st[ST_H] = h;
        __syncwarp(gmask);
        iter = 0;
        ++attempts;
        phase = PH_ITER;
        fresh = true;
    };

    int obj_rounds = 0;
    const int max_obj_rounds = a.max_loops * 11;
    for (;;) {
        if (phase == PH_STORE) {  // the finished object's outcome (the leader stores)
            if (leader) {
                double xs[3] = {st[ST_X], st[ST_X + 1], st[ST_X + 2]};
                double vs[3] = {st[ST_V], st[ST_V + 1], st[ST_V + 2]};
                if (!PREPARED && outcome == ST_OK)
                    outcome = from_ssb_equatorial(st[ST_TF], a.frame, a.chain, xs, vs);
                pool_store(a, obj, outcome, xs, vs, impact_id, st[ST_T], min_r2, cnt);
            }
            __syncwarp(gmask);  // st is read before the next object overwrites it
            phase = PH_DONE;
        }
        if (phase == PH_DONE) {  // take the next object (group-collective)
            obj_rounds = 0;
            if (!fetch()) phase = PH_FINISHED;
        }
        // every lane of the warp stays in the loop for the pool's collectives until all its
        // groups have run out of objects
        if (__all_sync(0xffffffffu, phase == PH_FINISHED)) break;
        bool active = phase == PH_ITER || phase == PH_EXACT_INIT;
        // the step loop's bound: step attempts (kete_b200_set_step_limit), and rounds as a
        // second guard
        if (active && (++obj_rounds > max_obj_rounds || attempts > a.max_loops)) {
            finish(ST_TIMEOUT);
            active = false;
        }
        const bool iter_round = phase == PH_ITER;
        // ---- the warp's record evaluations for every group at new times ----
        const bool need = active && fresh;
        const unsigned M = __ballot_sync(0xffffffffu, need);
        if (M) {
            if (need && sub == 0) {
                const double te = iter_round ? st[ST_T] + nrow[8].x * st[ST_H] : st[ST_T];
                ste[lane] = __dmul_rn(te - 2451545.0, 86400.0);
            }
            __syncwarp();
            pool_records<S, COLS, Sh::ROWS, KM>(T, M, gi, ste, s_cache);
            if (need && sub == 0) pool_chain<KM>(T, col, COLS);
            if (S > 1) __syncwarp();
            fresh = false;
        }
        if (!active) continue;
        double xe[3], ve[3];
        if (!iter_round) {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                xe[c] = st[ST_X + c];
                ve[c] = st[ST_V + c];
            }
        } else {
            pool_predict(nrow, sb, st, xe, ve);
        }
        const bool exact = !iter_round || se_lane;
        PoolExact ex;
        ex.impact_id = 0;
        ex.min_r2 = min_r2;
        double ev[3];  // S > 1: ev[0] is the sub-lane's component
        if (S > 1)
            ev[0] = pool_forces_wide<false, KM>(T.body, T.n_body, sub, col, COLS, term, exact, track, xe, ve, ex);
        else
            pool_forces<false, KM>(T.plan->b, T.n_vel, T.n_body, col, COLS, exact, track, xe, ve, ex, ev);
        if (ng.kind != 0) {
            // non_grav_accel relative to the Sun (acceleration.rs:161-165): inline for the
            // JPL comet model without delay; a call for the delayed model and dust
            double sx[3], sv[3];
            pool_body_position<KM>(T.plan->b[0], xe, col, COLS, sx);
            pool_body_velocity<KM>(T.plan->b[0], ve, col, COLS, sv);
            const double3 rp = make_double3(sx[0], sx[1], sx[2]);
            const double3 rv = make_double3(sv[0], sv[1], sv[2]);
            const double3 na = (ng.kind == 1 && ng.p(9) == 0.0) ? nongrav_terms<false>(ng, rp, rv)
                                                                : nongrav_accel(ng, rp, rv);
            if (S > 1) {
                ev[0] += sub == 0 ? na.x : (sub == 1 ? na.y : na.z);
            } else {
                ev[0] += na.x;
                ev[1] += na.y;
                ev[2] += na.z;
            }
        }
        // ---- exchange the node evaluations ----
        if (S > 1) {
            if (sub < 3) se[NODE_G * sub + lane] = ev[0];
        } else {
            se[lane] = ev[0];
            se[NODE_G + lane] = ev[1];
            se[2 * NODE_G + lane] = ev[2];
        }
        __syncwarp(gmask);
        if (!iter_round) {  // the initial exact evaluation (every lane evaluated one point)
            cnt.exact++;
            const double t = st[ST_T], tf = st[ST_TF];
            impact_id = ex.impact_id;
            min_r2 = ex.min_r2;
            if (impact_id != 0) {
                finish(ST_IMPACT);
                continue;
            }
            if (owner) st[ST_A + comp] = se[NODE_G * comp + lane];
            if (fabs(tf - t) < 1e-10) {
                __syncwarp(gmask);
                finish(ST_OK);
                continue;
            }
            failures = 0;
            start_step(copysign(0.1, tf - t), t, tf, false, 0.0);
            continue;
        }
        // ---- corrector iteration: form g and b (radau.rs:292-313); lanes 0-2 each own one
        // component ----
        cnt.iterations++;
        bool conv;
        {
            const double ac = st[ST_A + comp];
            double g[7], e7;
            pool_divided(se + NODE_G * comp, ac, g, e7);
            // converged when |b6 - b6_old| / (|a at node 7| + 1e-6) is below 1e-14 in every
            // component, as products; a NaN counts as below while another component is not one
            const double change = fabs(g[6] - sb[POOL_B * comp + 6]);
            const double limit = 1e-14 * (fabs(e7) + 1e-6);
            const unsigned above = __ballot_sync(gmask, owner && change >= limit);
            const unsigned number = __ballot_sync(gmask, owner && change == change);
            conv = above == 0 && number != 0;
            if (owner) pool_store_b(g, sb + POOL_B * comp);
        }
        __syncwarp(gmask);
        ++iter;
        if (conv) {
            const double h = st[ST_H], t = st[ST_T], tf = st[ST_TF];
            const double fem = fmax(fmax(fabs(se[6]), fabs(se[NODE_G + 6])), fabs(se[2 * NODE_G + 6]));
            const double mb6 =
                fmax(fmax(fabs(sb[6]), fabs(sb[POOL_B + 6])), fabs(sb[2 * POOL_B + 6]));
            __syncwarp(gmask);  // every lane has read the step before the leader replaces it
            if (owner) {
                // x += dx, v += dv with compensated (Kahan) summation; lane c owns component c
                const int c = comp;
                const double h2 = h * h;
                double dw = 0.0, du = 0.0;
#pragma unroll
                for (int k = 0; k < 7; ++k) {
                    const double bck = sb[POOL_B * c + k];
                    dw += bck * c_tab.w[k];
                    du += bck * c_tab.u[k];
                }
                const double xc = st[ST_X + c], vc = st[ST_V + c], ac = st[ST_A + c];
                const double dx = vc * h + h2 * (ac * 0.5 + dw);
                const double dv = h * (ac + du);
                const double yx = dx - scmp[c], yv = dv - scmp[3 + c];
                const double tx = xc + yx, tv = vc + yv;
                scmp[c] = (tx - xc) - yx;
                scmp[3 + c] = (tv - vc) - yv;
                st[ST_X + c] = tx;
                st[ST_V + c] = tv;
                // the step-end lane's evaluation is the exact evaluation of the new state
                st[ST_A + c] = se[NODE_G * c + 7];
            }
            const double next_h =
                h * clampd(pow(1e-6 * (fem + 1e-6) / mb6, 1.0 / 7.0), 0.25, 4.0);
            const double tn = t + h;
            if (leader) {
                st[ST_T] = tn;
                st[ST_HP] = h;
                st[ST_H] = next_h;
            }
            // the step-end lane's impact and closest approach count now that it converged
            impact_id = __shfl_sync(gmask, ex.impact_id, lane0 + 7);
            if (track) min_r2 = __shfl_sync(gmask, ex.min_r2, lane0 + 7);
            __syncwarp(gmask);
            cnt.exact++;
            if (impact_id != 0) {
                finish(ST_IMPACT);
                continue;
            }
            cnt.steps++;
            if (fabs(tn - tf) < 1e-12) {
                finish(ST_OK);
                continue;
            }
            failures = 0;
            start_step(next_h, tn, tf, true, h);
            continue;
        }
        if (iter >= 10) {  // step failed to converge (radau.rs:345) -> retry smaller
            failures += 1;
            if (failures > 10) {
                finish(ST_CONVERGENCE);
                continue;
            }
            const double h = st[ST_H] * 0.7, t = st[ST_T], tf = st[ST_TF];
            __syncwarp(gmask);  // read before the leader replaces the step
            start_step(h, t, tf, false, 0.0);
        }
    }
}

// Fills the block's tables (static shared memory of the kernels).
__device__ __forceinline__ PoolTables pool_tables(int n_force, double* s_node,
                                                  PoolSeries* s_src, PoolBody* s_body) {
    const PoolPlan& plan = n_force == c_eph.n_force_planets ? c_plans.planets : c_plans.all;
    for (int i = threadIdx.x; i < 9 * POOL_NODE; i += blockDim.x) {
        const int j = i / POOL_NODE, k = i % POOL_NODE;
        double val = 0.0;
        if (k < 7) val = j < 8 ? c_tab.w_pow[j][k] : c_tab.w[k];
        else if (k >= 8 && k < 15) val = j < 8 ? c_tab.u_pow[j][k - 8] : c_tab.u[k - 8];
        else if (k == 16) val = j < 8 ? c_tab.spacing[j] : 1.0;
        else if (k == 17) val = j < 8 ? c_tab.frac2[j] : 1.0;
        s_node[i] = val;
    }
    for (int i = threadIdx.x; i < plan.n_series; i += blockDim.x) s_src[i] = plan.s[i];
    for (int i = threadIdx.x; i <= plan.n_body; i += blockDim.x) s_body[i] = plan.b[i];
    __syncthreads();
    return PoolTables{s_node, s_src, s_body, plan.n_pos, plan.n_series, plan.n_body, plan.n_vel,
                      plan.n_slot, &plan};
}

// MINB: minimum resident blocks per SM requested from the compiler (3: 168 registers, 4:
// 128); the host picks the instantiation.  With a.queue the grid is persistent and groups take
// objects from the queues; without, each group integrates one object.
//
// The first blocks begin with the order's heavy objects, a warp each, and turn to the others when
// those are taken (without any, the counts are zero).  The objects with many times the steps of
// most (near the Earth, long spans) bound a launch of a few objects per lane group: see
// order_scan_kernel for the rule.
template <int MINB, bool KM>
__global__ void __launch_bounds__(NODES_BLOCK, MINB) nbody_pool_kernel(NBodyArgs a) {
    extern __shared__ __align__(16) double s_pool[];
    __shared__ __align__(16) double s_node[9 * POOL_NODE];
    __shared__ PoolSeries s_src[MAX_SERIES];
    __shared__ PoolBody s_body[MAX_FORCE + 2];
    const PoolTables T = pool_tables(a.n_force, s_node, s_src, s_body);
    if ((int)blockIdx.x * (NODES_BLOCK / 32) < a.wide[0] + a.wide[1])
        pool_run<4, NODES_BLOCK, true, KM>(a, T, s_pool);
    __syncthreads();
    pool_run<1, NODES_BLOCK, true, KM>(a, T, s_pool);
}

// A warp an object in the caller's order, blocks of one warp so that few objects spread over
// the SMs; centre and frame are changed here, and the objects whose span leaves the window are
// left to the general form.
constexpr int WIDE_BLOCK = 32;
template <int MINB, bool KM>
__global__ void __launch_bounds__(WIDE_BLOCK, MINB) nbody_wide_kernel(NBodyArgs a) {
    extern __shared__ __align__(16) double s_pool[];
    __shared__ __align__(16) double s_node[9 * POOL_NODE];
    __shared__ PoolSeries s_src[MAX_SERIES];
    __shared__ PoolBody s_body[MAX_FORCE + 2];
    const PoolTables T = pool_tables(a.n_force, s_node, s_src, s_body);
    pool_run<4, WIDE_BLOCK, false, KM>(a, T, s_pool);
}

}  // namespace kb
