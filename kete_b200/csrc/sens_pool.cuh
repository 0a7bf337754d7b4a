// sens_pool.cuh -- the differentiation passes on the warp-pooled step machinery of
// radau_pool.cuh: the checkpointed forward pass, the replays of its checkpoint blocks and the
// forward sensitivities.
//
// The step loop is sens_rounds's (adjoint.cuh) in the same arithmetic: the exact evaluation at
// the updated state in a round of its own, plain state updates, the non-gravitational term after
// the Sun's.  What differs is who evaluates what: a step's records are evaluated once by the
// whole warp for the seven node times and the step end (the exact evaluation reads the step end's
// column, where every lane evaluated the same eleven records again), and a group's state lives
// in shared memory.  S = 4 gives an object a warp (few objects: every step is waited for), S = 1
// eight lanes (many checkpoint blocks).  KM: unscaled columns for the plan with the asteroid masses,
// as in radau_pool.cuh, so that the sums are the general kernels'.
//
// The forward kernels take the objects inside the fast plan's window and mark the others ST_PENDING
// for the kernels of adjoint.cuh and stm_nodes.cuh; the replays take the blocks whose checkpoint
// says that the forward pass was the one here, and mark the others SENS_PENDING.
#pragma once
#include "adjoint.cuh"
#include "radau_pool.cuh"
#include "stm_nodes.cuh"

namespace kb {

// Shared memory of a block: cache columns, then per group the b of this and the previous
// iteration, the evaluations, the state and the times, then TANGENTS doubles per group, then
// (S = 4) the warps' scalars.
template <int S, int THREADS, int TANGENTS>
struct SensPoolShared {
    static constexpr int GROUPS = THREADS / (NODE_G * S);
    static constexpr int COLS = GROUPS * NODE_G;
    static constexpr int ROWS = 2 * 3 * POOL_B + 3 * NODE_G + ST_ROW + 1 + NODE_G + TANGENTS;
    static constexpr int TERMS = S > 1 ? GROUPS * TERM_SLOTS * NODE_G : 0;
    static_assert(ROWS % 2 == 0, "rows of double pairs");
    __host__ __device__ static constexpr int doubles(int slots) {
        return slots * COLS + GROUPS * ROWS + TERMS;
    }
};

enum SensPoolPhase : int {
    SQ_FETCH = 0, SQ_BEGIN = 1, SQ_INIT = 2, SQ_ITER = 3, SQ_EXACT = 4, SQ_SEGMENT = 5, SQ_END = 6,
    SQ_FINISHED = 7
};

// What the policies see of a group.
struct SensPoolGroup {
    int lane, sub;  // node and sub-lane
    unsigned gmask;
    bool leader, owner;
    double* st;      // ST_T .. (radau_pool.cuh)
    double* sb;      // the current b, POOL_B a component
    double* tan;     // the policy's doubles
    const double* col;       // this lane's cache column
    const double* col_end;   // the step end's column
    int stride;
    const PoolTables* T;
    NonGrav ng;
    int rc;
};

// d force / d(x, v) and d force / d(A1, A2) from a cache column (TangentForce::jacobian_cached on
// the pooled plan).
template <bool KM>
__device__ __forceinline__ void pool_jacobian(const PoolTables& T, const double* col, int stride,
                                              const NonGrav& ng, const double x[3],
                                              const double v[3], double J[18], double jp[6]) {
#pragma unroll
    for (int i = 0; i < 18; ++i) J[i] = 0.0;
#pragma unroll
    for (int i = 0; i < 6; ++i) jp[i] = 0.0;
    double xx = 0.0, xy = 0.0, xz = 0.0, yy = 0.0, yz = 0.0, zz = 0.0;  // Newtonian part
#pragma unroll 1
    for (int i = 0; i < T.n_body; ++i) {
        const PoolBody& B = T.plan->b[i];
        double rp[3];
        pool_body_position<KM>(B, x, col, stride, rp);
        const double ir = rsqrt(pool_r2(rp));
        const double ir2 = ir * ir, kk = B.mass * ir2 * ir, k3 = 3.0 * kk * ir2;
        xx += k3 * rp[0] * rp[0] - kk;
        yy += k3 * rp[1] * rp[1] - kk;
        zz += k3 * rp[2] * rp[2] - kk;
        xy += k3 * rp[0] * rp[1];
        xz += k3 * rp[0] * rp[2];
        yz += k3 * rp[1] * rp[2];
        if (B.kind == FK_PLAIN) continue;
        const bool vel = B.kind != FK_EARTH;
        const double n[3] = {0.0, vel ? -c_tab.rot_s : 0.0, vel ? c_tab.rot_c : 1.0};
        TangentForce::j2_gradient(rp, ir, ir2, B.j2m * B.radius2, n, J);
        if (!vel) continue;
        double rv[3];
        pool_body_velocity<KM>(B, v, col, stride, rv);
        TangentForce::gr_gradient(rp, rv, ir, ir2, B.mass, J);
        if (B.kind == FK_SUN && ng.kind != 0) TangentForce::nongrav_gradient(ng, rp, rv, ir, J, jp);
    }
    J[0] += xx; J[1] += xy; J[2] += xz;
    J[6] += xy; J[7] += yy; J[8] += yz;
    J[12] += xz; J[13] += yz; J[14] += zz;
}

// The rounds of every group of the warp until the policies have no more work.
template <int S, int THREADS, int TANGENTS, bool KM, class Policy>
__device__ __forceinline__ void sens_pool_run(const PoolTables& T, double* smem, Policy& P,
                                              int max_rounds) {
    using Sh = SensPoolShared<S, THREADS, TANGENTS>;
    constexpr int GL = NODE_G * S, COLS = Sh::COLS;
    const int warp_lane = threadIdx.x & 31;
    const int gi = threadIdx.x / GL;
    SensPoolGroup G;
    G.lane = threadIdx.x & (NODE_G - 1);
    G.sub = S == 1 ? 0 : warp_lane / NODE_G;
    const int lane0 = S == 1 ? (warp_lane & ~(NODE_G - 1)) : 0;
    const unsigned gmask = S == 1 ? 0xFFu << lane0 : 0xffffffffu;
    G.gmask = gmask;
    const int lane = G.lane, sub = G.sub;
    double* rows = smem + T.n_slot * COLS + gi * Sh::ROWS;
    double* se = rows + 2 * 3 * POOL_B;
    double* st = se + 3 * NODE_G;
    double* ste = st + ST_ROW + 1;
    G.st = st;
    G.tan = ste + NODE_G;
    double* term = smem + T.n_slot * COLS + Sh::GROUPS * Sh::ROWS + gi * TERM_SLOTS * NODE_G + lane;
    double* col = smem + gi * NODE_G + lane;
    G.col = col;
    G.col_end = smem + gi * NODE_G + 7;
    G.stride = COLS;
    G.T = &T;
    G.leader = lane == 0 && sub == 0;
    G.owner = lane < 3 && sub == 0;
    const bool owner = G.owner, leader = G.leader;
    const int comp = lane < 3 ? lane : 0;
    const double2* nrow =
        reinterpret_cast<const double2*>(T.node + (lane < 7 ? lane + 1 : 8) * POOL_NODE);
    G.ng.base = nullptr;
    G.ng.stride = 0;
    G.ng.kind = 0;
    G.rc = ST_OK;
    int cur = 0;  // which of the two b rows is current
    G.sb = rows;
    int phase = SQ_FETCH, iter = 0, failures = 0, att = 0, rounds = 0;
    bool fresh = false, predict = false;
    double next_h = 0.0;

    for (;;) {
        if (phase == SQ_END) {
            P.job_done(G);
            __syncwarp(gmask);
            phase = SQ_FETCH;
        }
        if (phase == SQ_FETCH) {
            G.rc = ST_OK;
            att = iter = rounds = 0;
            predict = false;
            bool resume = false;
            if (!P.next(G, resume, failures, predict)) phase = SQ_FINISHED;
            else phase = G.rc != ST_OK ? SQ_END : (resume ? SQ_BEGIN : SQ_INIT);
            fresh = phase == SQ_INIT;
            __syncwarp(gmask);
        }
        if (__all_sync(0xffffffffu, phase == SQ_FINISHED)) break;
        if (phase == SQ_SEGMENT) {  // the epoch is reached: the next one, or done
            const bool more = P.segment_end(G, failures, predict);
            __syncwarp(gmask);
            phase = more ? SQ_INIT : SQ_END;
            fresh = more;
        }
        if (phase == SQ_BEGIN) {  // MIN_STEP, then truncate to the end (radau.rs:187-190,214-216)
            if (!P.begin_attempt(G, att, failures, predict)) {
                phase = SQ_END;
            } else {
                double h = st[ST_H];
                const double t = st[ST_T], tf = st[ST_TF];
                if (fabs(h) < 0.005) h = copysign(0.005, h);
                if (fabs(t - tf) <= fabs(h)) h = tf - t;
                double q = 0.0;
                if (predict) {
                    q = h / st[ST_HP];
                    if (owner) predict_b_row(G.sb + POOL_B * comp, q);
                }
                __syncwarp(gmask);  // every lane has read the proposed step
                if (leader) st[ST_H] = h;
                __syncwarp(gmask);
                P.attempt_predict(G, q);
                iter = 0;
                ++att;
                phase = SQ_ITER;
                fresh = true;
            }
        }
        bool active = phase == SQ_ITER || phase == SQ_INIT || phase == SQ_EXACT;
        if (active && rounds++ >= max_rounds) {
            G.rc = ST_TIMEOUT;
            phase = SQ_END;
            active = false;
        }
        const bool iter_round = phase == SQ_ITER;
        const bool need = active && fresh;
        const unsigned M = __ballot_sync(0xffffffffu, need);
        if (M) {
            if (need && sub == 0) {
                const double te = iter_round ? st[ST_T] + nrow[8].x * st[ST_H] : st[ST_T];
                ste[lane] = __dmul_rn(te - 2451545.0, 86400.0);
            }
            __syncwarp();
            pool_records<S, COLS, Sh::ROWS, KM>(T, M, gi, ste, smem);
            if (need && sub == 0) pool_chain<KM>(T, col, COLS);
            __syncwarp();
            fresh = false;
        }
        if (!active) continue;
        double xe[3], ve[3];
        if (iter_round) {
            pool_predict(nrow, G.sb, st, xe, ve);
        } else {
#pragma unroll
            for (int c = 0; c < 3; ++c) {
                xe[c] = st[ST_X + c];
                ve[c] = st[ST_V + c];
            }
        }
        // the exact evaluation of an accepted step is at the step end's time
        const double* cl = phase == SQ_EXACT ? G.col_end : G.col;
        PoolExact ex;
        ex.impact_id = 0;
        ex.min_r2 = 0.0;
        double na[3] = {0.0, 0.0, 0.0};
        if (G.ng.kind != 0) {
            const PoolBody& sun = T.plan->b[0];
            double rp[3], rv[3];
            pool_body_position<KM>(sun, xe, cl, COLS, rp);
            pool_body_velocity<KM>(sun, ve, cl, COLS, rv);
            const double3 p3 = make_double3(rp[0], rp[1], rp[2]), v3 = make_double3(rv[0], rv[1], rv[2]);
            const double3 r = (G.ng.kind == 1 && G.ng.p(9) == 0.0) ? nongrav_terms<false>(G.ng, p3, v3)
                                                                   : nongrav_accel(G.ng, p3, v3);
            na[0] = r.x; na[1] = r.y; na[2] = r.z;
        }
        if (S > 1) {
            const double own = sub == 0 ? na[0] : (sub == 1 ? na[1] : na[2]);
            const double e = pool_forces_wide<true, KM>(T.body, T.n_body, sub, cl, COLS, term,
                                                        !iter_round, false, xe, ve, ex, own);
            if (sub < 3) se[NODE_G * sub + lane] = e;
        } else {
            double ev[3];
            pool_forces<true, KM>(T.plan->b, T.n_vel, T.n_body, cl, COLS, !iter_round, false, xe, ve,
                                  ex, ev, na);
            se[lane] = ev[0];
            se[NODE_G + lane] = ev[1];
            se[2 * NODE_G + lane] = ev[2];
        }
        __syncwarp(gmask);
        if (!iter_round) {
            if (ex.impact_id != 0) {
                G.rc = ST_IMPACT;
                phase = SQ_END;
                continue;
            }
            const double t = st[ST_T], tf = st[ST_TF], h = st[ST_H];
            if (owner) st[ST_A + comp] = se[NODE_G * comp + lane];
            __syncwarp(gmask);
            if (phase == SQ_INIT) {
                if (fabs(tf - t) < 1e-10) {
                    phase = SQ_SEGMENT;
                    continue;
                }
                if (leader) st[ST_H] = copysign(0.1, tf - t);
                att = 0;
                predict = false;
            } else {
                P.end_attempt(G, iter, true);
                __syncwarp(gmask);
                if (leader) {
                    st[ST_HP] = h;
                    st[ST_H] = next_h;
                }
                predict = true;
                if (fabs(t - tf) < 1e-12) {
                    __syncwarp(gmask);
                    phase = SQ_SEGMENT;
                    continue;
                }
            }
            __syncwarp(gmask);
            failures = 0;
            phase = SQ_BEGIN;
            continue;
        }
        // corrector iteration (radau.rs:292-330); the new b goes to the other row
        double* old_b = G.sb;
        cur ^= 1;
        G.sb = rows + cur * 3 * POOL_B;
        double g[7], e7;
        pool_divided(se + NODE_G * comp, st[ST_A + comp], g, e7);
        const double change = fabs(g[6] - old_b[POOL_B * comp + 6]);
        const double limit = 1e-14 * (fabs(e7) + 1e-6);
        const unsigned above = __ballot_sync(gmask, owner && change >= limit);
        const unsigned number = __ballot_sync(gmask, owner && change == change);
        const bool conv = above == 0 && number != 0;
        if (owner) pool_store_b(g, G.sb + POOL_B * comp);
        __syncwarp(gmask);
        ++iter;
        if (conv || iter >= 10) P.last_iteration(G, old_b, xe, ve);
        if (conv) {
            const double h = st[ST_H], t = st[ST_T];
            const double fem = fmax(fmax(fabs(se[6]), fabs(se[NODE_G + 6])), fabs(se[2 * NODE_G + 6]));
            const double mb6 = fmax(fmax(fabs(G.sb[6]), fabs(G.sb[POOL_B + 6])), fabs(G.sb[2 * POOL_B + 6]));
            __syncwarp(gmask);
            if (owner) {
                const double h2 = h * h;
                double dw = 0.0, du = 0.0;
#pragma unroll
                for (int k = 0; k < 7; ++k) {
                    const double bck = G.sb[POOL_B * comp + k];
                    dw += bck * c_tab.w[k];
                    du += bck * c_tab.u[k];
                }
                const double vc = st[ST_V + comp], ac = st[ST_A + comp];
                st[ST_X + comp] += vc * h + h2 * (ac * 0.5 + dw);
                st[ST_V + comp] += h * (ac + du);
            }
            if (leader) st[ST_T] = t + h;
            next_h = h * clampd(pow(1e-6 * (fem + 1e-6) / mb6, 1.0 / 7.0), 0.25, 4.0);
            __syncwarp(gmask);
            phase = SQ_EXACT;
            continue;
        }
        if (iter >= 10) {  // not converged: retry with a smaller step (radau.rs:199-210)
            P.end_attempt(G, iter, false);
            const double h = st[ST_H] * 0.7;
            __syncwarp(gmask);
            if (leader) st[ST_H] = h;
            __syncwarp(gmask);
            predict = false;
            failures += 1;
            phase = SQ_BEGIN;
            if (failures > 10) {
                G.rc = ST_CONVERGENCE;
                phase = SQ_END;
            }
        }
    }
}

// ---------------------------------------------------------------------------------------
// What the forward passes share: one object per group, its checks and the epochs.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ void sens_pool_clear_b(const SensPoolGroup& G) {
    if (G.sub == 0) {
        G.sb[G.lane] = 0.0;
        G.sb[POOL_B + G.lane] = 0.0;
        G.sb[2 * POOL_B + G.lane] = 0.0;
    }
}

// The leader's start of object obj: the checks of nbody_sens_forward_kernel, the barycentric
// equatorial state into G.st; ST_PENDING when an epoch lies outside the window.
__device__ __forceinline__ int sens_pool_start(const SensPoolGroup& G, int64_t obj, int64_t n,
                                               const double* pos, const double* vel,
                                               const double* jd0, const double* epochs, int n_epochs,
                                               int frame, const CenterChain& chain) {
    const FastPlan& plan =
        G.T->n_body == c_plans.planets.n_body ? c_eph.fast_planets : c_eph.fast_all;
    const double t = jd0[obj];
    for (int k = 0; k < n_epochs; ++k)
        if (!in_window(t, epochs[k], plan.lo, plan.hi)) return ST_PENDING;
    double p[3], v[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        p[c] = pos[c * n + obj];
        v[c] = vel[c * n + obj];
    }
    int rc = ST_OK;
    if (!(isfinite(p[0]) && isfinite(p[1]) && isfinite(p[2]) && isfinite(v[0]) && isfinite(v[1]) &&
          isfinite(v[2]) && isfinite(t)))
        rc = ST_VALUE_ERROR;
    // the derivative of the comet model is taken with its time delay dt = 0
    if (G.ng.kind == 1 && G.ng.p(9) != 0.0) rc = ST_VALUE_ERROR;
    if (rc == ST_OK) rc = to_ssb_equatorial(t, frame, chain, p, v);
    G.st[ST_T] = t;
    G.st[ST_TF] = epochs[0];
    G.st[ST_H] = G.st[ST_HP] = 0.0;
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        G.st[ST_X + c] = p[c];
        G.st[ST_V + c] = v[c];
        G.st[ST_A + c] = 0.0;
    }
    return rc;
}

// The leader's store of the state at epoch k in the caller's frame; returns its outcome.
__device__ __forceinline__ int sens_pool_store_epoch(const SensPoolGroup& G, int64_t obj, int64_t n,
                                                     int k, int frame, const CenterChain& chain,
                                                     double* out_state) {
    double px[3], pv[3];
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        px[c] = G.st[ST_X + c];
        pv[c] = G.st[ST_V + c];
    }
    const int rc = from_ssb_equatorial(G.st[ST_TF], frame, chain, px, pv);
    double* o = out_state + (int64_t)k * 6 * n;
    const double nan = __longlong_as_double(0x7ff8000000000000LL);
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        o[c * n + obj] = rc == ST_OK ? px[c] : nan;
        o[(3 + c) * n + obj] = rc == ST_OK ? pv[c] : nan;
    }
    return rc;
}

// The group's state and b to a checkpoint or record slot (the layout of sens_store_state).
__device__ __forceinline__ void sens_pool_store_state(const SensPoolGroup& G, double* dst, double w2,
                                                      bool predict) {
    if (G.sub != 0) return;
    const double* st = G.st;
    const int lane = G.lane;
    if (lane == 0) {
        dst[0] = st[ST_T];
        dst[1] = st[ST_H];
        dst[2] = w2;
        dst[34] = predict ? st[ST_HP] : 0.0;
        dst[35] = SENS_BY_POOL;
    } else if (lane < 4) {
        const int from = lane == 1 ? ST_X : (lane == 2 ? ST_V : ST_A);
#pragma unroll
        for (int c = 0; c < 3; ++c) dst[1 + 3 * lane + c] = st[from + c];
    }
    if (lane < 7) {
        dst[13 + lane] = G.sb[lane];
        dst[20 + lane] = G.sb[POOL_B + lane];
        dst[27 + lane] = G.sb[2 * POOL_B + lane];
    }
}

// ---------------------------------------------------------------------------------------
// forward with checkpoints
// ---------------------------------------------------------------------------------------
struct SensPoolForward {
    const SensArgs& a;
    int64_t obj;  // the group's object; a.n or more: none
    bool first = true;
    int k = 0, nck = 0;

    __device__ bool next(SensPoolGroup& G, bool&, int& failures, bool&) {
        if (!first || obj >= a.n) return false;
        first = false;
        failures = 0;
        G.ng.base = a.nongrav ? a.nongrav + obj : nullptr;
        G.ng.stride = a.n;
        G.ng.kind = a.nongrav ? (int)a.nongrav[obj] : 0;
        sens_pool_clear_b(G);
        int rc = ST_OK;
        if (G.leader) {
            rc = sens_pool_start(G, obj, a.n, a.pos, a.vel, a.jd0, a.epochs, a.n_epochs, a.frame, a.chain);
            if (rc != ST_PENDING) a.ckpt_seg[obj] = 0;
        }
        G.rc = __shfl_sync(G.gmask, rc, __ffs(G.gmask) - 1);
        return true;
    }
    __device__ void job_done(SensPoolGroup& G) {
        if (!G.leader) return;
        int rc = G.rc;
        if (rc == ST_OK && nck > a.ckpt_cap) rc = ST_CHECKPOINT_FULL;
        a.status[obj] = rc;
        if (rc == ST_PENDING) return;
        a.ckpt_count[obj] = nck;
        if (G.rc != ST_OK) {  // epochs not reached are NaN
            const double nan = __longlong_as_double(0x7ff8000000000000LL);
            for (int e = k; e < a.n_epochs; ++e)
                for (int c = 0; c < 6; ++c) a.out_state[((int64_t)e * 6 + c) * a.n + obj] = nan;
            for (int e = k + 1; e < a.n_epochs; ++e) a.ckpt_seg[(int64_t)e * a.n + obj] = nck;
        }
    }
    __device__ bool begin_attempt(SensPoolGroup& G, int att, int failures, bool predict) {
        if (att % SENS_CK_ATTEMPTS == 0) {
            if (nck < a.ckpt_cap)
                sens_pool_store_state(G, a.ckpt + ((size_t)obj * a.ckpt_cap + nck) * SENS_STRIDE,
                                      (double)failures, predict);
            nck++;
            __syncwarp(G.gmask);
        }
        return true;
    }
    __device__ void attempt_predict(SensPoolGroup&, double) {}
    __device__ void last_iteration(SensPoolGroup&, const double*, const double*, const double*) {}
    __device__ void end_attempt(SensPoolGroup&, int, bool) {}
    __device__ bool segment_end(SensPoolGroup& G, int&, bool&) {
        int rc = ST_OK;
        if (G.leader) rc = sens_pool_store_epoch(G, obj, a.n, k, a.frame, a.chain, a.out_state);
        G.rc = __shfl_sync(G.gmask, rc, __ffs(G.gmask) - 1);
        if (G.rc != ST_OK || ++k >= a.n_epochs) return false;
        if (G.leader) {
            a.ckpt_seg[(int64_t)k * a.n + obj] = nck;
            G.st[ST_TF] = a.epochs[k];
        }
        sens_pool_clear_b(G);  // b restarts at zero in every fresh integration
        return true;
    }
};

template <int S, int THREADS, int MINB, bool KM>
__global__ void __launch_bounds__(THREADS, MINB) sens_pool_forward_kernel(SensArgs a) {
    extern __shared__ __align__(16) double s_pool[];
    __shared__ __align__(16) double s_node[9 * POOL_NODE];
    __shared__ PoolSeries s_src[MAX_SERIES];
    __shared__ PoolBody s_body[MAX_FORCE + 2];
    const PoolTables T = pool_tables(a.n_force, s_node, s_src, s_body);
    SensPoolForward P{a, ((int64_t)blockIdx.x * THREADS + threadIdx.x) / (NODE_G * S)};
    sens_pool_run<S, THREADS, 0, KM>(T, s_pool, P, a.max_loops * 12);
}

// ---------------------------------------------------------------------------------------
// the replays of every checkpoint block (nbody_sens_replay_kernel's work and layout)
// ---------------------------------------------------------------------------------------
struct SensPoolReplay {
    const SensArgs& a;
    int64_t total;
    int64_t item = 0;
    double* rec = nullptr;
    const double* after = nullptr;  // the checkpoint that the block leads to
    int na = 0;
    bool ended = false;

    __device__ bool next(SensPoolGroup& G, bool& resume, int& failures, bool& predict) {
        const int64_t n = a.n;
        for (;;) {
            int q = 0;
            if (G.leader) q = atomicAdd(a.rep_first + n + 1, 1);
            const int64_t idx = __shfl_sync(G.gmask, q, __ffs(G.gmask) - 1);
            if (idx >= total) return false;
            // the object holding block idx: the last o with rep_first[o] <= idx
            int64_t lo = 0, hi = n;
            while (hi - lo > 1) {
                const int64_t mid = (lo + hi) >> 1;
                if (a.rep_first[mid] <= idx) lo = mid;
                else hi = mid;
            }
            const int64_t obj = lo;
            const int at = (int)(idx - a.rep_first[obj]);
            const int cb = sens_pass_first(sens_block_count(a, obj), a.pass, a.window) + at;
            item = obj * a.window + at;
            int e0 = 0, e1 = a.n_epochs;  // the epoch segment: the last one starting at or before cb
            while (e1 - e0 > 1) {
                const int mid = (e0 + e1) >> 1;
                if (a.ckpt_seg[(int64_t)mid * n + obj] <= cb) e0 = mid;
                else e1 = mid;
            }
            const double* c = a.ckpt + ((size_t)obj * a.ckpt_cap + cb) * SENS_STRIDE;
            const double t = c[0], tf = a.epochs[e0];
            // (the window: checkpoints of another ephemeris than the present one)
            const FastPlan& plan = a.n_force == c_eph.n_force_planets ? c_eph.fast_planets : c_eph.fast_all;
            if (c[35] != SENS_BY_POOL || !in_window(t, tf, plan.lo, plan.hi)) {
                if (G.leader) {
                    a.rep_count[item] = SENS_PENDING;
                    atomicAdd(a.rep_first + n + 3, 1);
                }
                continue;
            }
            after = sens_next_checkpoint(a, obj, e0, cb);
            ended = false;
            G.ng.base = a.nongrav ? a.nongrav + obj : nullptr;
            G.ng.stride = n;
            G.ng.kind = a.nongrav ? (int)a.nongrav[obj] : 0;
            rec = a.rec_all + (size_t)item * (SENS_CK_ATTEMPTS + 1) * SENS_STRIDE;
            na = 0;
            failures = (int)c[2];
            predict = c[34] != 0.0;
            resume = true;
            if (G.leader) {
                G.st[ST_T] = t;
                G.st[ST_TF] = tf;
                G.st[ST_H] = c[1];
                G.st[ST_HP] = c[34];
            }
            if (G.sub == 0) {
                if (G.lane >= 1 && G.lane < 4) {
                    const int to = G.lane == 1 ? ST_X : (G.lane == 2 ? ST_V : ST_A);
#pragma unroll
                    for (int q3 = 0; q3 < 3; ++q3) G.st[to + q3] = c[1 + 3 * G.lane + q3];
                }
                const bool pad = G.lane == 7;
                G.sb[G.lane] = pad ? 0.0 : c[13 + G.lane];
                G.sb[POOL_B + G.lane] = pad ? 0.0 : c[20 + G.lane];
                G.sb[2 * POOL_B + G.lane] = pad ? 0.0 : c[27 + G.lane];
            }
            return true;
        }
    }
    __device__ void job_done(SensPoolGroup& G) {
        if (!G.leader) return;
        int rc = G.rc;
        if (rc == ST_OK && !sens_block_follows(after, ended, G.st[ST_T], G.st + ST_X))
            rc = ST_CHECKPOINT_MISMATCH;
        a.rep_count[item] = rc == ST_OK ? na : -1 - rc;
    }
    __device__ bool begin_attempt(SensPoolGroup& G, int, int, bool predict) {
        sens_pool_store_state(G, rec + (size_t)na * SENS_STRIDE, 0.0, predict);
        __syncwarp(G.gmask);
        if (na == SENS_CK_ATTEMPTS) return false;  // the block's end state is stored
        na++;
        return true;
    }
    __device__ void attempt_predict(SensPoolGroup& G, double q) {
        if (G.leader) rec[(size_t)(na - 1) * SENS_STRIDE + 34] = q;
    }
    __device__ void last_iteration(SensPoolGroup& G, const double* old_b, const double*, const double*) {
        if (G.sub == 0 && G.lane < 7) {  // the b that the last iteration's points came from
            double* d = rec + (size_t)(na - 1) * SENS_STRIDE;
            d[13 + G.lane] = old_b[G.lane];
            d[20 + G.lane] = old_b[POOL_B + G.lane];
            d[27 + G.lane] = old_b[2 * POOL_B + G.lane];
        }
    }
    __device__ void end_attempt(SensPoolGroup& G, int iter, bool converged) {
        if (G.leader) {
            double* d = rec + (size_t)(na - 1) * SENS_STRIDE;
            d[1] = G.st[ST_H];
            d[2] = (double)iter;
            d[3] = converged ? 1.0 : 0.0;
        }
    }
    __device__ bool segment_end(SensPoolGroup& G, int&, bool& predict) {
        sens_pool_store_state(G, rec + (size_t)na * SENS_STRIDE, 0.0, predict);
        ended = true;
        return false;
    }
};

template <int S, int THREADS, int MINB, bool KM>
__global__ void __launch_bounds__(THREADS, MINB) sens_pool_replay_kernel(SensArgs a) {
    extern __shared__ __align__(16) double s_pool[];
    __shared__ __align__(16) double s_node[9 * POOL_NODE];
    __shared__ PoolSeries s_src[MAX_SERIES];
    __shared__ PoolBody s_body[MAX_FORCE + 2];
    const PoolTables T = pool_tables(a.n_force, s_node, s_src, s_body);
    SensPoolReplay P{a, a.rep_first[a.n]};
    sens_pool_run<S, THREADS, 0, KM>(T, s_pool, P, a.max_loops * 12);
}

// ---------------------------------------------------------------------------------------
// forward sensitivities (stm_nodes.cuh's linearisation and tangent rows), a warp per object:
// the four sub-lanes of a node take two of the eight directions each, the 24 rows of db and of
// the state tangents a lane each.
// ---------------------------------------------------------------------------------------
template <bool KM>
struct SensPoolStm {
    const StmArgs& a;
    int64_t obj;
    bool first = true;
    int k = 0;
    double J[18], jp[6];  // the node's Jacobian at the last corrector iteration's point

    // da = J (dx, dv) + jp at the state, component sub and direction lane
    __device__ void tangent_acc(SensPoolGroup& G, const double Jn[18], const double jn[6]) {
        double* ts = G.tan;
        const int p = G.lane;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            if (c == G.sub) {
                double s = 0.0;
#pragma unroll
                for (int i = 0; i < 3; ++i)
                    s += Jn[6 * c + i] * ts[STM_DX + 8 * i + p] + Jn[6 * c + 3 + i] * ts[STM_DV + 8 * i + p];
                if (p == 6) s += jn[2 * c];
                if (p == 7) s += jn[2 * c + 1];
                ts[STM_DA + 8 * c + p] = s;
            }
        __syncwarp(G.gmask);
    }
    __device__ void state_jacobian(SensPoolGroup& G, const double* col, double Jn[18], double jn[6]) {
        const double x[3] = {G.st[ST_X], G.st[ST_X + 1], G.st[ST_X + 2]};
        const double v[3] = {G.st[ST_V], G.st[ST_V + 1], G.st[ST_V + 2]};
        pool_jacobian<KM>(*G.T, col, G.stride, G.ng, x, v, Jn, jn);
    }
    __device__ bool next(SensPoolGroup& G, bool&, int& failures, bool&) {
        if (!first || obj >= a.n) return false;
        first = false;
        failures = 0;
        G.ng.base = a.nongrav ? a.nongrav + obj : nullptr;
        G.ng.stride = a.n;
        G.ng.kind = a.nongrav ? (int)a.nongrav[obj] : 0;
        sens_pool_clear_b(G);
        int rc = ST_OK;
        if (G.leader)
            rc = sens_pool_start(G, obj, a.n, a.pos, a.vel, a.jd0, a.epochs, a.n_epochs, a.frame, a.chain);
        G.rc = __shfl_sync(G.gmask, rc, __ffs(G.gmask) - 1);
        // tangents of the initial state: d(equatorial state) / d(caller's state), A1, A2
        double R[3][3];
        sens_rotation(a.frame, R);
        const int p = G.lane;
#pragma unroll
        for (int c = 0; c < 3; ++c)
            if (c == G.sub) {
                double dx = 0.0, dv = 0.0;
#pragma unroll
                for (int q = 0; q < 3; ++q) {
                    if (p == q) dx = R[c][q];
                    if (p == 3 + q) dv = R[c][q];
                }
                G.tan[STM_DX + 8 * c + p] = dx;
                G.tan[STM_DV + 8 * c + p] = dv;
            }
        return true;
    }
    __device__ void job_done(SensPoolGroup& G) {
        if (G.leader) a.status[obj] = G.rc;
        if (G.rc == ST_OK || G.rc == ST_PENDING) return;
        const double nan = __longlong_as_double(0x7ff8000000000000LL);  // epochs not reached
        const int L = threadIdx.x & 31;
        for (int e = k; e < a.n_epochs; ++e) {
            if (L < 6) a.out_state[((int64_t)e * 6 + L) * a.n + obj] = nan;
            for (int r = L; r < 48; r += 32) a.out_stm[((int64_t)e * 48 + r) * a.n + obj] = nan;
        }
    }
    __device__ bool begin_attempt(SensPoolGroup& G, int att, int, bool) {
        if (att == 0) {  // a fresh integration: db = 0 and da at the start
            for (int i = threadIdx.x & 31; i < 168; i += 32) G.tan[STM_DB + i] = 0.0;
            double Jn[18], jn[6];
            state_jacobian(G, G.col, Jn, jn);
            tangent_acc(G, Jn, jn);
        }
        return true;
    }
    __device__ void attempt_predict(SensPoolGroup& G, double q) {
        if (q == 0.0) return;
        if (G.sub < 3) predict_b_row(G.tan + STM_DB + (8 * G.sub + G.lane) * 7, q);
        __syncwarp(G.gmask);
    }
    __device__ void last_iteration(SensPoolGroup& G, const double*, const double* xe, const double* ve) {
        pool_jacobian<KM>(*G.T, G.col, G.stride, G.ng, xe, ve, J, jp);
    }
    __device__ void end_attempt(SensPoolGroup& G, int M, bool converged) {
        double* ts = G.tan;
        const int lane = G.lane, sub = G.sub;
        // an accepted step has already moved to its end; h is the step taken
        const double h = G.st[ST_H], h2 = h * h;
        const double* node = G.T->node + (lane < 7 ? lane + 1 : 8) * POOL_NODE;
        const double f = node[16], frac2 = node[17];
        for (int m = 0; m < M; ++m) {
            if (lane < 7) {
#pragma unroll 1
                for (int pp = 0; pp < 2; ++pp) {
                    const int p = 2 * sub + pp;
                    double dX[3], dV[3];
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        const double* row = ts + STM_DB + (8 * c + p) * 7;
                        double bw = 0.0, bu = 0.0;
#pragma unroll
                        for (int kk = 0; kk < 7; ++kk) {
                            bw += node[kk] * row[kk];
                            bu += node[8 + kk] * row[kk];
                        }
                        const double dx = ts[STM_DX + 8 * c + p], dv = ts[STM_DV + 8 * c + p],
                                     da = ts[STM_DA + 8 * c + p];
                        dX[c] = dx + f * dv * h + frac2 * h2 * (da / 2.0 + bw);
                        dV[c] = dv + f * h * (da + bu);
                    }
#pragma unroll
                    for (int c = 0; c < 3; ++c) {
                        double s = 0.0;
#pragma unroll
                        for (int i = 0; i < 3; ++i) s += J[6 * c + i] * dX[i] + J[6 * c + 3 + i] * dV[i];
                        if (p == 6) s += jp[2 * c];
                        if (p == 7) s += jp[2 * c + 1];
                        ts[STM_DE + (lane * 3 + c) * 8 + p] = s;
                    }
                }
            }
            __syncwarp(G.gmask);
            if (sub < 3) {  // db = P (dE - da), component sub, direction lane
                const double da = ts[STM_DA + 8 * sub + lane];
                double e[7];
#pragma unroll
                for (int j = 0; j < 7; ++j) e[j] = ts[STM_DE + (j * 3 + sub) * 8 + lane] - da;
#pragma unroll
                for (int kk = 0; kk < 7; ++kk) {
                    double s = 0.0;
#pragma unroll
                    for (int j = 0; j < 7; ++j) s += c_tab.adj_p[kk][j] * e[j];
                    ts[STM_DB + (8 * sub + lane) * 7 + kk] = s;
                }
            }
            __syncwarp(G.gmask);
        }
        if (!converged) return;  // a failed attempt keeps the state; its b carries on
        if (sub < 3) {
            const double* row = ts + STM_DB + (8 * sub + lane) * 7;
            double dw = 0.0, du = 0.0;
#pragma unroll
            for (int kk = 0; kk < 7; ++kk) {
                dw += row[kk] * c_tab.w[kk];
                du += row[kk] * c_tab.u[kk];
            }
            double& dx = ts[STM_DX + 8 * sub + lane];
            double& dv = ts[STM_DV + 8 * sub + lane];
            const double da = ts[STM_DA + 8 * sub + lane];
            dx = dx + dv * h + h2 * (da * 0.5 + dw);
            dv = dv + h * (da + du);
        }
        __syncwarp(G.gmask);
        double Jn[18], jn[6];  // da' from the Jacobian at the accepted state
        state_jacobian(G, G.col_end, Jn, jn);
        tangent_acc(G, Jn, jn);
    }
    __device__ bool segment_end(SensPoolGroup& G, int&, bool&) {
        int rc = ST_OK;
        if (G.leader) rc = sens_pool_store_epoch(G, obj, a.n, k, a.frame, a.chain, a.out_state);
        G.rc = __shfl_sync(G.gmask, rc, __ffs(G.gmask) - 1);
        if (G.sub < 3) {  // back in the caller's frame: row sub of R^T d(state), column lane
            double R[3][3];
            sens_rotation(a.frame, R);
            double* phi = a.out_stm + (int64_t)k * 48 * a.n;
            const double nan = __longlong_as_double(0x7ff8000000000000LL);
            const int p = G.lane;
            double sx = 0.0, sv = 0.0;
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                const double r = G.sub == 0 ? R[q][0] : (G.sub == 1 ? R[q][1] : R[q][2]);
                sx += r * G.tan[STM_DX + 8 * q + p];
                sv += r * G.tan[STM_DV + 8 * q + p];
            }
            phi[(G.sub * TAN_DIRS + p) * a.n + obj] = G.rc == ST_OK ? sx : nan;
            phi[((3 + G.sub) * TAN_DIRS + p) * a.n + obj] = G.rc == ST_OK ? sv : nan;
        }
        if (G.rc != ST_OK || ++k >= a.n_epochs) return false;
        if (G.leader) G.st[ST_TF] = a.epochs[k];
        sens_pool_clear_b(G);
        return true;
    }
};

template <int MINB, bool KM>
__global__ void __launch_bounds__(WIDE_BLOCK, MINB) sens_pool_stm_kernel(StmArgs a) {
    extern __shared__ __align__(16) double s_pool[];
    __shared__ __align__(16) double s_node[9 * POOL_NODE];
    __shared__ PoolSeries s_src[MAX_SERIES];
    __shared__ PoolBody s_body[MAX_FORCE + 2];
    const PoolTables T = pool_tables(a.n_force, s_node, s_src, s_body);
    SensPoolStm<KM> P{a, (int64_t)blockIdx.x};
    sens_pool_run<4, WIDE_BLOCK, STM_ROW, KM>(T, s_pool, P, a.max_loops * 12);
}

}  // namespace kb
