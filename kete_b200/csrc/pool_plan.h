// pool_plan.h -- what the warp-pooled node kernels read of the ephemeris and the force model,
// built by the host (capi.cu) with every load and kept in pool.cu's constant memory.
#pragma once
#include "ephem.cuh"

namespace kb {

// Record series of the pooled node kernels (radau_pool.cuh): one per body or centre whose
// position enters the force, then one per body whose velocity does.  The host lays their
// records out in the pool for these kernels alone:
//   [mid_s, 1/radius_s, 86400/radius_s/AU_KM, 0, then per coefficient pair x0 x1 y0 y1 z0 z1]
// so that a pair's six coefficients are three consecutive 16-byte loads and series of fewer
// coefficients take fewer of them.
struct PoolSeries {
    int64_t offset;                     // pool offset of record 0
    double start_s, inv_intlen;         // record = clamp(floor((t - start_s) * inv_intlen))
    int32_t n_rec, rsize, pairs, slot;  // slot: doubles into a cache column
};
// One body of the pooled force sum, in the fast plan's order (the bodies with velocities, then
// the others; b[n_body] is a copy of the last one without mass or radius, the partner of an odd
// one).  j2m: 1.5 J2 mass; vscale: the velocity series' scale; chain: cache slot of the centre
// whose position the body's is relative to (-1: none).
struct PoolBody {
    double mass, radius, radius2, j2m, vscale;
    int32_t slot, vslot, chain, naif_id, kind, pad_;
};
constexpr int MAX_SERIES = 24;
constexpr int POOL_MAX_SLOTS = 57;  // doubles of a cache column (planets 39, with the asteroids 54)
constexpr int POOL_EARTH = 4;  // the Earth's place in the plan: Sun, Jupiter, Mercury, Venus, Earth
struct PoolPlan {
    int32_t ok, n_pos, n_series, n_body, n_vel, n_slot;
    int32_t km, pad_;  // 1: unscaled columns (radau_pool.cuh), for a plan too large for EPH_CACHE
    PoolSeries s[MAX_SERIES];  // n_pos positions (longest first), then velocities
    PoolBody b[MAX_FORCE + 2];
};
// The plans of PLANETS and MASSES, in the constant memory of pool.cu and sens_pool.cu.
struct PoolPlans {
    PoolPlan planets, all;
};
int upload_pool_plans(const PoolPlans& p);
int upload_pool_plans_sens(const PoolPlans& p);

}  // namespace kb
