// kernels.cu -- two-body, thread-per-object N-body Radau, ephemeris queries, processing
// order, flux, FOV and two-body STM kernels with their host launchers.  The node-parallel
// Radau launchers (nodes.cu), the sensitivity kernels (sens.cu, adjoint.cu) and system integration
// (long.cu) are translation units of their own; each carries its own copy of the device
// constants, which upload_tables / upload_ephem write to all of them.
#include <atomic>
#include <cstdio>

#include "common.cuh"
#include "ephem.cuh"
#include "facet_math.cuh"
#include "forces.cuh"
#include "internal.h"
#include "kepler.cuh"
#include "radau.cuh"

namespace kb {

// Kernels launched by this library since it was loaded (kete_b200_kernel_launches): every
// launch helper below adds the kernels it enqueued when it checks the launch.
std::atomic<int64_t> g_kernel_launches{0};
std::atomic<int64_t> g_device_allocations{0};

KB_CONSTANT_UPLOADER(kernels)

int upload_tables(const Tables& t) {
    int rc = 0;
    for (auto up : {upload_consts_kernels, upload_consts_nodes, upload_consts_pool,
                    upload_consts_sens, upload_consts_sens_nodes, upload_consts_sens_pool,
                    upload_consts_adjoint, upload_consts_long})
        if ((rc = up(&t, nullptr))) return rc;
    return 0;
}
int upload_ephem(const EphemConst& e) {
    int rc = 0;
    for (auto up : {upload_consts_kernels, upload_consts_nodes, upload_consts_pool,
                    upload_consts_sens, upload_consts_sens_nodes, upload_consts_sens_pool,
                    upload_consts_adjoint, upload_consts_long})
        if ((rc = up(nullptr, &e))) return rc;
    return 0;
}

// -------------------------------------------------------------------------------------------
// two-body (kete_core/propagation/kepler.rs:306-322 with the light-delay second pass of the
// PyO3 binding, src/kete/rust/kepler.rs:89-102).  One thread per object, SoA FP64.
// -------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128, 6) two_body_kernel(
    int64_t n, const double* __restrict__ pos, const double* __restrict__ vel,
    const double* __restrict__ jd0, const double* __restrict__ jd1,
    const double* __restrict__ obs, double* __restrict__ out_pos, double* __restrict__ out_vel,
    double* __restrict__ out_jd, int32_t* __restrict__ status) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double p[3] = {pos[i], pos[n + i], pos[2 * n + i]};
    double v[3] = {vel[i], vel[n + i], vel[2 * n + i]};
    const double t0 = jd0[i], t1 = jd1[i];
    double tj = t1;
    int rc = analytic_2_body(t1 - t0, p, v);
    if (rc == ST_OK && obs != nullptr) {
        const double o0 = obs[0], o1 = obs[1], o2 = obs[2];
        const double delay = -norm3(p[0] - o0, p[1] - o1, p[2] - o2) / C_AU_PER_DAY;
        const double t2 = tj + delay;
        rc = analytic_2_body(t2 - tj, p, v);
        tj = t2;
    }
    if (rc != ST_OK) {
        p[0] = p[1] = p[2] = v[0] = v[1] = v[2] = __longlong_as_double(0x7ff8000000000000LL);
        tj = t1;
    }
    out_pos[i] = p[0];
    out_pos[n + i] = p[1];
    out_pos[2 * n + i] = p[2];
    out_vel[i] = v[0];
    out_vel[n + i] = v[1];
    out_vel[2 * n + i] = v[2];
    if (out_jd) out_jd[i] = tj;
    status[i] = rc;
}

int launch_two_body(int64_t n, const double* pos, const double* vel, const double* jd0,
                    const double* jd1, const double* obs, double* out_pos, double* out_vel,
                    double* out_jd, int32_t* status, cudaStream_t stream) {
    if (n <= 0) return 0;
    const int block = 128;
    const int64_t grid = (n + block - 1) / block;
    two_body_kernel<<<(unsigned)grid, block, 0, stream>>>(n, pos, vel, jd0, jd1, obs, out_pos,
                                                          out_vel, out_jd, status);
    return launched(1, "two_body_kernel launch");
}

// -------------------------------------------------------------------------------------------
// N-body Radau, one object per thread (the plain form of propagate_n_body_spk,
// kete_core/propagation/mod.rs:70-118).
// -------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(128) nbody_thread_kernel(NBodyArgs a) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= a.n) return;
    const int64_t n = a.n;
    RadauObj s;
    s.t = a.jd0[i];
    const double tf = a.jd1[i];
    s.x[0] = a.pos[i]; s.x[1] = a.pos[n + i]; s.x[2] = a.pos[2 * n + i];
    s.v[0] = a.vel[i]; s.v[1] = a.vel[n + i]; s.v[2] = a.vel[2 * n + i];
    SpkForceUnrolled F;  // one object per thread: fully unrolled Chebyshev loops
    F.n_force = a.n_force;
    F.ng.base = a.nongrav ? a.nongrav + i : nullptr;
    F.ng.stride = n;
    F.ng.kind = a.nongrav ? (int)a.nongrav[i] : 0;
    F.impact_id = 0;
    F.min_dist = 1e300;
    F.min_id = 0;
    RadauCounters cnt;
    int rc = ST_OK;
    bool finite = isfinite(s.x[0]) && isfinite(s.x[1]) && isfinite(s.x[2]) && isfinite(s.v[0]) &&
                  isfinite(s.v[1]) && isfinite(s.v[2]) && isfinite(s.t);
    if (!finite) rc = ST_VALUE_ERROR;
    if (rc == ST_OK) rc = to_ssb_equatorial(s.t, a.frame, a.chain, s.x, s.v);
    if (rc == ST_OK) rc = radau_integrate(s, tf, F, cnt, a.max_loops);
    if (rc == ST_OK) rc = from_ssb_equatorial(tf, a.frame, a.chain, s.x, s.v);
    if (rc != ST_OK) {
        const double nan = __longlong_as_double(0x7ff8000000000000LL);
        s.x[0] = s.x[1] = s.x[2] = s.v[0] = s.v[1] = s.v[2] = nan;
    }
    a.out_pos[i] = s.x[0]; a.out_pos[n + i] = s.x[1]; a.out_pos[2 * n + i] = s.x[2];
    a.out_vel[i] = s.v[0]; a.out_vel[n + i] = s.v[1]; a.out_vel[2 * n + i] = s.v[2];
    a.status[i] = rc;
    if (a.impact_id) a.impact_id[i] = rc == ST_IMPACT ? F.impact_id : 0;
    if (a.impact_jd) a.impact_jd[i] = rc == ST_IMPACT ? s.t : 0.0;
    if (a.min_dist) a.min_dist[i] = F.min_dist;
    if (a.counters) {
        a.counters[i] = cnt.steps;
        a.counters[n + i] = cnt.iterations;
        a.counters[2 * n + i] = cnt.exact;
    }
}

int launch_nbody_thread(const NBodyArgs& a, int block, cudaStream_t stream) {
    if (a.n <= 0) return 0;
    if (block <= 0) block = 128;
    const int64_t grid = (a.n + block - 1) / block;
    nbody_thread_kernel<<<(unsigned)grid, block, 0, stream>>>(a);
    return launched(1, "nbody_thread_kernel launch");
}

// -------------------------------------------------------------------------------------------
// Radau with the central force only (propagate_two_body_radau / propagation_central,
// kete_core/propagation/mod.rs:35-46,126-138): checks the integrator in isolation.
// -------------------------------------------------------------------------------------------
__global__ void radau_central_kernel(int64_t n, const double* pos, const double* vel,
                                     const double* t0, const double* t1, double* out_pos,
                                     double* out_vel, int32_t* status) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    RadauObj s;
    s.t = t0[i];
    s.x[0] = pos[i]; s.x[1] = pos[n + i]; s.x[2] = pos[2 * n + i];
    s.v[0] = vel[i]; s.v[1] = vel[n + i]; s.v[2] = vel[2 * n + i];
    CentralForce F;
    F.impact_id = 0;
    F.min_dist = 0.0;
    F.min_id = 0;
    RadauCounters cnt;
    int rc = radau_integrate(s, t1[i], F, cnt, 1 << 20);
    out_pos[i] = s.x[0]; out_pos[n + i] = s.x[1]; out_pos[2 * n + i] = s.x[2];
    out_vel[i] = s.v[0]; out_vel[n + i] = s.v[1]; out_vel[2 * n + i] = s.v[2];
    status[i] = rc;
}

int launch_radau_central(int64_t n, const double* pos, const double* vel, const double* t0,
                         const double* t1, double* out_pos, double* out_vel, int32_t* status,
                         cudaStream_t stream) {
    if (n <= 0) return 0;
    const int block = 128;
    radau_central_kernel<<<(unsigned)((n + block - 1) / block), block, 0, stream>>>(
        n, pos, vel, t0, t1, out_pos, out_vel, status);
    return launched(1, "radau_central_kernel launch");
}

// -------------------------------------------------------------------------------------------
// batched SpkCollection::try_get_state (spk.rs:87-96): state of body `slot` (chained to the
// barycentre) minus the centre chain, in `frame`.
// -------------------------------------------------------------------------------------------
constexpr int SPK_BLOCK = 64;
__global__ void __launch_bounds__(SPK_BLOCK) spk_states_kernel(int64_t n, int32_t slot,
                                                               const double* jd,
                                                               CenterChain center_chain,
                                                               int frame, double* out6,
                                                               int32_t* status) {
    // the modified-difference work arrays of types 1/21 (76 doubles a thread) in shared
    // memory rather than local memory
    __shared__ double s_work[76 * SPK_BLOCK];
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double t = jd[i];
    double p[3] = {0, 0, 0}, v[3] = {0, 0, 0};
    int rc = ST_OK;
    // the body's own chain: raw(body) + raw(parent) ...
    int s = slot;
    for (int k = 0; k < 3 && s >= 0 && rc == ST_OK; ++k) {
        double sp[3], sv[3];
        rc = eph_raw(c_eph, s, t, sp, sv, s_work + threadIdx.x, SPK_BLOCK);
        for (int q = 0; q < 3; ++q) {
            p[q] += sp[q];
            v[q] += sv[q];
        }
        s = c_eph.slot[s].parent_slot;
    }
    if (s < -1 || s >= 0) rc = ST_DAF_LIMITS;  // centre chain not complete
    if (rc == ST_OK) rc = from_ssb_equatorial(t, frame, center_chain, p, v);
    for (int q = 0; q < 3; ++q) {
        out6[q * n + i] = p[q];
        out6[(3 + q) * n + i] = v[q];
    }
    status[i] = rc;
}

int launch_spk_states(int64_t n, int32_t slot, const double* jd,
                      const CenterChain& center_chain, int frame, double* out6, int32_t* status,
                      cudaStream_t stream) {
    if (n <= 0) return 0;
    const int block = SPK_BLOCK;
    spk_states_kernel<<<(unsigned)((n + block - 1) / block), block, 0, stream>>>(
        n, slot, jd, center_chain, frame, out6, status);
    return launched(1, "spk_states_kernel launch");
}

}  // namespace kb

namespace kb {

// -------------------------------------------------------------------------------------------
// FP64 pipe probe: independent DFMA chains, for the roofline denominator.  Each thread
// runs 16 independent accumulators for `iters` iterations (2 flops per FMA).
// -------------------------------------------------------------------------------------------
__global__ void __launch_bounds__(256) dfma_probe_kernel(int64_t iters, double seed, double* out) {
    double a[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) a[k] = seed + threadIdx.x * 1e-9 + k * 1e-7;
    const double m = 0.999999999, c = 1e-9;
    for (int64_t i = 0; i < iters; ++i) {
#pragma unroll
        for (int k = 0; k < 16; ++k) a[k] = fma(a[k], m, c);
    }
    double s = 0.0;
#pragma unroll
    for (int k = 0; k < 16; ++k) s += a[k];
    if (s == 12345.678) out[0] = s;  // practically never true; keeps the chains live
}

int fp64_probe(int64_t iters, double* tflops, float* ms_out) {
    int dev = 0, sms = 0;
    int rc = cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc) return rc;
    if ((rc = cuda_check(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev), "attr")))
        return rc;
    double* d_out = nullptr;
    if ((rc = cuda_check(counted_malloc((void**)&d_out, sizeof(double)), "cudaMalloc probe"))) return rc;
    const int block = 256, grid = sms * 8;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    dfma_probe_kernel<<<grid, block>>>(iters / 10, 1.0, d_out);  // warm-up
    cudaEventRecord(e0);
    dfma_probe_kernel<<<grid, block>>>(iters, 1.0, d_out);
    cudaEventRecord(e1);
    rc = cuda_check(cudaEventSynchronize(e1), "probe synchronize");
    float ms = 0.f;
    cudaEventElapsedTime(&ms, e0, e1);
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    cudaFree(d_out);
    if (rc) return rc;
    const double flops = 2.0 * 16.0 * (double)iters * (double)grid * (double)block;
    *tflops = flops / (ms * 1e-3) / 1e12;
    if (ms_out) *ms_out = ms;
    return 0;
}

}  // namespace kb

namespace kb {

// -------------------------------------------------------------------------------------------
// Processing order of the node kernel: objects with the most work first, where the work is
// the integration span in units of the object's orbital period (span x two-body mean motion
// from the vis-viva energy; r^-1.5 for unbound orbits), since the Radau steps scale with
// the orbit.  With a persistent grid the groups that finish early pick up the small ones
// and the tail is short; with one group per object, neighbours in a warp get similar work,
// so the warp-synchronous forms' groups wait less for each other.  Work is bucketed on a
// log2 scale (quarter-octave classes from 2^-8 to 2^7 radians); within a bucket the order is
// whatever the atomics give -- it does not affect any object's result.
//
// The warp-pooled node kernel evaluates the ephemeris from the fast plan's records alone, so
// the objects whose span [jd0, jd1] does not lie inside the plan's window (with a margin of
// 1e-6 day: every evaluation time of a Radau integration lies between jd0 and jd1 up to
// rounding) go to one last bucket.  Before it, the objects with a non-gravitational model (given
// ng) have the work classes to themselves: the pooled kernel integrates them on a few SMs of
// their own (the model's code, fetched by any warp of an SM, evicts the step loop from the
// SM's instruction cache), also most work first.  (In one bucket, unsorted, their long ones
// started late: 100,000 objects of the +-5 yr mix took 19.6 ms with a third of the SM time
// idle at the end.)  The header's range {0, ng start, outside start, n} splits the order.
// Callers without a window pass [-inf, inf] and ng = null.
// -------------------------------------------------------------------------------------------
static_assert(ORDER_WIDE + 3 <= ORDER_SCRATCH_HEADER, "order header too small");

__device__ __forceinline__ int work_bucket(int64_t i, int64_t n, const double* __restrict__ pos,
                                           const double* __restrict__ vel, double jd0, double jd1) {
    const double span = fabs(jd1 - jd0);
    const double px = pos[i], py = pos[n + i], pz = pos[2 * n + i];
    const double vx = vel[i], vy = vel[n + i], vz = vel[2 * n + i];
    const double r = sqrt(px * px + py * py + pz * pz);
    const double inv_a = 2.0 / r - (vx * vx + vy * vy + vz * vz) / GMS;
    const double mean_motion = inv_a > 0.0 ? sqrt(GMS * inv_a * inv_a * inv_a) : sqrt(GMS / (r * r * r));
    const double work = span * mean_motion;
    if (!(work > 0.0) || !isfinite(work)) return ORDER_CLASSES - 1;  // no work, NaN last
    const int b = (int)floor(log2(work) * 4.0) + 32;
    return ORDER_CLASSES - 1 - (b < 0 ? 0 : (b > ORDER_CLASSES - 1 ? ORDER_CLASSES - 1 : b));
}

__device__ __forceinline__ int order_bucket(int64_t i, int64_t n, const double* __restrict__ pos,
                                            const double* __restrict__ vel, double t0, double t1,
                                            double lo, double hi, const double* __restrict__ ng) {
    if (!in_window(t0, t1, lo, hi)) return ORDER_OUT_BUCKET;
    return work_bucket(i, n, pos, vel, t0, t1) + (ng && ng[i] != 0.0 ? ORDER_NG_BUCKET : 0);
}

__global__ void order_hist_kernel(int64_t n, const double* __restrict__ pos,
                                  const double* __restrict__ vel, const double* __restrict__ jd0,
                                  const double* __restrict__ jd1, double lo, double hi,
                                  const double* __restrict__ ng, int* __restrict__ scratch) {
    __shared__ int h[ORDER_ALL_BUCKETS];
    for (int i = threadIdx.x; i < ORDER_ALL_BUCKETS; i += blockDim.x) h[i] = 0;
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n;
         i += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(&h[order_bucket(i, n, pos, vel, jd0[i], jd1[i], lo, hi, ng)], 1);
    __syncthreads();
    for (int i = threadIdx.x; i < ORDER_ALL_BUCKETS; i += blockDim.x)
        if (h[i]) atomicAdd(&scratch[1 + i], h[i]);
}

constexpr int ORDER_BLOCK = 256;

// Bucket starts (the cursors) and the range from the histogram: one block, one bucket a thread.
//
// groups > 0 (a persistent pooled launch with that many lane groups): the objects of the classes
// whose work is over a group's share of all the work would still run when the others are done;
// the pooled kernel gives them a warp each (at most half its warps' worth).
__global__ void __launch_bounds__(ORDER_BLOCK) order_scan_kernel(int groups,
                                                                 int* __restrict__ scratch) {
    __shared__ int start[ORDER_BLOCK];
    __shared__ float total;
    const int t = threadIdx.x;
    const int own = t < ORDER_ALL_BUCKETS ? scratch[1 + t] : 0;
    start[t] = own;
    __syncthreads();
    for (int o = 1; o < ORDER_BLOCK; o <<= 1) {  // inclusive sums
        const int v = t >= o ? start[t - o] : 0;
        __syncthreads();
        start[t] += v;
        __syncthreads();
    }
    if (t < ORDER_ALL_BUCKETS) scratch[1 + ORDER_ALL_BUCKETS + t] = start[t] - own;
    if (t == 0) {
        scratch[ORDER_RANGE] = 0;
        scratch[ORDER_RANGE + 1] = start[ORDER_NG_BUCKET - 1];
        scratch[ORDER_RANGE + 2] = start[ORDER_OUT_BUCKET - 1];
        scratch[ORDER_RANGE + 3] = start[ORDER_OUT_BUCKET];
        total = 0.0f;
    }
    if (groups <= 0) return;
    __syncthreads();
    const int cls = t < ORDER_NG_BUCKET ? t : t - ORDER_NG_BUCKET;
    const float work = exp2f((float)(ORDER_CLASSES - 1 - 32 - cls) * 0.25f);  // the class's least
    if (t < ORDER_OUT_BUCKET) atomicAdd(&total, (float)own * work * 1.09f);
    __syncthreads();
    if (t == 0 || t == ORDER_NG_BUCKET) {
        const float limit = total / (float)groups;
        const int most = groups / 16;  // of each part: a quarter of the warps
        int heavy = 0;
        for (int c = 0; c < ORDER_CLASSES; ++c) {
            const int add = scratch[1 + t + c];
            if (exp2f((float)(ORDER_CLASSES - 1 - 32 - c) * 0.25f) <= limit || heavy + add > most) break;
            heavy += add;
        }
        scratch[ORDER_WIDE + (t ? 1 : 0)] = heavy;
        scratch[t ? ORDER_QUEUE3 : 0] = heavy;
    }
}

// Tiles of one object per thread: ranks inside a tile come from shared-memory counters and a
// tile takes its place in each bucket with one global atomic (one per object on a few hot
// cursors took 223 us on 1M objects).
__global__ void __launch_bounds__(ORDER_BLOCK) order_scatter_kernel(
    int64_t n, const double* __restrict__ pos, const double* __restrict__ vel,
    const double* __restrict__ jd0, const double* __restrict__ jd1, double lo, double hi,
    const double* __restrict__ ng, int* __restrict__ scratch, int32_t* __restrict__ order) {
    __shared__ int count[ORDER_ALL_BUCKETS], base[ORDER_ALL_BUCKETS];
    const int t = threadIdx.x;
    for (int64_t first = (int64_t)blockIdx.x * ORDER_BLOCK; first < n;
         first += (int64_t)gridDim.x * ORDER_BLOCK) {
        if (t < ORDER_ALL_BUCKETS) count[t] = 0;
        __syncthreads();
        const int64_t i = first + t;
        int b = 0, rank = 0;
        if (i < n) {
            b = order_bucket(i, n, pos, vel, jd0[i], jd1[i], lo, hi, ng);
            rank = atomicAdd(&count[b], 1);
        }
        __syncthreads();
        if (t < ORDER_ALL_BUCKETS && count[t])
            base[t] = atomicAdd(&scratch[1 + ORDER_ALL_BUCKETS + t], count[t]);
        __syncthreads();
        if (i < n) {
            const int p = base[b] + rank;
            if (p >= 0 && p < n) order[p] = (int32_t)i;
        }
    }
}

int preload_order_kernels() {
    cudaFuncAttributes fa;
    int rc = 0;
    for (const void* f : {(const void*)order_hist_kernel, (const void*)order_scan_kernel,
                          (const void*)order_scatter_kernel})
        if ((rc = cuda_check(cudaFuncGetAttributes(&fa, f), "load ordering kernels"))) return rc;
    return 0;
}

// Zero the header, histogram the work, scan, scatter.  scratch must hold
// ORDER_SCRATCH_HEADER + n ints; order = scratch + ORDER_SCRATCH_HEADER.  [lo, hi]: the fast
// plan's window whose outsiders are ordered last, ng: the non-gravitational rows whose
// objects are ordered just before them ([-inf, inf] and null: no split).
int launch_span_order(int64_t n, const double* pos, const double* vel, const double* jd0,
                      const double* jd1, double lo, double hi, const double* ng, int groups,
                      int* scratch, cudaStream_t stream) {
    int rc = cuda_check(cudaMemsetAsync(scratch, 0, ORDER_SCRATCH_HEADER * sizeof(int), stream),
                        "clear order header");
    if (rc || n <= 0) return rc;
    const int64_t g = (n + ORDER_BLOCK - 1) / ORDER_BLOCK;
    const int grid = (int)(g > 1184 ? 1184 : g);
    order_hist_kernel<<<grid, ORDER_BLOCK, 0, stream>>>(n, pos, vel, jd0, jd1, lo, hi, ng, scratch);
    order_scan_kernel<<<1, ORDER_BLOCK, 0, stream>>>(groups, scratch);
    order_scatter_kernel<<<grid, ORDER_BLOCK, 0, stream>>>(
        n, pos, vel, jd0, jd1, lo, hi, ng, scratch, (int32_t*)(scratch + ORDER_SCRATCH_HEADER));
    return launched(3, "span order launch");
}

}  // namespace kb

#include "flux.cuh"

namespace kb {

// -------------------------------------------------------------------------------------------
// hg_apparent_mag for n geometries (src/kete/rust/flux/reflected.rs:120-132)
// -------------------------------------------------------------------------------------------
__global__ void hg_mag_kernel(int64_t n, const double* __restrict__ s2obj,
                              const double* __restrict__ s2obs, const double* __restrict__ h,
                              const double* __restrict__ g, double* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double a[3] = {s2obj[i], s2obj[n + i], s2obj[2 * n + i]};
    const double b[3] = {s2obs[i], s2obs[n + i], s2obs[2 * n + i]};
    out[i] = hg_apparent_mag(a, b, h[i], g[i]);
}

int launch_hg_mag(int64_t n, const double* s2obj, const double* s2obs, const double* h,
                  const double* g, double* out, cudaStream_t stream) {
    if (n <= 0) return 0;
    hg_mag_kernel<<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(n, s2obj, s2obs, h, g, out);
    return launched(1, "hg_mag_kernel launch");
}

// -------------------------------------------------------------------------------------------
// NEATM and FRM total flux (NeatmParams / FrmParams::apparent_total_flux, flux/neatm.rs:143-185,
// flux/frm.rs:137-185).  One warp per geometry.  A facet adds to the thermal sum only when
// the observer sees it and its temperature is above black_body_flux's 30 K floor
// (common.rs:139-154), and on a sphere that is a scattered half or less of the 2048 facets.
// So the warp first tests 32 facets at a time (two dot products), appends the survivors'
// (cos, seen) pairs to a per-warp queue in shared memory, and evaluates the black bodies
// only in full 32-facet batches: every lane busy on the exp-heavy part.  Band sums are
// reduced across the warp at the end.
// -------------------------------------------------------------------------------------------
constexpr int THERMAL_WARPS = 4;

// The WISE colour corrections at temperature t in [100, 400] (constants/wise.rs:40-85): the
// first three divide, the fourth, of l = log(t), multiplies.
__device__ __forceinline__ void wise_factors(double t, double l, double& d0, double& d1, double& d2,
                                             double& w4) {
    const double t2 = t * t, t3 = t * t2, t4 = t2 * t2, l2 = l * l;
    const FacetConst& C = c_fc;
    w4 = C.w4[0] + C.w4[1] * l + C.w4[2] * l2 + C.w4[3] * (l * l2) + C.w4[4] * (l2 * l2);
    d0 = C.w1[0] + C.w1[1] * t + C.w1[2] * t2 + C.w1[3] * t3 + C.w1[4] * t4;
    d1 = C.w2[0] + C.w2[1] * t + C.w2[2] * t2 + C.w2[3] * t3 + C.w2[4] * t4;
    d2 = C.w3[0] + C.w3[1] * t + C.w3[2] * t2 + C.w3[3] * t3 + C.w3[4] * t4;
}

// Black-body sum of one surviving facet into th[]: temperature from the cos term, then per
// band coef / (exp(k / T) - 1) (common.rs:139-154) with the WISE colour correction folded
// into the same division.  Bands the caller does not have carry coef = 0, k = 1.
//
// Bound by instruction issue and the FP64 pipe (60% and 55% busy; 11,300 warp instructions a
// geometry, 21,300 with the library's functions and all of a geometry in one warp; 100,000
// geometries with four WISE bands 2.27 -> 1.44 ms, with two NEOS bands 1.24 -> 0.80): T = Tss cos^(1/4) and 1 / T
// come from two reciprocal square roots, the bands' divisions from one reciprocal of their
// product.  That holds while the exponentials' product stays below e^600 (the WISE and NEOS
// bands at 30 K: e^311) and no denominator vanishes (an infinite temperature, a band whose
// exponential rounds to one: inv_ss is NaN there); other facets take the plain form, a division
// a band.
template <int NB, bool CC>
static __device__ __noinline__ void thermal_facet_plain(const NeatmArgs& a, double temp, double seen,
                                                       double (&th)[NB]) {
    double d[3], w4;
    if (CC) {
        const double t = clampd(temp, 100.0, 400.0);
        wise_factors(t, log(t), d[0], d[1], d[2], w4);
    }
    for (int b = 0; b < NB; ++b) {
        if (a.bb_coef[b] == 0.0) continue;  // 0, also over a vanishing denominator
        const double em1 = exp(a.bb_k[b] / temp) - 1.0;
        const double ff = a.bb_coef[b] / (CC && b < 3 ? em1 * d[b < 3 ? b : 0] : em1);
        th[b] += seen * (CC && b == 3 ? ff * w4 : ff);
    }
}

template <int NB, bool CC>
__device__ __forceinline__ void thermal_facet(const NeatmArgs& a, double tmp, double seen,
                                              double ss_temp, double inv_ss,
                                              const double* __restrict__ table, double (&th)[NB]) {
    const double root = tmp * rsqrt3(tmp), w = rsqrt3(root);  // tmp^(1/2), tmp^(-1/4)
    const double temp = root * w * ss_temp;
    if (!(temp >= 30.0)) return;
    const double inv_t = w * inv_ss;
    if (!(a.bb_ksum * inv_t < 600.0)) {
        thermal_facet_plain<NB, CC>(a, temp, seen, th);
        return;
    }
    double den[NB];
#pragma unroll
    for (int b = 0; b < NB; ++b) den[b] = exp_positive(a.bb_k[b] * inv_t, table) - 1.0;
    double w4 = 1.0;
    if (CC) {
        const double t = clampd(temp, 100.0, 400.0);
        double d0, d1, d2;
        wise_factors(t, log_kelvin(t), d0, d1, d2, w4);
        den[0] *= d0;
        den[1] *= d1;
        den[2] *= d2;
    }
    // seen / (product of all), then each band's by the product of the others
    double pre[NB];
    pre[0] = den[0];
#pragma unroll
    for (int b = 1; b < NB; ++b) pre[b] = pre[b - 1] * den[b];
    double r = seen * recip3(pre[NB - 1]);
#pragma unroll
    for (int b = NB - 1; b >= 0; --b) {
        const double inv = b ? r * pre[b ? b - 1 : 0] : r;
        r *= den[b];
        const double ff = a.bb_coef[b] * inv;
        th[b] = CC && b == 3 ? fma(ff, w4, th[b]) : th[b] + ff;
    }
}

// A block takes per_block geometries (a power of two up to THERMAL_MAX): what each needs before
// the facets and the reflected light after them run one geometry (and band) a thread, the facet
// sums one geometry a warp.  (With all of it one geometry a warp, the trigonometry of four lanes
// cost a sixth of the instructions.)
constexpr int THERMAL_MAX = 16;
template <int NB, bool CC>
__global__ void __launch_bounds__(32 * THERMAL_WARPS, 8) thermal_kernel(NeatmArgs a, int per_block) {
    __shared__ double2 queue[THERMAL_WARPS][96];
    __shared__ double s_geo[10][THERMAL_MAX];  // to the Sun, to the observer, T, 1 / T, cos, sin
    __shared__ double s_th[NB][THERMAL_MAX];
    __shared__ double s_exp[EXP_TABLE];  // 2^(j / 32)
    if (threadIdx.x < EXP_TABLE) s_exp[threadIdx.x] = exp2(threadIdx.x * (1.0 / EXP_TABLE));
    const int lane = threadIdx.x & 31;
    const int64_t n = a.n, first = (int64_t)blockIdx.x * per_block;
    const int count_geo = (int)(n - first < per_block ? n - first : per_block);
    if ((int)threadIdx.x < count_geo) {
        const int g = threadIdx.x;
        const int64_t i = first + g;
        const double s2obj[3] = {a.sun2obj[i], a.sun2obj[n + i], a.sun2obj[2 * n + i]};
        const double s2obs[3] = {a.sun2obs[i], a.sun2obs[n + i], a.sun2obs[2 * n + i]};
        const double obj2sun[3] = {-s2obj[0], -s2obj[1], -s2obj[2]};
        const double obs2obj[3] = {s2obj[0] - s2obs[0], s2obj[1] - s2obs[1], s2obj[2] - s2obs[2]};
        const double obs2obj_r = norm3(obs2obj[0], obs2obj[1], obs2obj[2]);
        // sub_solar_temperature (common.rs:220-236); the FRM's beaming is pi (frm.rs:95-101)
        const double emis = a.emissivity[i];
        const double phase_integral = 0.29 + 0.684 * a.g_param[i];
        const double bond_albedo = a.vis_albedo[i] * phase_integral;
        const double r2 = obj2sun[0] * obj2sun[0] + obj2sun[1] * obj2sun[1] + obj2sun[2] * obj2sun[2];
        const double reflected = (1.0 - bond_albedo) * SOLAR_FLUX / r2;
        const double beam = a.model == 1 ? PI : a.beaming[i];
        double ss_temp = reflected / (beam * emis * STEFAN_BOLTZMANN);
        ss_temp = ss_temp <= 0.0 ? 0.0 : sqrt(sqrt(ss_temp));
        const double ns = norm3(obj2sun[0], obj2sun[1], obj2sun[2]);
        for (int c = 0; c < 3; ++c) {
            s_geo[c][g] = obj2sun[c] / ns;
            s_geo[3 + c][g] = obs2obj[c] / obs2obj_r;
        }
        s_geo[6][g] = ss_temp;
        // used where the temperature is at least 30 K; no facet is hotter than ss_temp
        const double inv_ss = 1.0 / ss_temp;
        s_geo[7][g] = a.bb_kmin * inv_ss > 1e-15 ? inv_ss : __longlong_as_double(0x7ff8000000000000LL);
        // FRM: cos(lat_facet - lat_sun) (frm_facet_temperature, frm.rs:19-30) expanded with
        // the facet's cos/sin of latitude from the table
        if (a.model == 1) {
            const double sun_lat = asin(obj2sun[2] / ns);
            s_geo[8][g] = cos(sun_lat);
            s_geo[9][g] = sin(sun_lat);
        }
    }
    __syncthreads();
    double2* q = queue[threadIdx.x >> 5];
    const unsigned below = (1u << lane) - 1u;
    const double *t0 = a.facets + (a.model == 1 ? 3 * N_FACETS : 0), *t1 = t0 + N_FACETS;
    for (int g = threadIdx.x >> 5; g < count_geo; g += THERMAL_WARPS) {
        const double o0 = s_geo[3][g], o1 = s_geo[4][g], o2 = s_geo[5][g];
        const double ss_temp = s_geo[6][g], inv_ss = s_geo[7][g];
        // the temperature's cosine: a table row pair by (c0, c1) plus, NEATM, nz by c2
        const double c0 = s_geo[a.model == 1 ? 8 : 0][g], c1 = s_geo[a.model == 1 ? 9 : 1][g];
        const double c2 = a.model == 1 ? 0.0 : s_geo[2][g];
        double th[NB];
#pragma unroll
        for (int b = 0; b < NB; ++b) th[b] = 0.0;
        int count = 0;  // queued facets, warp-uniform
        for (int base = 0; base < N_FACETS; base += 64) {
#pragma unroll
            for (int half = 0; half < 2; ++half) {
                const int f = base + 32 * half + lane;
                const double nx = __ldg(a.facets + f), ny = __ldg(a.facets + N_FACETS + f),
                             nz = __ldg(a.facets + 2 * N_FACETS + f);
                const double seen = -(nx * o0 + ny * o1 + nz * o2);
                const double tmp = a.model == 1 ? __ldg(t0 + f) * c0 + __ldg(t1 + f) * c1
                                                : nx * c0 + ny * c1 + nz * c2;
                const bool keep = seen > 0.0 && tmp > 0.0;
                const unsigned m = __ballot_sync(0xffffffffu, keep);
                if (keep) q[count + __popc(m & below)] = make_double2(tmp, seen);
                count += __popc(m);
            }
            __syncwarp();
            while (count >= 32) {  // the queue's last 32
                count -= 32;
                const double2 e = q[count + lane];
                thermal_facet<NB, CC>(a, e.x, e.y, ss_temp, inv_ss, s_exp, th);
            }
            __syncwarp();
        }
        if (lane < count) {
            const double2 e = q[lane];
            thermal_facet<NB, CC>(a, e.x, e.y, ss_temp, inv_ss, s_exp, th);
        }
#pragma unroll
        for (int b = 0; b < NB; ++b) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) th[b] += __shfl_xor_sync(0xffffffffu, th[b], o);
            if (lane == 0) s_th[b][g] = th[b];
        }
        __syncwarp();
    }
    __syncthreads();
    for (int k = threadIdx.x; k < per_block * a.n_bands; k += blockDim.x) {
        const int b = k / per_block, g = k - b * per_block;
        if (g >= count_geo) continue;
        const int64_t i = first + g;
        const double s2obj[3] = {a.sun2obj[i], a.sun2obj[n + i], a.sun2obj[2 * n + i]};
        const double s2obs[3] = {a.sun2obs[i], a.sun2obs[n + i], a.sun2obs[2 * n + i]};
        const double gp = a.g_param[i], diam = a.diam[i];
        // Lambertian scale emissivity * pi * (r / D)^-2 (common.rs:190-205) and the facet area
        const double obs2obj_r = norm3(s2obj[0] - s2obs[0], s2obj[1] - s2obs[1], s2obj[2] - s2obs[2]);
        const double dscale = obs2obj_r * AU_KM / diam;
        const double thb =
            s_th[b][g] * (a.emissivity[i] * PI * (1.0 / (dscale * dscale)) * a.facet_area);
        const double refl = hg_apparent_flux(s2obj, s2obs, gp, diam, a.wavelength[b],
                                             a.band_albedo[(int64_t)b * n + i]) *
                            a.sun_correction[b];
        const double total = thb + refl;
        a.thermal[(int64_t)b * n + i] = thb;
        a.hg_fluxes[(int64_t)b * n + i] = refl;
        a.fluxes[(int64_t)b * n + i] = total;
        if (a.mags) a.mags[(int64_t)b * n + i] = a.have_zero_mags ? -2.5 * log10(total / a.zero_mag[b])
                                                                  : __longlong_as_double(0x7ff8000000000000LL);
        if (b == 0) {
            const double vm = hg_apparent_mag(s2obj, s2obs, a.h_mag[i], gp);
            a.v_mag[i] = vm;
            a.v_flux[i] = -2.5 * log10(vm / V_MAG_ZERO);  // flux_to_mag(v_mag, V_MAG_ZERO), neatm.rs:167
        }
    }
}

int launch_neatm(const NeatmArgs& a, cudaStream_t stream) {
    if (a.n <= 0) return 0;
    // a warp per geometry until the GPU is full of them (8 blocks an SM) twice, then up to
    // THERMAL_MAX a block
    int sms = 0;
    const int rc = sm_count(&sms);
    if (rc) return rc;
    int per_block = THERMAL_WARPS;
    while (per_block < THERMAL_MAX && a.n >= (int64_t)per_block * sms * 8 * 2) per_block *= 2;
    const unsigned grid = (unsigned)((a.n + per_block - 1) / per_block);
    const unsigned block = 32 * THERMAL_WARPS;
    if (a.wise_cc)  // the capi admits colour corrections only with the 4 WISE bands
        thermal_kernel<4, true><<<grid, block, 0, stream>>>(a, per_block);
    else if (a.n_bands <= 2)
        thermal_kernel<2, false><<<grid, block, 0, stream>>>(a, per_block);
    else if (a.n_bands <= 4)
        thermal_kernel<4, false><<<grid, block, 0, stream>>>(a, per_block);
    else
        thermal_kernel<MAX_BANDS, false><<<grid, block, 0, stream>>>(a, per_block);
    return launched(1, "thermal_kernel launch");
}

}  // namespace kb

#include "fov.cuh"

namespace kb {

int launch_fov_prefilter(const FovArgs& a, cudaStream_t stream) {
    if (a.n_obj <= 0 || a.n_fov <= 0) return 0;
    fov_prefilter_kernel<<<(unsigned)((a.n_obj + 127) / 128), 128, 0, stream>>>(a);
    return launched(1, "fov_prefilter_kernel launch");
}

int launch_fov_screen(const FovArgs& a, cudaStream_t stream) {
    if (a.n_obj <= 0 || a.n_fov <= 0) return 0;
    fov_screen_kernel<<<(unsigned)((a.n_obj + 127) / 128), 128, 0, stream>>>(a);
    return launched(1, "fov_screen_kernel launch");
}

int launch_fov_pairs(const FovArgs& a, int64_t m, cudaStream_t stream) {
    if (m <= 0) return 0;
    fov_pairs_kernel<<<(unsigned)((m + 127) / 128), 128, 0, stream>>>(a, m);
    return launched(1, "fov_pairs_kernel launch");
}

int launch_fov_gather(const FovArgs& a, int64_t m, double* gpos, double* gvel, double* gjd0,
                      double* gjd1, cudaStream_t stream) {
    if (m <= 0) return 0;
    fov_gather_kernel<<<(unsigned)((m + 127) / 128), 128, 0, stream>>>(a, m, gpos, gvel, gjd0, gjd1);
    return launched(1, "fov_gather_kernel launch");
}

int launch_fov_contains(int64_t n_vec, const double* vec, int64_t n_fov, const double* fov,
                        int64_t capacity, unsigned long long* counter, int32_t* out_fov,
                        int32_t* out_idx, cudaStream_t stream) {
    if (n_vec <= 0 || n_fov <= 0) return 0;
    fov_contains_kernel<<<(unsigned)((n_vec + 127) / 128), 128, 0, stream>>>(
        n_vec, vec, n_fov, fov, capacity, counter, out_fov, out_idx);
    return launched(1, "fov_contains_kernel launch");
}

int launch_fov_finish(const FovArgs& a, int64_t m, const double* npos, const double* nvel,
                      const int32_t* nst, cudaStream_t stream) {
    if (m <= 0) return 0;
    fov_nbody_finish_kernel<<<(unsigned)((m + 127) / 128), 128, 0, stream>>>(a, m, npos, nvel, nst);
    return launched(1, "fov_nbody_finish_kernel launch");
}

}  // namespace kb

// -------------------------------------------------------------------------------------------
// Two-body state-transition matrices with covariance propagation (compute_stm,
// propagate_covariance: src/kete/state_transition.py:8-59, corrected as kepler_stm.cuh
// describes), and the covariance sandwich Phi C Phi^T on its own for other matrices.
// -------------------------------------------------------------------------------------------
#include "kepler_stm.cuh"

namespace kb {

// out (rows x rows) = Phi (rows x cols) C (cols x cols) Phi^T for object i; SoA with the
// object index fastest.
__device__ __forceinline__ void covariance_sandwich(int64_t n, int64_t i, int rows, int cols,
                                                    const double* Phi, const double* C,
                                                    double* out) {
    for (int r = 0; r < rows; ++r)
        for (int q = r; q < rows; ++q) {
            double acc = 0.0;
            for (int a = 0; a < cols; ++a) {
                double inner = 0.0;
                for (int b = 0; b < cols; ++b)
                    inner += C[(int64_t)(a * cols + b) * n + i] * Phi[(int64_t)(q * cols + b) * n + i];
                acc += Phi[(int64_t)(r * cols + a) * n + i] * inner;
            }
            out[(int64_t)(r * rows + q) * n + i] = acc;
            out[(int64_t)(q * rows + r) * n + i] = acc;
        }
}

// The same for the 6x6 case with Phi in registers: every row of C is read once, the 21 distinct
// sums grow row by row.
__device__ __forceinline__ void covariance_sandwich6(int64_t n, int64_t i, const double Phi[36],
                                                     const double* __restrict__ C,
                                                     double* __restrict__ out) {
    double acc[21];
#pragma unroll
    for (int k = 0; k < 21; ++k) acc[k] = 0.0;
#pragma unroll
    for (int a = 0; a < 6; ++a) {
        double row[6], inner[6];
#pragma unroll
        for (int b = 0; b < 6; ++b) row[b] = __ldg(C + (int64_t)(6 * a + b) * n + i);
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            inner[q] = 0.0;
#pragma unroll
            for (int b = 0; b < 6; ++b) inner[q] += row[b] * Phi[6 * q + b];
        }
        int k = 0;
#pragma unroll
        for (int r = 0; r < 6; ++r)
#pragma unroll
            for (int q = r; q < 6; ++q) acc[k++] += Phi[6 * r + a] * inner[q];
    }
    int k = 0;
#pragma unroll
    for (int r = 0; r < 6; ++r)
#pragma unroll
        for (int q = r; q < 6; ++q, ++k) {
            out[(int64_t)(6 * r + q) * n + i] = acc[k];
            if (q != r) out[(int64_t)(6 * q + r) * n + i] = acc[k];
        }
}

__global__ void __launch_bounds__(128, 3) two_body_stm_kernel(
    int64_t n, const double* __restrict__ pos, const double* __restrict__ vel,
    const double* __restrict__ jd0, const double* __restrict__ jd1, double mu,
    const double* __restrict__ cov, double* __restrict__ out_pos, double* __restrict__ out_vel,
    double* __restrict__ out_stm, double* __restrict__ out_cov, int32_t* __restrict__ status) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double p[3] = {pos[i], pos[n + i], pos[2 * n + i]};
    double v[3] = {vel[i], vel[n + i], vel[2 * n + i]};
    double Phi[36];
    // analytic_2_body with its matrix: the whole interval at once, then halves
    const double time = jd1[i] - jd0[i];
    int rc = ST_OK;
    if (fabs(time) < 1e-10) {
#pragma unroll
        for (int k = 0; k < 36; ++k) Phi[k] = (k % 7 == 0) ? 1.0 : 0.0;
    } else if (!two_body_state_ok(p, v)) {
        rc = ST_CONVERGENCE;
    } else if (two_body_leaf_stm(time, p, v, mu, Phi) != ST_OK) {
        double p2[3] = {p[0], p[1], p[2]}, v2[3] = {v[0], v[1], v[2]}, M[36];
        rc = analytic_2_body_stm_halved(time, p2, v2, mu, M);
#pragma unroll
        for (int c = 0; c < 3; ++c) {
            p[c] = p2[c];
            v[c] = v2[c];
        }
#pragma unroll
        for (int k = 0; k < 36; ++k) Phi[k] = M[k];
    }
    if (rc != ST_OK) {
        const double nan = __longlong_as_double(0x7ff8000000000000LL);
        p[0] = p[1] = p[2] = v[0] = v[1] = v[2] = nan;
#pragma unroll
        for (int k = 0; k < 36; ++k) Phi[k] = nan;
    }
#pragma unroll
    for (int c = 0; c < 3; ++c) {
        out_pos[c * n + i] = p[c];
        out_vel[c * n + i] = v[c];
    }
    if (out_stm)
#pragma unroll
        for (int k = 0; k < 36; ++k) out_stm[k * n + i] = Phi[k];
    if (cov && out_cov) covariance_sandwich6(n, i, Phi, cov, out_cov);
    status[i] = rc;
}

__global__ void __launch_bounds__(128) covariance_kernel(int64_t n, int rows, int cols,
                                                         const double* __restrict__ phi,
                                                         const double* __restrict__ cov,
                                                         double* __restrict__ out) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    covariance_sandwich(n, i, rows, cols, phi, cov, out);
}

int launch_two_body_stm(int64_t n, const double* pos, const double* vel, const double* jd0,
                        const double* jd1, double mu, const double* cov, double* out_pos,
                        double* out_vel, double* out_stm, double* out_cov, int32_t* status,
                        cudaStream_t stream) {
    if (n <= 0) return 0;
    two_body_stm_kernel<<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(
        n, pos, vel, jd0, jd1, mu, cov, out_pos, out_vel, out_stm, out_cov, status);
    return launched(1, "two_body_stm_kernel launch");
}

int launch_covariance(int64_t n, int rows, int cols, const double* phi, const double* cov,
                      double* out, cudaStream_t stream) {
    if (n <= 0) return 0;
    covariance_kernel<<<(unsigned)((n + 127) / 128), 128, 0, stream>>>(n, rows, cols, phi, cov, out);
    return launched(1, "covariance_kernel launch");
}

}  // namespace kb
