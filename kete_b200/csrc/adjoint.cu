// adjoint.cu -- reverse-mode gradients: the checkpointed forward pass and the discrete
// adjoint pass (adjoint.cuh) with their host launchers.
// every object of the differentiation workloads carries the comet model: inline it
#define KB_FORCE_NG_INLINE 1
#include "common.cuh"
#include "forces.cuh"
#include "internal.h"
#include "adjoint.cuh"

namespace kb {
KB_CONSTANT_UPLOADER(adjoint)
}  // namespace kb

namespace kb {

// Exclusive prefix sums of the blocks each object replays in this pass (none when its forward pass
// failed) into a.rep_first[0 .. n], and the counters behind them cleared; one thread block, each
// thread a contiguous run of objects.
constexpr int OFFSETS_THREADS = 1024;
__global__ void __launch_bounds__(OFFSETS_THREADS) sens_replay_offsets_kernel(SensArgs a) {
    __shared__ int64_t s_sum[OFFSETS_THREADS];
    const int64_t n = a.n;
    const int64_t per = (n + OFFSETS_THREADS - 1) / OFFSETS_THREADS;
    const int64_t o0 = (int64_t)threadIdx.x * per;
    const int64_t o1 = o0 + per < n ? o0 + per : n;
    auto blocks = [&](int64_t o) -> int64_t {
        if (a.status[o] != ST_OK) return 0;
        const int c = sens_block_count(a, o);
        return (a.pass > 0 ? sens_pass_first(c, a.pass - 1, a.window) : c) -
               sens_pass_first(c, a.pass, a.window);
    };
    int64_t own = 0;
    for (int64_t o = o0; o < o1; ++o) own += blocks(o);
    s_sum[threadIdx.x] = own;
    __syncthreads();
    for (int d = 1; d < OFFSETS_THREADS; d <<= 1) {  // inclusive scan (Hillis-Steele)
        const int64_t add = threadIdx.x >= (unsigned)d ? s_sum[threadIdx.x - d] : 0;
        __syncthreads();
        s_sum[threadIdx.x] += add;
        __syncthreads();
    }
    int64_t run = s_sum[threadIdx.x] - own;
    for (int64_t o = o0; o < o1; ++o) {
        a.rep_first[o] = (int32_t)run;
        run += blocks(o);
    }
    if (threadIdx.x == OFFSETS_THREADS - 1) {
        a.rep_first[n] = (int32_t)s_sum[threadIdx.x];
        a.rep_first[n + 1] = a.rep_first[n + 2] = a.rep_first[n + 3] = 0;
    }
}

int launch_sens_forward(const SensArgs& args, cudaStream_t stream) {
    if (args.n <= 0) return 0;
    SensArgs a = args;
    a.pending = a.pool_slots > 0;
    if (a.pending) {
        const int rc = launch_sens_pool_forward(a, stream);
        if (rc) return rc;
    }
    const int64_t threads = a.n * SG;
    nbody_sens_forward_kernel<1><<<(unsigned)((threads + SENS_BLOCK - 1) / SENS_BLOCK), SENS_BLOCK, 0, stream>>>(a);
    return launched(1, "nbody_sens_forward_kernel launch");
}

// One pass: the replays of its blocks, then the sweep over them.
static int launch_sens_pass(SensArgs a, bool passes, cudaStream_t stream) {
    constexpr int cache_bytes = EPH_CACHE * SENS_BLOCK * (int)sizeof(double);
    int rc = 0;
    sens_replay_offsets_kernel<<<1, OFFSETS_THREADS, 0, stream>>>(a);
    if ((rc = launched(1, "sens_replay_offsets_kernel launch"))) return rc;
    a.pending = a.pool_slots > 0;
    if (a.pending && (rc = launch_sens_pool_replay(a, stream))) return rc;
    // persistent grid: as many thread blocks as are resident at once, and no more than the
    // blocks to replay could occupy
    int sms = 0, per_sm = 0;
    if ((rc = sm_count(&sms)) ||
        (rc = cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                             &per_sm, nbody_sens_replay_kernel<3>, SENS_BLOCK, cache_bytes),
                         "occupancy")))
        return rc;
    const int64_t resident = (int64_t)sms * (per_sm > 0 ? per_sm : 1);
    const int64_t rthreads = a.n * (int64_t)a.window * SG;
    const int64_t need = (rthreads + SENS_BLOCK - 1) / SENS_BLOCK;
    const unsigned rgrid = (unsigned)(need < resident ? need : resident);
    nbody_sens_replay_kernel<3><<<rgrid, SENS_BLOCK, cache_bytes, stream>>>(a);
    if ((rc = launched(1, "nbody_sens_replay_kernel launch"))) return rc;
    const unsigned grid = (unsigned)((a.n * SG + SENS_BLOCK - 1) / SENS_BLOCK);
    if (passes) nbody_sens_backward_kernel<1, true><<<grid, SENS_BLOCK, cache_bytes, stream>>>(a);
    else nbody_sens_backward_kernel<1, false><<<grid, SENS_BLOCK, cache_bytes, stream>>>(a);
    return launched(1, "nbody_sens_backward_kernel launch");
}

int launch_sens_backward(const SensArgs& args, cudaStream_t stream) {
    if (args.n <= 0) return 0;
    SensArgs a = args;
    // the per-lane ephemeris cache takes the block past the 48 KB of shared memory a kernel
    // gets without opting in (a function attribute, not a stream operation).  The replay is
    // throughput bound (every block of every object), so it is capped at 168 registers for 12
    // resident warps per SM; the sweep is one partial wave and keeps the full register file.
    constexpr int cache_bytes = EPH_CACHE * SENS_BLOCK * (int)sizeof(double);
    int rc = 0;
    for (const void* f : {(const void*)nbody_sens_replay_kernel<3>,
                          (const void*)nbody_sens_backward_kernel<1, false>,
                          (const void*)nbody_sens_backward_kernel<1, true>})
        if ((rc = cuda_check(cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  cache_bytes),
                             "cudaFuncSetAttribute")))
            return rc;
    for (a.pass = 0; (int64_t)a.pass * a.window < a.ckpt_cap; ++a.pass)
        if ((rc = launch_sens_pass(a, a.window < a.ckpt_cap, stream))) return rc;
    return 0;
}

}  // namespace kb
