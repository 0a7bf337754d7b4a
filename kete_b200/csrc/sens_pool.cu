// sens_pool.cu -- launchers of the differentiation passes on the warp-pooled step machinery
// (sens_pool.cuh).  Each takes the work inside the fast plan's window and marks the rest for the
// kernels of adjoint.cu and sens_nodes.cu, which the callers launch after it.
#include <atomic>

#include "common.cuh"
#include "forces.cuh"
#include "internal.h"
#include "sens_pool.cuh"

namespace kb {
KB_CONSTANT_UPLOADER(sens_pool)

int upload_pool_plans_sens(const PoolPlans& p) {
    return cuda_check(cudaMemcpyToSymbol(c_plans, &p, sizeof(PoolPlans)), "upload pooled plans");
}

// Dynamic shared memory past 48 KB has to be allowed once per device (a function attribute, not
// a stream operation).
static int allow_smem(const void* kernel, int slot, int bytes) {
    static std::atomic<unsigned long long> done[4];
    int dev = 0;
    int rc = cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc) return rc;
    const unsigned long long bit = 1ull << (dev & 63);
    if (done[slot].load() & bit) return 0;
    if ((rc = cuda_check(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes),
                         "sensitivity kernel shared memory")))
        return rc;
    done[slot].fetch_or(bit);
    return 0;
}

constexpr int SENS_POOL_BLOCK = 128;
using Shared1 = SensPoolShared<1, SENS_POOL_BLOCK, 0>;
using Shared4 = SensPoolShared<4, WIDE_BLOCK, 0>;
using SharedStm = SensPoolShared<4, WIDE_BLOCK, STM_ROW>;

// A warp per object while one wave of blocks (12 per SM) takes them all (1,776 on 148 SMs), eight
// lanes above: what counts is then the slowest object's chain of steps, afterwards how many run at a time.
// Measured, 400 days: 50 objects 2.87 ms and 3.73, 1000 objects 3.66 and 4.49, 2048 objects 5.05
// and 4.45; 730 days, 4096 objects: 14.06 and 8.96 (thread groups that replay per node: 12.8).
constexpr int SENS_WIDE_PER_SM = 12;

template <bool KM>
static int launch_forward(const SensArgs& a, cudaStream_t stream) {
    int sms = 0;
    const int src = sm_count(&sms);
    if (src) return src;
    if (a.n <= (int64_t)SENS_WIDE_PER_SM * sms) {
        const int smem = Shared4::doubles(a.pool_slots) * (int)sizeof(double);
        sens_pool_forward_kernel<4, WIDE_BLOCK, SENS_WIDE_PER_SM, KM><<<(unsigned)a.n, WIDE_BLOCK, smem, stream>>>(a);
    } else {
        const auto kernel = sens_pool_forward_kernel<1, SENS_POOL_BLOCK, 3, KM>;
        const int smem = Shared1::doubles(a.pool_slots) * (int)sizeof(double);
        const int rc = allow_smem((const void*)kernel, 2 * KM,
                                  Shared1::doubles(POOL_MAX_SLOTS) * (int)sizeof(double));
        if (rc) return rc;
        const int64_t grid = (a.n * NODE_G + SENS_POOL_BLOCK - 1) / SENS_POOL_BLOCK;
        kernel<<<(unsigned)grid, SENS_POOL_BLOCK, smem, stream>>>(a);
    }
    return launched(1, "sens_pool_forward_kernel launch");
}

int launch_sens_pool_forward(const SensArgs& a, cudaStream_t stream) {
    return a.pool_km ? launch_forward<true>(a, stream) : launch_forward<false>(a, stream);
}

// Persistent grids; a.n * a.window bounds the blocks to replay.
template <bool KM>
static int launch_replay(const SensArgs& a, cudaStream_t stream) {
    int sms = 0, per_sm = 0;
    int rc = sm_count(&sms);
    if (rc) return rc;
    const int64_t most = a.n * (int64_t)a.window;
    const bool wide = most <= 8192;
    const auto k4 = sens_pool_replay_kernel<4, WIDE_BLOCK, 12, KM>;
    const auto k1 = sens_pool_replay_kernel<1, SENS_POOL_BLOCK, 3, KM>;
    const int smem = (wide ? Shared4::doubles(a.pool_slots) : Shared1::doubles(a.pool_slots)) *
                     (int)sizeof(double);
    if (!wide && (rc = allow_smem((const void*)k1, 1 + 2 * KM,
                                  Shared1::doubles(POOL_MAX_SLOTS) * (int)sizeof(double))))
        return rc;
    const int block = wide ? WIDE_BLOCK : SENS_POOL_BLOCK;
    if ((rc = cuda_check(wide ? cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k4, block, smem)
                              : cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k1, block, smem),
                         "occupancy")))
        return rc;
    const int64_t resident = (int64_t)sms * (per_sm > 0 ? per_sm : 1);
    const int64_t need = wide ? most : (most * NODE_G + block - 1) / block;
    const unsigned grid = (unsigned)(need < resident ? need : resident);
    if (wide) k4<<<grid, block, smem, stream>>>(a);
    else k1<<<grid, block, smem, stream>>>(a);
    return launched(1, "sens_pool_replay_kernel launch");
}

int launch_sens_pool_replay(const SensArgs& a, cudaStream_t stream) {
    return a.pool_km ? launch_replay<true>(a, stream) : launch_replay<false>(a, stream);
}

template <bool KM>
static int launch_stm(const StmArgs& a, cudaStream_t stream) {
    const int smem = SharedStm::doubles(a.pool_slots) * (int)sizeof(double);
    // Eight blocks an SM leave a thread 255 registers, which pays while that is one wave: 1021
    // objects 6.46 ms and 6.81 with twelve, 4096 objects 38.8 ms and 34.3
    // (sixteen: 38.4).
    int sms = 0;
    const int rc = sm_count(&sms);
    if (rc) return rc;
    if (a.n <= (int64_t)8 * sms) sens_pool_stm_kernel<8, KM><<<(unsigned)a.n, WIDE_BLOCK, smem, stream>>>(a);
    else sens_pool_stm_kernel<12, KM><<<(unsigned)a.n, WIDE_BLOCK, smem, stream>>>(a);
    return launched(1, "sens_pool_stm_kernel launch");
}

int launch_sens_pool_stm(const StmArgs& a, cudaStream_t stream) {
    return a.pool_km ? launch_stm<true>(a, stream) : launch_stm<false>(a, stream);
}

}  // namespace kb
