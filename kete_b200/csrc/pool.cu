// pool.cu -- the warp-pooled Radau kernels (radau_pool.cuh) and their launchers; a translation
// unit of its own beside nodes.cu so that the instantiations compile in parallel.
#include <algorithm>
#include <atomic>

#include "../../include/kete_b200.h"

#include "common.cuh"
#include "forces.cuh"
#include "internal.h"
#include "radau_nodes.cuh"
#include "radau_pool.cuh"

namespace kb {
KB_CONSTANT_UPLOADER(pool)

int upload_pool_plans(const PoolPlans& p) {
    return cuda_check(cudaMemcpyToSymbol(c_plans, &p, sizeof(PoolPlans)), "upload pooled plans");
}

static const void* kernel_ptr(int variant, bool km) {
    switch (variant) {
        case NODES_WIDE:
            return km ? (const void*)nbody_wide_kernel<16, true> : (const void*)nbody_wide_kernel<16, false>;
        case 9:
            return km ? (const void*)nbody_pool_kernel<3, true>
                      : (const void*)nbody_pool_kernel<3, false>;
        default:
            return km ? (const void*)nbody_pool_kernel<4, true>
                      : (const void*)nbody_pool_kernel<4, false>;
    }
}
const void* pool_kernel_ptr(int variant) { return kernel_ptr(variant, false); }

// Dynamic shared memory of a variant for cache columns of `slots` doubles.  Above the 48 KB
// static limit it has to be allowed once per device (a function attribute, not a stream
// operation).
static int pool_bytes(int variant, int slots) {
    const int n = variant == NODES_WIDE ? PoolShared<4, WIDE_BLOCK>::doubles(slots)
                                        : std::max(PoolShared<1, NODES_BLOCK>::doubles(slots),
                                                   PoolShared<4, NODES_BLOCK>::doubles(slots));
    return n * (int)sizeof(double);
}

int pool_smem(int variant, int slots, int* bytes) {
    static std::atomic<unsigned long long> done[2];
    *bytes = pool_bytes(variant, slots);
    if (variant == NODES_WIDE) return 0;
    int dev = 0;
    int rc = cuda_check(cudaGetDevice(&dev), "cudaGetDevice");
    if (rc) return rc;
    const unsigned long long bit = 1ull << (dev & 63);
    auto& d = done[variant - 9];
    if (d.load() & bit) return 0;
    for (bool km : {false, true})
        if ((rc = cuda_check(cudaFuncSetAttribute(kernel_ptr(variant, km),
                                                  cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                  pool_bytes(variant, POOL_MAX_SLOTS)),
                             "pooled kernel shared memory")))
            return rc;
    d.fetch_or(bit);
    return 0;
}

int launch_pool(const NBodyArgs& a, int variant, int grid, cudaStream_t stream) {
    int smem = 0;
    const int rc = pool_smem(variant, a.pool_slots, &smem);
    if (rc) return rc;
    if (variant == NODES_WIDE && a.pool_km)
        nbody_wide_kernel<16, true><<<grid, WIDE_BLOCK, smem, stream>>>(a);
    else if (variant == NODES_WIDE)
        nbody_wide_kernel<16, false><<<grid, WIDE_BLOCK, smem, stream>>>(a);
    else if (variant == 9 && a.pool_km)
        nbody_pool_kernel<3, true><<<grid, NODES_BLOCK, smem, stream>>>(a);
    else if (variant == 9)
        nbody_pool_kernel<3, false><<<grid, NODES_BLOCK, smem, stream>>>(a);
    else if (a.pool_km)
        nbody_pool_kernel<4, true><<<grid, NODES_BLOCK, smem, stream>>>(a);
    else
        nbody_pool_kernel<4, false><<<grid, NODES_BLOCK, smem, stream>>>(a);
    return launched(1, "nbody_pool_kernel launch");
}

int launch_pool_centre(const NBodyArgs& a, bool before, cudaStream_t stream) {
    const int grid = (int)std::min<int64_t>((a.n + 255) / 256, 1184);
    if (before) pool_prepare_kernel<<<grid, 256, 0, stream>>>(a);
    else pool_finish_kernel<<<grid, 256, 0, stream>>>(a);
    return launched(1, before ? "pool_prepare_kernel launch" : "pool_finish_kernel launch");
}

int preload_pool_kernels() {
    cudaFuncAttributes fa;
    int rc = 0, smem = 0;
    for (const void* f : {(const void*)pool_prepare_kernel, (const void*)pool_finish_kernel,
                          kernel_ptr(NODES_WIDE, false), kernel_ptr(NODES_WIDE, true)})
        if ((rc = cuda_check(cudaFuncGetAttributes(&fa, f), "load pooled kernels"))) return rc;
    for (int v : {9, 10})
        if ((rc = pool_smem(v, POOL_MAX_SLOTS, &smem))) return rc;
    return 0;
}

}  // namespace kb
