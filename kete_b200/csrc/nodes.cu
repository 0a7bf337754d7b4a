// nodes.cu -- host launchers of the node-parallel Radau kernels (radau_nodes.cuh here, the
// warp-pooled forms in pool.cu): every register-cap / step-end / warp-synchronous /
// pooled instantiation the tuner chooses from.  Its own translation unit so the
// instantiations compile in parallel with the other kernels.
#include "../../include/kete_b200.h"

#include "common.cuh"
#include "forces.cuh"
#include "internal.h"
#include "radau_nodes.cuh"

namespace kb {
KB_CONSTANT_UPLOADER(nodes)
}  // namespace kb

namespace kb {

// Node-parallel Radau: 8 lanes per object.  With a.queue == null each group integrates one
// object (grid covers n groups); with a queue the grid is persistent and groups refill.
// variant: 0 = no register cap, 1 = >= 3 blocks/SM (168 registers), 2 = >= 4 blocks/SM;
// +3: the step-end lane form (exact evaluations taken from lane 7, see radau_nodes.cuh);
// 6-8: the step-end form with warp-synchronous steps and the per-lane ephemeris cache;
// 9, 10: the warp-pooled record evaluations (radau_pool.cuh) at 168 / 128 registers.
static const void* nodes_kernel_ptr(int variant) {
    switch (variant) {
        case NODES_WIDE:
        case 9:
        case 10: return pool_kernel_ptr(variant);
        case 1: return (const void*)nbody_nodes_kernel<3, false>;
        case 2: return (const void*)nbody_nodes_kernel<4, false>;
        case 3: return (const void*)nbody_nodes_kernel<1, true>;
        case 4: return (const void*)nbody_nodes_kernel<3, true>;
        case 5: return (const void*)nbody_nodes_kernel<4, true>;
        case 6: return (const void*)nbody_nodes_kernel<1, true, true>;
        case 7: return (const void*)nbody_nodes_kernel<3, true, true>;
        case 8: return (const void*)nbody_nodes_kernel<4, true, true>;
        default: return (const void*)nbody_nodes_kernel<1, false>;
    }
}

int launch_nbody_nodes(const NBodyArgs& a, int variant, int grid, cudaStream_t stream) {
    if (a.n <= 0) return 0;
    if (variant >= 9 && !a.range)
        return set_error(KETE_B200_E_ARGUMENT,
                         "the warp-pooled node kernels take the window split of the processing "
                         "order (launch_nodes_ordered)");
    const int block = NODES_BLOCK;
    if (grid <= 0) grid = (int)((a.n * NODE_G + block - 1) / block);
    if (variant >= 9) return launch_pool(a, variant, grid, stream);
    switch (variant) {
        case 1: nbody_nodes_kernel<3, false><<<grid, block, 0, stream>>>(a); break;
        case 2: nbody_nodes_kernel<4, false><<<grid, block, 0, stream>>>(a); break;
        case 3: nbody_nodes_kernel<1, true><<<grid, block, 0, stream>>>(a); break;
        case 4: nbody_nodes_kernel<3, true><<<grid, block, 0, stream>>>(a); break;
        case 5: nbody_nodes_kernel<4, true><<<grid, block, 0, stream>>>(a); break;
        case 6: nbody_nodes_kernel<1, true, true><<<grid, block, 0, stream>>>(a); break;
        case 7: nbody_nodes_kernel<3, true, true><<<grid, block, 0, stream>>>(a); break;
        case 8: nbody_nodes_kernel<4, true, true><<<grid, block, 0, stream>>>(a); break;
        default: nbody_nodes_kernel<1, false><<<grid, block, 0, stream>>>(a); break;
    }
    return launched(1, "nbody_nodes_kernel launch");
}

// Persistent grid of a variant, capped at one lane group per object.
static int refill_grid(int variant, int64_t n, int slots, int* grid) {
    int rc = nodes_grid_size(variant, slots, grid);
    if (rc) return rc;
    const int64_t need = (n * NODE_G + NODES_BLOCK - 1) / NODES_BLOCK;
    if (*grid > need) *grid = (int)need;
    return 0;
}

int pool_groups(int variant, int64_t n, int slots, bool refill, int* groups) {
    *groups = 0;
    if (variant < 9 || !refill) return 0;
    int grid = 0;
    const int rc = refill_grid(variant, n, slots, &grid);
    *groups = grid * (NODES_BLOCK / NODE_G);
    return rc;
}

int launch_nodes_ordered(NBodyArgs a, int variant, int general_variant, bool refill,
                         int* scratch, cudaStream_t stream) {
    a.order = (const int32_t*)(scratch + ORDER_SCRATCH_HEADER);
    int grid = 0, rc = 0;
    if (variant < 9) {  // one launch over the whole order
        a.range = nullptr;
        a.queue = refill ? scratch : nullptr;
        if (refill && (rc = refill_grid(variant, a.n, a.pool_slots, &grid))) return rc;
        return launch_nbody_nodes(a, variant, grid, stream);
    }
    // objects inside the window: the pooled kernel between its centre-change kernels; the
    // others: the general form.  The counts are on the device, so every grid covers every
    // object (threads and groups past their part exit).
    a.range = scratch + ORDER_RANGE;
    a.queue = refill ? scratch : nullptr;
    a.queue_ng = refill ? scratch + ORDER_QUEUE3 : nullptr;
    a.wide = scratch + ORDER_WIDE;
    if ((rc = launch_pool_centre(a, true, stream))) return rc;
    if (refill && (rc = refill_grid(variant, a.n, a.pool_slots, &grid))) return rc;
    if ((rc = launch_nbody_nodes(a, variant, grid, stream))) return rc;
    if ((rc = launch_pool_centre(a, false, stream))) return rc;
    a.range = scratch + ORDER_RANGE + 2;
    a.queue = refill ? scratch + ORDER_QUEUE2 : nullptr;
    a.queue_ng = nullptr;
    grid = 0;
    if (refill && (rc = refill_grid(general_variant, a.n, 0, &grid))) return rc;
    return launch_nbody_nodes(a, general_variant, grid, stream);
}

int launch_nodes_wide(NBodyArgs a, int general_variant, cudaStream_t stream) {
    a.order = nullptr;
    a.range = nullptr;
    a.queue = a.queue_ng = nullptr;
    int rc = launch_pool(a, NODES_WIDE, (int)a.n, stream);
    if (rc) return rc;
    a.pending = 1;
    return launch_nbody_nodes(a, general_variant, 0, stream);
}

int preload_nodes_kernels() {
    cudaFuncAttributes fa;
    int rc = 0;
    for (int v = 0; v <= NODES_WIDE; ++v)
        if ((rc = cuda_check(cudaFuncGetAttributes(&fa, nodes_kernel_ptr(v)), "load node kernels")))
            return rc;
    return preload_pool_kernels();
}

// Resident grid for the persistent (refill) form: blocks per SM from the occupancy API.
int nodes_grid_size(int variant, int slots, int* grid) {
    int sms = 0, per_sm = 0;
    int rc = sm_count(&sms);
    if (rc) return rc;
    int smem = 0;
    if (variant >= 9 && (rc = pool_smem(variant, slots, &smem))) return rc;
    if ((rc = cuda_check(cudaOccupancyMaxActiveBlocksPerMultiprocessor(
                             &per_sm, nodes_kernel_ptr(variant), NODES_BLOCK, smem),
                         "occupancy")))
        return rc;
    *grid = sms * (per_sm > 0 ? per_sm : 1);
    return 0;
}

}  // namespace kb
