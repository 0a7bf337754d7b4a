// sens_nodes.cu -- N-body forward sensitivities, node-parallel (nbody_stm_nodes_kernel,
// stm_nodes.cuh), with the launcher of both forms.
// every object of the differentiation workloads carries the comet model: inline it
#define KB_FORCE_NG_INLINE 1
#include "common.cuh"
#include "forces.cuh"
#include "internal.h"
#include "radau.cuh"
#include "stm_nodes.cuh"
#include "tangent.cuh"

namespace kb {
KB_CONSTANT_UPLOADER(sens_nodes)

int launch_nbody_stm(const StmArgs& args, int form, cudaStream_t stream) {
    if (args.n <= 0) return 0;
    StmArgs a = args;
    a.pending = 0;
    if (form == 1) return launch_nbody_stm_thread(a, stream);
    if (a.pool_slots > 0) {
        const int prc = launch_sens_pool_stm(a, stream);
        if (prc) return prc;
        a.pending = 1;
    }
    // node-parallel: tangents in dynamic shared memory above the 48 KB static limit (a
    // function attribute, set on every launch: it is not a stream operation)
    int rc = cuda_check(cudaFuncSetAttribute(nbody_stm_nodes_kernel<1>,
                                             cudaFuncAttributeMaxDynamicSharedMemorySize,
                                             STM_DYN_SMEM),
                        "sensitivity kernel shared memory");
    if (rc) return rc;
    const int64_t grid = (a.n * SG + STM_BLOCK - 1) / STM_BLOCK;
    nbody_stm_nodes_kernel<1><<<(unsigned)grid, STM_BLOCK, STM_DYN_SMEM, stream>>>(a);
    return launched(1, "nbody_stm_nodes_kernel launch");
}

}  // namespace kb
