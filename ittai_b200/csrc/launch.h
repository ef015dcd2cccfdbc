// Host helper: kernel launches that let the NEXT kernel of the stream begin its prologue before this one has drained
// (programmatic dependent launch).  Every kernel launched through launch_pdl calls pdl_wait() before its first access to global
// memory that another kernel of the run may have written or may still read, and pdl_trigger() on entry, or once the resources
// that it shares with its successors are its own.  So a kernel may be resident while several kernels in front of it still run
// (each of them triggers before it waits): what it reads ahead of its wait has to be complete before the FIRST of them starts.
// Ahead of the wait run barrier initialisation, tensor-memory allocation and descriptor prefetch, and in some kernels loads of
// such data: weights in the split-K GEMM, the decode chain and the projections of short forwards (there the norms' gains, too); in the
// chain also positions and older cache rows, which the late trigger of a token's first kernel makes safe; sequence records in the
// key-loop attention and the one for few queries, where the caller vouches for them.  (The one-SM GEMM only asks for weights to be
// brought into L2, which hands no data over.)  ITTAI_PDL=0 in the environment turns the attribute off (plain stream order).
#pragma once
#include <cuda_runtime.h>

#include <cstdlib>
#include <utility>

namespace ittai {

inline bool pdl_enabled() {
    static const bool on = [] { const char* e = std::getenv("ITTAI_PDL"); return !(e && e[0] == '0'); }();
    return on;
}

template <typename... KArgs, typename... Args>
inline cudaError_t launch_pdl(void (*kernel)(KArgs...), dim3 grid, dim3 block, size_t smem, cudaStream_t st, int cluster_x, Args&&... args) {
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = grid;
    cfg.blockDim = block;
    cfg.dynamicSmemBytes = smem;
    cfg.stream = st;
    cudaLaunchAttribute attr[2];
    unsigned n = 0;
    if (cluster_x > 1) {
        attr[n].id = cudaLaunchAttributeClusterDimension;
        attr[n].val.clusterDim.x = (unsigned)cluster_x; attr[n].val.clusterDim.y = 1; attr[n].val.clusterDim.z = 1;
        ++n;
    }
    if (pdl_enabled()) {
        attr[n].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        attr[n].val.programmaticStreamSerializationAllowed = 1;
        ++n;
    }
    cfg.attrs = attr;
    cfg.numAttrs = n;
    return cudaLaunchKernelEx(&cfg, kernel, std::forward<Args>(args)...);
}

}  // namespace ittai
