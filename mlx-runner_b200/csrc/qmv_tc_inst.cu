// One instantiation set of the tensor-memory decode matvec per bit width: compiled six times with -DMLXQ_BITS=n.
#include <mutex>

#include "dependent_launch.h"
#include "qmv_tc.cuh"

#ifndef MLXQ_BITS
#error "compile with -DMLXQ_BITS=2|3|4|5|6|8"
#endif

#define MLXQ_CAT2(a, b) a##b
#define MLXQ_CAT(a, b) MLXQ_CAT2(a, b)

namespace mlxq {

template <int NTK, int SPLIT>
static cudaError_t launch_one(const MmaParams& p, const TcPlan& tp, size_t smem, int device, cudaStream_t st) {
    if constexpr (!tc_compiled(MLXQ_BITS, NTK, SPLIT)) {
        return cudaErrorNotSupported;
    } else {
        // the shared-memory opt-in is an attribute of the function in one device's context
        static std::mutex mu;
        static bool done[64] = {};
        if (device < 0 || device >= 64) return cudaErrorInvalidDevice;
        {
            std::lock_guard<std::mutex> lk(mu);
            if (!done[device]) {
                const cudaError_t e = cudaFuncSetAttribute(qmv_tc_kernel<MLXQ_BITS, NTK, SPLIT>, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_WHOLE);
                if (e != cudaSuccess) return e;
                done[device] = true;
            }
        }
        cudaLaunchConfig_t cfg = {};
        cfg.gridDim = dim3(static_cast<unsigned>(tp.clusters * tp.kz));
        cfg.blockDim = dim3(TC_THREADS);
        cfg.dynamicSmemBytes = smem;
        cfg.stream = st;
        cudaLaunchAttribute la[2];
        la[0].id = cudaLaunchAttributeProgrammaticStreamSerialization;
        la[0].val.programmaticStreamSerializationAllowed = 1;
        int n = pdl_enabled() ? 1 : 0;
        if (tp.kz > 1) {
            la[n].id = cudaLaunchAttributeClusterDimension;
            la[n].val.clusterDim.x = static_cast<unsigned>(tp.kz);
            la[n].val.clusterDim.y = la[n].val.clusterDim.z = 1;
            n++;
        }
        cfg.attrs = la;
        cfg.numAttrs = static_cast<unsigned>(n);
        return cudaLaunchKernelEx(&cfg, qmv_tc_kernel<MLXQ_BITS, NTK, SPLIT>, p, tp);
    }
}

template <int SPLIT>
static cudaError_t launch_tokens(const MmaParams& p, const TcPlan& tp, size_t smem, int device, cudaStream_t st) {
    switch (tc_tokens(p.q.T)) {
        case 2: return launch_one<2, SPLIT>(p, tp, smem, device, st);
        case 4: return launch_one<4, SPLIT>(p, tp, smem, device, st);
        case 8: return launch_one<8, SPLIT>(p, tp, smem, device, st);
        default: return launch_one<16, SPLIT>(p, tp, smem, device, st);
    }
}

#if MLXQ_BITS == 4
// (an empty kernel of the same block and shared memory: for one that allocates tensor memory the occupancy calls say one CTA an
// SM whatever its shared memory, although two of these run side by side -- 24576 x 2048, 4 bits, 16 fp32 tokens, planned for one
// CTA an SM 44.7 us, for two 24.6)
static __global__ void __launch_bounds__(TC_THREADS, 2) qmv_tc_shape() {}

int qmv_tc_clusters(int kz, size_t smem) {
    const auto kernel = qmv_tc_shape;
    int dev = 0, sms = 0, n = 0;
    cudaLaunchConfig_t cfg = {};
    cudaLaunchAttribute la[1];
    la[0].id = cudaLaunchAttributeClusterDimension;
    la[0].val.clusterDim.x = static_cast<unsigned>(kz);
    la[0].val.clusterDim.y = la[0].val.clusterDim.z = 1;
    cfg.blockDim = dim3(TC_THREADS);
    cfg.dynamicSmemBytes = smem;
    cfg.attrs = la;
    cfg.numAttrs = 1;
    if (cudaGetDevice(&dev) != cudaSuccess || cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
        cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, TC_SMEM_WHOLE) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    cfg.gridDim = dim3(static_cast<unsigned>(2 * sms / kz * kz));
    if (cudaOccupancyMaxActiveClusters(&n, kernel, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}
#endif

cudaError_t MLXQ_CAT(launch_qmv_tc_b, MLXQ_BITS)(const MmaParams& p, const TcPlan& tp, size_t smem, int device, cudaStream_t st) {
    return p.split == 2 ? launch_tokens<2>(p, tp, smem, device, st) : launch_tokens<1>(p, tp, smem, device, st);
}

}  // namespace mlxq
