// ksfused_multi.cu -- the one-kernel key switch (ksfused.cuh), keys in prepared form.
#include "ksfused.cuh"

namespace afhe {
namespace ksf {

cudaError_t launch_multi(int log_n, const KsFusedArgs& a, uint32_t nz, cudaStream_t st) {
#define LAUNCH(Q, C) launch_fused<Q, C, true, false>(a, nz, st)
    AFHE_KS_BY_DEGREE(log_n, LAUNCH, cudaErrorInvalidValue)
#undef LAUNCH
}

namespace {
// Ciphertexts the GPU can hold at once for the kernel at N = 2^(LOGQ + LOGCL)
// (0 when it cannot place even one: the multi-kernel path is used then).
template <int LOGQ, int LOGCL>
int fused_capacity() {
    auto kern = ks_fused_kernel<LOGQ, LOGCL, 16, true, false>;
    constexpr size_t smem = fused_smem<LOGQ, false>();
    constexpr uint32_t T = Geo<LOGQ, LOGCL, 16>::T;
    if (cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    int n = 0;
    if constexpr (LOGCL == 0) {
        int dev = 0, sms = 0;
        if (cudaGetDevice(&dev) != cudaSuccess ||
            cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess ||
            cudaOccupancyMaxActiveBlocksPerMultiprocessor(&n, kern, (int)T, smem) != cudaSuccess) {
            cudaGetLastError();
            return 0;
        }
        return n * sms;
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3(1u << LOGCL, 1, 1);
    cfg.blockDim = dim3(T, 1, 1);
    cfg.dynamicSmemBytes = smem;
    cudaLaunchAttribute attr[1];
    attr[0].id = cudaLaunchAttributeClusterDimension;
    attr[0].val.clusterDim.x = 1u << LOGCL;
    attr[0].val.clusterDim.y = 1;
    attr[0].val.clusterDim.z = 1;
    cfg.attrs = attr;
    cfg.numAttrs = 1;
    if (cudaOccupancyMaxActiveClusters(&n, kern, &cfg) != cudaSuccess) {
        cudaGetLastError();
        return 0;
    }
    return n;
}

}  // namespace

int capacity(int log_n) {
#define CAPACITY(Q, C) fused_capacity<Q, C>()
    AFHE_KS_BY_DEGREE(log_n, CAPACITY, 0)
#undef CAPACITY
}

}  // namespace ksf
}  // namespace afhe
