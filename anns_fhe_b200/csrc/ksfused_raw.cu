// ksfused_raw.cu -- the one-kernel key switch (ksfused.cuh), keys as they lie in key_gmem (not registered): rarely
// used, so compiled for size.
#define AFHE_KS_FN __noinline__
#include "ksfused.cuh"

namespace afhe {
namespace ksf {

cudaError_t launch_raw(int log_n, const KsFusedArgs& a, uint32_t nz, cudaStream_t st) {
#define LAUNCH(Q, C) launch_fused<Q, C, false, false>(a, nz, st)
    AFHE_KS_BY_DEGREE(log_n, LAUNCH, cudaErrorInvalidValue)
#undef LAUNCH
}

}  // namespace ksf
}  // namespace afhe
