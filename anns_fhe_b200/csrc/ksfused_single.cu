// ksfused_single.cu -- the one-kernel key switch (ksfused.cuh), keys in prepared form, every entry's level a single digit.
#include "ksfused.cuh"

namespace afhe {
namespace ksf {

cudaError_t launch_single(int log_n, const KsFusedArgs& a, uint32_t nz, cudaStream_t st) {
#define LAUNCH(Q, C) launch_fused<Q, C, true, true>(a, nz, st)
    AFHE_KS_BY_DEGREE(log_n, LAUNCH, cudaErrorInvalidValue)
#undef LAUNCH
}

}  // namespace ksf
}  // namespace afhe
