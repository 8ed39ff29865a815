// Lane-dense kernel (gx_dense.cuh): one class in a launch, FP32 entries.
#include "gx_dense.cuh"

namespace gx {
namespace dense {

cudaError_t run_one_f32(int pair, const EriDev& d, const QuartetClass& qc, int smem, cudaStream_t s) {
    switch (pair) {
#define GX_CASE(A, B)                                                                                             \
    case A * 4 + B: {                                                                                             \
        static PerDevice limit;                                                                                   \
        return launch_with_smem(dense_kernel<A, B, kDenseF32>, limit, dim3(qc.ngroup, qc.nchunk), smem, s, d, qc);     \
    }
        GX_DENSE_PAIRS
#undef GX_CASE
        default:
            return cudaErrorInvalidValue;
    }
}

}  // namespace dense
}  // namespace gx
