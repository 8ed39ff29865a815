// Lane-dense kernel (gx_dense.cuh): a list of classes in one launch, FP64 entries.
#include "gx_dense.cuh"

namespace gx {
namespace dense {

cudaError_t run_list_f64(int pair, const EriDev& d, const ClassList& list, int smem, cudaStream_t s) {
    switch (pair) {
#define GX_CASE(A, B)                                                                                             \
    case A * 4 + B: {                                                                                             \
        static PerDevice limit;                                                                                   \
        return launch_with_smem(dense_list_kernel<A, B, kDenseF64>, limit, dim3(list.first[list.n]), smem, s, d, list); \
    }
        GX_DENSE_PAIRS
#undef GX_CASE
        default:
            return cudaErrorInvalidValue;
    }
}

}  // namespace dense
}  // namespace gx
