// Lane-dense kernel (gx_dense.cuh): the entries that FP32 leaves to FP64, of many
// classes in one launch.  There are few of them (twelve atoms: none of 11.5 M FP32
// entries), so a small grid looks through the units (the tasks of classes without
// unit arrays), a thread each, for those in which the FP32 launch met one.
#include <algorithm>

#include "gx_dense.cuh"

namespace gx {

namespace {

constexpr int kMaxWide = 48;
struct WideList {
    int n;
    int pair[kMaxWide];
    QuartetClass cls[kMaxWide];
};

__global__ void __launch_bounds__(32 * dense::kWarps) wide_kernel(const __grid_constant__ EriDev d,
                                                                  const __grid_constant__ WideList list) {
    constexpr int THREADS = 32 * dense::kWarps;
    __shared__ int4 queue[64];
    __shared__ long long hits[THREADS];
    __shared__ int nhit, wide[kMaxWide];
    if (threadIdx.x < (unsigned)list.n) wide[threadIdx.x] = *list.cls[threadIdx.x].wide;
    __syncthreads();
    for (int c = 0; c < list.n; ++c) {
        if (wide[c] == 0) continue;
        const QuartetClass& qc = list.cls[c];
        // items: (unit or task, share of its components)
        const long long items = (long long)(qc.unit_start32 ? qc.ngroup : qc.ntask) * qc.nchunk;
        for (long long i0 = blockIdx.x; i0 < items; i0 += (long long)THREADS * gridDim.x) {
            if (threadIdx.x == 0) nhit = 0;
            __syncthreads();
            const long long i = i0 + (long long)threadIdx.x * gridDim.x;
            // (any order: they write disjoint elements)
            const int u = (int)(i / qc.nchunk);
            if (i < items && (qc.unit_start32 ? qc.unit_start32[u] < 0 : qc.wide[1 + u / 32] >> (u & 31) & 1))
                hits[atomicAdd(&nhit, 1)] = i;
            __syncthreads();
            const int n = nhit;
            for (int k = 0; k < n; ++k) {
                switch (list.pair[c]) {
#define GX_CASE(A, B)                                                              \
    case A * 4 + B:                                                                \
        dense::dense_block<A, B, kDenseWide>(d, qc, (int)(hits[k] / qc.nchunk),    \
                                             (int)(hits[k] % qc.nchunk), queue);   \
        break;
                    GX_DENSE_PAIRS
#undef GX_CASE
                }
                __syncthreads();
            }
        }
    }
}

}  // namespace

int wide_lists(size_t n) { return (int)((n + kMaxWide - 1) / kMaxWide); }

cudaError_t launch_wide(const EriDev& d, const std::vector<std::pair<int, QuartetClass>>& classes, int sms,
                        cudaStream_t s) {
    static PerDevice limit;
    WideList list;
    for (size_t k = 0; k < classes.size();) {
        long long units = 0;
        int smem = 0;
        for (list.n = 0; k < classes.size() && list.n < kMaxWide; ++k) {
            const auto& [pair, qc] = classes[k];
            if (qc.ntask <= 0 || qc.ngroup <= 0 || !qc.wide) continue;
            list.pair[list.n] = pair;
            list.cls[list.n] = qc;
            // (blocks that share a unit's components: few units have anything to do,
            // and the launch is the end of its plan)
            const int nchunk = dense_chunks(qc.bra.la, qc.bra.lb, qc.ket.la, qc.ket.lb, 8, true);
            list.cls[list.n++].nchunk = nchunk;
            units += (long long)(qc.unit_start32 ? qc.ngroup : qc.ntask) * nchunk;
            smem = std::max(smem, dense_smem(pair, qc, d.all_real ? 8 : 16));
        }
        if (list.n == 0) continue;
        const dim3 grid((unsigned)std::min<long long>(units, 2ll * std::max(sms, 1)));
        const cudaError_t e = dense::launch_with_smem(wide_kernel, limit, grid, smem, s, d, list);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

}  // namespace gx
