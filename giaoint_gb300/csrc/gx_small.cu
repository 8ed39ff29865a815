// Instantiations and dispatch of the register-resident small-class kernel
// (all (la, lb, lc, ld) with la + lb + lc + ld <= 2).
#include "gx_small.cuh"

namespace gx {

namespace {
template <int A, int B, int C, int D>
cudaError_t go(const EriDev& d, const QuartetClass& qc, cudaStream_t s) {
    small::small_kernel<A, B, C, D>
        <<<(qc.ngroup + small::kWarps - 1) / small::kWarps, 32 * small::kWarps, 0, s>>>(d, qc);
    return cudaGetLastError();
}
}  // namespace

// all classes with la + lb + lc + ld <= 2
#define GX_SMALL_CLASSES \
    GX_CASE(0, 0, 0, 0)  \
    GX_CASE(1, 0, 0, 0)  \
    GX_CASE(0, 1, 0, 0)  \
    GX_CASE(0, 0, 1, 0)  \
    GX_CASE(0, 0, 0, 1)  \
    GX_CASE(2, 0, 0, 0)  \
    GX_CASE(0, 2, 0, 0)  \
    GX_CASE(0, 0, 2, 0)  \
    GX_CASE(0, 0, 0, 2)  \
    GX_CASE(1, 1, 0, 0)  \
    GX_CASE(1, 0, 1, 0)  \
    GX_CASE(1, 0, 0, 1)  \
    GX_CASE(0, 1, 1, 0)  \
    GX_CASE(0, 1, 0, 1)  \
    GX_CASE(0, 0, 1, 1)

bool small_class(int la, int lb, int lc, int ld) { return la + lb + lc + ld <= 2; }

cudaError_t launch_small(int la, int lb, int lc, int ld, const EriDev& d, const QuartetClass& qc, cudaStream_t s) {
    if (qc.ntask <= 0 || qc.ngroup <= 0) return cudaSuccess;
    const int key = ((la * 3 + lb) * 3 + lc) * 3 + ld;
    switch (key) {
#define GX_CASE(A, B, C, D) \
    case ((A * 3 + B) * 3 + C) * 3 + D: return go<A, B, C, D>(d, qc, s);
        GX_SMALL_CLASSES
#undef GX_CASE
        default:
            return cudaErrorInvalidValue;
    }
}

namespace {

__global__ void __launch_bounds__(32 * small::kWarps) small_list_kernel(const __grid_constant__ EriDev d,
                                                                        const __grid_constant__ small::ClassList list) {
    __shared__ small::WarpBuffers<9> s_buf[small::kWarps];
    char* smem = reinterpret_cast<char*>(s_buf);
    int c = 0;
    while (c + 1 < list.n && (int)blockIdx.x >= list.first[c + 1]) ++c;
    const QuartetClass& qc = list.cls[c];
    const int block = (int)blockIdx.x - list.first[c];
    switch (list.key[c]) {
#define GX_CASE(A, B, C, D) \
    case ((A * 3 + B) * 3 + C) * 3 + D: small::small_block<A, B, C, D>(d, qc, block, smem); break;
        GX_SMALL_CLASSES
#undef GX_CASE
    }
}

}  // namespace

cudaError_t launch_small_list(const EriDev& d, const std::vector<int>& keys, const std::vector<QuartetClass>& classes,
                              cudaStream_t s) {
    small::ClassList list;
    list.n = 0;
    list.first[0] = 0;
    for (size_t k = 0; k < classes.size(); ++k) {
        const QuartetClass& qc = classes[k];
        if (qc.ntask <= 0 || qc.ngroup <= 0) continue;
        if (list.n == 15) return cudaErrorInvalidValue;
        list.key[list.n] = keys[k];
        list.cls[list.n] = qc;
        list.first[list.n + 1] = list.first[list.n] + (qc.ngroup + small::kWarps - 1) / small::kWarps;
        ++list.n;
    }
    if (list.n == 0) return cudaSuccess;
    small_list_kernel<<<(unsigned)list.first[list.n], 32 * small::kWarps, 0, s>>>(d, list);
    return cudaGetLastError();
}

}  // namespace gx
