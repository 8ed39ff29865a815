// Dispatch of the lane-dense kernel (gx_dense.cuh) and the kernels that cut a
// plan's classes into its FP64 work units.
#include "gx_dense.cuh"

#include <algorithm>
#include <cstdint>

namespace gx {

namespace {

using dense::kMaxOrder;
using dense::kMaxOrderReal;
using dense::kMaxSmem;

// template pairs: (l, 0) runs as (0, l), whose components, boxes and Hermite
// records are the same in the same order
bool template_pair(int la, int lb) {
    return la + lb <= 4 && la <= 3 && lb <= 3;
}

// multiply-adds per primitive quartet with (la, lb) as the template side
long long work(int la, int lb, int lc, int ld) {
    return (long long)small::hc(la + lb) * small::etot(lc, ld) +
           (long long)small::nc(lc) * small::nc(ld) * small::etot(la, lb);
}

int smem_bytes(int la, int lb, int lc, int ld, int word) {
    return dense::layout(small::hc(la + lb), small::nc(la) * small::nc(lb), small::hc(lc + ld), small::etot(lc, ld),
                         small::nc(lc) * small::nc(ld), la + lb + lc + ld, word)
        .total;
}

// 0: not this kernel's class, 1: (la, lb) is the template side, 2: (lc, ld) is.
// The run-time side is the one whose components fill the block's warps; between
// two such sides, the choice with fewer multiply-adds ((01|12): 532 with (01)
// as the template side, 438 with (12)).
int side_of(int la, int lb, int lc, int ld) {
    const int L = la + lb + lc + ld;
    if (L < 3 || L > kMaxOrderReal) return 0;
    const int word = L <= kMaxOrder ? 16 : 8;
    const bool ab = template_pair(la, lb) && smem_bytes(la, lb, lc, ld, word) <= kMaxSmem;
    const bool cd = template_pair(lc, ld) && smem_bytes(lc, ld, la, lb, word) <= kMaxSmem;
    if (!ab || !cd) return ab ? 1 : (cd ? 2 : 0);
    auto groups = [](int a, int b, int c, int d) {
        const int cg = dense::group_of(small::nc(a) * small::nc(b));
        return std::min(dense::kWarps, (small::nc(c) * small::nc(d) + cg - 1) / cg);
    };
    const int g1 = groups(la, lb, lc, ld), g2 = groups(lc, ld, la, lb);
    if (g1 != g2) return g1 > g2 ? 1 : 2;
    return work(la, lb, lc, ld) <= work(lc, ld, la, lb) ? 1 : 2;
}

}  // namespace

bool dense_class(int la, int lb, int lc, int ld, bool real) {
    return la + lb + lc + ld <= (real ? kMaxOrderReal : kMaxOrder) && side_of(la, lb, lc, ld) != 0;
}

// Blocks that share a work unit's components when `want` would fill the GPU:
// at most as many as have components for their warps, and (unless the class
// has a single batch, whose latency is all that counts) as keep a block's
// transforms at twice the Boys function and table that each of them repeats.
int dense_chunks(int la, int lb, int lc, int ld, int want, bool single) {
    if (side_of(la, lb, lc, ld) == 2) {
        std::swap(la, lc);
        std::swap(lb, ld);
    }
    const int L = la + lb + lc + ld, ncd = small::nc(lc) * small::nc(ld);
    const int cg = dense::group_of(small::nc(la) * small::nc(lb));
    const int groups = (ncd + cg - 1) / cg;
    const double repeated = 150.0 + 12.0 * L + 5.0 * small::rsteps(L);
    int most = (groups + dense::kWarps - 1) / dense::kWarps;
    if (!single) most = std::min(most, (int)(4.0 * (double)work(la, lb, lc, ld) / (2.0 * repeated)));
    return std::max(1, std::min(want, most));
}

int dense_orient(int la, int lb, int lc, int ld, QuartetClass& qc) {
    const int side = side_of(la, lb, lc, ld);
    int a = 0, b = 1, c = 2, e = 3;  // task strides of the template and the other side
    if (side == 2) {
        std::swap(la, lc);
        std::swap(lb, ld);
        std::swap(a, c);
        std::swap(b, e);
        std::swap(qc.bra, qc.ket);
    }
    if (lb == 0 && la > 0) {
        std::swap(la, lb);
        std::swap(a, b);
    }
    qc.swap = side == 2;
    qc.axis = a | b << 2 | c << 4 | e << 6;
    return la * 4 + lb;
}

int dense_lists(size_t n) { return (int)((n + dense::kMaxClasses - 1) / dense::kMaxClasses); }

int dense_smem(int pair, const QuartetClass& qc, int word) {
    return smem_bytes(pair / 4, pair % 4, qc.ket.la, qc.ket.lb, word);
}

cudaError_t launch_dense(int pair, const EriDev& d, const std::vector<QuartetClass>& classes, bool f32, cudaStream_t s) {
    dense::ClassList list;
    for (size_t k = 0; k < classes.size();) {
        list.n = 0;
        list.first[0] = 0;
        int smem = 0;
        for (; k < classes.size() && list.n < dense::kMaxClasses; ++k) {
            const QuartetClass& qc = classes[k];
            const long long blocks = (long long)qc.ngroup * qc.nchunk;
            if (qc.ntask <= 0 || blocks <= 0) continue;
            if (list.n > 0 && list.first[list.n] + blocks > INT32_MAX) break;
            list.cls[list.n] = qc;
            list.first[list.n + 1] = (int)(list.first[list.n] + blocks);
            ++list.n;
            smem = std::max(smem, dense_smem(pair, qc, f32 || d.all_real ? 8 : 16));
        }
        if (list.n == 0) continue;
        cudaError_t e;
        if (list.n == 1)
            e = f32 ? dense::run_one_f32(pair, d, list.cls[0], smem, s) : dense::run_one_f64(pair, d, list.cls[0], smem, s);
        else
            e = f32 ? dense::run_list_f32(pair, d, list, smem, s) : dense::run_list_f64(pair, d, list, smem, s);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// ---------------------------------------------------------------------------
// Work units.  How many primitive quartets of a task survive depends on the
// field, so the units are cut on the device at every execution: unit u of a
// class starts at the first task whose weight prefix (task_weight) within the
// class reaches u * target.  Two launches for the classes with many tasks:
// counts with prefixes over tiles of tasks (the last block to finish turns the
// tile sums into a prefix), then the starts; the others' blocks cut their units
// themselves (cut_units).  A large plan is bound by memory: 48 bytes read and 16
// written per task, and the blocks of the tasks without an FP64 survivor, which
// are cleared here (the kernels store the first batch of every other block).  A
// small one waits for a warp's chain of dependent loads (a task's shells, their
// primitives, the walk over its pair factors) once per row of 32 tasks: up to
// kFewTasks tasks a warp takes one row and a tile is 256 tasks (300,000 tasks:
// 122 us with four rows, 63 with one); beyond, four rows and tiles of 1024, which
// leave the last block a quarter of the tile sums.
// ---------------------------------------------------------------------------

namespace {

constexpr int kUnitThreads = 256, kNoTask = 0x7f7f7f7f;
constexpr long long kFewTasks = 1 << 20;

__device__ __forceinline__ int class_of(const UnitClass* cls, int n, long long v) {
    int lo = 0, hi = n - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) / 2;
        if (cls[mid].vfirst <= v)
            lo = mid;
        else
            hi = mid - 1;
    }
    return lo;
}

// block-wide exclusive prefix of one value per thread; *total receives the sum
__device__ long long block_prefix(long long x, long long* smem, long long* total) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    long long inc = x;
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const long long v = __shfl_up_sync(0xffffffffu, inc, off);
        if (lane >= off) inc += v;
    }
    if (lane == 31) smem[warp] = inc;
    __syncthreads();
    long long before = 0, sum = 0;
    for (int w = 0; w < kUnitThreads / 32; ++w) {
        if (w < warp) before += smem[w];
        sum += smem[w];
    }
    __syncthreads();
    *total = sum;
    return before + inc - x;
}

// ROWS: rows of 32 tasks per warp; a block's tile is ROWS * kUnitThreads tasks
template <int ROWS>
__global__ void __launch_bounds__(kUnitThreads) unit_count_kernel(UnitPlan u, const Task* tasks, PairData pp,
                                                                  const int* nprim, float skip, float cut32,
                                                                  int all_real, double2* out) {
    __shared__ long long smem[kUnitThreads / 32];
    __shared__ bool last;
    for (long long i = (long long)blockIdx.x * kUnitThreads + threadIdx.x; i < u.nunit;
         i += (long long)gridDim.x * kUnitThreads)
        u.start[i] = kNoTask;
    const int lane = threadIdx.x & 31;
    // a warp takes consecutive tasks, 32 at a time: lane-coalesced, and the
    // lanes' weights are put in order by the prefix below
    const long long v0 = ((long long)blockIdx.x * kUnitThreads + (threadIdx.x & ~31)) * ROWS;
    long long w[ROWS], before[ROWS], sum = 0;
#pragma unroll
    for (int k = 0; k < ROWS; ++k) {
        const long long v = v0 + 32 * k + lane;
        w[k] = 0;
        const Task* t = nullptr;
        int dims = 0;
        bool clear = false;
        if (v < u.ntask) {
            const UnitClass c = u.cls[class_of(u.cls, u.ncls, v)];
            if (!c.real_only || all_real) {
                t = tasks + c.first + (v - c.vfirst);
                dims = c.dims;
                int n64, n32;
                w[k] = task_weight(c.mode, t, pp, nprim, skip, cut32, n64, n32);
                u.count[v] = c.mode == 1 ? n32 : n64;
                clear = c.mode != 1 && n64 == 0;
            }
        }
        // clear this row's empty blocks, the warp together on each
        unsigned m = __ballot_sync(0xffffffffu, clear);
        while (m) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            const Task* ts = reinterpret_cast<const Task*>(
                __shfl_sync(0xffffffffu, (unsigned long long)(uintptr_t)t, src));
            clear_block(out, ts, __shfl_sync(0xffffffffu, dims, src), lane);
        }
        // exclusive prefix over the row
        long long inc = w[k];
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const long long x = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += x;
        }
        before[k] = sum + inc - w[k];
        sum += __shfl_sync(0xffffffffu, inc, 31);
    }
    long long total;
    const long long at = block_prefix(lane == 0 ? sum : 0, smem, &total);
    const long long base = __shfl_sync(0xffffffffu, at, 0);
#pragma unroll
    for (int k = 0; k < ROWS; ++k)
        if (v0 + 32 * k + lane < u.ntask) u.prefix[v0 + 32 * k + lane] = base + before[k];
    if (threadIdx.x == 0) {
        u.tile[blockIdx.x] = total;
        __threadfence();
        last = atomicAdd(u.done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    // exclusive prefix of the tile sums, 256 at a time
    __threadfence();
    long long carry = 0;
    for (int t0 = 0; t0 < (int)gridDim.x; t0 += kUnitThreads) {
        const int t = t0 + threadIdx.x;
        const long long x = t < (int)gridDim.x ? __ldcg(u.tile + t) : 0;
        const long long p = block_prefix(x, smem, &total);
        if (t < (int)gridDim.x) u.tile[t] = carry + p;
        carry += total;
    }
    if (threadIdx.x == 0) *u.done = 0;
}

__global__ void unit_start_kernel(UnitPlan u, int tile) {
    const long long v = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (v >= u.ntask) return;
    const UnitClass c = u.cls[class_of(u.cls, u.ncls, v)];
    auto at = [&](long long x) { return u.tile[x / tile] + u.prefix[x]; };
    const long long base = at(c.vfirst);
    const int here = (int)((at(v) - base) / c.target);
    const int prev = v == c.vfirst ? -1 : (int)((at(v - 1) - base) / c.target);
    for (int k = prev + 1; k <= here; ++k) u.start[c.base + k] = (int)(v - c.vfirst);
}

}  // namespace

long long unit_tiles(long long ntask) { return (ntask + kUnitThreads - 1) / kUnitThreads; }

cudaError_t launch_units(const UnitPlan& plan, const Task* tasks, const EriDev& d, cudaStream_t s) {
    UnitPlan u = plan;
    if (!(d.fp32_cut > 0.0f)) {  // (the FP32 unit classes come last)
        u.ntask = plan.ntask64;
        u.nunit = plan.nunit64;
    }
    if (u.ntask <= 0) return cudaSuccess;
    const int tile = (u.ntask <= kFewTasks ? 1 : 4) * kUnitThreads;
    auto* count = u.ntask <= kFewTasks ? unit_count_kernel<1> : unit_count_kernel<4>;
    count<<<(unsigned)((u.ntask + tile - 1) / tile), kUnitThreads, 0, s>>>(u, tasks, d.pairs, d.basis.nprim, d.skip_cut,
                                                                           d.fp32_cut, d.all_real, d.out);
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) return e;
    unit_start_kernel<<<(unsigned)((u.ntask + 255) / 256), 256, 0, s>>>(u, tile);
    return cudaGetLastError();
}

}  // namespace gx
