// Surviving primitive quartets of a work unit as a stream of full batches, for
// the kernels that give a primitive quartet to a lane (gx_small.cuh,
// gx_dense.cuh).
#pragma once

#include "gx_internal.h"

namespace gx {

__device__ __forceinline__ double plus(double a, double b) { return a + b; }
__device__ __forceinline__ double2 plus(double2 a, double2 b) { return cadd(a, b); }

// Number of primitive quartets of a task with lo <= B_P B_Q < hi (FP32
// products of the sorted factors, so that for every bra pair they are a run of
// ket pairs whose ends move down as the bra pair's factor decreases).
__device__ __forceinline__ int survivors(const float* __restrict__ sp, int Kab, const float* __restrict__ sq, int Kcd,
                                         float lo, float hi) {
    int qb = Kcd, qa = hi < 3.0e38f ? Kcd : 0, n = 0;
    for (int P = 0; P < Kab; ++P) {
        const float b = sp[P];
        while (qb > 0 && !(b * sq[qb - 1] >= lo)) --qb;
        while (qa > 0 && b * sq[qa - 1] < hi) --qa;
        n += qb - qa > 0 ? qb - qa : 0;
    }
    return n;
}

// Where a survivor lies: its bra pair, the ends of that one's run of ket pairs, and
// the survivors of the bra pairs before it.
struct Row {
    int P, qb, qa, before;
};
// The row of a stream's last entry, of the task it is in (-1: not kept).
struct Walk {
    Row row;
    int task;
};

// The j-th of them in stream order (bra pair, then ket pair), from `row` on (of the
// task's start, or of an earlier survivor), which is left at the survivor's.
__device__ __forceinline__ int2 survivor(const float* __restrict__ sp, int Kab, const float* __restrict__ sq, float lo,
                                         float hi, int j, Row& row) {
    int qb = row.qb, qa = row.qa, before = row.before;
    for (int P = row.P; P < Kab; ++P) {
        const float b = sp[P];
        while (qb > 0 && !(b * sq[qb - 1] >= lo)) --qb;
        while (qa > 0 && b * sq[qa - 1] < hi) --qa;
        const int n = qb - qa > 0 ? qb - qa : 0;
        if (j - before < n) {
            row = Row{P, qb, qa, before};
            return make_int2(P, qa + j - before);
        }
        before += n;
    }
    return make_int2(0, 0);
}

// Weight of a task in its class's work units: 64 per FP64 survivor (modes 0 and
// 2), 64 (mode 1) or 24 (mode 2, whose kernel takes both) per FP32 one, plus 1.
// n64 and n32 receive the survivors that the mode counts.
__device__ __forceinline__ long long task_weight(int mode, const Task* t, const PairData& pp,
                                                 const int* __restrict__ nprim, float skip, float cut32, int& n64,
                                                 int& n32) {
    const int Kab = nprim[t->sa] * nprim[t->sb], Kcd = nprim[t->sc] * nprim[t->sd];
    const float *sp = pp.sbound + t->pab, *sq = pp.sbound + t->pcd;
    n64 = mode == 1 ? 0 : survivors(sp, Kab, sq, Kcd, fmaxf(skip, cut32), 3.4e38f);
    n32 = mode == 0 || !(cut32 > 0.0f) ? 0 : survivors(sp, Kab, sq, Kcd, skip, cut32);
    return 64ll * n64 + (mode == 1 ? 64ll : 24ll) * n32 + 1;
}

// clears the block of one task with all lanes of a warp (dims: the components
// of its shells, one byte each)
__device__ __forceinline__ void clear_block(double2* out, const Task* t, int dims, int lane) {
    const int nb = (dims >> 8) & 255, nc = (dims >> 16) & 255, nd = (dims >> 24) & 255;
    const int per = (dims & 255) * nb * nc * nd;
    double2* o = out + t->out_off;
    const int s0 = t->st[0], s1 = t->st[1], s2 = t->st[2], s3 = t->st[3];
    if (s3 == 1 && s2 == nd && s1 == nc * nd && s0 == nb * nc * nd) {
        for (int e = lane; e < per; e += 32) o[e] = c2(0.0, 0.0);
        return;
    }
    for (int e = lane; e < per; e += 32) {
        const int ab = e / (nc * nd), cd = e - ab * (nc * nd);
        o[(long long)(ab / nb) * s0 + (long long)(ab % nb) * s1 + (long long)(cd / nd) * s2 + (long long)(cd % nd) * s3] =
            c2(0.0, 0.0);
    }
}

// Units of a class with few tasks, cut by every block for itself (all its
// threads call this): bounds[k] = the number of tasks whose weight prefix lies
// below (first + k) * target, k = 0 .. n, i.e. the first task of unit first + k.
// Units first .. first + n - 1 of the class are the block's; their tasks
// without an FP64 survivor are cleared when `clear` is set.  THREADS: block size.
template <int THREADS>
__device__ __forceinline__ void cut_units(const EriDev& d, const QuartetClass& qc, int mode, int first, int n,
                                          bool clear, int* bounds, long long* warp_sum) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (threadIdx.x <= (unsigned)n) bounds[threadIdx.x] = 0;
    __syncthreads();
    long long base = 0;
    for (int i0 = 0; i0 < qc.ntask; i0 += THREADS) {
        const int i = i0 + threadIdx.x;
        int n64 = 1, n32 = 0;
        long long w = 0;
        if (i < qc.ntask)
            w = task_weight(mode, qc.tasks + i, d.pairs, d.basis.nprim, d.skip_cut, d.fp32_cut, n64, n32);
        long long inc = w;
#pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            const long long v = __shfl_up_sync(0xffffffffu, inc, off);
            if (lane >= off) inc += v;
        }
        if (lane == 31) warp_sum[warp] = inc;
        __syncthreads();
        long long before = base + inc - w;
        for (int k = 0; k < THREADS / 32; ++k) {
            if (k < warp) before += warp_sum[k];
            base += warp_sum[k];
        }
        for (int k = 0; k <= n; ++k) {
            const unsigned m = __ballot_sync(0xffffffffu, i < qc.ntask && before < (long long)(first + k) * qc.target);
            if (lane == 0 && m) atomicAdd(&bounds[k], __popc(m));
        }
        unsigned m = __ballot_sync(0xffffffffu, clear && i < qc.ntask && n64 == 0 &&
                                                    before >= (long long)first * qc.target &&
                                                    before < (long long)(first + n) * qc.target);
        while (m) {
            const int src = __ffs(m) - 1;
            m &= m - 1;
            clear_block(d.out, qc.tasks + i0 + warp * 32 + src, qc.dims, lane);
        }
        __syncthreads();
    }
}

// A task's FP64 values are summed in runs of entries, and the run sums one
// after the other, so that the rounding of a deep contraction grows with the
// number of runs; batches never split a run, so the sums do not depend on how
// the stream is cut into batches.  Runs of 8 cost a batch two lanes on average;
// a task of 256 entries or more has room for runs of 32, which start at lane 0 and
// are four sums of 8.
__device__ __forceinline__ int run_length(int survivors) { return survivors >= 256 ? 32 : 8; }

// The surviving primitive quartets of the tasks t0 .. t1 - 1 in stream order
// (task, bra pair, ket pair), up to 32 at a time, one per lane.  32 tasks are
// looked at together: their survivor counts as an inclusive prefix over the
// lanes, and how many of those have been handed out.  Entries with
// lo <= B_P B_Q < hi; counts: their number in every task of the class (may be
// null).  FP64 batches hold tasks
// of one kind (bit 0: template pair real, bit 1: other pair real), so that a
// task's arithmetic does not depend on its neighbours.
template <bool F32>
struct Stream {
    const EriDev& d;
    const QuartetClass& qc;
    float lo, hi;
    const int* counts;
    int t1, next_task, chunk = 0, incl = 0, cnt = 0, kind = 0, total = 0, used = 0, batch_kind = 0;
    int run = 8;  // run length of the lane's task
    // The last entry handed out, when its task goes on and the walk to it was a long
    // one: the next entry is sought from there (from the task's start every batch of
    // a deep contraction walked over all its bra pairs: one (ss|ss) of 20 primitives
    // a shell, 1.6e5 entries, 141 instead of 29.5 ms).  In shared memory: held in
    // registers it cost the (pp| template an occupancy step, 1% of twelve atoms.
    Walk* walk;

    __device__ __forceinline__ Stream(const EriDev& dev, const QuartetClass& cls, int first, int last, float from,
                                      float below, const int* task_counts, Walk* kept)
        : d(dev), qc(cls), lo(from), hi(below), counts(task_counts), t1(last), next_task(first), walk(kept) {
        __syncwarp();
        walk->task = -1;  // (every lane of the stream's warp)
        __syncwarp();
    }
    // Returns the number of entries; every lane below it has its task, the
    // entry's rank within the task, and its bra and ket pair.
    __device__ __forceinline__ int next(int lane, int& task, int& rank, int2& pq) {
        const PairData& pp = d.pairs;
        const int* np = d.basis.nprim;
        int got = 0;
        task = -1;
        int left = 0;  // entries of the lane's task after its own
        while (got < 32) {
            if (used == total) {
                if (next_task >= t1) break;
                chunk = next_task;
                next_task += 32;
                cnt = 0;
                kind = 0;
                if (chunk + lane < t1) {
                    const Task* tg = qc.tasks + chunk + lane;
                    if constexpr (!F32) {
                        const double *pb = pp.Pi + 3 * (size_t)tg->pab, *pk = pp.Pi + 3 * (size_t)tg->pcd;
                        kind = (pb[0] == 0.0 && pb[1] == 0.0 && pb[2] == 0.0 ? (qc.swap ? 2 : 1) : 0) |
                               (pk[0] == 0.0 && pk[1] == 0.0 && pk[2] == 0.0 ? (qc.swap ? 1 : 2) : 0);
                        if (d.all_real) kind = 3;  // (every pair has q = 0; the table is sized for that)
                    }
                    if (!counts)
                        cnt = survivors(pp.sbound + tg->pab, np[tg->sa] * np[tg->sb], pp.sbound + tg->pcd,
                                        np[tg->sc] * np[tg->sd], lo, hi);
                    else
                        cnt = counts[chunk + lane];
                }
                if (__any_sync(0xffffffffu, cnt > 1 << 25)) {  // (the sum of 32 might not fit)
                    if (lane > 0) cnt = 0;
                    next_task = chunk + 1;
                }
                incl = cnt;
#pragma unroll
                for (int off = 1; off < 32; off <<= 1) {
                    const int v = __shfl_up_sync(0xffffffffu, incl, off);
                    if (lane >= off) incl += v;
                }
                total = __shfl_sync(0xffffffffu, incl, 31);
                used = 0;
                continue;
            }
            int end = total;
            if constexpr (!F32) {
                const bool open = cnt > 0 && incl > used;
                const unsigned left = __ballot_sync(0xffffffffu, open);
                const int kd = __shfl_sync(0xffffffffu, kind, __ffs(left) - 1);
                if (got > 0 && kd != batch_kind) break;
                batch_kind = kd;
                const unsigned other = __ballot_sync(0xffffffffu, open && kind != kd);
                const int stop = __shfl_sync(0xffffffffu, incl - cnt, other ? __ffs(other) - 1 : 31);
                if (other) end = stop;
            }
            int take = min(32 - got, end - used);
            bool full = false;
            if constexpr (!F32) {
                // a batch that ends within a task ends after a whole run
                if (used + take < end) {
                    int at = 0;
#pragma unroll
                    for (int h = 16; h > 0; h >>= 1) {
                        const int v = __shfl_sync(0xffffffffu, incl, at + h - 1);
                        if (v <= used + take) at += h;
                    }
                    const int out = used + take - __shfl_sync(0xffffffffu, incl - cnt, at);
                    take -= out % run_length(__shfl_sync(0xffffffffu, cnt, at));
                    full = true;
                }
            }
            const int e = used + lane - got;
            int src = 0;
#pragma unroll
            for (int h = 16; h > 0; h >>= 1) {
                const int v = __shfl_sync(0xffffffffu, incl, src + h - 1);
                if (v <= e) src += h;
            }
            const int before = __shfl_sync(0xffffffffu, incl - cnt, src & 31);
            const int whole = __shfl_sync(0xffffffffu, cnt, src & 31);
            if (lane >= got && lane < got + take) {
                task = chunk + src;
                rank = e - before;
                run = run_length(whole);
                left = whole - 1 - rank;
            }
            used += take;
            got += take;
            if (full) break;
        }
        if (got == 0) return 0;
        Row r{};
        if (lane < got) {
            const Task* tg = qc.tasks + task;
            if (task == walk->task) {
                r = walk->row;
            } else {
                const int Kcd = np[tg->sc] * np[tg->sd];
                r = Row{0, Kcd, hi < 3.0e38f ? Kcd : 0, 0};
            }
            pq = survivor(pp.sbound + tg->pab, np[tg->sa] * np[tg->sb], pp.sbound + tg->pcd, lo, hi, rank, r);
        }
        // (a kept row stays valid until the stream has left its task: entries are only
        // sought further on)
        const bool keep = lane == got - 1 && left > 0 && r.P >= 16;
        if (__any_sync(0xffffffffu, keep)) {
            __syncwarp();
            if (keep) *walk = Walk{r, task};
            __syncwarp();
        }
        return got;
    }
};

// Flags of a batch's segment beside its first lane: the batch holds the shell
// quartet's first FP64 entry, which stores instead of adding; long runs.
// kSingle: entry by entry (entries queued over several batches of the stream).
constexpr int kStore = 256, kLongRuns = 512, kSingle = 1024;

// A segment's values v(l0) .. v(l1 - 1) by runs, added to sum (or, with
// kStore, in its place).
template <typename T, typename Get>
__device__ __forceinline__ T add_by_runs(T sum, int flags, int l0, int l1, Get&& v) {
    const int run = flags & kSingle ? 1 : (flags & kLongRuns ? 32 : 8);
    bool fresh = flags & kStore;
    for (int l = l0; l < l1; l += run) {
        const int end = l + run < l1 ? l + run : l1;
        T whole{};
        for (int l8 = l; l8 < end; l8 += 8) {
            T part = v(l8);
            for (int k = l8 + 1; k < l8 + 8 && k < end; ++k) part = plus(part, v(k));
            whole = l8 == l ? part : plus(whole, part);
        }
        sum = fresh ? whole : plus(sum, whole);
        fresh = false;
    }
    return sum;
}

// v 2^shift as a double by integer work (a conversion is an FP64 instruction);
// results below the normal range become zero.
__device__ __forceinline__ double widen(float v, int shift) {
    const unsigned u = __float_as_uint(v);
    const int e = (int)((u >> 23) & 255u), x = e + 896 + shift;
    if (e == 255) return (double)v;
    if (e == 0 || x <= 0) return 0.0;
    if (x >= 2047) return __hiloint2double((int)((u & 0x80000000u) | 0x7ff00000u), 0);
    return __hiloint2double((int)((u & 0x80000000u) | ((unsigned)x << 20) | ((u & 0x7fffffu) >> 3)), (int)(u << 29));
}

}  // namespace gx
