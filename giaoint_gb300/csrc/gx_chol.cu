// Device kernels of the streamed pivoted Cholesky (K6-K9):
//
//   chol_diag_kernel     (mu nu|nu mu) diagonal from packed (ab|ba) blocks,
//                        placed as src/cholesky.cpp:305-311
//   chol_cols_kernel     pivot columns (mu nu|p1 p0) from packed
//                        (ab|sb sa) blocks; zero-phase real path mirrored and
//                        same-shell averaged as src/cholesky.cpp:245-279
//   chol_gemv_kernel     column -= conj(L[:rank, piv]) L[:rank]
//                        (python/giao_integrals/cholesky.py:268)
//   chol_update_kernel   real symmetrisation, 1/sqrt(residual) scale, new
//                        factor row, residual -= |column|^2, PSD minimum,
//                        clamp, zeroed pivot and the next argmax, fused
//                        (cholesky.py:269-281)
//   argmax reductions    lowest flat index on ties (NumPy argmax order)
#include <algorithm>
#include <type_traits>

#include "gx_internal.h"

namespace gx {

// ---- diagonal --------------------------------------------------------------

// info per block: ao_a, ao_b, na, nb
__global__ void chol_diag_kernel(const double2* packed, const long long* boff, const int* info, int nblocks, int n,
                                 double* D) {
    const int bi = blockIdx.x;
    if (bi >= nblocks) return;
    const int oa = info[4 * bi], ob = info[4 * bi + 1], na = info[4 * bi + 2], nb = info[4 * bi + 3];
    const double2* blk = packed + boff[bi];
    for (int e = threadIdx.x; e < na * nb; e += blockDim.x) {
        const int i = e / nb, j = e - i * nb;
        const double v = blk[(((long long)i * nb + j) * nb + j) * na + i].x;
        const long long mu = oa + i, nu = ob + j;
        D[nu * n + mu] = v;
        if (oa != ob) D[mu * n + nu] = v;
    }
}

cudaError_t launch_chol_diag(const double2* packed, const long long* boff, const int* info, int nblocks, int n,
                             double* D, cudaStream_t s) {
    if (nblocks <= 0) return cudaSuccess;
    chol_diag_kernel<<<nblocks, 128, 0, s>>>(packed, boff, info, nblocks, n, D);
    return cudaGetLastError();
}

// ---- columns ---------------------------------------------------------------

// info per block: ao_a, ao_b, na, nb, same_shell; cand[2*k] = (c, d) local
// indices in shells (sb, sa); dst[k] = column k (n*n values).  flip[block]
// (may be null): the block was evaluated as (sb sa | a b), laid out
// (nc, nd, na, nb), which equals (a b | sb sa) by the exchange of the two
// electrons.
template <bool REAL>
__global__ void chol_cols_kernel(const double2* packed, const long long* boff, const int* info, const int* flip,
                                 int nblocks, const int* cand, int ncand, int nc, int nd, int n, void* const* dst) {
    const int bi = blockIdx.x;
    if (bi >= nblocks) return;
    const int oa = info[5 * bi], ob = info[5 * bi + 1], na = info[5 * bi + 2], nb = info[5 * bi + 3];
    const bool same = info[5 * bi + 4] != 0;
    const bool flipped = flip != nullptr && flip[bi] != 0;
    const double2* blk = packed + boff[bi];
    const int per = na * nb;
    auto at = [&](int i, int j, int c, int d) -> double2 {
        return flipped ? blk[(((long long)c * nd + d) * na + i) * nb + j]
                       : blk[(((long long)i * nb + j) * nc + c) * nd + d];
    };
    for (int e = threadIdx.x; e < per * ncand; e += blockDim.x) {
        const int k = e / per, r = e - k * per;
        const int i = r / nb, j = r - i * nb;
        const int c = cand[2 * k], d = cand[2 * k + 1];
        const double2 v = at(i, j, c, d);
        const long long mu = oa + i, nu = ob + j;
        if (REAL) {
            double s = v.x;
            if (same) s = (s + at(j, i, c, d).x) * 0.5;
            double* out = static_cast<double*>(dst[k]);
            out[mu * n + nu] = s;
            if (!same) out[nu * n + mu] = s;
        } else {
            double2* out = static_cast<double2*>(dst[k]);
            out[mu * n + nu] = v;
        }
    }
}

cudaError_t launch_chol_cols(bool real, const double2* packed, const long long* boff, const int* info,
                             const int* flip, int nblocks, const int* cand, int ncand, int nc, int nd, int n,
                             void* const* dst, cudaStream_t s) {
    if (nblocks <= 0) return cudaSuccess;
    if (real)
        chol_cols_kernel<true><<<nblocks, 256, 0, s>>>(packed, boff, info, flip, nblocks, cand, ncand, nc, nd, n,
                                                       dst);
    else
        chol_cols_kernel<false><<<nblocks, 256, 0, s>>>(packed, boff, info, flip, nblocks, cand, ncand, nc, nd, n,
                                                        dst);
    return cudaGetLastError();
}

// ---- argmax / min reductions -------------------------------------------------

// Largest value (the lowest index among equals) and smallest value.  The
// reductions compare order-preserving integer keys: an FP64 comparison occupies
// its sub-partition for 64 cycles, and the butterflies over (value, index,
// minimum) were most of a 9 us step end (chain_update_kernel, 1,600 entries).
struct Red {
    double maxv;
    long long idx;
    double minv;
};
struct RedKey {
    long long maxk, idx, mink;
};

__device__ __forceinline__ long long red_order(long long bits) { return bits ^ ((bits >> 63) & 0x7fffffffffffffffll); }
// (NaN takes part in neither, as in a comparison; -0 counts as 0)
__device__ __forceinline__ RedKey red_key(double v, long long j, double low) {
    const long long v0 = __double_as_longlong(v), l0 = __double_as_longlong(low);
    constexpr long long kInf = 0x7ff0000000000000ll, kAbs = 0x7fffffffffffffffll;
    RedKey k;
    k.maxk = (v0 & kAbs) > kInf ? red_order(kInf | (1ll << 63)) : red_order((v0 & kAbs) == 0 ? 0 : v0);
    k.idx = j;
    k.mink = (l0 & kAbs) > kInf ? kInf : red_order((l0 & kAbs) == 0 ? 0 : l0);
    return k;
}
__device__ __forceinline__ RedKey red_none() { return red_key(-1.0 / 0.0, (long long)1 << 62, 1.0 / 0.0); }
__device__ __forceinline__ Red red_value(const RedKey& k) {
    return Red{__longlong_as_double(red_order(k.maxk)), k.idx, __longlong_as_double(red_order(k.mink))};
}

__device__ __forceinline__ void red_merge(RedKey& a, const RedKey& b) {
    if (b.maxk > a.maxk || (b.maxk == a.maxk && b.idx < a.idx)) {
        a.maxk = b.maxk;
        a.idx = b.idx;
    }
    a.mink = min(a.mink, b.mink);
}

__device__ __forceinline__ RedKey warp_reduce(RedKey r, int lanes) {
    for (int o = lanes / 2; o > 0; o >>= 1) {
        RedKey t;
        t.maxk = __shfl_down_sync(0xffffffffu, r.maxk, o);
        t.idx = __shfl_down_sync(0xffffffffu, r.idx, o);
        t.mink = __shfl_down_sync(0xffffffffu, r.mink, o);
        red_merge(r, t);
    }
    return r;
}

// (blocks of at most eight warps)
__device__ RedKey block_reduce(RedKey r) {
    __shared__ RedKey sh[8];
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    r = warp_reduce(r, 32);
    if (lane == 0) sh[w] = r;
    __syncthreads();
    if (w == 0) r = warp_reduce(lane < (int)(blockDim.x >> 5) ? sh[lane] : red_none(), 8);
    return r;
}

// Blocks of the reductions over N entries, at most as many as one block merges:
// an entry a thread, in blocks of 128 (of 1,000 entries every warp then has a
// sub-partition to itself).
constexpr int RED_BLOCKS = 256, RED_THREADS = 128;
int red_blocks(long long N) {
    return (int)std::max<long long>(1, std::min<long long>((N + RED_THREADS - 1) / RED_THREADS, RED_BLOCKS));
}

__global__ void chol_scan_kernel(const double* res, long long N, RedKey* partial) {
    RedKey r = red_none();
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < N; j += (long long)gridDim.x * blockDim.x) {
        const double v = res[j];
        red_merge(r, red_key(v, j, v));
    }
    r = block_reduce(r);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
}

__global__ void chol_final_kernel(const RedKey* partial, int np, Red* out) {
    RedKey r = red_none();
    for (int i = threadIdx.x; i < np; i += blockDim.x) red_merge(r, partial[i]);
    r = block_reduce(r);
    if (threadIdx.x == 0) *out = red_value(r);
}

cudaError_t launch_chol_scan(const double* res, long long N, void* partial, void* out, cudaStream_t s) {
    chol_scan_kernel<<<red_blocks(N), RED_THREADS, 0, s>>>(res, N, static_cast<RedKey*>(partial));
    chol_final_kernel<<<1, 256, 0, s>>>(static_cast<const RedKey*>(partial), red_blocks(N), static_cast<Red*>(out));
    return cudaGetLastError();
}

// ---- small copies ------------------------------------------------------------

// The loop's transfers are a few words to a few hundred KB each; as copies of
// their own every one took the stream 3 us and its call 3.5 us of the host
// (four to the host after a step, three before an evaluation).
struct WordCopies {
    WordCopy c[4];
    long long first[5];
    int n;
};

__global__ void __launch_bounds__(256) copy_words_kernel(const __grid_constant__ WordCopies a) {
    for (long long i = blockIdx.x * 256ll + threadIdx.x; i < a.first[a.n]; i += gridDim.x * 256ll) {
        int k = 0;
        while (i >= a.first[k + 1]) ++k;
        const long long w = i - a.first[k];
        static_cast<unsigned long long*>(a.c[k].dst)[w] = static_cast<const unsigned long long*>(a.c[k].src)[w];
    }
}

cudaError_t launch_copy_words(std::initializer_list<WordCopy> copies, int sms, cudaStream_t s) {
    WordCopies a;
    a.n = 0;
    a.first[0] = 0;
    for (const WordCopy& c : copies) {
        if (c.words <= 0) continue;
        if (a.n == 4) return cudaErrorInvalidValue;
        a.c[a.n] = c;
        a.first[a.n + 1] = a.first[a.n] + c.words;
        ++a.n;
    }
    if (a.n == 0) return cudaSuccess;
    const long long blocks = std::min<long long>((a.first[a.n] + 255) / 256, 4ll * std::max(sms, 1));
    copy_words_kernel<<<(unsigned)blocks, 256, 0, s>>>(a);
    return cudaGetLastError();
}

// ---- factor update -----------------------------------------------------------

// acc +/- conj(a) * b as four dependent-pair FMAs (the complex update is
// FP64-pipe bound: 4 DFMA per 16-byte element instead of 4 + 2 adds)
__device__ __forceinline__ double2 conj_mul_add(double2 acc, double2 a, double2 b) {
    return c2(fma(a.y, b.y, fma(a.x, b.x, acc.x)), fma(-a.y, b.x, fma(a.x, b.y, acc.y)));
}
__device__ __forceinline__ double2 conj_mul_sub(double2 acc, double2 a, double2 b) {
    return c2(fma(-a.y, b.y, fma(-a.x, b.x, acc.x)), fma(a.y, b.x, fma(-a.x, b.y, acc.y)));
}

// What a thread of the factor update sums: a column entry, or with HALVES the
// real or imaginary part of one.  The rows of a few thousand entries come from
// the L2 cache, and an entry's four dependent-pair FMAs per complex row, 31 ns
// each for a warp alone on its sub-partition, are most of the time of the update:
// two threads share them, with the same operations in the same order (the 223
// updates of two atoms in a field, 900 entries, 5.66 -> 5.36 ms, the 348 of
// three, 2,025 entries, 8.87 -> 8.45 ms, each twice within 0.02; one atom, 225
// entries, and six, 8,100, are the same either way).  Long columns, bound by
// memory, keep whole entries.
template <typename T, bool HALVES>
struct Entry {
    using Acc = std::conditional_t<HALVES, double, T>;
    long long j;
    int part = 0;
    __device__ __forceinline__ explicit Entry(long long t) : j(HALVES ? t >> 1 : t) {
        if (HALVES) part = (int)(t & 1);
    }
    __device__ __forceinline__ static Acc zero() {
        if constexpr (std::is_same_v<Acc, double>)
            return 0.0;
        else
            return c2(0.0, 0.0);
    }
    __device__ __forceinline__ long long at(long long row) const { return HALVES ? 2 * row + part : row; }
};

// acc +/- the sum of conj(L[r, piv]) L[r, j] over rows rbeg .. rend - 1, in
// order (all threads of a block call this; coef: 256 entries of shared memory)
template <typename T, bool HALVES, bool SUB>
__device__ __forceinline__ typename Entry<T, HALVES>::Acc gemv_rows(typename Entry<T, HALVES>::Acc acc,
                                                                   const Entry<T, HALVES>& e, const T* L,
                                                                   long long ld, int rbeg, int rend, long long piv,
                                                                   long long N, T* coef) {
    for (int r0 = rbeg; r0 < rend; r0 += 256) {
        const int nr = min(256, rend - r0);
        __syncthreads();
        for (int i = threadIdx.x; i < nr; i += blockDim.x) coef[i] = L[(long long)(r0 + i) * ld + piv];
        __syncthreads();
        if (e.j < N) {
            // eight independent row loads in flight per thread: the GEMV of a
            // long column is bound by HBM bandwidth, not by load latency
#pragma unroll 8
            for (int r = 0; r < nr; ++r) {
                const T lv = __ldg(&L[(long long)(r0 + r) * ld + e.j]);
                if constexpr (sizeof(T) == 8) {
                    acc = fma(SUB ? -coef[r] : coef[r], lv, acc);
                } else if constexpr (HALVES) {
                    // re: fma(a.y, b.y, fma(a.x, b.x, acc)); im: fma(-a.y, b.x, fma(a.x, b.y, acc))
                    const double2 a = SUB ? c2(-coef[r].x, -coef[r].y) : coef[r];
                    const double u = e.part ? lv.y : lv.x;
                    const double w = e.part ? __hiloint2double(__double2hiint(lv.x) ^ 0x80000000, __double2loint(lv.x))
                                            : lv.y;
                    acc = fma(a.y, w, fma(a.x, u, acc));
                } else {
                    acc = SUB ? conj_mul_sub(acc, coef[r], lv) : conj_mul_add(acc, coef[r], lv);
                }
            }
        }
    }
    return acc;
}

template <typename T, bool HALVES>
__global__ void chol_gemv_kernel(const T* L, long long ld, int rank, long long piv, const T* col_in, T* col_out,
                                 long long N) {
    __shared__ T coef[256];
    using Acc = typename Entry<T, HALVES>::Acc;
    const Entry<T, HALVES> e((long long)blockIdx.x * blockDim.x + threadIdx.x);
    Acc acc = e.j < N ? reinterpret_cast<const Acc*>(col_in)[e.at(e.j)] : Entry<T, HALVES>::zero();
    acc = gemv_rows<T, HALVES, true>(acc, e, L, ld, 0, rank, piv, N, coef);
    if (e.j < N) reinterpret_cast<Acc*>(col_out)[e.at(e.j)] = acc;
}

// The same update with the rank split over blockIdx.y: block (x, y) sums
// conj(L[r, piv]) L[r, j] over its rows into partials[y][j], and
// chol_gemv_sum_kernel subtracts the chunks in order.  Small n (few column
// entries) otherwise leaves too few loads in flight to stream L at HBM speed.
template <typename T, bool HALVES>
__global__ void chol_gemv_split_kernel(const T* L, long long ld, int rank, long long piv, int chunk, T* partials,
                                       long long N) {
    __shared__ T coef[256];
    using Acc = typename Entry<T, HALVES>::Acc;
    const Entry<T, HALVES> e((long long)blockIdx.x * blockDim.x + threadIdx.x);
    const int rbeg = blockIdx.y * chunk, rend = min(rank, rbeg + chunk);
    const Acc acc = gemv_rows<T, HALVES, false>(Entry<T, HALVES>::zero(), e, L, ld, rbeg, rend, piv, N, coef);
    if (e.j < N) reinterpret_cast<Acc*>(partials)[e.at((long long)blockIdx.y * N + e.j)] = acc;
}

// Two threads per complex entry while the doubled grid leaves at most two
// warps on a sub-partition.
bool gemv_halves(bool real, int blocks, int nchunks, int sms) { return !real && 2 * blocks * nchunks <= 2 * sms; }

template <typename T>
__global__ void chol_gemv_sum_kernel(const T* col_in, const T* partials, int nchunks, long long N, T* col_out) {
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < N; j += (long long)gridDim.x * blockDim.x) {
        T acc = col_in[j];
        for (int y = 0; y < nchunks; ++y) {
            if constexpr (sizeof(T) == 8) {
                acc -= partials[(long long)y * N + j];
            } else {
                acc = csub(acc, partials[(long long)y * N + j]);
            }
        }
        col_out[j] = acc;
    }
}

// entry (nu mu) of entry j = (mu nu)
__device__ __forceinline__ long long transposed(long long j, int n) {
    const unsigned mu = (unsigned long long)j >> 32 ? (unsigned)(j / n) : (unsigned)j / (unsigned)n;
    return (j - (long long)mu * n) * n + mu;
}

// scale = 1/sqrt(residual[piv]) (read before the update)
__global__ void chol_scale_kernel(const double* res, long long piv, double* scale) { *scale = rsqrt(res[piv]); }

template <typename T>
__global__ void chol_update_kernel(const T* col, int n, long long piv, const double* scale, T* Lrow, double* res,
                                   RedKey* partial) {
    const long long N = (long long)n * n;
    const double sc = *scale;
    RedKey r = red_none();
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < N; j += (long long)gridDim.x * blockDim.x) {
        double mag2;
        if constexpr (sizeof(T) == 8) {
            const double c = (col[j] + col[transposed(j, n)]) * 0.5 * sc;
            Lrow[j] = c;
            mag2 = c * c;
        } else {
            const double2 c = cscale(col[j], sc);
            Lrow[j] = c;
            mag2 = c.x * c.x + c.y * c.y;
        }
        const double nr = res[j] - mag2;
        const double kept = j == piv ? 0.0 : fmax(nr, 0.0);
        res[j] = kept;
        red_merge(r, red_key(kept, j, nr));
    }
    r = block_reduce(r);
    if (threadIdx.x == 0) partial[blockIdx.x] = r;
}

cudaError_t launch_chol_step(bool real, const void* L, long long ld, int rank, long long piv, const void* column,
                             void* work, int n, double* res, double* scale, void* Lrow, void* partial, void* out,
                             cudaStream_t s, void* gemv_partials, int max_chunks, int sms) {
    const long long N = (long long)n * n;
    const int blocks = (int)((N + 127) / 128);
    // rank chunks: enough blocks for about eight per SM, at least 32 rows each
    int nchunks = 1;
    if (gemv_partials && max_chunks > 1 && rank >= 64 && sms > 0) {
        nchunks = std::max(1, std::min({max_chunks, (8 * sms) / std::max(blocks, 1), (rank + 31) / 32}));
    }
    if (nchunks > 1) {
        const int chunk = (rank + nchunks - 1) / nchunks;
        const dim3 grid(blocks, nchunks);
        const int sblocks = (int)std::min<long long>((N + 255) / 256, 8LL * sms);
        if (real) {
            chol_gemv_split_kernel<double, false><<<grid, 128, 0, s>>>(
                static_cast<const double*>(L), ld, rank, piv, chunk, static_cast<double*>(gemv_partials), N);
            chol_gemv_sum_kernel<double><<<sblocks, 256, 0, s>>>(static_cast<const double*>(column),
                                                                  static_cast<const double*>(gemv_partials), nchunks,
                                                                  N, static_cast<double*>(work));
        } else {
            const bool halves = gemv_halves(real, blocks, nchunks, sms);
            auto* gemv = halves ? chol_gemv_split_kernel<double2, true> : chol_gemv_split_kernel<double2, false>;
            gemv<<<halves ? dim3(2 * blocks, nchunks) : grid, 128, 0, s>>>(
                static_cast<const double2*>(L), ld, rank, piv, chunk, static_cast<double2*>(gemv_partials), N);
            chol_gemv_sum_kernel<double2><<<sblocks, 256, 0, s>>>(static_cast<const double2*>(column),
                                                                   static_cast<const double2*>(gemv_partials), nchunks,
                                                                   N, static_cast<double2*>(work));
        }
    } else if (real) {
        chol_gemv_kernel<double, false><<<blocks, 128, 0, s>>>(static_cast<const double*>(L), ld, rank, piv,
                                                               static_cast<const double*>(column),
                                                               static_cast<double*>(work), N);
    } else {
        const bool halves = gemv_halves(real, blocks, 1, sms);
        auto* gemv = halves ? chol_gemv_kernel<double2, true> : chol_gemv_kernel<double2, false>;
        gemv<<<halves ? 2 * blocks : blocks, 128, 0, s>>>(static_cast<const double2*>(L), ld, rank, piv,
                                                          static_cast<const double2*>(column),
                                                          static_cast<double2*>(work), N);
    }
    chol_scale_kernel<<<1, 1, 0, s>>>(res, piv, scale);
    if (real)
        chol_update_kernel<double><<<red_blocks(N), RED_THREADS, 0, s>>>(static_cast<const double*>(work), n, piv,
                                                                         scale, static_cast<double*>(Lrow), res,
                                                                         static_cast<RedKey*>(partial));
    else
        chol_update_kernel<double2><<<red_blocks(N), RED_THREADS, 0, s>>>(static_cast<const double2*>(work), n, piv,
                                                                          scale, static_cast<double2*>(Lrow), res,
                                                                          static_cast<RedKey*>(partial));
    chol_final_kernel<<<1, 256, 0, s>>>(static_cast<const RedKey*>(partial), red_blocks(N), static_cast<Red*>(out));
    return cudaGetLastError();
}

// ---- chained steps: pivots taken on the device while their columns are cached ----
//
// After a step the next pivot is the argmax of the residual.  When its raw
// column is already in the column cache (slot_of[pivot] >= 0), the next step
// needs no host decision, so the host enqueues up to K steps at once and
// synchronises once: chain_select_kernel takes the argmax of the previous
// step, stops the chain (active = 0, with the reason) when the residual has
// converged, the rank limit is reached, the PSD check failed or the column is
// not cached, and otherwise records the pivot and its slot; the step kernels
// below read the pivot, rank and column from that state and return at once
// when the chain has stopped.

// Select logic shared by the chain's first step and the fused end of every
// step: stop the chain, or take the argmax as the next pivot (its column
// slot, its scale 1/sqrt(residual), its place in the log).
__device__ void chain_select(ChainState* st, const Red& r, int* slot_of, long long* log, double tol, double psd) {
    int stop = 0;
    int slot = -1;
    if (r.minv < -psd)
        stop = 4;
    else if (!(r.maxv > tol))
        stop = 2;
    else if (st->rank >= st->rank_limit)
        stop = 3;
    else if ((slot = slot_of[r.idx]) < 0)
        stop = 1;
    if (stop) {
        st->active = 0;
        st->stop = stop;
        return;
    }
    st->pivot = r.idx;
    st->slot = slot;
    st->scale = rsqrt(r.maxv);  // r.maxv is the stored residual of the pivot
    slot_of[r.idx] = -1;
    log[st->rank] = r.idx;
}

__global__ void chain_select_kernel(ChainState* st, const Red* red, int* slot_of, long long* log, double tol,
                                    double psd) {
    if (!st->active) return;
    chain_select(st, *red, slot_of, log, tol, psd);
}

template <typename T, bool HALVES>
__global__ void chain_gemv_split_kernel(const T* L, long long ld, const ChainState* st, int nchunks, T* partials,
                                        long long N) {
    if (!st->active) return;
    __shared__ T coef[256];
    using Acc = typename Entry<T, HALVES>::Acc;
    const int rank = st->rank;
    const int chunk = (rank + nchunks - 1) / nchunks;
    const Entry<T, HALVES> e((long long)blockIdx.x * blockDim.x + threadIdx.x);
    const int rbeg = blockIdx.y * chunk, rend = min(rank, rbeg + chunk);
    const Acc acc = gemv_rows<T, HALVES, false>(Entry<T, HALVES>::zero(), e, L, ld, rbeg, rend, st->pivot, N, coef);
    if (e.j < N) reinterpret_cast<Acc*>(partials)[e.at((long long)blockIdx.y * N + e.j)] = acc;
}

// Updated column entry j: the cached raw column minus the rank-chunk partial
// sums, in chunk order.
template <typename T>
__device__ __forceinline__ T chain_column(const T* col_in, const T* partials, int nchunks, long long N, long long j) {
    T acc = col_in[j];
    for (int y = 0; y < nchunks; ++y) {
        if constexpr (sizeof(T) == 8) {
            acc -= partials[(long long)y * N + j];
        } else {
            acc = csub(acc, partials[(long long)y * N + j]);
        }
    }
    return acc;
}

// The new factor row (the updated column times the pivot's scale; the real
// path symmetrises (mu nu) with (nu mu)), the residual update and its
// argmax/minimum.  Each block reduces its entries into partial[block]; the
// last block to finish (counted in st->done) merges the partials in block
// order, as a separate reduction kernel would, ends the step (rank, step
// count) and, unless this is the chain's last step, selects the next pivot.
template <typename T>
__global__ void chain_update_kernel(ChainState* st, const T* pool, const T* partials, int nchunks, int n, T* L,
                                    double* res, RedKey* partial, Red* out, int* slot_of, long long* log, double tol,
                                    double psd, int select_next) {
    if (!st->active) return;
    const long long N = (long long)n * n;
    const long long piv = st->pivot;
    const T* col_in = pool + (long long)st->slot * N;
    T* Lrow = L + (long long)st->rank * N;
    const double sc = st->scale;
    RedKey r = red_none();
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < N; j += (long long)gridDim.x * blockDim.x) {
        double mag2;
        if constexpr (sizeof(T) == 8) {
            const double wj = chain_column(col_in, partials, nchunks, N, j);
            const double wt = chain_column(col_in, partials, nchunks, N, transposed(j, n));
            const double c = (wj + wt) * 0.5 * sc;
            Lrow[j] = c;
            mag2 = c * c;
        } else {
            const double2 c = cscale(chain_column(col_in, partials, nchunks, N, j), sc);
            Lrow[j] = c;
            mag2 = c.x * c.x + c.y * c.y;
        }
        const double nr = res[j] - mag2;
        const double kept = j == piv ? 0.0 : fmax(nr, 0.0);
        res[j] = kept;
        red_merge(r, red_key(kept, j, nr));
    }
    r = block_reduce(r);
    __shared__ int last;
    if (threadIdx.x == 0) {
        partial[blockIdx.x] = r;
        __threadfence();
        last = atomicAdd(&st->done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    RedKey k = red_none();
    const volatile RedKey* vp = partial;
    for (int i = threadIdx.x; i < (int)gridDim.x; i += blockDim.x)
        red_merge(k, RedKey{vp[i].maxk, vp[i].idx, vp[i].mink});
    k = block_reduce(k);
    if (threadIdx.x == 0) {
        const Red q = red_value(k);
        *out = q;
        st->done = 0;
        st->rank += 1;
        st->steps += 1;
        if (select_next) chain_select(st, q, slot_of, log, tol, psd);
    }
}

cudaError_t launch_chol_chain(bool real, void* L, long long N, int n, int rank_hi, int steps, ChainState* st,
                              int* slot_of, long long* log, const void* pool, double* res, void* partial, void* out,
                              void* gemv_partials, int max_chunks, int sms, double tol, double psd, cudaStream_t s) {
    const int blocks = (int)((N + 127) / 128);
    int nchunks = 1;
    if (gemv_partials && max_chunks > 1 && rank_hi >= 64 && sms > 0)
        nchunks = std::max(1, std::min(max_chunks, (8 * sms) / std::max(blocks, 1)));
    const dim3 grid(blocks, nchunks);
    Red* red = static_cast<Red*>(out);
    if (steps > 0) chain_select_kernel<<<1, 1, 0, s>>>(st, red, slot_of, log, tol, psd);
    for (int k = 0; k < steps; ++k) {
        const int select_next = k + 1 < steps ? 1 : 0;
        if (real) {
            chain_gemv_split_kernel<double, false><<<grid, 128, 0, s>>>(static_cast<const double*>(L), N, st, nchunks,
                                                                        static_cast<double*>(gemv_partials), N);
            chain_update_kernel<double><<<red_blocks(N), RED_THREADS, 0, s>>>(
                st, static_cast<const double*>(pool), static_cast<const double*>(gemv_partials), nchunks, n,
                static_cast<double*>(L), res, static_cast<RedKey*>(partial), red, slot_of, log, tol, psd, select_next);
        } else {
            const bool halves = gemv_halves(real, blocks, nchunks, sms);
            auto* gemv = halves ? chain_gemv_split_kernel<double2, true> : chain_gemv_split_kernel<double2, false>;
            gemv<<<halves ? dim3(2 * blocks, nchunks) : grid, 128, 0, s>>>(
                static_cast<const double2*>(L), N, st, nchunks, static_cast<double2*>(gemv_partials), N);
            chain_update_kernel<double2><<<red_blocks(N), RED_THREADS, 0, s>>>(
                st, static_cast<const double2*>(pool), static_cast<const double2*>(gemv_partials), nchunks, n,
                static_cast<double2*>(L), res, static_cast<RedKey*>(partial), red, slot_of, log, tol, psd, select_next);
        }
    }
    return cudaGetLastError();
}

// Real factor rows widened to complex128 (imaginary parts zero), for the
// copy to the caller.
__global__ void widen_real_kernel(const double* __restrict__ src, double2* __restrict__ dst, long long n) {
    for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (long long)gridDim.x * blockDim.x)
        dst[i] = make_double2(src[i], 0.0);
}

cudaError_t launch_widen_real(const double* src, double2* dst, long long n, int sms, cudaStream_t s) {
    if (n <= 0) return cudaSuccess;
    const int grid = (int)std::max<long long>(1, std::min<long long>((n + 255) / 256, 8LL * std::max(sms, 1)));
    widen_real_kernel<<<grid, 256, 0, s>>>(src, dst, n);
    return cudaGetLastError();
}

// residual = D - sum_P |L_P|^2 (used when screened diagonal blocks are measured at the end)
template <typename T>
__global__ void chol_final_residual_kernel(const double* D, const T* L, int rank, long long N, double* res) {
    for (long long j = (long long)blockIdx.x * blockDim.x + threadIdx.x; j < N; j += (long long)gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int r = 0; r < rank; ++r) {
            const T v = L[(long long)r * N + j];
            if constexpr (sizeof(T) == 8)
                s += v * v;
            else
                s += v.x * v.x + v.y * v.y;
        }
        res[j] = D[j] - s;
    }
}

cudaError_t launch_chol_final_residual(bool real, const double* D, const void* L, int rank, long long N, double* res,
                                       cudaStream_t s) {
    const int blocks = (int)((N + 255) / 256);
    if (real)
        chol_final_residual_kernel<double><<<blocks, 256, 0, s>>>(D, static_cast<const double*>(L), rank, N, res);
    else
        chol_final_residual_kernel<double2><<<blocks, 256, 0, s>>>(D, static_cast<const double2*>(L), rank, N, res);
    return cudaGetLastError();
}

size_t chol_red_bytes() { return sizeof(Red); }
size_t chol_partial_bytes() { return sizeof(RedKey) * RED_BLOCKS; }

}  // namespace gx
