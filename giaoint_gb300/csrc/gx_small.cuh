// Register-resident kernel for the small quartet classes (L = la+lb+lc+ld <= 2).
//
// One lane evaluates one primitive quartet completely: Boys values, Hermite
// table Rh, ket transform W[K][cd] and bra transform into its contribution
// v[ab][cd], all in registers; every loop is expanded at compile time from
// constexpr plans (index-sequence folds), so all register indices are
// constants.  The kernel is bound by the number of FP64 warp instructions (one
// per 64 cycles and SM sub-partition, whatever the number of active lanes).  A
// warp takes a work unit of consecutive shell quartets with about as many
// surviving primitive quartets as any other (units cut on the device,
// gx_dense.cu) and walks them in full batches of 32 (gx_stream.cuh); the lanes'
// values go through shared memory, where a lane adds the entries of an output
// element in stream order.  Against a segmented shuffle sum (ten FP64
// instructions per element and batch) that costs about two per 32 additions,
// and the result does not depend on the batches.  Batches both of whose pairs have
// q = 0 (zero field, shells on one centre) run in real arithmetic.
#pragma once

#include <utility>

#include "gx_internal.h"
#include "gx_stream.cuh"

namespace gx {
namespace small {

__host__ __device__ constexpr int nc(int l) { return (l + 1) * (l + 2) / 2; }
__host__ __device__ constexpr int hc(int L) { return (L + 1) * (L + 2) * (L + 3) / 6; }
__host__ __device__ constexpr int hi(int k, int l, int m) {
    const int s = k + l + m;
    return s * (s + 1) * (s + 2) / 6 + (s - k) * (s - k + 1) / 2 + m;
}
struct I3 {
    int x, y, z;
};
__host__ __device__ constexpr I3 comp(int l, int idx) {  // x-major Cartesian component
    int k = 0;
    for (int x = l; x >= 0; --x)
        for (int y = l - x; y >= 0; --y) {
            if (k == idx) return I3{x, y, l - x - y};
            ++k;
        }
    return I3{0, 0, 0};
}
__host__ __device__ constexpr I3 herm(int idx) {  // Hermite multi-index of enumeration position idx
    for (int s = 0;; ++s)
        for (int k = s; k >= 0; --k)
            for (int l = s - k; l >= 0; --l)
                if (hi(k, l, s - k - l) == idx) return I3{k, l, s - k - l};
}
// box of component pair ab of pair class (la, lb)
__host__ __device__ constexpr I3 boxdim(int la, int lb, int ab) {
    const I3 a = comp(la, ab / nc(lb)), b = comp(lb, ab % nc(lb));
    return I3{a.x + b.x + 1, a.y + b.y + 1, a.z + b.z + 1};
}
__host__ __device__ constexpr int boxsize(int la, int lb, int ab) {
    const I3 d = boxdim(la, lb, ab);
    return d.x * d.y * d.z;
}
__host__ __device__ constexpr int boxoff(int la, int lb, int ab) {
    int o = 0;
    for (int i = 0; i < ab; ++i) o += boxsize(la, lb, i);
    return o;
}
__host__ __device__ constexpr I3 boxent(int la, int lb, int ab, int e) {
    const I3 d = boxdim(la, lb, ab);
    return I3{e / (d.y * d.z), (e / d.z) % d.y, e % d.z};
}
__host__ __device__ constexpr int etot(int la, int lb) { return boxoff(la, lb, nc(la) * nc(lb)); }

// Rh recurrence plan: step s of the in-place descending scheme.
struct RStep {
    int kind;  // 0 = recurrence entry, 1 = seed of level n
    int dst, s1, s2, axis, coef, n;
};
__host__ __device__ constexpr int rsteps(int L) {
    int c = 0;
    for (int n = L - 1; n >= 0; --n) {
        for (int d = L - n; d >= 1; --d) c += (d + 1) * (d + 2) / 2;
        ++c;
    }
    return c;
}
__host__ __device__ constexpr RStep rstep(int L, int idx) {
    int c = 0;
    for (int n = L - 1; n >= 0; --n) {
        for (int d = L - n; d >= 1; --d)
            for (int k = d; k >= 0; --k)
                for (int l = d - k; l >= 0; --l) {
                    const int m = d - k - l;
                    if (c++ == idx) {
                        if (k > 0) return RStep{0, hi(k, l, m), hi(k - 1, l, m), k > 1 ? hi(k - 2, l, m) : 0, 0, k - 1, n};
                        if (l > 0) return RStep{0, hi(0, l, m), hi(0, l - 1, m), l > 1 ? hi(0, l - 2, m) : 0, 1, l - 1, n};
                        return RStep{0, hi(0, 0, m), hi(0, 0, m - 1), m > 1 ? hi(0, 0, m - 2) : 0, 2, m - 1, n};
                    }
                }
        if (c++ == idx) return RStep{1, 0, 0, 0, 0, 0, n};
    }
    return RStep{1, 0, 0, 0, 0, 0, 0};
}

// ket-transform MAC t over (cd, e, K): W[K][cd] += s(e) Ecd[off(cd)+e] Rh[K + ent(e)]
struct KMac {
    int w, eoff, r, neg;
};
template <int LA, int LB, int LC, int LD>
__host__ __device__ constexpr int kmacs() {
    int c = 0;
    for (int cd = 0; cd < nc(LC) * nc(LD); ++cd) c += boxsize(LC, LD, cd) * hc(LA + LB);
    return c;
}
template <int LA, int LB, int LC, int LD>
__host__ __device__ constexpr KMac kmac(int idx) {
    constexpr int NH = hc(LA + LB), NCD = nc(LC) * nc(LD);
    int c = 0;
    for (int cd = 0; cd < NCD; ++cd)
        for (int e = 0; e < boxsize(LC, LD, cd); ++e)
            for (int K = 0; K < NH; ++K)
                if (c++ == idx) {
                    const I3 h = herm(K), t = boxent(LC, LD, cd, e);
                    return KMac{K * NCD + cd, boxoff(LC, LD, cd) + e, hi(h.x + t.x, h.y + t.y, h.z + t.z),
                                (t.x + t.y + t.z) & 1};
                }
    return KMac{0, 0, 0, 0};
}
// bra-transform MAC t over (ab, e, cd): out[ab][cd] += Eab[off(ab)+e] W[ent(e)][cd]
struct BMac {
    int o, eoff, w;
};
template <int LA, int LB, int LC, int LD>
__host__ __device__ constexpr int bmacs() {
    int c = 0;
    for (int ab = 0; ab < nc(LA) * nc(LB); ++ab) c += boxsize(LA, LB, ab) * nc(LC) * nc(LD);
    return c;
}
template <int LA, int LB, int LC, int LD>
__host__ __device__ constexpr BMac bmac(int idx) {
    constexpr int NCD = nc(LC) * nc(LD);
    int c = 0;
    for (int ab = 0; ab < nc(LA) * nc(LB); ++ab)
        for (int e = 0; e < boxsize(LA, LB, ab); ++e)
            for (int cd = 0; cd < NCD; ++cd)
                if (c++ == idx) {
                    const I3 t = boxent(LA, LB, ab, e);
                    return BMac{ab * NCD + cd, boxoff(LA, LB, ab) + e, hi(t.x, t.y, t.z) * NCD + cd};
                }
    return BMac{0, 0, 0};
}

__device__ __forceinline__ float2 fmul2(float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, -a.y * b.y), fmaf(a.x, b.y, a.y * b.x));
}
__device__ __forceinline__ float2 fmac2(float2 c, float2 a, float2 b) {
    return make_float2(fmaf(a.x, b.x, fmaf(-a.y, b.y, c.x)), fmaf(a.x, b.y, fmaf(a.y, b.x, c.y)));
}

template <int L, int... S>
__device__ __forceinline__ void run_rec32(float2* R, const float2* seed, const float2* X,
                                          std::integer_sequence<int, S...>) {
    (
        [&] {
            constexpr RStep st = rstep(L, S);
            if constexpr (st.kind == 1) {
                R[0] = seed[st.n];
            } else {
                float2 v = fmul2(X[st.axis], R[st.s1]);
                if constexpr (st.coef > 0) {
                    v.x = fmaf((float)st.coef, R[st.s2].x, v.x);
                    v.y = fmaf((float)st.coef, R[st.s2].y, v.y);
                }
                R[st.dst] = v;
            }
        }(),
        ...);
}

template <int LA, int LB, int LC, int LD, int... S>
__device__ __forceinline__ void run_k32(float2* W, const float2* R, const float2* __restrict__ Ecd,
                                        std::integer_sequence<int, S...>) {
    (
        [&] {
            constexpr KMac m = kmac<LA, LB, LC, LD>(S);
            float2 e = __ldg(&Ecd[m.eoff]);
            if constexpr (m.neg) e = make_float2(-e.x, -e.y);
            W[m.w] = fmac2(W[m.w], e, R[m.r]);
        }(),
        ...);
}

template <int LA, int LB, int LC, int LD, int... S>
__device__ __forceinline__ void run_b32(float2* out, const float2* W, const float2* __restrict__ Eab,
                                        std::integer_sequence<int, S...>) {
    (
        [&] {
            constexpr BMac m = bmac<LA, LB, LC, LD>(S);
            out[m.o] = fmac2(out[m.o], __ldg(&Eab[m.eoff]), W[m.w]);
        }(),
        ...);
}

template <int L, int... S>
__device__ __forceinline__ void run_rec(double2* R, const double2* seed, const double2* X,
                                        std::integer_sequence<int, S...>) {
    (
        [&] {
            constexpr RStep st = rstep(L, S);
            if constexpr (st.kind == 1) {
                R[0] = seed[st.n];
            } else {
                double2 v = cmul(X[st.axis], R[st.s1]);
                if constexpr (st.coef > 0) v = cmacr(v, (double)st.coef, R[st.s2]);
                R[st.dst] = v;
            }
        }(),
        ...);
}

template <int LA, int LB, int LC, int LD, int... S>
__device__ __forceinline__ void run_k(double2* W, const double2* R, const double2* __restrict__ Ecd,
                                      std::integer_sequence<int, S...>) {
    (
        [&] {
            constexpr KMac m = kmac<LA, LB, LC, LD>(S);
            double2 e = __ldg(&Ecd[m.eoff]);
            if constexpr (m.neg) e = c2(-e.x, -e.y);
            W[m.w] = cmac(W[m.w], e, R[m.r]);
        }(),
        ...);
}

template <int LA, int LB, int LC, int LD, int... S>
__device__ __forceinline__ void run_b(double2* out, const double2* W, const double2* __restrict__ Eab,
                                      std::integer_sequence<int, S...>) {
    (
        [&] {
            constexpr BMac m = bmac<LA, LB, LC, LD>(S);
            out[m.o] = cmac(out[m.o], __ldg(&Eab[m.eoff]), W[m.w]);
        }(),
        ...);
}

// Seeds C (-2 rho)^n F_n for one primitive quartet; zero seeds on a Boys
// failure, which is reported through the status word.
template <int L>
__device__ __forceinline__ void quartet_seeds(const EriDev& d, long long item, double2 C, double rho, double tre,
                                              double tim, double2* Sh) {
    double2 e0;
    if (const int rc = boys_eval(tre, tim, L, d.boys, d.gl, Sh, e0)) {
        report(d.status, rc, item, L, tre, tim);
        C = c2(0.0, 0.0);
        e0 = c2(0.0, 0.0);
    }
    C = cmul(C, e0);
    const double m2r = -2.0 * rho;
#pragma unroll
    for (int n = 0; n <= L; ++n) {
        Sh[n] = cmul(C, Sh[n]);
        C = cscale(C, m2r);
    }
}

// Real forms of the recurrence and the transforms, for batches both of whose
// pairs have q = 0 (E: the real parts of the complex records).
template <int L, int... S>
__device__ __forceinline__ void run_rec_real(double* R, const double* seed, const double* X,
                                             std::integer_sequence<int, S...>) {
    (
        [&] {
            constexpr RStep st = rstep(L, S);
            if constexpr (st.kind == 1) {
                R[0] = seed[st.n];
            } else {
                double v = X[st.axis] * R[st.s1];
                if constexpr (st.coef > 0) v = fma((double)st.coef, R[st.s2], v);
                R[st.dst] = v;
            }
        }(),
        ...);
}
template <int LA, int LB, int LC, int LD, int... S>
__device__ __forceinline__ void run_k_real(double* W, const double* R, const double2* __restrict__ Ecd,
                                           std::integer_sequence<int, S...>) {
    (
        [&] {
            constexpr KMac m = kmac<LA, LB, LC, LD>(S);
            const double e = __ldg(&Ecd[m.eoff].x);
            W[m.w] = fma(m.neg ? -e : e, R[m.r], W[m.w]);
        }(),
        ...);
}
template <int LA, int LB, int LC, int LD, int... S>
__device__ __forceinline__ void run_b_real(double* out, const double* W, const double2* __restrict__ Eab,
                                           std::integer_sequence<int, S...>) {
    (
        [&] {
            constexpr BMac m = bmac<LA, LB, LC, LD>(S);
            out[m.o] = fma(__ldg(&Eab[m.eoff].x), W[m.w], out[m.o]);
        }(),
        ...);
}

constexpr int kWarps = 4;  // warps of a block, each with its own work unit

// Shared memory of a warp: the values of a batch (33 columns: free of bank
// conflicts both ways), the segments (lanes with one shell quartet), and the
// queue of FP32 entries that wait for a full batch.
template <int NOUT>
struct WarpBuffers {
    double2 v[NOUT * 33];
    long long seg_off[32];
    int4 seg_st[32];
    int seg_lane[36];  // first lane and flags of each segment, and the end
    int2 queue[64];    // task, bra pair * ket pairs of the task + ket pair
    Walk walk;
};

// Notes the segments; flags: those of the lane's task.  Returns their number.
template <int NOUT>
__device__ __forceinline__ int segments(WarpBuffers<NOUT>& w, const QuartetClass& qc, int task, int flags, int nb,
                                        int lane) {
    const int tp = __shfl_up_sync(0xffffffffu, task, 1);
    const bool head = lane < nb && (lane == 0 || tp != task);
    const unsigned heads = __ballot_sync(0xffffffffu, head);
    const int nseg = __popc(heads);
    if (head) {
        const int s = __popc(heads & ((1u << lane) - 1u));
        const Task* t = qc.tasks + task;
        w.seg_off[s] = t->out_off;
        w.seg_st[s] = make_int4(t->st[0], t->st[1], t->st[2], t->st[3]);
        w.seg_lane[s] = lane | flags;
    }
    if (lane == 0) w.seg_lane[nseg] = nb;
    return nseg;
}

// Adds the buffered values of every shell quartet's lanes to its block in
// stream order: the result does not depend on how the stream was cut into
// batches.  kReal: the imaginary parts are zero.  A lane takes the real or the
// imaginary part of an element, or a quarter of a long run: a batch of a deep
// contraction has few elements, and its sums, one lane after 32 entries, were two
// of the 13 us of a batch of (ss|ss).
enum AddMode { kReal, kComplex, kFP32 };
template <int LA, int LB, int LC, int LD, AddMode MODE>
__device__ __forceinline__ void add_runs(double2* out, const WarpBuffers<nc(LA) * nc(LB) * nc(LC) * nc(LD)>& w, int nseg,
                                         int lane) {
    constexpr int NCD = nc(LC) * nc(LD), NOUT = nc(LA) * nc(LB) * NCD, NCB = nc(LB), NCDD = nc(LD);
    constexpr int PARTS = MODE == kReal ? 1 : 2;
    auto element = [&](int s, int o, int part) {
        const int ab = o / NCD, cd = o - ab * NCD;
        const int4 st = w.seg_st[s];
        return reinterpret_cast<double*>(out + w.seg_off[s] + (long long)(ab / NCB) * st.x + (long long)(ab % NCB) * st.y +
                                         (long long)(cd / NCDD) * st.z + (long long)(cd % NCDD) * st.w) +
               part;
    };
    auto put = [&](double* p, bool store, double sum) {
        if (MODE == kReal && store)
            *reinterpret_cast<double2*>(p) = c2(sum, 0.0);
        else
            *p = sum;
    };
    int first = 0;
    if (MODE != kFP32 && nseg > 0 && (w.seg_lane[0] & kLongRuns)) {
        first = 1;
        const bool store = w.seg_lane[0] & kStore;
        const int l1 = w.seg_lane[1] & 255, quarter = lane & 3, l0 = 8 * quarter;
        for (int i0 = 0; i0 < NOUT * PARTS; i0 += 8) {
            const int i = i0 + lane / 4, o = i / PARTS, part = i - o * PARTS;
            const bool valid = i < NOUT * PARTS;
            const double* v = reinterpret_cast<const double*>(w.v + (valid ? o : 0) * 33) + (valid ? part : 0);
            double sum = 0.0;
            if (valid && l0 < l1) {
                sum = v[2 * l0];
                for (int k = l0 + 1; k < l0 + 8 && k < l1; ++k) sum += v[2 * k];
            }
#pragma unroll
            for (int j = 1; j < 4; ++j) {
                const double other = __shfl_down_sync(0xffffffffu, sum, j);
                if (quarter == 0 && 8 * j < l1) sum += other;
            }
            if (valid && quarter == 0) {
                double* p = element(0, o, part);
                put(p, store, store ? sum : *p + sum);
            }
        }
    }
    for (int it = lane; it < (nseg - first) * NOUT * PARTS; it += 32) {
        const int s = it / (NOUT * PARTS), i = it - s * (NOUT * PARTS), o = i / PARTS, part = i - o * PARTS;
        double* p = element(first + s, o, part);
        const double* v = reinterpret_cast<const double*>(w.v + o * 33) + part;
        const int flags = w.seg_lane[first + s], l0 = flags & 255, l1 = w.seg_lane[first + s + 1] & 255;
        if constexpr (MODE == kFP32) {
            // (FP32 values: their passes cut the stream where the Boys paths part)
            double sum = *p;
            for (int l = l0; l < l1; ++l) sum += v[2 * l];
            *p = sum;
        } else {
            const bool store = flags & kStore;
            const double old = store ? 0.0 : *p;
            put(p, store, add_by_runs(old, flags, l0, l1, [&](int k) { return v[2 * k]; }));
        }
    }
}

template <int LA, int LB, int LC, int LD>
__device__ __forceinline__ void small_block(const EriDev& d, const QuartetClass& qc, int block, char* smem) {
    constexpr int L = LA + LB + LC + LD;
    constexpr int NL = hc(L), NH = hc(LA + LB);
    constexpr int NCD = nc(LC) * nc(LD), NOUT = nc(LA) * nc(LB) * NCD;
    const int lane = threadIdx.x & 31;
    WarpBuffers<NOUT>& w = reinterpret_cast<WarpBuffers<NOUT>*>(smem)[threadIdx.x >> 5];
    const int unit = block * kWarps + (threadIdx.x >> 5);
    int t0, t1;
    if (qc.unit_start) {
        if (unit >= qc.ngroup) return;
        // (entries past the last unit lie beyond the class)
        t0 = qc.unit_start[unit];
        t1 = min(qc.unit_start[unit + 1], qc.ntask);
    } else {
        __shared__ int bounds[kWarps + 1];
        __shared__ long long sums[kWarps];
        cut_units<32 * kWarps>(d, qc, 2, block * kWarps, kWarps, true, bounds, sums);
        t0 = bounds[threadIdx.x >> 5];
        t1 = bounds[(threadIdx.x >> 5) + 1];
    }
    if (t0 >= t1) return;
    const PairData& pp = d.pairs;
    unsigned n64 = 0, n32 = 0;
    // FP64 form of one entry into the value buffer
    auto complex_entry = [&](const double2* X, const double2* Sh, int ip, int iq) {
        double2 R[NL];
        if constexpr (L == 0) {
            R[0] = Sh[0];
        } else {
            R[0] = Sh[L];
            run_rec<L>(R, Sh, X, std::make_integer_sequence<int, rsteps(L)>{});
        }
        double2 W[NH * NCD], v[NOUT];
#pragma unroll
        for (int i = 0; i < NH * NCD; ++i) W[i] = c2(0.0, 0.0);
#pragma unroll
        for (int i = 0; i < NOUT; ++i) v[i] = c2(0.0, 0.0);
        run_k<LA, LB, LC, LD>(W, R, pp.Epool + pp.Eoff[iq],
                              std::make_integer_sequence<int, kmacs<LA, LB, LC, LD>()>{});
        run_b<LA, LB, LC, LD>(v, W, pp.Epool + pp.Eoff[ip], std::make_integer_sequence<int, bmacs<LA, LB, LC, LD>()>{});
#pragma unroll
        for (int i = 0; i < NOUT; ++i) w.v[i * 33 + lane] = v[i];
    };
    {
        Stream<false> stream(d, qc, t0, t1, fmaxf(d.skip_cut, d.fp32_cut), 3.4e38f, qc.unit_count, &w.walk);
        for (;;) {
            int task, rank = 0;
            int2 pq;
            const int nb = stream.next(lane, task, rank, pq);
            if (nb == 0) break;
            const int nseg = segments<NOUT>(
                w, qc, task, (rank == 0 ? kStore : 0) | (stream.run == 32 ? kLongRuns : 0), nb, lane);
            const bool real = stream.batch_kind == 3;
            if (lane < nb) {
                const Task* tg = qc.tasks + task;
                const int ip = pp.order[tg->pab + pq.x], iq = pp.order[tg->pcd + pq.y];
                const double p = pp.p[ip], q = pp.p[iq];
                const double rs = rsqrt(p + q);
                const double rho = p * q * rs * rs;
                const double x0 = pp.Pr[3 * ip] - pp.Pr[3 * iq], x1 = pp.Pr[3 * ip + 1] - pp.Pr[3 * iq + 1],
                             x2 = pp.Pr[3 * ip + 2] - pp.Pr[3 * iq + 2];
                if (real) {
                    const double t = rho * fma(x0, x0, fma(x1, x1, x2 * x2));
                    double Sh[L + 1], e0;
                    double C = pp.F[ip].x * pp.F[iq].x * rs;
                    if (const int rc = boys_eval_real(t, L, d.boys, Sh, e0)) {
                        report(d.status, rc, task, L, t, 0.0);
                        C = e0 = 0.0;
#pragma unroll
                        for (int n = 0; n <= L; ++n) Sh[n] = 0.0;
                    }
                    C *= e0;
                    const double m2r = -2.0 * rho;
#pragma unroll
                    for (int n = 0; n <= L; ++n) {
                        Sh[n] *= C;
                        C *= m2r;
                    }
                    const double X[3] = {x0, x1, x2};
                    double R[NL];
                    if constexpr (L == 0) {
                        R[0] = Sh[0];
                    } else {
                        R[0] = Sh[L];
                        run_rec_real<L>(R, Sh, X, std::make_integer_sequence<int, rsteps(L)>{});
                    }
                    double W[NH * NCD], v[NOUT];
#pragma unroll
                    for (int i = 0; i < NH * NCD; ++i) W[i] = 0.0;
#pragma unroll
                    for (int i = 0; i < NOUT; ++i) v[i] = 0.0;
                    run_k_real<LA, LB, LC, LD>(W, R, pp.Epool + pp.Eoff[iq],
                                               std::make_integer_sequence<int, kmacs<LA, LB, LC, LD>()>{});
                    run_b_real<LA, LB, LC, LD>(v, W, pp.Epool + pp.Eoff[ip],
                                               std::make_integer_sequence<int, bmacs<LA, LB, LC, LD>()>{});
#pragma unroll
                    for (int i = 0; i < NOUT; ++i) w.v[i * 33 + lane].x = v[i];
                } else {
                    const double2 X[3] = {c2(x0, pp.Pi[3 * ip] - pp.Pi[3 * iq]),
                                          c2(x1, pp.Pi[3 * ip + 1] - pp.Pi[3 * iq + 1]),
                                          c2(x2, pp.Pi[3 * ip + 2] - pp.Pi[3 * iq + 2])};
                    const double tre = rho * (fma(X[0].x, X[0].x, fma(X[1].x, X[1].x, X[2].x * X[2].x)) -
                                              fma(X[0].y, X[0].y, fma(X[1].y, X[1].y, X[2].y * X[2].y)));
                    const double tim = 2.0 * rho * fma(X[0].x, X[0].y, fma(X[1].x, X[1].y, X[2].x * X[2].y));
                    const double2 C = cscale(cmul(pp.F[ip], pp.F[iq]), rs);
                    double2 Sh[L + 1];
                    quartet_seeds<L>(d, task, C, rho, tre, tim, Sh);
                    complex_entry(X, Sh, ip, iq);
                }
                ++n64;
            }
            __syncwarp();
            if (real)
                add_runs<LA, LB, LC, LD, kReal>(d.out, w, nseg, lane);
            else
                add_runs<LA, LB, LC, LD, kComplex>(d.out, w, nseg, lane);
            __syncwarp();
        }
    }
    // Mixed precision: pass 0 evaluates the FP32 entries whose Boys argument
    // lies in the asymptotic sector (FP32 Boys), pass 1 the others (FP64 Boys,
    // FP32 recurrence), so that every batch follows one Boys path.
    for (int pass = 0; pass < (d.fp32_cut > 0.0f ? 2 : 0); ++pass) {
        Stream<true> stream(d, qc, t0, t1, d.skip_cut, d.fp32_cut, qc.unit_count32, &w.walk);
        int waiting = 0;
        bool more = true;
        while (more || waiting > 0) {
            while (more && waiting < 32) {
                int task, rank;
                int2 pq = make_int2(0, 0);
                const int n = stream.next(lane, task, rank, pq);
                more = n > 0;
                bool mine = lane < n;
                int at = 0;
                if (mine) {
                    const Task* tg = qc.tasks + task;
                    at = pq.x * (d.basis.nprim[tg->sc] * d.basis.nprim[tg->sd]) + pq.y;
                    mine = (pass == 0) ==
                           boys_asymptotic32(pp, pp.order[tg->pab + pq.x], pp.order[tg->pcd + pq.y], L);
                }
                const unsigned m = __ballot_sync(0xffffffffu, mine);
                if (mine) w.queue[waiting + __popc(m & ((1u << lane) - 1u))] = make_int2(task, at);
                waiting += __popc(m);
            }
            __syncwarp();
            const int nb = min(waiting, 32);
            if (nb == 0) break;
            const int2 en = w.queue[min(lane, nb - 1)];
            const int2 rest = w.queue[32 + lane];
            __syncwarp();
            if (lane < waiting - nb) w.queue[lane] = rest;
            waiting -= nb;
            const int nseg = segments<NOUT>(w, qc, en.x, 0, nb, lane);
            if (lane < nb) {
                const Task* tg = qc.tasks + en.x;
                const int Kcd = d.basis.nprim[tg->sc] * d.basis.nprim[tg->sd], P = en.y / Kcd;
                const int ip = pp.order[tg->pab + P], iq = pp.order[tg->pcd + en.y - P * Kcd];
                const double p = pp.p[ip], q = pp.p[iq];
                const double2 X[3] = {c2(pp.Pr[3 * ip] - pp.Pr[3 * iq], pp.Pi[3 * ip] - pp.Pi[3 * iq]),
                                      c2(pp.Pr[3 * ip + 1] - pp.Pr[3 * iq + 1], pp.Pi[3 * ip + 1] - pp.Pi[3 * iq + 1]),
                                      c2(pp.Pr[3 * ip + 2] - pp.Pr[3 * iq + 2], pp.Pi[3 * ip + 2] - pp.Pi[3 * iq + 2])};
                const double rs = rsqrt(p + q);
                const double rho = p * q * rs * rs;
                const double tre = rho * (fma(X[0].x, X[0].x, fma(X[1].x, X[1].x, X[2].x * X[2].x)) -
                                          fma(X[0].y, X[0].y, fma(X[1].y, X[1].y, X[2].y * X[2].y)));
                const double tim = 2.0 * rho * fma(X[0].x, X[0].y, fma(X[1].x, X[1].y, X[2].x * X[2].y));
                const double2 C = cscale(cmul(pp.F[ip], pp.F[iq]), rs);
                double2 Sh[L + 1];
                float2 S32[L + 1];
                bool ok32 = pass == 0 && seeds32(C, rho, tre, tim, L, S32);
                if (!ok32) {
                    // FP64 Boys; FP32 recurrence when the seeds fit
                    quartet_seeds<L>(d, en.x, C, rho, tre, tim, Sh);
                    ok32 = true;
#pragma unroll
                    for (int n = 0; n <= L; ++n) {
                        ok32 = ok32 && fabs(Sh[n].x) + fabs(Sh[n].y) < 1.0e25;
                        S32[n] = make_float2((float)Sh[n].x, (float)Sh[n].y);
                    }
                }
                if (ok32) {
                    const float2 X32[3] = {make_float2((float)X[0].x, (float)X[0].y),
                                           make_float2((float)X[1].x, (float)X[1].y),
                                           make_float2((float)X[2].x, (float)X[2].y)};
                    float2 R32[NL];
                    if constexpr (L == 0) {
                        R32[0] = S32[0];
                    } else {
                        R32[0] = S32[L];
                        run_rec32<L>(R32, S32, X32, std::make_integer_sequence<int, rsteps(L)>{});
                    }
                    float2 W32[NH * NCD], v32[NOUT];
#pragma unroll
                    for (int i = 0; i < NH * NCD; ++i) W32[i] = make_float2(0.0f, 0.0f);
#pragma unroll
                    for (int i = 0; i < NOUT; ++i) v32[i] = make_float2(0.0f, 0.0f);
                    run_k32<LA, LB, LC, LD>(W32, R32, pp.Epool32 + pp.Eoff[iq],
                                            std::make_integer_sequence<int, kmacs<LA, LB, LC, LD>()>{});
                    run_b32<LA, LB, LC, LD>(v32, W32, pp.Epool32 + pp.Eoff[ip],
                                            std::make_integer_sequence<int, bmacs<LA, LB, LC, LD>()>{});
#pragma unroll
                    for (int i = 0; i < NOUT; ++i) w.v[i * 33 + lane] = c2(widen(v32[i].x, 0), widen(v32[i].y, 0));
                    ++n32;
                } else {
                    complex_entry(X, Sh, ip, iq);
                    ++n64;
                }
            }
            __syncwarp();
            add_runs<LA, LB, LC, LD, kFP32>(d.out, w, nseg, lane);
            __syncwarp();
        }
    }
    if (qc.counters) {
        const unsigned a64 = __reduce_add_sync(0xffffffffu, n64);
        const unsigned a32 = __reduce_add_sync(0xffffffffu, n32);
        if (lane == 0) {
            if (a64) atomicAdd(&qc.counters[0], (unsigned long long)a64);
            if (a32) atomicAdd(&qc.counters[1], (unsigned long long)a32);
        }
    }
}

template <int LA, int LB, int LC, int LD>
__global__ void __launch_bounds__(32 * kWarps) small_kernel(const __grid_constant__ EriDev d,
                                                            const __grid_constant__ QuartetClass qc) {
    __shared__ WarpBuffers<nc(LA) * nc(LB) * nc(LC) * nc(LD)> s_buf[kWarps];
    small_block<LA, LB, LC, LD>(d, qc, blockIdx.x, reinterpret_cast<char*>(s_buf));
}

// The small classes of a small plan in one launch: block b works on class c with
// first[c] <= b < first[c + 1].
struct ClassList {
    int n;
    int key[15];
    int first[16];
    QuartetClass cls[15];
};

}  // namespace small
}  // namespace gx
