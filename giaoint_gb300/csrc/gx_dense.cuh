// Lane-dense kernel of the shell-quartet classes one side of which is a
// template pair (dense_class in gx_dense.cu): a lane owns a primitive quartet
// from the Boys function to its block contribution.
//
// What bounds it.  Each SM sub-partition issues one FP64 warp instruction per
// 64 cycles, whatever the number of active lanes and already with one warp and
// no instruction-level parallelism (measured: 31.0 ns per dependent DFMA for
// one warp, 7.75 ns per SM for four warps, the same with 1 or 32 active
// lanes).  The time of a class is therefore its number of FP64 warp
// instructions: idle lanes cost as much as working ones, while loads, integer
// work and shared-memory traffic fit between two FP64 issues.  The
// class-generic kernel gives a primitive quartet to a whole warp, whose
// transforms (items rounded up to 32, butterfly sums, recurrence levels of 4 or
// 10 entries) leave about half of the lanes idle.
//
// Split.  A block of four warps takes a work unit -- consecutive shell quartets
// with about `target` surviving primitive quartets, found on the device from
// the current field's Schwarz factors (unit kernels below), so that the batches
// of 32 are full whatever share of the quartets is screened.  Per batch one
// warp (another one from block to block: each sub-partition gets its share)
// forms the Boys values and seeds; the warps together build the Hermite table
// of every lane in a column of shared memory (conflict-free) and then share the
// components of the run-time side: per component the first
// transform accumulates W[K] for the template side's Hermite rows in
// registers, and the second one, unrolled from constexpr boxes, writes the
// values to a shared buffer, from which the lanes of each shell quartet are
// added to its block in stream order.  One table serves four warps, so that a
// dozen warps fit an SM even at L = 6.
//
// Real arithmetic.  A pair with q = 0 (zero field, or both shells on one
// centre) has real Hermite coefficients, and two such pairs have a real
// separation and a real table.  A batch whose pairs on one side are of that
// kind uses two DFMA per multiply-add on that side instead of four, and a batch
// with both sides real uses one; batches do not mix the kinds, and plans order
// the tasks of a class so that this rarely shortens a batch.  The dropped terms
// are products with exact zeros.
//
// FP32.  The same kernel evaluates the FP32 entries of mixed precision (tables,
// transforms in FP32; separation, T, prefactor, Boys function outside its
// asymptotic sector, seeds and every sum into the blocks in FP64), after the FP64
// one on the same stream.  Entries whose seeds may leave the FP32 range (tight
// primitives on one centre at high orders) are skipped there and evaluated in
// FP64 by a launch for all classes (gx_dense_wide.cu).
#pragma once

#include <type_traits>
#include <utility>

#include "gx_internal.h"
#include "gx_per_device.h"
#include "gx_small.cuh"
#include "gx_stream.cuh"

namespace gx {
namespace dense {

using small::boxent;
using small::boxoff;
using small::boxsize;
using small::etot;
using small::hc;
using small::hi;
using small::I3;
using small::nc;

__device__ __forceinline__ double2 mac(double2 c, double2 a, double2 b) { return cmac(c, a, b); }
__device__ __forceinline__ double2 mac(double2 c, double a, double2 b) { return cmacr(c, a, b); }
__device__ __forceinline__ double mac(double c, double a, double b) { return fma(a, b, c); }
__device__ __forceinline__ float2 mac(float2 c, float2 a, float2 b) { return small::fmac2(c, a, b); }
__device__ __forceinline__ float2 mac(float2 c, float a, float2 b) {
    return make_float2(fmaf(a, b.x, c.x), fmaf(a, b.y, c.y));
}
__device__ __forceinline__ double2 mul(double2 a, double2 b) { return cmul(a, b); }
__device__ __forceinline__ double mul(double a, double b) { return a * b; }
__device__ __forceinline__ float2 mul(float2 a, float2 b) { return small::fmul2(a, b); }
__device__ __forceinline__ double2 add(double2 a, double2 b) { return cadd(a, b); }
__device__ __forceinline__ double add(double a, double b) { return a + b; }
__device__ __forceinline__ float2 add(float2 a, float2 b) { return make_float2(a.x + b.x, a.y + b.y); }
template <typename T>
__device__ __forceinline__ T zero() {
    return T{};
}
// EV: the part of a Hermite coefficient that is used (its real part for a real pair)
template <typename EV, typename EP>
__device__ __forceinline__ EV load(const EP* p) {
    if constexpr (std::is_same_v<EV, double>)
        return __ldg(&p->x);
    else
        return __ldg(p);
}
// v with its sign flipped when bit 31 of s is set (no FP64 instruction)
__device__ __forceinline__ double flip(double v, int s) {
    return __hiloint2double(__double2hiint(v) ^ (s & 0x80000000), __double2loint(v));
}
__device__ __forceinline__ double2 flip(double2 v, int s) { return c2(flip(v.x, s), flip(v.y, s)); }
__device__ __forceinline__ float2 flip(float2 v, int s) {
    return make_float2(__int_as_float(__float_as_int(v.x) ^ (s & 0x80000000)),
                       __int_as_float(__float_as_int(v.y) ^ (s & 0x80000000)));
}
__device__ __forceinline__ double coef_of(double2*, int k) { return c_dev.ints[k]; }
__device__ __forceinline__ double coef_of(double*, int k) { return c_dev.ints[k]; }
__device__ __forceinline__ float coef_of(float2*, int k) { return (float)k; }

constexpr int kWarps = 4;
// Highest order of an execution, and of one whose pairs are all real.  The table
// of order 8 takes 84 KB a block (165 rows), two blocks an SM; at 9 and 10 there
// is room for one, and five atoms with f shells in a field took 35.2 ms instead
// of the class-generic kernel's 29.6.  A real table has half the bytes: 73 KB at
// order 10, and the same atoms at zero field take 11.7 ms instead of 13.4.
constexpr int kMaxOrder = 8, kMaxOrderReal = 10;
constexpr int kMaxSeeds = kMaxOrderReal + 1;

// Value buffer of a warp: the components ab of `group` components of the other
// side, or of a slice of one, 9 to 12 rows of 33 columns (the odd width keeps
// both the lanes' stores and the sums over a row's lanes free of conflicts).
__host__ __device__ constexpr int slice_of(int nab) { return nab <= 12 ? nab : (nab % 9 == 0 ? 9 : 10); }
__host__ __device__ constexpr int group_of(int nab) { return nab == 1 ? 9 : (nab <= 6 ? (nab == 3 ? 3 : 2) : 1); }
__host__ __device__ constexpr int rows_of(int nab) { return slice_of(nab) * group_of(nab); }

// Shared layout of a block, in bytes; word: bytes of a table entry (16 complex
// FP64, 8 complex FP32 or an execution all of whose pairs are real).  hsum rows are padded to four entries so
// that the table rows of one Hermite index of the other side are read as int4.
struct Layout {
    int hsum, kh, kb, R, v, seed, eb, ek, seg_off, seg_st, shift, seg_lane, info, walk, total;
};
__host__ __device__ inline Layout layout(int NH, int NAB, int ncdh, int etot_ket, int ncd, int L, int word) {
    const int NHP = (NH + 3) / 4 * 4, NL = (L + 1) * (L + 2) * (L + 3) / 6;
    Layout w;
    w.hsum = 0;
    w.kb = w.hsum + ncdh * NHP * 4;
    w.kh = w.kb + ncd * 8;
    w.R = (w.kh + etot_ket * 4 + 15) / 16 * 16;
    w.v = w.R + NL * 32 * word;
    w.seed = w.v + (kWarps * rows_of(NAB) * 33 * word + 15) / 16 * 16;
    w.eb = w.seed + (L + 4) * 32 * word;
    w.ek = w.eb + 32 * 8;
    w.seg_off = w.ek + 32 * 8;
    w.seg_st = w.seg_off + 32 * 8;
    w.shift = w.seg_st + 32 * 16;
    w.seg_lane = w.shift + 32 * 4;
    w.info = w.seg_lane + 36 * 4;
    w.walk = w.info + 16;
    w.total = w.walk + 32;
    return w;
}

// Hermite recurrence of every lane's column (32 columns) by the step list of
// order L, in place: level by level, and within a level degree by degree from
// the top, whose entries only read lower degrees of the previous level and are
// shared by the block's warps.  seeds: [L + 1] seeds and X'[3] of every lane.
// (seeds, col: of the lane's entry; part, parts: its share of every degree, over
// the block's warps and the lanes that share the entry.)
template <typename T>
__device__ __forceinline__ void recurrence(const int2* __restrict__ plan, int L, const T* seeds, T* col, int part,
                                           int parts) {
    const T X0 = seeds[(L + 1) * 32], X1 = seeds[(L + 2) * 32], X2 = seeds[(L + 3) * 32];
    if (part == 0) col[0] = seeds[L * 32];
    int pos = 0;
    for (int n = L - 1; n >= 0; --n) {
        __syncthreads();
        for (int dg = L - n; dg >= 1; --dg) {
            const int cnt = (dg + 1) * (dg + 2) / 2;
            for (int i = part; i < cnt; i += parts) {
                const int2 st = __ldg(&plan[pos + i]);
                const int dst = st.x & 0xffff, s1 = (st.x >> 16) & 0xffff;
                const int s2 = st.y & 0x3fff, axis = (st.y >> 14) & 3, coef = (st.y >> 16) & 63;
                const T xa = axis == 0 ? X0 : (axis == 1 ? X1 : X2);
                T v = mul(xa, col[s1 * 32]);
                if (coef > 0) v = mac(v, coef_of((T*)nullptr, coef), col[s2 * 32]);
                col[dst * 32] = v;
            }
            pos += cnt;
            __syncthreads();
        }
        if (part == 0) col[0] = seeds[n * 32];
        ++pos;  // (the list's seed step)
    }
    __syncthreads();
}

// First transform of one component of the other side:
//   W[K] = sum_e (+-) E[e] R[K + K'_e], e over the component's box.
template <int NH, typename EV, typename RT, typename EP>
__device__ __forceinline__ void ket(RT* W, const RT* col, const EP* __restrict__ E, const int* kh, int nbox,
                                    const int* hsum) {
#pragma unroll
    for (int k = 0; k < NH; ++k) W[k] = zero<RT>();
    EV next = load<EV>(&E[0]);
    for (int e = 0; e < nbox; ++e) {
        const int kk = kh[e];
        const EV ev = flip(next, kk);
        next = load<EV>(&E[min(e + 1, nbox - 1)]);
        const int4* h = reinterpret_cast<const int4*>(hsum + (kk & 0x7fffffff));
#pragma unroll
        for (int k = 0; k < NH; k += 4) {
            const int4 r = h[k / 4];
            W[k] = mac(W[k], ev, col[r.x]);
            if (k + 1 < NH) W[k + 1 < NH ? k + 1 : 0] = mac(W[k + 1 < NH ? k + 1 : 0], ev, col[r.y]);
            if (k + 2 < NH) W[k + 2 < NH ? k + 2 : 0] = mac(W[k + 2 < NH ? k + 2 : 0], ev, col[r.z]);
            if (k + 3 < NH) W[k + 3 < NH ? k + 3 : 0] = mac(W[k + 3 < NH ? k + 3 : 0], ev, col[r.w]);
        }
    }
}

// Second transform: v[ab] = sum_{K in box(ab)} E[K] W[K] of the components
// AB0 + AB into the lane's column of the value buffer.
template <int LA, int LB, int AB, typename EA, typename RT, typename EP, int... I>
__device__ __forceinline__ RT bra_component(const RT* W, const EP* __restrict__ E, std::integer_sequence<int, I...>) {
    RT v = zero<RT>();
    (
        [&] {
            constexpr I3 t = boxent(LA, LB, AB, I);
            v = mac(v, load<EA>(&E[boxoff(LA, LB, AB) + I]), W[hi(t.x, t.y, t.z)]);
        }(),
        ...);
    return v;
}
template <int LA, int LB, int AB0, typename EA, typename RT, typename EP, int... AB>
__device__ __forceinline__ void bra(RT* vb, const RT* W, const EP* __restrict__ E, std::integer_sequence<int, AB...>) {
    ((vb[AB * 33] = bra_component<LA, LB, AB0 + AB, EA, RT>(
          W, E, std::make_integer_sequence<int, boxsize(LA, LB, AB0 + AB)>{})),
     ...);
}

// What a warp needs for the sums into the blocks.
struct Out {
    double2* out;
    const long long* seg_off;   // block of each segment (run of lanes with one shell quartet)
    const int4* seg_st;         // its strides: template a, b, other c, d
    const int* shift;           // FP32: per lane, the power of two that undoes its seed scale
    const int* seg_lane;        // first lane and flags of each segment, and the end
    int nseg, cbegin, cend, ndd, lane;  // (components of this block)
    int width, parts;           // lanes of an entry set, and how many sets (with their own components) fill the warp
    bool inner_c;               // the other side's components are the inner ones of the block
};

// The lanes of each segment over the value buffer (components ab0 .. of the
// other side's components c .. c + cg - 1 of lane set 0, the following groups of
// `stride` components of the other sets), added to its block in stream order
// and in FP64: the result depends neither on where the batches of a unit begin
// or end, nor on what else they hold.
template <int LB, typename RT>
__device__ __forceinline__ void reduce_out(const Out& o, const RT* vb, int ab0, int nab, int c, int cg, int stride) {
    constexpr int NCB = nc(LB);
    const int one = nab * cg, per = one * o.parts;
    for (int it = o.lane; it < o.nseg * per; it += 32) {
        const int s = it / per, rest = it - s * per;
        const int set = rest / one, m = rest - set * one;
        // neighbouring lanes take neighbouring elements of the block
        const int i = o.inner_c ? m / cg : m % nab, u = o.inner_c ? m - i * cg : m / nab;
        const int ab = ab0 + i, cx = c + set * stride + u;
        if (cx >= o.cend) continue;
        const int cc = cx / o.ndd, cdd = cx - cc * o.ndd;
        const int4 st = o.seg_st[s];
        double2* p = o.out + o.seg_off[s] + (long long)(ab / NCB) * st.x + (long long)(ab % NCB) * st.y +
                     (long long)cc * st.z + (long long)cdd * st.w;
        const RT* v = vb + (u * nab + i) * 33 + set * o.width;
        const int flags = o.seg_lane[s], l0 = flags & 255, l1 = o.seg_lane[s + 1] & 255;
        const bool store = flags & kStore;
        auto at = [&](int k) { return v[k]; };
        if constexpr (std::is_same_v<RT, double2>) {
            const double2 old = store ? c2(0.0, 0.0) : *p;
            *p = add_by_runs(old, flags, l0, l1, at);
        } else if constexpr (std::is_same_v<RT, double>) {
            const double old = store ? 0.0 : p->x;
            const double sum = add_by_runs(old, flags, l0, l1, at);
            if (store)
                *p = c2(sum, 0.0);
            else
                p->x = sum;
        } else {
            double2 sum = *p;
            for (int l = l0; l < l1; ++l) sum = cadd(sum, c2(widen(v[l].x, o.shift[l]), widen(v[l].y, o.shift[l])));
            *p = sum;
        }
    }
}

// Second transform and sums of a component group, slice by slice (only: the
// slices of one warp, when the block's warps share the group; -1: all).
template <int LA, int LB, typename RT, typename EP, int... S>
__device__ __forceinline__ void slices(const Out& o, const RT* W, RT* vb, const EP* Eb, bool bra_real, int c,
                                       int only, std::integer_sequence<int, S...>) {
    constexpr int SL = slice_of(nc(LA) * nc(LB));
    (
        [&] {
            if (sizeof...(S) > 1 && !std::is_same_v<RT, float2> && only >= 0 && S % kWarps != only) return;
            if constexpr (std::is_same_v<RT, double>) {
                bra<LA, LB, S * SL, double, RT>(vb + o.lane, W, Eb, std::make_integer_sequence<int, SL>{});
            } else if constexpr (std::is_same_v<RT, double2>) {
                if (bra_real)
                    bra<LA, LB, S * SL, double, RT>(vb + o.lane, W, Eb, std::make_integer_sequence<int, SL>{});
                else
                    bra<LA, LB, S * SL, double2, RT>(vb + o.lane, W, Eb, std::make_integer_sequence<int, SL>{});
            } else {
                bra<LA, LB, S * SL, float2, RT>(vb + o.lane, W, Eb, std::make_integer_sequence<int, SL>{});
            }
            if constexpr (group_of(nc(LA) * nc(LB)) == 1) {
                __syncwarp();
                reduce_out<LB, RT>(o, vb, S * SL, SL, c, 1, 1);
                __syncwarp();
            }
        }(),
        ...);
}

// The component groups of one batch: sets of o.parts consecutive groups, dealt
// out to the block's warps; each lane set takes one group of a set.  When one
// set holds all of them, the warps share the slices of the second transform
// instead (each forms W): of the latency of a short batch, which is all that a
// plan of a few quartets waits for, that is a third with d shells.
template <int LA, int LB, typename RT, typename EP>
__device__ __forceinline__ void transforms(const Out& o, const RT* R, RT* vb, const int* hsum, const int* kh,
                                           const int2* kb, const EP* Ek, const EP* Eb, bool ket_real, bool bra_real,
                                           int warp) {
    constexpr int NH = hc(LA + LB), NAB = nc(LA) * nc(LB), CG = group_of(NAB);
    const RT* col = R + (o.lane & (o.width - 1));
    const int set = o.lane / o.width;
    constexpr int NS = NAB / slice_of(NAB);
    // (FP32 transforms are short beside the rest of a batch)
    constexpr bool SHARED = NS > 1 && !std::is_same_v<RT, float2>;
    const bool share = SHARED && o.cend - o.cbegin <= o.parts * CG;
    for (int c1 = o.cbegin + (share ? 0 : warp * o.parts * CG); c1 < o.cend; c1 += kWarps * o.parts * CG) {
        const int cg = min(CG, o.cend - c1);
        for (int u = 0; u < cg; ++u) {
            // (a set beyond the last component repeats it; it is not added)
            const int2 box = kb[min(c1 + set * CG + u, o.cend - 1)];
            RT W[NH];
            if constexpr (std::is_same_v<RT, double>) {
                ket<NH, double, RT>(W, col, Ek + box.x, kh + box.x, box.y, hsum);
            } else if constexpr (std::is_same_v<RT, double2>) {
                if (ket_real)
                    ket<NH, double, RT>(W, col, Ek + box.x, kh + box.x, box.y, hsum);
                else
                    ket<NH, double2, RT>(W, col, Ek + box.x, kh + box.x, box.y, hsum);
            } else {
                ket<NH, float2, RT>(W, col, Ek + box.x, kh + box.x, box.y, hsum);
            }
            slices<LA, LB, RT>(o, W, vb + u * NAB * 33, Eb, bra_real, c1, SHARED && share ? warp : -1,
                               std::make_integer_sequence<int, NS>{});
        }
        if constexpr (CG > 1) {
            __syncwarp();
            reduce_out<LB, RT>(o, vb, 0, NAB, c1, cg, CG);
            __syncwarp();
        }
    }
}

// 2^e as a double (|e| <= 1000)
__device__ __forceinline__ double pow2(int e) { return __hiloint2double((e + 1023) << 20, 0); }

// FP32 seeds of a lane, scaled by a power of two.  Asymptotic sector (T and
// X'.X' formed in FP64, then rounded): F_0 = sqrt(pi) / (2 sqrt T) and
// S_{n+1} = -(2n + 1) S_n / X'.X'.  Elsewhere, and where |C| is not between 1e-30
// and 1e30, FP64 Boys values and seeds, which are then rounded.  seed32[0 .. L];
// `e_lane`: a binary exponent that bounds the seeds.  used: the lane's entry is
// evaluated here (C is zero otherwise).
struct Seeds32 {
    float2 F0, iXX;
    bool asymptotic;
    int e_lane;
};
__device__ __forceinline__ Seeds32 seeds32_begin(double2 XX64, double tre, double tim, double2 C, bool used, int L) {
    Seeds32 s{};
    s.e_lane = -1000;
    const float2 XX = make_float2((float)XX64.x, (float)XX64.y);
    const float tr = (float)tre, ti = (float)tim;
    const float r2 = fmaf(tr, tr, ti * ti);
    s.asymptotic = tr >= 2.0f * L + 24.0f && fabsf(ti) <= 0.5f * tr && (r2 <= 160.0f * 160.0f || tr >= 2.0f * L + 60.0f);
    if (!s.asymptotic) return s;
    const float ir = rsqrtf(r2);
    const float sq = sqrtf(0.5f * (r2 * ir + tr));
    const float k0 = 0.886226925452758f * ir;  // sqrt(pi) / 2 / |T|
    s.F0 = make_float2(k0 * sq, -k0 * (0.5f * ti / sq));
    const float m2 = fmaf(XX.x, XX.x, XX.y * XX.y);
    const float ixx = rsqrtf(m2);
    s.iXX = make_float2(XX.x * ixx * ixx, -XX.y * ixx * ixx);
    float gm = 1.0f, gmax = 1.0f;
    for (int n = 0; n < L; ++n) {
        gm *= (2.0f * n + 1.0f) * ixx;
        gmax = fmaxf(gmax, gm);
    }
    const int ec = max((__double2hiint(C.x) >> 20) & 0x7ff, (__double2hiint(C.y) >> 20) & 0x7ff);
    const int ef = (__float_as_int(fmaxf(fabsf(s.F0.x), fabsf(s.F0.y))) >> 23) & 0xff;
    const int eg = (__float_as_int(gmax) >> 23) & 0xff;
    if (used && (ec < 1023 - 99 || ec > 1023 + 99 || eg == 0xff)) s.asymptotic = false;
    if (ec > 0 && ec < 0x7ff && ef > 0 && ef < 0xff && eg < 0xff) s.e_lane = (ec - 1023) + (ef - 127) + (eg - 127) + 2;
    if (!s.asymptotic) s.e_lane = -1000;
    return s;
}

// The entries of a stream that FP32 leaves to FP64, in stream order and up to 32
// at a time, of tasks of one kind (see Stream): they are few among the stream's,
// so they wait in a queue until there are 32, the kind changes or the stream ends.
struct WideEntries {
    int waiting = 0, kind = 0;  // queued entries and their kind
    unsigned held = 0;          // lanes whose entry of the last batch has yet to be queued
    int htask = 0;
    int2 hpq = make_int2(0, 0);
    bool done = false;

    __device__ __forceinline__ int next(Stream<false>& stream, int4* queue, int lane, int L, int& task, int2& pq,
                                        int& batch_kind) {
        const PairData& pp = stream.d.pairs;
        for (;;) {
            if (held && (waiting == 0 || kind == stream.batch_kind)) {
                if (held >> lane & 1)
                    queue[waiting + __popc(held & ((1u << lane) - 1u))] = make_int4(htask, hpq.x, hpq.y, 0);
                waiting += __popc(held);
                kind = stream.batch_kind;
                held = 0;
                __syncwarp();
            }
            if (waiting >= 32 || (waiting > 0 && (held || done))) {
                const int nb = min(waiting, 32);
                const int4 e = queue[min(lane, nb - 1)], rest = queue[32 + lane];
                __syncwarp();
                if (lane < waiting - nb) queue[lane] = rest;
                __syncwarp();
                waiting -= nb;
                task = e.x;
                pq = make_int2(e.y, e.z);
                batch_kind = kind;
                return nb;
            }
            if (done) return 0;
            int rank;
            const int n = stream.next(lane, htask, rank, hpq);
            done = n == 0;
            bool wide = false;
            if (lane < n) {
                const Task* tg = stream.qc.tasks + htask;
                const int op = pp.order[tg->pab + hpq.x], oq = pp.order[tg->pcd + hpq.y];
                wide = stream.qc.swap ? seeds_exceed_fp32(pp, oq, op, L) : seeds_exceed_fp32(pp, op, oq, L);
            }
            held = __ballot_sync(0xffffffffu, wide);
        }
    }
};

// The classes of one launch: all have the same template pair; block b works on
// class c with first[c] <= b < first[c + 1], on unit (b - first[c]) / nchunk and
// that unit's share (b - first[c]) % nchunk of the components.
constexpr int kMaxClasses = 24;
struct ClassList {
    int n;
    int first[kMaxClasses + 1];
    QuartetClass cls[kMaxClasses];
};

// Unit `unit` of a class; share_of: which of the nchunk blocks that share it;
// queue: 64 entries of shared memory (kDenseWide, where `unit` is a task in
// classes without unit arrays).
template <int LA, int LB, DenseMode MODE>
__device__ __forceinline__ void dense_block(const EriDev& d, const QuartetClass& qc, int unit, int share_of,
                                            int4* queue = nullptr) {
    constexpr bool F32 = MODE == kDenseF32, WIDE = MODE == kDenseWide;
    constexpr int NH = hc(LA + LB), NHP = (NH + 3) / 4 * 4;
    constexpr int NAB = nc(LA) * nc(LB), NCB = nc(LB), CG = group_of(NAB);
    extern __shared__ double2 dsm[];
    char* base = reinterpret_cast<char*>(dsm);
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int L = qc.L;
    const int ncd = qc.ket.nab, ndd = ncart(qc.ket.lb), ncdh = herm_count(qc.ket.Lab);
    const int word = F32 || d.all_real ? 8 : 16;
    const Layout lay = layout(NH, NAB, ncdh, qc.ket.Etot, ncd, L, word);
    int* hsum = reinterpret_cast<int*>(base + lay.hsum);
    int* kh = reinterpret_cast<int*>(base + lay.kh);
    int2* kb = reinterpret_cast<int2*>(base + lay.kb);
    char* R = base + lay.R;
    char* vb = base + lay.v + warp * rows_of(NAB) * 33 * word;
    char* seeds = base + lay.seed;
    long long* s_eb = reinterpret_cast<long long*>(base + lay.eb);
    long long* s_ek = reinterpret_cast<long long*>(base + lay.ek);
    long long* seg_off = reinterpret_cast<long long*>(base + lay.seg_off);
    int4* seg_st = reinterpret_cast<int4*>(base + lay.seg_st);
    int* s_shift = reinterpret_cast<int*>(base + lay.shift);
    int* seg_lane = reinterpret_cast<int*>(base + lay.seg_lane);
    int* info = reinterpret_cast<int*>(base + lay.info);  // entries, segments, real sides
    // (set by the FP32 launch, which follows the FP64 one)
    if (MODE == kDenseF64 && qc.wide && unit == 0 && share_of == 0 && threadIdx.x < kWideWords) qc.wide[threadIdx.x] = 0;
    // the unit's tasks (entries past the last unit lie beyond the class)
    const int* start = MODE == kDenseF64 ? qc.unit_start : qc.unit_start32;
    int t0, t1;
    if (start) {
        t0 = start[unit] & 0x7fffffff;
        t1 = min(start[unit + 1] & 0x7fffffff, qc.ntask);
    } else if (WIDE) {
        t0 = unit;
        t1 = unit + 1;
    } else {
        __shared__ int bounds[2];
        __shared__ long long sums[kWarps];
        cut_units<32 * kWarps>(d, qc, MODE == kDenseF64 ? 0 : 1, unit, 1, MODE == kDenseF64 && share_of == 0, bounds,
                               sums);
        t0 = bounds[0];
        t1 = bounds[1];
    }
    if (t0 >= t1) return;
    // class tables: table row (in columns of 32) of K + K' by K', the other
    // side's box entries (first row of K' in hsum, sign (-1)^{|K'|} in bit 31)
    // and boxes
    for (int i = threadIdx.x; i < ncdh * NHP; i += 32 * kWarps) {
        const int Kp = i / NHP, K = i - Kp * NHP;
        int row = 0;
        if (K < NH) {
            const uint32_t a = d.herm_xyz[K], b = d.herm_xyz[Kp];
            row = herm_index((a & 255) + (b & 255), ((a >> 8) & 255) + ((b >> 8) & 255),
                             ((a >> 16) & 255) + ((b >> 16) & 255));
        }
        hsum[i] = row * 32;
    }
    for (int i = threadIdx.x; i < qc.ket.Etot; i += 32 * kWarps) {
        const uint32_t ke = qc.ket.ent[i];
        const int k = ke & 255, l = (ke >> 8) & 255, m = (ke >> 16) & 255;
        kh[i] = herm_index(k, l, m) * NHP | (int)((uint32_t)((k + l + m) & 1) << 31);
    }
    for (int i = threadIdx.x; i < ncd; i += 32 * kWarps) {
        const int bd = qc.ket.boxdim[i];
        kb[i] = make_int2(qc.ket.boxoff[i], (bd & 255) * ((bd >> 8) & 255) * ((bd >> 16) & 255));
    }
    const PairData& pp = d.pairs;
    auto strides = [&](const Task* t) {
        return make_int4(t->st[qc.axis & 3], t->st[(qc.axis >> 2) & 3], t->st[(qc.axis >> 4) & 3],
                         t->st[(qc.axis >> 6) & 3]);
    };
    // component groups of this block (of nchunk that share the unit)
    const int groups = (ncd + CG - 1) / CG, share = (groups + qc.nchunk - 1) / qc.nchunk * CG;
    const int cbegin = share_of * share, cend = min(ncd, cbegin + share);
    const int2* plan = d.rec_plan + d.rec_plan_off[L];
    const bool leader = warp == (int)(blockIdx.x % kWarps);
    unsigned count = 0;
    Stream<F32> stream(d, qc, t0, t1, MODE == kDenseF64 ? fmaxf(d.skip_cut, d.fp32_cut) : d.skip_cut,
                       MODE == kDenseF64 ? 3.4e38f : d.fp32_cut, MODE == kDenseF64 ? qc.unit_count : qc.unit_count32,
                       reinterpret_cast<Walk*>(base + lay.walk));
    WideEntries wide;
    bool skipped = false;  // FP32: the lane met an entry left to FP64
    __syncthreads();
    for (;;) {
        if (leader) {
            int task, rank = 0, kind;
            int2 pq;
            int nb;
            if constexpr (WIDE) {
                nb = wide.next(stream, queue, lane, L, task, pq, kind);
            } else {
                nb = stream.next(lane, task, rank, pq);
                kind = stream.batch_kind;
            }
            if (nb > 0) {
                // the lanes past a short batch repeat its last entry with a zero prefactor
                const bool active = lane < nb;
                task = __shfl_sync(0xffffffffu, task, active ? lane : nb - 1);
                rank = __shfl_sync(0xffffffffu, rank, active ? lane : nb - 1);
                pq.x = __shfl_sync(0xffffffffu, pq.x, active ? lane : nb - 1);
                pq.y = __shfl_sync(0xffffffffu, pq.y, active ? lane : nb - 1);
                const Task* tg = qc.tasks + task;
                const int op = pp.order[tg->pab + pq.x], oq = pp.order[tg->pcd + pq.y];
                const int ip = qc.swap ? oq : op, iq = qc.swap ? op : oq;
                const int tp = __shfl_up_sync(0xffffffffu, task, 1);
                const bool head = active && (lane == 0 || tp != task);
                const unsigned heads = __ballot_sync(0xffffffffu, head);
                const int nseg = __popc(heads);
                if (head) {
                    const int s = __popc(heads & ((1u << lane) - 1u));
                    seg_off[s] = tg->out_off;
                    seg_st[s] = strides(tg);
                    seg_lane[s] = lane | (MODE == kDenseF64 && rank == 0 ? kStore : 0) |
                                  (WIDE ? kSingle : (stream.run == 32 ? kLongRuns : 0));
                }
                const double pi0 = pp.Pi[3 * ip], pi1 = pp.Pi[3 * ip + 1], pi2 = pp.Pi[3 * ip + 2];
                const double qi0 = pp.Pi[3 * iq], qi1 = pp.Pi[3 * iq + 1], qi2 = pp.Pi[3 * iq + 2];
                const bool bra_real = kind & 1, ket_real = kind & 2;
                bool mine = active;
                if constexpr (F32) {
                    if (L >= kWideOrder && seeds_exceed_fp32(pp, ip, iq, L)) mine = false;
                    if (active && !mine) {
                        skipped = true;
                        if (!start && share_of == 0) atomicOr(&qc.wide[1 + task / 32], 1 << (task & 31));
                    }
                }
                const double p = pp.p[ip], q = pp.p[iq];
                const double rs = rsqrt(p + q);
                const double x0 = pp.Pr[3 * ip] - pp.Pr[3 * iq], x1 = pp.Pr[3 * ip + 1] - pp.Pr[3 * iq + 1],
                             x2 = pp.Pr[3 * ip + 2] - pp.Pr[3 * iq + 2];
                s_eb[lane] = pp.Eoff[ip];
                s_ek[lane] = pp.Eoff[iq];
                if (lane == 0) {
                    seg_lane[nseg] = nb;
                    info[0] = nb;
                    info[1] = nseg;
                    info[2] = kind;
                }
                count += mine && share_of == 0;
                if (!F32 && bra_real && ket_real) {
                    const double rho = p * q * rs * rs;
                    const double t = rho * fma(x0, x0, fma(x1, x1, x2 * x2));
                    double Sh[kMaxSeeds];
                    double e0;
                    double C = active ? pp.F[ip].x * pp.F[iq].x * rs : 0.0;
                    if (const int rc = boys_eval_real(t, L, d.boys, Sh, e0)) {
                        report(d.status, rc, task, L, t, 0.0);
                        C = e0 = 0.0;
                        for (int n = 0; n <= L; ++n) Sh[n] = 0.0;
                    }
                    C *= e0;
                    const double m2r = -2.0 * rho;
                    for (int n = 0; n <= L; ++n) {
                        Sh[n] *= C;
                        C *= m2r;
                    }
                    double* sd = reinterpret_cast<double*>(seeds) + lane;
                    for (int n = 0; n <= L; ++n) sd[n * 32] = Sh[n];
                    sd[(L + 1) * 32] = x0;
                    sd[(L + 2) * 32] = x1;
                    sd[(L + 3) * 32] = x2;
                } else {
                    const double2 X[3] = {c2(x0, pi0 - qi0), c2(x1, pi1 - qi1), c2(x2, pi2 - qi2)};
                    double2 C = mine ? cscale(cmul(pp.F[ip], pp.F[iq]), rs) : c2(0.0, 0.0);
                    const double rho = p * q * rs * rs;
                    const double2 XX = c2(fma(X[0].x, X[0].x, fma(X[1].x, X[1].x, X[2].x * X[2].x)) -
                                              fma(X[0].y, X[0].y, fma(X[1].y, X[1].y, X[2].y * X[2].y)),
                                          2.0 * fma(X[0].x, X[0].y, fma(X[1].x, X[1].y, X[2].x * X[2].y)));
                    const double tre = rho * XX.x, tim = rho * XX.y;
                    float2 X32[3];
                    Seeds32 s32{};
                    if constexpr (F32) {
                        for (int k = 0; k < 3; ++k) X32[k] = make_float2((float)X[k].x, (float)X[k].y);
                        s32 = seeds32_begin(XX, tre, tim, C, mine, L);
                    }
                    double2 Sh[kMaxSeeds];
                    if (!F32 || !s32.asymptotic) {
                        double2 e0;
                        if (const int rc = boys_eval(tre, tim, L, d.boys, d.gl, Sh, e0)) {
                            report(d.status, rc, task, L, tre, tim);
                            C = e0 = c2(0.0, 0.0);
                            for (int n = 0; n <= L; ++n) Sh[n] = c2(0.0, 0.0);
                        }
                        C = cmul(C, e0);
                        const double m2r = -2.0 * rho;
                        for (int n = 0; n <= L; ++n) {
                            Sh[n] = cmul(C, Sh[n]);
                            C = cscale(C, m2r);
                            if constexpr (F32) {
                                const int ex = (__double2hiint(Sh[n].x) >> 20) & 0x7ff;
                                const int ey = (__double2hiint(Sh[n].y) >> 20) & 0x7ff;
                                const int em = max(ex, ey);
                                if (em > 0 && em < 0x7ff) s32.e_lane = max(s32.e_lane, em - 1023);
                            }
                        }
                    }
                    if constexpr (F32) {
                        // one power of two per lane: its largest seed becomes 2^60
                        const int shift = max(-900, min(900, s32.e_lane - 60));
                        s_shift[lane] = shift;
                        const double sc = pow2(-shift);
                        float2 S32[kMaxSeeds];
                        if (s32.asymptotic) {
                            S32[0] = mul(make_float2((float)(C.x * sc), (float)(C.y * sc)), s32.F0);
                            for (int n = 0; n < L; ++n) {
                                const float2 t = mul(S32[n], s32.iXX);
                                S32[n + 1] = make_float2(-(2.0f * n + 1.0f) * t.x, -(2.0f * n + 1.0f) * t.y);
                            }
                        } else {
                            for (int n = 0; n <= L; ++n)
                                S32[n] = make_float2((float)(Sh[n].x * sc), (float)(Sh[n].y * sc));
                        }
                        float2* sd = reinterpret_cast<float2*>(seeds) + lane;
                        for (int n = 0; n <= L; ++n) sd[n * 32] = S32[n];
                        for (int k = 0; k < 3; ++k) sd[(L + 1 + k) * 32] = X32[k];
                    } else {
                        double2* sd = reinterpret_cast<double2*>(seeds) + lane;
                        for (int n = 0; n <= L; ++n) sd[n * 32] = Sh[n];
                        for (int k = 0; k < 3; ++k) sd[(L + 1 + k) * 32] = X[k];
                    }
                }
            } else if (lane == 0) {
                info[0] = 0;
            }
        }
        __syncthreads();
        if (info[0] == 0) break;
        const bool bra_real = info[2] & 1, ket_real = info[2] & 2;
        // a batch of at most 16 entries is repeated over the lanes, and the
        // sets of lanes share the recurrence and the components
        int width = 32;
        while (width > 1 && info[0] <= width / 2) width /= 2;
        const Out o{d.out, seg_off, seg_st,  s_shift, seg_lane,   info[1],
                    cbegin, cend,  ndd,     lane,    width,      32 / width, !qc.swap};
        const int ent = lane & (width - 1), part = warp * o.parts + lane / width, parts = kWarps * o.parts;
        if constexpr (F32) {
            recurrence<float2>(plan, L, reinterpret_cast<const float2*>(seeds) + ent,
                               reinterpret_cast<float2*>(R) + ent, part, parts);
            transforms<LA, LB, float2>(o, reinterpret_cast<const float2*>(R), reinterpret_cast<float2*>(vb), hsum, kh,
                                       kb, pp.Epool32 + s_ek[ent], pp.Epool32 + s_eb[ent], false, false, warp);
        } else {
            const double2 *Ek = pp.Epool + s_ek[ent], *Eb = pp.Epool + s_eb[ent];
            if (bra_real && ket_real) {
                recurrence<double>(plan, L, reinterpret_cast<const double*>(seeds) + ent,
                                   reinterpret_cast<double*>(R) + ent, part, parts);
                transforms<LA, LB, double>(o, reinterpret_cast<const double*>(R), reinterpret_cast<double*>(vb), hsum,
                                           kh, kb, Ek, Eb, true, true, warp);
            } else {
                recurrence<double2>(plan, L, reinterpret_cast<const double2*>(seeds) + ent,
                                    reinterpret_cast<double2*>(R) + ent, part, parts);
                transforms<LA, LB, double2>(o, reinterpret_cast<const double2*>(R), reinterpret_cast<double2*>(vb),
                                            hsum, kh, kb, Ek, Eb, ket_real, bra_real, warp);
            }
        }
        __syncthreads();  // the next batch overwrites the table
    }
    if constexpr (F32) {
        if (leader && __any_sync(0xffffffffu, skipped) && lane == 0) {
            *qc.wide = 1;
            if (start) const_cast<int*>(start)[unit] = t0 | (int)0x80000000;
        }
    }
    if (qc.counters && leader && share_of == 0) {
        const unsigned a = __reduce_add_sync(0xffffffffu, count);
        if (lane == 0 && a) atomicAdd(&qc.counters[F32 ? 1 : 0], (unsigned long long)a);
    }
}

template <int LA, int LB, DenseMode MODE>
__global__ void __launch_bounds__(32 * kWarps) dense_kernel(const __grid_constant__ EriDev d,
                                                            const __grid_constant__ QuartetClass qc) {
    dense_block<LA, LB, MODE>(d, qc, blockIdx.x, blockIdx.y);
}

// (reading the class through the list costs the FP64-bound plans 1.5%, so a
// class with a launch of its own has the kernel above)
template <int LA, int LB, DenseMode MODE>
__global__ void __launch_bounds__(32 * kWarps) dense_list_kernel(const __grid_constant__ EriDev d,
                                                                 const __grid_constant__ ClassList list) {
    int ci = 0;
    while (ci + 1 < list.n && (int)blockIdx.x >= list.first[ci + 1]) ++ci;
    const int b = (int)blockIdx.x - list.first[ci], nchunk = list.cls[ci].nchunk;
    dense_block<LA, LB, MODE>(d, list.cls[ci], b / nchunk, b % nchunk);
}

constexpr int kMaxSmem = 200 * 1024;

// Launches of the template pair LA * 4 + LB, one translation unit for each
// pair of (one class or a list, FP64 or FP32).
cudaError_t run_one_f64(int pair, const EriDev& d, const QuartetClass& qc, int smem, cudaStream_t s);
cudaError_t run_one_f32(int pair, const EriDev& d, const QuartetClass& qc, int smem, cudaStream_t s);
cudaError_t run_list_f64(int pair, const EriDev& d, const ClassList& list, int smem, cudaStream_t s);
cudaError_t run_list_f32(int pair, const EriDev& d, const ClassList& list, int smem, cudaStream_t s);

template <class Arg>
cudaError_t launch_with_smem(void (*kernel)(EriDev, Arg), PerDevice& limit, dim3 grid, int smem, cudaStream_t s,
                             const EriDev& d, const Arg& arg) {
    int device = 0;
    cudaError_t e = cudaGetDevice(&device);
    if (e != cudaSuccess) return e;
    if (limit.needs(device, kMaxSmem)) {
        e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kMaxSmem);
        if (e != cudaSuccess) return e;
        limit.done(device, kMaxSmem);
    }
    kernel<<<grid, 32 * kWarps, smem, s>>>(d, arg);
    return cudaGetLastError();
}

#define GX_DENSE_PAIRS \
    GX_CASE(0, 0)      \
    GX_CASE(0, 1)      \
    GX_CASE(0, 2)      \
    GX_CASE(0, 3)      \
    GX_CASE(1, 1)      \
    GX_CASE(1, 2)      \
    GX_CASE(2, 1)      \
    GX_CASE(1, 3)      \
    GX_CASE(3, 1)      \
    GX_CASE(2, 2)

}  // namespace dense
}  // namespace gx
