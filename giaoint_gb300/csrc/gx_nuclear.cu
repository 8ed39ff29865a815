// GIAO nuclear-attraction matrix V[mu][nu] = sum_C -Z_C <mu| 1/|r - C| |nu>
// (src/nuclear.cpp:27-170, 207-330 of the reference).
//
// Same formulation as the electron-repulsion kernels: the London phase lives
// in the complex Hermite expansion E~ of the primitive pair (K1 records), so
// per (primitive pair, nucleus)
//   V = -Z (2 pi / p) K_ab sum_K E~_K R^_K(X' = P' - C),
// with R^ the three-index MD table of the complex separation seeded by
// (-2p)^n F_n(p X'.X').  With the pair prefactor F = sqrt(2 pi^{5/2}) K_ab / p
// of the K1 record this is -Z F (2 pi / sqrt(2 pi^{5/2})) sum_K E~_K R^_K.
//
// Bound by FP64 warp instructions (one per 64 cycles and SM sub-partition,
// whatever the number of active lanes).  nuclear_dense_kernel: a lane holds one
// (primitive pair, nucleus) of a shell pair, so the Boys function and the
// recurrence (a table column per lane in shared memory, 33 columns: free of
// bank conflicts both ways) run on full warps; E~ does not depend on the nucleus,
// so the columns of one primitive pair are summed row by row before the boxes
// are contracted, with a lane per component pair.  V is Hermitian: one
// orientation of every shell pair is evaluated and written twice.  Pairs with
// q = 0 run in real arithmetic.  216 functions and 12 nuclei: 3.4 -> 0.2 ms
// against nuclear_kernel, which evaluates one (primitive pair, nucleus) of an
// ordered shell pair at a time with the Boys function on lane 0 and the
// recurrence level by level across the lanes; it remains for pairs with
// la + lb > 8, whose columns do not fit.
#include <algorithm>
#include <type_traits>

#include "gx_internal.h"

namespace gx {

namespace {

constexpr int kDenseOrder = 8;

// (value types of the dense kernel: complex, or real for pairs with q = 0)
__device__ __forceinline__ double2 nmul(double2 a, double2 b) { return cmul(a, b); }
__device__ __forceinline__ double nmul(double a, double b) { return a * b; }
__device__ __forceinline__ double2 nmacr(double2 c, double s, double2 a) { return cmacr(c, s, a); }
__device__ __forceinline__ double nmacr(double c, double s, double a) { return fma(s, a, c); }
__device__ __forceinline__ double2 nadd(double2 a, double2 b) { return cadd(a, b); }
__device__ __forceinline__ double nadd(double a, double b) { return a + b; }

// In-place descending-level recurrence of one lane's column (33 columns), the
// entries of a level from the highest index down: they only read lower degrees.
template <typename T>
__device__ __forceinline__ void column_rec(int L, const T* seed, const T* X, T* col,
                                           const uint32_t* __restrict__ herm_xyz) {
    col[0] = seed[L];
    for (int n = L - 1; n >= 0; --n) {
        for (int e = herm_count(L - n) - 1; e >= 1; --e) {
            const uint32_t kx = __ldg(&herm_xyz[e]);
            const int k = kx & 255, l = (kx >> 8) & 255, m = (kx >> 16) & 255;
            const int axis = k > 0 ? 0 : (l > 0 ? 1 : 2), pw = k > 0 ? k : (l > 0 ? l : m);
            const int dk = axis == 0, dl = axis == 1, dm = axis == 2;
            T v = nmul(axis == 0 ? X[0] : (axis == 1 ? X[1] : X[2]), col[33 * herm_index(k - dk, l - dl, m - dm)]);
            if (pw > 1) v = nmacr(v, c_dev.ints[pw - 1], col[33 * herm_index(k - 2 * dk, l - 2 * dl, m - 2 * dm)]);
            col[33 * e] = v;
        }
        col[0] = seed[n];
    }
}

struct NuclearArgs {
    BasisDev bs;
    PairData pp;
    BoysTable boys;
    const GLRules* gl;
    const uint32_t* herm_xyz;
    const PairClassDev* classes;
    const int* pp_class;
    int nnuc, group;  // nuclei; primitive pairs at a time (their entries are counted in 32 bits)
    const double* charge;
    const double* center;
    const long long* seg_ao;
    long long n;
    double2* out;
    DevStatus* status;
};

// The block of shell pair (sa, sb) into acc[nab] (shared, cleared).
template <typename T>
__device__ __forceinline__ void nuclear_block(const NuclearArgs& a, int sa, int sb, const PairClassDev& pc, T* R,
                                              double2* acc, int lane) {
    constexpr bool REAL = std::is_same_v<T, double>;
    const BasisDev& bs = a.bs;
    const PairData& pp = a.pp;
    const int L = pc.la + pc.lb, NL = herm_count(L);
    const int pairs = bs.nprim[sa] * bs.nprim[sb];
    const double scale = -6.283185307179586 / 5.914967172795613;  // -2 pi / sqrt(2 pi^{5/2})
    for (int g0 = 0; g0 < pairs; g0 += a.group) {
        const int p0 = bs.sp_off[sa * bs.ns + sb] + g0, total = min(a.group, pairs - g0) * a.nnuc;
        for (int first = 0; first < total; first += 32) {
            const int nb = min(32, total - first);
            const int it = first + min(lane, nb - 1);
            const int ip = p0 + it / a.nnuc, c = it - (it / a.nnuc) * a.nnuc;
            const double p = pp.p[ip];
            double x[3];
            for (int k = 0; k < 3; ++k) x[k] = pp.Pr[3 * ip + k] - a.center[3 * c + k];
            const double z = a.charge[c] * scale;
            if constexpr (REAL) {
                const double t = p * (x[0] * x[0] + x[1] * x[1] + x[2] * x[2]);
                double Sh[kDenseOrder + 1], e0;
                if (const int rc = boys_eval_real(t, L, a.boys, Sh, e0)) {
                    report(a.status, rc, blockIdx.x, L, t, 0.0);
                    e0 = 0.0;
                    for (int k = 0; k <= L; ++k) Sh[k] = 0.0;
                }
                double s = e0 * z;
                for (int k = 0; k <= L; ++k) {
                    Sh[k] *= s;
                    s *= -2.0 * p;
                }
                column_rec<double>(L, Sh, x, R + lane, a.herm_xyz);
            } else {
                const double2 X[3] = {c2(x[0], pp.Pi[3 * ip]), c2(x[1], pp.Pi[3 * ip + 1]), c2(x[2], pp.Pi[3 * ip + 2])};
                const double tre = p * (X[0].x * X[0].x + X[1].x * X[1].x + X[2].x * X[2].x -
                                        (X[0].y * X[0].y + X[1].y * X[1].y + X[2].y * X[2].y));
                const double tim = 2.0 * p * (X[0].x * X[0].y + X[1].x * X[1].y + X[2].x * X[2].y);
                double2 Sh[kDenseOrder + 1], e0;
                if (const int rc = boys_eval(tre, tim, L, a.boys, a.gl, Sh, e0)) {
                    report(a.status, rc, blockIdx.x, L, tre, tim);
                    e0 = c2(0.0, 0.0);
                    for (int k = 0; k <= L; ++k) Sh[k] = c2(0.0, 0.0);
                }
                double2 s = cscale(e0, z);
                for (int k = 0; k <= L; ++k) {
                    Sh[k] = cmul(s, Sh[k]);
                    s = cscale(s, -2.0 * p);
                }
                column_rec<double2>(L, Sh, X, R + lane, a.herm_xyz);
            }
            __syncwarp();
            // rows summed over the nuclei of each primitive pair; the sum of the
            // batch's j-th pair goes to column j, which has been read by then
            const int k0 = first / a.nnuc, k1 = (first + nb - 1) / a.nnuc;
            for (int row = lane; row < NL; row += 32) {
                T* r = R + 33 * row;
                int l = 0;
                for (int k = k0; k <= k1; ++k) {
                    const int end = min(nb, (k + 1) * a.nnuc - first);
                    T sum = r[l++];
                    for (; l < end; ++l) sum = nadd(sum, r[l]);
                    r[k - k0] = sum;
                }
            }
            __syncwarp();
            for (int ab = lane; ab < pc.nab; ab += 32) {
                const int bo = pc.boxoff[ab], bd = pc.boxdim[ab];
                const int nbox = (bd & 255) * ((bd >> 8) & 255) * ((bd >> 16) & 255);
                double2 sum = acc[ab];
                for (int k = k0; k <= k1; ++k) {
                    const double2* E = pp.Epool + pp.Eoff[p0 + k] + bo;
                    const double2 F = pp.F[p0 + k];
                    T v{};
                    for (int e = 0; e < nbox; ++e) {
                        const uint32_t ke = pc.ent[bo + e];
                        const T rv = R[33 * herm_index(ke & 255, (ke >> 8) & 255, (ke >> 16) & 255) + (k - k0)];
                        if constexpr (REAL)
                            v = fma(__ldg(&E[e].x), rv, v);
                        else
                            v = cmac(v, __ldg(&E[e]), rv);
                    }
                    if constexpr (REAL)
                        sum.x = fma(F.x, v, sum.x);
                    else
                        sum = cmac(sum, F, v);
                }
                acc[ab] = sum;
            }
            __syncwarp();  // the next batch overwrites the table
        }
    }
}

// One warp per shell pair (sa <= sb) with lo < la + lb <= hi.
__global__ void __launch_bounds__(32) nuclear_dense_kernel(NuclearArgs a, int lo, int hi) {
    extern __shared__ double2 ndm[];
    const int lane = threadIdx.x;
    const int sa = blockIdx.x / a.bs.ns, sb = blockIdx.x - sa * a.bs.ns;
    if (sa > sb) return;
    const int la = a.bs.l[sa], lb = a.bs.l[sb], L = la + lb;
    if (L <= lo || L > hi) return;
    const int p0 = a.bs.sp_off[sa * a.bs.ns + sb];
    const PairClassDev pc = a.classes[a.pp_class[p0]];
    double2* R = ndm;
    double2* acc = R + 33 * herm_count(L);
    for (int i = lane; i < pc.nab; i += 32) acc[i] = c2(0.0, 0.0);
    __syncwarp();
    if (a.pp.Pi[3 * p0] == 0.0 && a.pp.Pi[3 * p0 + 1] == 0.0 && a.pp.Pi[3 * p0 + 2] == 0.0)
        nuclear_block<double>(a, sa, sb, pc, reinterpret_cast<double*>(R), acc, lane);
    else
        nuclear_block<double2>(a, sa, sb, pc, R, acc, lane);
    const int ncb = ncart(lb);
    for (int ab = lane; ab < pc.nab; ab += 32) {
        const long long i = a.seg_ao[sa] + ab / ncb, j = a.seg_ao[sb] + ab % ncb;
        a.out[i * a.n + j] = acc[ab];
        if (sa != sb) a.out[j * a.n + i] = cconj(acc[ab]);
    }
}

// Level-parallel recurrence between columns 0 and 1 (stride 2) of R, level
// 0 ending in column 0.
__device__ void nuclear_rec(int L, const double2* seed, const double2* X, double2* R, const uint32_t* herm_xyz,
                            int lane) {
    int cur = (L % 2 == 0) ? 0 : 1;
    if (lane == 0) R[cur] = seed[L];
    __syncwarp();
    for (int n = L - 1; n >= 0; --n) {
        const int nxt = cur ^ 1;
        const int cnt = herm_count(L - n);
        for (int e = lane; e < cnt; e += 32) {
            double2 v;
            if (e == 0) {
                v = seed[n];
            } else {
                const uint32_t kx = __ldg(&herm_xyz[e]);
                const int k = kx & 255, l = (kx >> 8) & 255, m = (kx >> 16) & 255;
                int axis, pw, i1, i2;
                if (k > 0) {
                    axis = 0, pw = k, i1 = herm_index(k - 1, l, m), i2 = k > 1 ? herm_index(k - 2, l, m) : 0;
                } else if (l > 0) {
                    axis = 1, pw = l, i1 = herm_index(0, l - 1, m), i2 = l > 1 ? herm_index(0, l - 2, m) : 0;
                } else {
                    axis = 2, pw = m, i1 = herm_index(0, 0, m - 1), i2 = m > 1 ? herm_index(0, 0, m - 2) : 0;
                }
                v = cmul(X[axis], R[2 * i1 + cur]);
                if (pw > 1) v = cmacr(v, (double)(pw - 1), R[2 * i2 + cur]);
            }
            R[2 * e + nxt] = v;
        }
        __syncwarp();
        cur = nxt;
    }
}

__global__ void __launch_bounds__(32) nuclear_kernel(BasisDev bs, PairData pp, BoysTable boys, const GLRules* gl,
                                                     const uint32_t* herm_xyz, const PairClassDev* classes,
                                                     const int* pp_class, int nnuc, const double* charge,
                                                     const double* center, const long long* seg_ao, long long n,
                                                     double2* out, DevStatus* status) {
    extern __shared__ double2 nsm[];
    const int lane = threadIdx.x;
    const int ns = bs.ns;
    const int sa = blockIdx.x / ns, sb = blockIdx.x - (blockIdx.x / ns) * ns;
    const int la = bs.l[sa], lb = bs.l[sb];
    const int L = la + lb;
    if (L <= kDenseOrder) return;
    const int nab = ncart(la) * ncart(lb);
    const int NL = herm_count(L);
    double2* R = nsm;                 // 2 columns x NL
    double2* seed = R + 2 * NL;       // L + 1 seeds, then X'[3]
    double2* acc = seed + L + 4;      // nab accumulators
    for (int i = lane; i < nab; i += 32) acc[i] = c2(0.0, 0.0);
    const int p0 = bs.sp_off[sa * ns + sb];
    const int kab = bs.nprim[sa] * bs.nprim[sb];
    const PairClassDev pc = classes[pp_class[p0]];
    const double scale = 6.283185307179586 / 5.914967172795613;  // 2 pi / sqrt(2 pi^{5/2})
    for (int it = 0; it < kab * nnuc; ++it) {
        const int ip = p0 + it / nnuc, c = it - (it / nnuc) * nnuc;
        const double p = pp.p[ip];
        if (lane == 0) {
            double2 X[3];
            for (int x = 0; x < 3; ++x) X[x] = c2(pp.Pr[3 * ip + x] - center[3 * c + x], pp.Pi[3 * ip + x]);
            const double tre = p * (X[0].x * X[0].x + X[1].x * X[1].x + X[2].x * X[2].x -
                                    (X[0].y * X[0].y + X[1].y * X[1].y + X[2].y * X[2].y));
            const double tim = 2.0 * p * (X[0].x * X[0].y + X[1].x * X[1].y + X[2].x * X[2].y);
            double2 Sh[BOYS_MAX_ORDER + 1], e0;
            if (const int rc = boys_eval(tre, tim, L, boys, gl, Sh, e0)) {
                report(status, rc, blockIdx.x, L, tre, tim);
                e0 = c2(0.0, 0.0);
            }
            double2 s = e0;
            for (int k = 0; k <= L; ++k) {
                seed[k] = cmul(s, Sh[k]);
                s = cscale(s, -2.0 * p);
            }
            for (int x = 0; x < 3; ++x) seed[L + 1 + x] = X[x];
        }
        __syncwarp();
        nuclear_rec(L, seed, seed + L + 1, R, herm_xyz, lane);
        const double2 pref = cscale(pp.F[ip], -charge[c] * scale);
        const double2* E = pp.Epool + pp.Eoff[ip];
        for (int ab = lane; ab < nab; ab += 32) {
            const int bo = pc.boxoff[ab];
            const int bd = pc.boxdim[ab];
            const int nbox = (bd & 255) * ((bd >> 8) & 255) * ((bd >> 16) & 255);
            double2 v = c2(0.0, 0.0);
            for (int e = 0; e < nbox; ++e) {
                const uint32_t ke = pc.ent[bo + e];
                v = cmac(v, E[bo + e], R[2 * herm_index(ke & 255, (ke >> 8) & 255, (ke >> 16) & 255)]);
            }
            acc[ab] = cmac(acc[ab], pref, v);
        }
        __syncwarp();  // R and seed are rewritten by the next entry
    }
    const int ncb = ncart(lb);
    for (int ab = lane; ab < nab; ab += 32) {
        const int ca = ab / ncb, cb = ab - ca * ncb;
        out[(seg_ao[sa] + ca) * n + seg_ao[sb] + cb] = acc[ab];
    }
}

}  // namespace

cudaError_t launch_nuclear(const BasisDev& bs, const PairData& pp, const BoysTable& boys, const GLRules* gl,
                           const uint32_t* herm_xyz, const PairClassDev* classes, const int* pp_class, int nnuc,
                           const double* charge, const double* center, const long long* seg_ao, long long n,
                           int max_pair_L, int max_nab, double2* out, DevStatus* status, cudaStream_t s) {
    const long long blocks = (long long)bs.ns * bs.ns;
    if (blocks == 0) return cudaSuccess;
    // pairs by order, so that the low ones do not carry the shared memory of the highest
    const int group = std::max(1, (1 << 30) / std::max(1, nnuc));
    const NuclearArgs args{bs,     pp,    boys,   gl,     herm_xyz, classes, pp_class, nnuc,
                           group, charge, center, seg_ao, n,        out,     status};
    const int steps[] = {-1, 2, 4, 6, kDenseOrder};
    for (int k = 0; k < 4 && steps[k] < max_pair_L; ++k) {
        const int hi = steps[k + 1];
        const size_t smem = (size_t)(33 * herm_count(hi) + std::min(max_nab, ncart(hi / 2) * ncart(hi - hi / 2))) *
                            sizeof(double2);
        if (smem > 48 * 1024) {
            cudaError_t e = cudaFuncSetAttribute(nuclear_dense_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                 (int)smem);
            if (e != cudaSuccess) return e;
        }
        nuclear_dense_kernel<<<(unsigned)blocks, 32, smem, s>>>(args, steps[k], hi);
        cudaError_t e = cudaGetLastError();
        if (e != cudaSuccess) return e;
    }
    if (max_pair_L <= kDenseOrder) return cudaSuccess;
    const size_t smem = (size_t)(2 * herm_count(max_pair_L) + max_pair_L + 4 + max_nab) * sizeof(double2);
    if (smem > 48 * 1024) {
        cudaError_t e = cudaFuncSetAttribute(nuclear_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem);
        if (e != cudaSuccess) return e;
    }
    nuclear_kernel<<<(unsigned)blocks, 32, smem, s>>>(bs, pp, boys, gl, herm_xyz, classes, pp_class, nnuc, charge,
                                                      center, seg_ao, n, out, status);
    return cudaGetLastError();
}

}  // namespace gx
