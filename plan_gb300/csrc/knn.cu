// KNN density and densest-neighbour search with the reference's exact traversal.
//
// The reference's KNN (KNN_Search_OpenMP, src/tree.hpp:3198-3251) is not an exact k-nearest
// search: it starts from a radius given by the tree (the half width of the smallest
// ancestor of the query's leaf holding >= k/4 points), collects every point of every node
// the sphere contains or intersects (the intersect test keeps the reference's comparison of
// a squared distance against r at src/tree.hpp:3030), doubles the radius until >= k points
// were visited and keeps the k closest visited points in a heap. The visited set and, without
// distance ties, the k kept do not depend on the order of the walk: a warp per query finds them
// in FP32 with error bounds (knn_warp.cuh). Queries with ties go to a thread per query that
// reproduces the reference point for point in FP64: a count-only traversal per radius (node
// tests, no per-point work), then one collecting traversal at the final radius that feeds a heap
// with the library's sifting order. No contraction.
#include <cmath>
#include <cstdlib>
#include <type_traits>

#include "exact64.cuh"
#include "pipeline.h"
#include "tree_walk.cuh"
#include "knn_warp.cuh"

namespace plan {

namespace {

template <int KMAX>
__global__ void __launch_bounds__(128) k_knn_positions(KTree t, const double *q3, const uint32_t *list, const uint32_t *nlist, uint32_t k,
                                                       double est, uint32_t *oidx, double *odr2, unsigned *err) {
    extern __shared__ unsigned char smem[];
    double *sd = reinterpret_cast<double *>(smem);
    uint32_t *si = reinterpret_cast<uint32_t *>(sd + KMAX * blockDim.x);
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < *nlist; u += gridDim.x * blockDim.x) {
    const uint32_t i = list[u];
    SlabHeap h{sd + threadIdx.x, si + threadIdx.x, (int)blockDim.x};
    double qx = q3[3 * i], qy = q3[3 * i + 1], qz = q3[3 * i + 2];
    double r = est != 0 ? est : knn_first_radius(t, qx, qy, qz, 0xffffffffu, k, err);
    int got = knn_query(t, qx, qy, qz, r, k, h, err);
    for (int j = 0; j < (int)k; ++j) {
        oidx[(size_t)i * k + j] = j < got ? h.iget(j) : 0xffffffffu;
        odr2[(size_t)i * k + j] = j < got ? h.dget(j) : -1.0;
    }
    }
}


// ---------------------------------------------------------------- exact heap path
// Thread per query, FP64, over a list on the device: what the warp kernels hand on because two
// distances tie, which the library's heap order decides.
template <int KMAX, int SPL>
__global__ void __launch_bounds__(128) k_density_at(KTree t, const double *q3, const double *est, const uint32_t *list, const uint32_t *nlist,
                                                    uint32_t k, double four_pi_over_three, SplineCells sc, double *out, unsigned *err) {
    extern __shared__ unsigned char smem[];
    double *sd = reinterpret_cast<double *>(smem);
    uint32_t *si = reinterpret_cast<uint32_t *>(sd + KMAX * blockDim.x);
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < *nlist; u += gridDim.x * blockDim.x) {
        const uint32_t i = list[u];
        SlabHeap h{sd + threadIdx.x, si + threadIdx.x, (int)blockDim.x};
        double qx = q3[3 * i], qy = q3[3 * i + 1], qz = q3[3 * i + 2];
        double r = est[i] != 0 ? est[i] : knn_first_radius(t, qx, qy, qz, 0xffffffffu, k, err);
        int got = knn_query(t, qx, qy, qz, r, k, h, err);
        if (got != (int)k) {
            out[i] = 0.0;
        } else if constexpr (SPL) {
            // the reference passes self_id = 0: offsets are taken from tree point 0 (src/tree.hpp:4889, 4905)
            const double4_32a p0 = t.pos[0];
            out[i] = spline_density(t.pos, [&](int j) { return h.iget(j); }, (int)k, p0.x, p0.y, p0.z, sc);
        } else {
            out[i] = knn_median_density(t, h, (int)k, four_pi_over_three);
        }
    }
}

template <int KMAX, int SPL>
__global__ void __launch_bounds__(128) k_density_list(KTree t, const uint32_t *list, const uint32_t *nlist, uint32_t k, double fpo3,
                                                      SplineCells sc, double *dens, unsigned *err) {
    extern __shared__ unsigned char smem[];
    double *sd = reinterpret_cast<double *>(smem);
    uint32_t *si = reinterpret_cast<uint32_t *>(sd + KMAX * blockDim.x);
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < *nlist; u += gridDim.x * blockDim.x) {
        const uint32_t i = list[u];
        SlabHeap h{sd + threadIdx.x, si + threadIdx.x, (int)blockDim.x};
        double4_32a q = t.pos[i];
        double r = knn_first_radius(t, q.x, q.y, q.z, t.leaf_of[i], k, err);
        int got = knn_query(t, q.x, q.y, q.z, r, k, h, err);
        if (got < (int)k) {
            atomicOr(err, (unsigned)kDevErrCapacity);
            dens[i] = 0;
            continue;
        }
        if constexpr (SPL) dens[i] = spline_density(t.pos, [&](int jj) { return h.iget(jj); }, (int)k, q.x, q.y, q.z, sc);
        else dens[i] = knn_median_density(t, h, (int)k, fpo3);
    }
}

template <int KMAX>
__global__ void __launch_bounds__(128) k_densest_list(KTree t, const uint32_t *list, const uint32_t *nlist, uint32_t k, const double *dens,
                                                      uint32_t *densest, unsigned *err) {
    extern __shared__ unsigned char smem[];
    double *sd = reinterpret_cast<double *>(smem);
    uint32_t *si = reinterpret_cast<uint32_t *>(sd + KMAX * blockDim.x);
    for (uint32_t u = blockIdx.x * blockDim.x + threadIdx.x; u < *nlist; u += gridDim.x * blockDim.x) {
        const uint32_t i = list[u];
        SlabHeap h{sd + threadIdx.x, si + threadIdx.x, (int)blockDim.x};
        double4_32a q = t.pos[i];
        double r = knn_first_radius(t, q.x, q.y, q.z, t.leaf_of[i], k, err);
        int got = knn_query(t, q.x, q.y, q.z, r, k, h, err);
        uint32_t best = i;
        double bd = dens[i];
        for (int jj = 0; jj < got; ++jj) {
            uint32_t c = h.iget(jj);
            double dc = dens[c];
            if (bd < dc) { best = c; bd = dc; }
            else if (bd == dc && best > c) best = c;
        }
        densest[i] = best;
    }
}

// ---------------------------------------------------------------- warp per query
// Densities of the tree points from the FP32 keys (median kernel). The density needs, of the
// sorted k-set, the masses up to the last distance that is not beyond twice the median one
// (MedianSphericalDensityKernel, src/tree.hpp:3473-3491) and that distance itself: the point
// there and the number of masses go to at and cnt, and k_density_finish forms the density in
// FP64, a thread per point. Where the tree's masses differ and those of a query do, their sum in
// ascending order goes to dens and kMixed marks it. A query whose k-set, median cut, last point
// or order is too close to tell in FP32 is listed for the exact warp kernel.
constexpr uint32_t kMixed = 0x80000000u, kNoPoint = 0xffffffffu;

__global__ void __launch_bounds__(32 * kWkWarps) k_density_w(KTree t, FTree f, uint32_t n, uint32_t k, bool uniform, uint32_t *at, uint32_t *cnt,
                                                             double *dens, uint32_t *redo, uint32_t *nredo, unsigned *err) {
    __shared__ WkBuf s_buf[kWkWarps];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, full = 0xffffffffu;
    const uint32_t i = blockIdx.x * kWkWarps + w;
    if (i >= n) return;
    WkBuf &s = s_buf[w];
    const double4_32a p = t.pos[i];
    WkQuery q{p.x, p.y, p.z, f.phi[i], f.plo[i]};
    uint32_t m, visited, tau;
    bool ok = wk_collect(t, f, q, wk_first_radius(t, q, t.leaf_of[i], k, err), k, s, m, visited, tau, err) && visited >= k && wk_kset(s, k, m, tau, f.tol);
    uint32_t last = 0, c = 0;
    if (ok) {
        __syncwarp();
        // the median, and which members lie within twice its distance (four times its square)
        uint32_t count, med = 0;
        const uint32_t T = wk_select(s.key, k, k / 2 + 1, count);
        for (uint32_t j = lane; j < k; j += 32)
            if (s.key[j] <= T) med = max(med, s.key[j]);
        med = __reduce_max_sync(full, med);
        const float lo4 = 4.f * f_lo(__uint_as_float(med), f.tol), hi4 = 4.f * f_hi(__uint_as_float(med), f.tol);
        uint32_t far = 0, second = 0;
        bool clear = true;
        for (uint32_t j = lane; j < k; j += 32) {
            const float v = __uint_as_float(s.key[j]);
            const bool in = f_hi(v, f.tol) <= lo4;
            clear = clear && (in || f_lo(v, f.tol) > hi4);
            if (in) {
                ++c;
                second = max(second, min(far, s.key[j]));
                far = max(far, s.key[j]);
            }
        }
        c = __reduce_add_sync(full, c);
        const uint32_t top = __reduce_max_sync(full, far);
        const unsigned holders = __ballot_sync(full, far == top);
        // the last point: no other as far, within the error bound
        second = __reduce_max_sync(full, (far == top && lane == (uint32_t)(__ffs(holders) - 1)) ? second : far);
        ok = __all_sync(full, clear) && c > 0 && f_hi(__uint_as_float(second), f.tol) < f_lo(__uint_as_float(top), f.tol);
        if (c == 1) ok = __all_sync(full, clear);
        for (uint32_t j = lane; j < k; j += 32)
            if (s.key[j] == top) last = s.ix[j];
        last = __reduce_max_sync(full, last);
        if (ok && !uniform) {
            // all the summed masses the same? then k_density_finish adds them
            const double m0 = t.pos[last].w;
            bool same = true;
            for (uint32_t j = lane; j < k; j += 32)
                if (s.key[j] <= top) same = same && t.pos[s.ix[j]].w == m0;
            if (!__all_sync(full, same)) {
                // by rank, in ascending order; every neighbour in the order must be clear
                double *ms = reinterpret_cast<double *>(s.xkey);
                bool order = true;
                for (uint32_t j = lane; j < k; j += 32) {
                    const uint32_t v = s.key[j];
                    if (v > top) continue;
                    uint32_t rank = 0;
                    for (uint32_t o = 0; o < k; ++o) {
                        const uint32_t u = s.key[o];
                        rank += u < v ? 1u : 0u;
                        order = order && (o == j || u > top || f_hi(__uint_as_float(min(u, v)), f.tol) < f_lo(__uint_as_float(max(u, v)), f.tol));
                    }
                    ms[rank] = t.pos[s.ix[j]].w;
                }
                ok = __all_sync(full, order);
                __syncwarp();
                if (ok && lane == 0) {
                    double sum = 0;
                    for (int j = (int)c - 1; j >= 0; j--) sum = sum + ms[j];
                    dens[i] = sum;
                }
                c |= kMixed;
            }
        }
    }
    if (lane == 0) {
        at[i] = last;
        cnt[i] = ok ? c : 0u;
        if (!ok) redo[atomicAdd(nredo, 1u)] = i;
    }
}

__global__ void k_density_finish(const double4_32a *pos, uint32_t n, double fpo3, const uint32_t *at, const uint32_t *cnt, double *dens) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint32_t c = cnt[i];
    if (!c) return;  // listed
    const double4_32a q = pos[i], p = pos[at[i]];
    const double r2 = point_dr2(q.x, q.y, q.z, p);
    double sum = 0;
    if (c & kMixed) sum = dens[i];
    else
        for (uint32_t j = 0; j < c; ++j) sum = sum + p.w;
    dens[i] = sum / (fpo3 * cr_pow15(r2));
}

// The densest of a point's k nearest and itself (src/tree.hpp:3719-3735): the largest density,
// the smallest index among equal ones, whatever the order. Densities are positive (their bits
// order like their values). At the points below the threshold, themselves.
__device__ __forceinline__ void wk_densest(const uint32_t *ix, uint32_t k, uint32_t i, double di, const double *dens, uint32_t *densest) {
    const uint32_t lane = threadIdx.x & 31, full = 0xffffffffu;
    double bd = di;
    uint32_t best = i;
    for (uint32_t j = lane; j < k; j += 32) {
        const uint32_t c = ix[j];
        const double dc = dens[c];
        if (dbits(bd) < dbits(dc)) { best = c; bd = dc; }
        else if (dbits(bd) == dbits(dc) && best > c) best = c;
    }
    const uint32_t hi = __reduce_max_sync(full, (uint32_t)(dbits(bd) >> 32));
    const uint32_t lo = __reduce_max_sync(full, (uint32_t)(dbits(bd) >> 32) == hi ? (uint32_t)dbits(bd) : 0u);
    best = __reduce_min_sync(full, dbits(bd) == (((uint64_t)hi << 32) | lo) ? best : 0xffffffffu);
    if (lane == 0) densest[i] = best;
}

__global__ void __launch_bounds__(32 * kWkWarps) k_densest_w(KTree t, FTree f, uint32_t n, uint32_t k, double threshold, const double *dens,
                                                             uint32_t *densest, uint32_t *redo, uint32_t *nredo, unsigned *err) {
    __shared__ WkBuf s_buf[kWkWarps];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const uint32_t i = blockIdx.x * kWkWarps + w;
    if (i >= n) return;
    WkBuf &s = s_buf[w];
    const double di = dens[i];
    if (!(di >= threshold)) {  // src/tree.hpp:3719-3735
        if (lane == 0) densest[i] = i;
        return;
    }
    const double4_32a p = t.pos[i];
    WkQuery q{p.x, p.y, p.z, f.phi[i], f.plo[i]};
    uint32_t m, visited, tau;
    if (wk_collect(t, f, q, wk_first_radius(t, q, t.leaf_of[i], k, err), k, s, m, visited, tau, err) && visited >= k && wk_kset(s, k, m, tau, f.tol)) {
        __syncwarp();
        wk_densest(s.ix, k, i, di, dens, densest);
    } else if (lane == 0) {
        redo[atomicAdd(nredo, 1u)] = i;
    }
}

// The exact k-set in FP64 order, for queries at given positions (q3; est: the first radius, 0
// for the reference's own) or at the tree points of a list, counted on the device (nlist) or by
// the host. What it makes of them:
enum WkOp {
    kOpMedian,   // the median density
    kOpSpline,   // the spline density (offsets from tree point 0 at given positions: self_id = 0, as in the heap path)
    kOpDensest,  // the densest neighbour
    kOpKnn,      // indices and squared distances
};
struct WkOut {
    double *dens;             // kOpMedian, kOpSpline: the result; kOpDensest: the densities
    uint32_t *idx;            // kOpDensest: the result; kOpKnn: k per query
    double *dr2;              // kOpKnn
    uint32_t *redo, *nredo;   // queries for the heap path
};

// What a query's sorted k-set (xkey, xix) becomes. p: the query point, at_q3: whether it was given.
template <int OP>
__device__ __forceinline__ void wk_finish(const KTree &t, WkBuf &s, const double4_32a &p, bool at_q3, uint32_t i, uint32_t k, double fpo3,
                                          const SplineCells &sc, const WkOut &out) {
    const uint32_t lane = threadIdx.x & 31;
    if constexpr (OP == kOpKnn) {
        for (uint32_t j = lane; j < k; j += 32) {
            out.idx[(size_t)i * k + j] = s.xix[j];
            out.dr2[(size_t)i * k + j] = dfrom(s.xkey[j]);
        }
    } else if constexpr (OP == kOpDensest) {
        wk_densest(s.xix, k, i, out.dens[i], out.dens, out.idx);
    } else if constexpr (OP == kOpSpline) {
        // the terms by the lanes, their sum in ascending order by one
        const double4_32a o = at_q3 ? t.pos[0] : p;
        double *term = reinterpret_cast<double *>(s.key);
        static_assert(sizeof(s.key) + sizeof(s.ix) >= 128 * sizeof(double), "terms");
        for (uint32_t j = lane; j < k; j += 32) {
            const double4_32a c = t.pos[s.xix[j]];
            term[j] = c.w / sc.volume * spline_weight(c.x - o.x, c.y - o.y, c.z - o.z, sc);
        }
        __syncwarp();
        if (lane == 0) {
            double dens = 0;
            for (uint32_t j = 0; j < k; ++j) dens = dens + term[j];
            out.dens[i] = dens;
        }
    } else {
        double *ms = reinterpret_cast<double *>(s.key);
        for (uint32_t j = lane; j < k; j += 32) ms[j] = t.pos[s.xix[j]].w;
        __syncwarp();
        if (lane == 0) {  // MedianSphericalDensityKernel on the sorted k-set, as knn_median_density
            int j = (int)k;
            const double m2 = 4 * dfrom(s.xkey[j / 2]);
            for (j = j - 1; j >= 0; j--)
                if (!(dfrom(s.xkey[j]) > m2)) break;
            const double r2 = dfrom(s.xkey[j]);
            double dens = 0;
            for (; j >= 0; j--) dens = dens + ms[j];
            out.dens[i] = dens / (fpo3 * cr_pow15(r2));
        }
    }
}

template <int OP>
__global__ void __launch_bounds__(32 * kWkWarps) k_exact_w(KTree t, FTree f, const double *q3, const double *est, double est0, const uint32_t *list,
                                                           const uint32_t *nlist, uint32_t nq, uint32_t k, double fpo3, SplineCells sc, WkOut out,
                                                           unsigned *err) {
    __shared__ WkBuf s_buf[kWkWarps];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    WkBuf &s = s_buf[w];
    if (nlist) nq = *nlist;
    for (uint32_t u = blockIdx.x * kWkWarps + w; u < nq; u += gridDim.x * kWkWarps) {
        const uint32_t i = list ? list[u] : u;
        double4_32a p;
        if (q3) p = make_double4_32a(q3[3 * (size_t)i], q3[3 * (size_t)i + 1], q3[3 * (size_t)i + 2], 0.0);
        else p = t.pos[i];
        const WkQuery q = wk_query(p.x, p.y, p.z);
        double r = q3 ? (est ? est[i] : est0) : 0.0;
        if (q3) r = r != 0 ? r : knn_first_radius(t, p.x, p.y, p.z, 0xffffffffu, k, err);
        else r = wk_first_radius(t, q, t.leaf_of[i], k, err);
        uint32_t m, visited, tau;
        __syncwarp();
        bool ok = wk_collect(t, f, q, r, k, s, m, visited, tau, err);
        if (ok && visited < k && (OP == kOpMedian || OP == kOpSpline) && q3) {  // fewer points than neighbours: the reference's zero
            if (lane == 0) out.dens[i] = 0.0;
            continue;
        }
        ok = ok && visited >= k && wk_sorted(t, q, s, k, m, tau, f.tol);
        if (!ok) {
            if (lane == 0) out.redo[atomicAdd(out.nredo, 1u)] = i;
            continue;
        }
        wk_finish<OP>(t, s, p, q3 != nullptr, i, k, fpo3, sc, out);
        __syncwarp();
    }
}

// The same for queries that may visit 10^5 points (the Hill sweeps' saddles: tens of queries from a
// Hill radius): a block per query. Its threads walk the tree a level at a time, listing the
// visited ranges; the points are shared out evenly over all warps, each with a buffer of its own
// and the smallest bound any of them has found, and warp 0 merges what is left. Measured on 48 to
// 72 such queries of 262,144 particles: 1.6 -> 0.15 ms per sweep against a warp per query. Queries
// that overflow a list go to the warp kernel.
constexpr int kBkThreads = 256, kBkWarps = kBkThreads / 32;
constexpr uint32_t kBkNodes = 4096, kBkRanges = 4096, kBkPart = 256;
constexpr uint32_t kBkMaxK = 48;       // eight warps' bounds must fit the merged buffer
// Queries of one call from which on a warp takes each. Measured, a block and a warp per query: 236
// queries 0.04 and 0.10 ms, 1,292 0.16 and 0.21, 5,460 0.64 and 0.76, 10,018 1.29 and 1.74, 15,634
// 1.95 and 1.82 ms.
constexpr uint32_t kBkQueries = 12000;

struct BkShared {
    WkBuf merged;
    uint32_t node[2][kBkNodes], first[kBkRanges], cum[kBkRanges];
    uint32_t key[kBkWarps][kBkPart], ix[kBkWarps][kBkPart];
    uint32_t nnode[2], nrange, over, tau, nmerged, wsum[kBkWarps];
};

template <int OP>
__global__ void __launch_bounds__(kBkThreads) k_exact_block(KTree t, FTree f, const double *q3, const double *est, uint32_t nq, uint32_t k,
                                                            double fpo3, SplineCells sc, WkOut out, unsigned *err) {
    extern __shared__ __align__(16) unsigned char bk_dyn[];
    BkShared &sh = *reinterpret_cast<BkShared *>(bk_dyn);
    const uint32_t tid = threadIdx.x, lane = tid & 31, w = tid >> 5, full = 0xffffffffu, i = blockIdx.x;
    const double4_32a p = make_double4_32a(q3[3 * (size_t)i], q3[3 * (size_t)i + 1], q3[3 * (size_t)i + 2], 0.0);
    const WkQuery q = wk_query(p.x, p.y, p.z);
    double r = est[i] != 0 ? est[i] : knn_first_radius(t, p.x, p.y, p.z, 0xffffffffu, k, err);
    uint32_t visited = 0, nr = 0;
    bool over = false;
    for (int it = 0; it < 200; ++it, r = r * 2) {
        const float rf = (float)r;
        if (tid == 0) {
            sh.node[0][0] = 0;
            sh.nnode[0] = 1;
            sh.nnode[1] = 0;
            sh.nrange = 0;
            sh.over = 0;
        }
        __syncthreads();
        for (int side = 0, level = 0; sh.nnode[side]; side ^= 1) {
            if (++level > 40) {  // a tree has 33 levels at most
                if (tid == 0) atomicOr(err, (unsigned)kDevErrLoopLimit);
                break;
            }
            const uint32_t na = sh.nnode[side];
            for (uint32_t j = tid; j < na; j += kBkThreads) {
                const uint32_t node = sh.node[side][j];
                int cls = 0;
                if (node < t.nodes) cls = wk_class(t, f, node, q, r, rf);
                else atomicOr(err, (unsigned)kDevErrBadNode);
                if (!cls) continue;
                const uint32_t nd = cls == 2 ? t.nnd[node] : 0u;
                if (nd) {
                    const uint32_t at = atomicAdd(&sh.nnode[side ^ 1], nd), c0 = t.nfd[node];
                    if (at + nd <= kBkNodes)
                        for (uint32_t c = 0; c < nd; ++c) sh.node[side ^ 1][at + c] = c0 + c;
                    else sh.over = 1;
                } else {
                    const uint32_t at = atomicAdd(&sh.nrange, 1u), b = t.nbeg[node];
                    if (at < kBkRanges) {
                        sh.first[at] = b;
                        sh.cum[at] = t.nend[node] - b;
                    } else {
                        sh.over = 1;
                    }
                }
            }
            __syncthreads();
            if (sh.over) break;
            if (tid == 0) sh.nnode[side] = 0;
            __syncthreads();
        }
        over = sh.over != 0;
        __syncthreads();
        if (over) break;
        // the ranges' lengths become their ends
        nr = sh.nrange;
        visited = 0;
        for (uint32_t j0 = 0; j0 < nr; j0 += kBkThreads) {
            const uint32_t j = j0 + tid;
            uint32_t v = j < nr ? sh.cum[j] : 0u;
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(full, v, d);
                if (lane >= (uint32_t)d) v += o;
            }
            if (lane == 31) sh.wsum[w] = v;
            __syncthreads();
            uint32_t before = visited, all = visited;
            for (uint32_t u = 0; u < kBkWarps; ++u) {
                if (u < w) before += sh.wsum[u];
                all += sh.wsum[u];
            }
            if (j < nr) sh.cum[j] = before + v;
            visited = all;
            __syncthreads();
        }
        if (visited >= k) break;
        if (it == 199 && tid == 0) atomicOr(err, (unsigned)kDevErrLoopLimit);
    }
    if (!over && visited < k) {  // fewer points than neighbours: the reference's zero
        if (tid == 0) out.dens[i] = 0.0;
        return;
    }
    if (tid == 0) {
        sh.tau = 0x7f800000u;
        sh.nmerged = 0;
        sh.over = over ? 1u : 0u;
    }
    __syncthreads();
    uint32_t n = 0, tau = 0x7f800000u;
    uint32_t *key = sh.key[w], *ix = sh.ix[w];
    constexpr int kIn = 4;
    for (uint32_t t0 = 0; !over && t0 < visited; t0 += kIn * kBkThreads) {
        uint32_t pt[kIn], v[kIn];
#pragma unroll
        for (int j = 0; j < kIn; ++j) {
            const uint32_t at = t0 + j * kBkThreads + tid;
            uint32_t lo = 0, hi = at < visited ? nr : 1;  // the first range that ends beyond it
            while (lo < hi) {
                const uint32_t mid = (lo + hi) >> 1;
                if (sh.cum[mid] <= at) lo = mid + 1;
                else hi = mid;
            }
            pt[j] = at < visited ? sh.first[lo] + at - (lo ? sh.cum[lo - 1] : 0u) : kNoPoint;
        }
#pragma unroll
        for (int j = 0; j < kIn; ++j)
            v[j] = pt[j] != kNoPoint ? __float_as_uint(f_dr2(q.h, q.l, f.phi[pt[j]], f.plo[pt[j]])) : 0xffffffffu;
        tau = min(tau, *(volatile uint32_t *)&sh.tau);
#pragma unroll
        for (int j = 0; j < kIn; ++j) {
            unsigned m = __ballot_sync(full, v[j] <= tau);
            if (!m) continue;
            if (n + __popc(m) > kBkPart) {
                wk_compact(key, ix, k, n, tau, f.tol);
                if (lane == 0) atomicMin(&sh.tau, tau);
                m = __ballot_sync(full, v[j] <= tau);
                if (n + __popc(m) > kBkPart) {
                    sh.over = 1;
                    m = 0;
                }
            }
            if ((m >> lane) & 1u) {
                const uint32_t at = n + __popc(m & ((1u << lane) - 1u));
                key[at] = v[j];
                ix[at] = pt[j];
            }
            n += __popc(m);
            __syncwarp();
        }
    }
    wk_compact(key, ix, k, n, tau, f.tol);
    if (lane == 0) atomicMin(&sh.tau, tau);
    __syncthreads();
    tau = sh.tau;
    n = wk_filter(key, ix, n, tau);
    uint32_t at = 0;
    if (lane == 0) at = atomicAdd(&sh.nmerged, n);
    at = __shfl_sync(full, at, 0);
    if (at + n <= kWkPoints) {
        for (uint32_t j = lane; j < n; j += 32) {
            sh.merged.key[at + j] = key[j];
            sh.merged.ix[at + j] = ix[j];
        }
    } else if (lane == 0) {
        sh.over = 1;
    }
    __syncthreads();
    if (w != 0) return;
    const uint32_t all = sh.nmerged;
    if (!sh.over && wk_sorted(t, q, sh.merged, k, all, tau, f.tol)) wk_finish<OP>(t, sh.merged, p, true, i, k, fpo3, sc, out);
    else if (lane == 0) out.redo[atomicAdd(out.nredo, 1u)] = i;
}

template <class F>
int launch_by_k(uint32_t k, F f) {
    if (k <= 32) return f(std::integral_constant<int, 32>(), 128);
    if (k <= 64) return f(std::integral_constant<int, 64>(), 64);
    if (k <= 128) return f(std::integral_constant<int, 128>(), 32);
    return kErrUnsupported;
}

}  // namespace

// Blocks for a list whose length only the device knows: enough to fill the GPU.
static unsigned list_blocks(Context &c) {
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
    return (unsigned)sms * 4u;
}

// Two redo lists (for the exact warp kernel, then for the heap path) and their counts.
struct RedoLists {
    uint32_t *warp, *heap, *n;  // n[0], n[1]
    int take(Context &c, size_t most, cudaStream_t s) {
        warp = c.scratch.get<uint32_t>(most + 1);
        heap = c.scratch.get<uint32_t>(most + 1);
        n = c.scratch.get<uint32_t>(4);
        if (!warp || !heap || !n) return kErrOutOfMemory;
        PLAN_CUDA(cudaMemsetAsync(n, 0, 8, s));
        return kOk;
    }
};

int launch_density(Context &c, const plan_params &p, uint32_t k, cudaStream_t s) {
    if (k > 64) return kErrUnsupported;
    KTree t = ktree_of(c.tree);
    const double fpo3 = 3.14159265358979323846 * 4. / 3.;
    const FTree f = ftree_of(c.tree);
    const uint32_t n = c.tree.Tu;
    const size_t mark = c.scratch.used;
    RedoLists redo;
    int rc = redo.take(c, n, s);
    if (rc) return rc;
    const SplineCells sc = c.fs.spline;
    const unsigned lb = list_blocks(c);
    WkOut out{c.tree.dens, nullptr, nullptr, redo.heap, redo.n + 1};
    PLAN_CUDA(cudaEventRecord(c.kev[0], s));
    if (c.fs.median_kernel) {
        uint32_t *at = c.scratch.get<uint32_t>(n), *cnt = c.scratch.get<uint32_t>(n);
        if (!at || !cnt) return kErrOutOfMemory;
        const bool uniform = c.tree.nsinks == 0 && p.ntypes <= 1;
        k_density_w<<<(n + kWkWarps - 1) / kWkWarps, 32 * kWkWarps, 0, s>>>(t, f, n, k, uniform, at, cnt, c.tree.dens, redo.warp, redo.n, c.d_err);
        k_density_finish<<<grid_for(n, 256), 256, 0, s>>>(t.pos, n, fpo3, at, cnt, c.tree.dens);
        k_exact_w<kOpMedian><<<lb, 32 * kWkWarps, 0, s>>>(t, f, nullptr, nullptr, 0.0, redo.warp, redo.n, 0, k, fpo3, sc, out, c.d_err);
        c.launches += 3;
    } else {
        k_exact_w<kOpSpline><<<(n + kWkWarps - 1) / kWkWarps, 32 * kWkWarps, 0, s>>>(t, f, nullptr, nullptr, 0.0, nullptr, nullptr, n, k, fpo3, sc,
                                                                                  out, c.d_err);
        c.launches++;
    }
    rc = launch_by_k(k, [&](auto km, int threads) {
        constexpr int KM = decltype(km)::value;
        size_t sm = (size_t)KM * threads * 12;
        auto kern = c.fs.median_kernel ? k_density_list<KM, 0> : k_density_list<KM, 1>;
        kern<<<lb, threads, sm, s>>>(t, redo.heap, redo.n + 1, k, fpo3, sc, c.tree.dens, c.d_err);
        c.launches++;
        PLAN_CUDA(cudaGetLastError());
        return (int)kOk;
    });
    if (rc) return rc;
    PLAN_CUDA(cudaEventRecord(c.kev[1], s));
    uint32_t h[2] = {0, 0};
    PLAN_CUDA(cudaMemcpyAsync(h, redo.n, 8, cudaMemcpyDeviceToHost, s));
    PLAN_CUDA(cudaStreamSynchronize(s));
    float kms = 0;
    cudaEventElapsedTime(&kms, c.kev[0], c.kev[1]);
    c.stage_ms[20] = kms;  // the density kernels
    c.counters[17] = h[0] + h[1];
    c.scratch.used = mark;
    return kOk;
}

int launch_densest(Context &c, const plan_params &p, uint32_t k, double threshold, uint32_t *densest, cudaStream_t s) {
    if (k > 64) return kErrUnsupported;
    KTree t = ktree_of(c.tree);
    const FTree f = ftree_of(c.tree);
    const uint32_t n = c.tree.Tu;
    const size_t mark = c.scratch.used;
    RedoLists redo;
    int rc = redo.take(c, n, s);
    if (rc) return rc;
    const unsigned lb = list_blocks(c);
    PLAN_CUDA(cudaEventRecord(c.kev[0], s));
    k_densest_w<<<(n + kWkWarps - 1) / kWkWarps, 32 * kWkWarps, 0, s>>>(t, f, n, k, threshold, c.tree.dens, densest, redo.warp, redo.n, c.d_err);
    k_exact_w<kOpDensest><<<lb, 32 * kWkWarps, 0, s>>>(t, f, nullptr, nullptr, 0.0, redo.warp, redo.n, 0, k, 0.0, c.fs.spline,
                                                       WkOut{c.tree.dens, densest, nullptr, redo.heap, redo.n + 1}, c.d_err);
    c.launches += 2;
    rc = launch_by_k(k, [&](auto km, int threads) {
        constexpr int KM = decltype(km)::value;
        size_t sm = (size_t)KM * threads * 12;
        k_densest_list<KM><<<lb, threads, sm, s>>>(t, redo.heap, redo.n + 1, k, c.tree.dens, densest, c.d_err);
        c.launches++;
        PLAN_CUDA(cudaGetLastError());
        return (int)kOk;
    });
    if (rc) return rc;
    PLAN_CUDA(cudaEventRecord(c.kev[1], s));
    uint32_t h[2] = {0, 0};
    PLAN_CUDA(cudaMemcpyAsync(h, redo.n, 8, cudaMemcpyDeviceToHost, s));
    PLAN_CUDA(cudaStreamSynchronize(s));
    float kms = 0;
    cudaEventElapsedTime(&kms, c.kev[0], c.kev[1]);
    c.stage_ms[21] = kms;  // the densest-neighbour kernels
    c.counters[18] = h[0] + h[1];
    c.scratch.used = mark;
    return kOk;
}

int launch_density_at(Context &c, const double *d_q3, const double *d_est, uint32_t nq, uint32_t k, double *d_out, cudaStream_t s) {
    if (nq == 0) return kOk;
    KTree t = ktree_of(c.tree);
    const double fpo3 = 3.14159265358979323846 * 4. / 3.;
    const bool spl = !c.fs.median_kernel;
    const FTree f = ftree_of(c.tree);
    const size_t mark = c.scratch.used;
    uint32_t *heap = c.scratch.get<uint32_t>(nq + 1), *warp = c.scratch.get<uint32_t>(nq + 1), *nheap = c.scratch.get<uint32_t>(4);
    if (!heap || !warp || !nheap) {
        c.scratch.used = mark;
        return kErrOutOfMemory;
    }
    PLAN_CUDA(cudaMemsetAsync(nheap, 0, 8, s));
    // a block per query where there are few, else a warp; what overflows a block goes to a warp,
    // the queries with distance ties to the exact heap path
    int rc = launch_by_k(k, [&](auto km, int threads) {
        constexpr int KM = decltype(km)::value;
        const bool blocks = nq < kBkQueries && k <= kBkMaxK;
        auto kern = spl ? k_exact_w<kOpSpline> : k_exact_w<kOpMedian>;
        const WkOut to_heap{d_out, nullptr, nullptr, heap, nheap};
        if (blocks) {
            auto bk = spl ? k_exact_block<kOpSpline> : k_exact_block<kOpMedian>;
            PLAN_CUDA(cudaFuncSetAttribute(bk, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)sizeof(BkShared)));
            bk<<<nq, kBkThreads, sizeof(BkShared), s>>>(t, f, d_q3, d_est, nq, k, fpo3, c.fs.spline, WkOut{d_out, nullptr, nullptr, warp, nheap + 1},
                                                      c.d_err);
            c.launches++;
        }
        kern<<<blocks ? list_blocks(c) : (nq + kWkWarps - 1) / kWkWarps, 32 * kWkWarps, 0, s>>>(
            t, f, d_q3, d_est, 0.0, blocks ? warp : nullptr, blocks ? nheap + 1 : nullptr, nq, k, fpo3, c.fs.spline, to_heap, c.d_err);
        size_t sm = (size_t)KM * threads * 12;
        auto list = spl ? k_density_at<KM, 1> : k_density_at<KM, 0>;
        list<<<list_blocks(c), threads, sm, s>>>(t, d_q3, d_est, heap, nheap, k, fpo3, c.fs.spline, d_out, c.d_err);
        c.launches += 2;
        PLAN_CUDA(cudaGetLastError());
        return (int)kOk;
    });
    uint32_t h = 0;
    if (!rc) {
        PLAN_CUDA(cudaMemcpyAsync(&h, nheap, 4, cudaMemcpyDeviceToHost, s));
        PLAN_CUDA(cudaStreamSynchronize(s));  // the list is scratch, released here
        c.counters[27] += h;
    }
    c.scratch.used = mark;
    return rc;
}

int knn_positions(Context &c, const double *pos3, uint32_t nq, uint32_t k, double est, uint32_t *idx, double *dr2) {
    if (!c.tree.Tu || k == 0 || k > c.tree.Tu) return kErrArgument;
    if (k > 128) return kErrUnsupported;
    if (nq == 0) return kOk;
    cudaStream_t s = c.stream;
    StreamBuf<double> d_q(s), d_d(s);
    StreamBuf<uint32_t> d_i(s), d_redo(s);
    PLAN_CUDA(d_q.alloc((size_t)nq * 3));
    PLAN_CUDA(d_d.alloc((size_t)nq * k));
    PLAN_CUDA(d_i.alloc((size_t)nq * k));
    PLAN_CUDA(d_redo.alloc((size_t)nq + 1));
    PLAN_CUDA(cudaMemsetAsync(d_redo.p, 0, 4, s));
    PLAN_CUDA(cudaMemcpyAsync(d_q.p, pos3, (size_t)nq * 3 * 8, cudaMemcpyHostToDevice, s));
    KTree t = ktree_of(c.tree);
    const FTree f = ftree_of(c.tree);
    int rc = launch_by_k(k, [&](auto km, int threads) {
        constexpr int KM = decltype(km)::value;
        k_exact_w<kOpKnn><<<(nq + kWkWarps - 1) / kWkWarps, 32 * kWkWarps, 0, s>>>(t, f, d_q.p, nullptr, est, nullptr, nullptr, nq, k, 0.0,
                                                                                c.fs.spline, WkOut{nullptr, d_i.p, d_d.p, d_redo.p + 1, d_redo.p},
                                                                                c.d_err);
        size_t sm = (size_t)KM * threads * 12;
        k_knn_positions<KM><<<list_blocks(c), threads, sm, s>>>(t, d_q.p, d_redo.p + 1, d_redo.p, k, est, d_i.p, d_d.p, c.d_err);
        c.launches += 2;
        PLAN_CUDA(cudaGetLastError());
        return (int)kOk;
    });
    if (rc) return rc;
    PLAN_CUDA(cudaMemcpyAsync(idx, d_i.p, (size_t)nq * k * 4, cudaMemcpyDeviceToHost, s));
    PLAN_CUDA(cudaMemcpyAsync(dr2, d_d.p, (size_t)nq * k * 8, cudaMemcpyDeviceToHost, s));
    PLAN_CUDA(cudaStreamSynchronize(s));
    return kOk;
}

}  // namespace plan
