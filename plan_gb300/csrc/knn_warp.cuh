// Nearest neighbours with the reference's exact results, one warp per query.
//
// The visited set of a query (tree_walk.cuh: every point of every node that the sphere contains
// or meets, the radius doubled until k points are visited) does not depend on the order of the
// walk. The warp keeps a last-in first-out list of nodes in shared memory; its lanes classify up
// to 32 of them at a time (FP32 with the error bounds of knn_f32.cuh, the FP64 test where that
// cannot tell), append the children of the met ones, and share the points of the contained nodes
// and met leaves. A point's FP32 squared distance (non-negative: its bits order like its value)
// and index go to a buffer; when that is full, the k-th smallest is found by bisection on the
// bits and everything beyond its error bound is dropped for good.
//
// Why a warp: a thread per query kept 3.3 of 32 lanes active (the walks of neighbouring queries
// diverge at every node, and a heap insertion runs for one lane at a time), 27 ns per tree point.
// What bounds this form: integer and FP32 instructions of the node tests and the selection.
// FP64 is kept out of it because an FP64 instruction costs the SM 19 cycles however few lanes
// work: the FP64 density of a query is formed afterwards, a thread per query.
#pragma once

#include "exact64.cuh"
#include "tree_walk.cuh"

namespace plan {

constexpr int kWkWarps = 4;           // warps (queries) per block
constexpr uint32_t kWkNodes = 704;    // nodes to classify: 32 at a time up to kWkWide, then one at a time,
constexpr uint32_t kWkWide = 256;     // when each of the tree's 32 levels adds at most seven (256 + 224 + 224)
constexpr uint32_t kWkPoints = 512;   // buffered candidates (at least four times the largest k, 128)
constexpr uint32_t kWkSmall = 8;      // ranges up to this length share the lanes (the default leaf size)
constexpr uint32_t kWkExact = 256;    // candidates whose FP64 distances are sorted

struct WkBuf {
    union {
        struct {
            uint32_t node[kWkNodes], pts[32 * kWkSmall];  // during the walk
        };
        struct {
            unsigned long long xkey[kWkExact];            // after it
            uint32_t xix[kWkExact];
        };
    };
    uint32_t key[kWkPoints], ix[kWkPoints];
};
static_assert(sizeof(WkBuf) * kWkWarps <= 48 * 1024, "one block's buffers");

struct WkQuery {
    double x, y, z;
    float4 h, l;
};

__device__ __forceinline__ WkQuery wk_query(double x, double y, double z) {
    WkQuery q;
    q.x = x; q.y = y; q.z = z;
    q.h = make_float4((float)x, (float)y, (float)z, 0.f);
    q.l = make_float4((float)(x - (double)q.h.x), (float)(y - (double)q.h.y), (float)(z - (double)q.h.z), 0.f);
    return q;
}

// The first radius of a tree point (knn_first_radius): the half width of the smallest node
// above it with at least k/4 points. The root of a half width's rounded square is the half
// width. Points near the root box's faces, which might lie outside it, take the FP64 form.
__device__ __forceinline__ double wk_first_radius(const KTree &t, const WkQuery &q, uint32_t leaf, uint32_t k, unsigned *err) {
    const float hw = (float)t.box.half_width * 0.999f;
    if (fabsf(q.h.x - (float)t.box.root_center[0]) < hw && fabsf(q.h.y - (float)t.box.root_center[1]) < hw &&
        fabsf(q.h.z - (float)t.box.root_center[2]) < hw) {
        uint32_t node = leaf;
        for (int guard = 0; guard < 40 && (t.nend[node] - t.nbeg[node]) < k / 4; ++guard) {
            if (node == 0) break;
            node = t.npar[node];
        }
        return t.ncf[node].w;
    }
    return knn_first_radius(t, q.x, q.y, q.z, leaf, k, err);
}

// 1 contained, 2 met, 0 neither
__device__ __forceinline__ int wk_class(const KTree &t, const FTree &f, uint32_t node, const WkQuery &q, double r, float rf) {
    const float4 nh = f.nhi[node], nl = f.nlo[node];
    const int c = f_contained(nh, nl, q.h, q.l, rf, f.tol);
    if (c > 0) return 1;
    const int m = f_intersects(nh, nl, q.h, q.l, rf, f.tol);
    if (c < 0 || m < 0) return node_class(t.ncf + node, q.x, q.y, q.z, r);
    return m ? 2 : 0;
}

// A threshold with at least want of the n keys at or below it, exactly want where equal keys
// allow; count is how many. n >= want >= 1.
__device__ __forceinline__ uint32_t wk_select(const uint32_t *key, uint32_t n, uint32_t want, uint32_t &count) {
    const uint32_t lane = threadIdx.x & 31;
    uint32_t lo = 0xffffffffu, hi = 0;
    for (uint32_t j = lane; j < n; j += 32) {
        const uint32_t v = key[j];
        lo = min(lo, v);
        hi = max(hi, v);
    }
    lo = __reduce_min_sync(0xffffffffu, lo);
    hi = __reduce_max_sync(0xffffffffu, hi);
    count = n;
    while (lo < hi && count != want) {
        const uint32_t mid = lo + (hi - lo) / 2;
        uint32_t c = 0;
        for (uint32_t j = lane; j < n; j += 32) c += key[j] <= mid ? 1u : 0u;
        c = __reduce_add_sync(0xffffffffu, c);
        if (c >= want) {
            hi = mid;
            count = c;
        } else {
            lo = mid + 1;
        }
    }
    return hi;
}

// Keeps the buffered candidates with keys at or below limit, in place; returns their number.
__device__ __forceinline__ uint32_t wk_filter(uint32_t *key, uint32_t *ix, uint32_t n, uint32_t limit) {
    const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u;
    uint32_t m = 0;
    for (uint32_t j = 0; j < n; j += 32) {
        const uint32_t v = j + lane < n ? key[j + lane] : 0xffffffffu, p = j + lane < n ? ix[j + lane] : 0u;
        const bool keep = j + lane < n && v <= limit;
        const unsigned b = __ballot_sync(0xffffffffu, keep);
        if (keep) {
            key[m + __popc(b & below)] = v;
            ix[m + __popc(b & below)] = p;
        }
        m += __popc(b);
        __syncwarp();
    }
    return m;
}

// Drops the candidates that cannot be among the k nearest: tau becomes a key that no member of
// the exact k-set exceeds.
__device__ __forceinline__ void wk_compact(uint32_t *key, uint32_t *ix, uint32_t k, uint32_t &n, uint32_t &tau, Tol tol) {
    __syncwarp();
    if (n < k) return;
    uint32_t count;
    const float thr = f_hi(__uint_as_float(wk_select(key, n, k, count)), tol);
    tau = min(tau, __float_as_uint((thr + 2.f * tol.sq) * (1.f + 4.f * kRel)));
    n = wk_filter(key, ix, n, tau);
}

// The walk. False when candidates at equal distances overflow the buffer. visited < k only
// where doubling the radius 200 times does not reach k points (an error flag is set).
__device__ inline bool wk_collect(const KTree &t, const FTree &f, const WkQuery &q, double r, uint32_t k, WkBuf &s, uint32_t &n,
                                  uint32_t &visited, uint32_t &tau, unsigned *err) {
    const uint32_t lane = threadIdx.x & 31, below = (1u << lane) - 1u;
    const unsigned full = 0xffffffffu;
    for (int it = 0; it < 200; ++it, r = r * 2) {
        n = 0;
        visited = 0;
        tau = 0x7f800000u;
        const float rf = (float)r;
        bool over = false;
        auto take_point = [&](uint32_t p, bool have) {
            uint32_t v = 0xffffffffu;
            if (have) v = __float_as_uint(f_dr2(q.h, q.l, f.phi[p], f.plo[p]));
            unsigned m = __ballot_sync(full, v <= tau);
            if (!m) return;
            if (n + __popc(m) > kWkPoints) {
                wk_compact(s.key, s.ix, k, n, tau, f.tol);
                m = __ballot_sync(full, v <= tau);
                if (n + __popc(m) > kWkPoints) {
                    over = true;
                    return;
                }
            }
            if ((m >> lane) & 1u) {
                const uint32_t at = n + __popc(m & below);
                s.key[at] = v;
                s.ix[at] = p;
            }
            n += __popc(m);
            __syncwarp();
        };
        uint32_t top = 1;
        __syncwarp();
        if (lane == 0) s.node[0] = 0;
        __syncwarp();
        while (top) {
            const uint32_t take = min(top, top > kWkWide ? 1u : 32u);
            uint32_t node = 0;
            int cls = 0;
            if (lane < take) {
                node = s.node[top - 1 - lane];
                if (node < t.nodes) cls = wk_class(t, f, node, q, r, rf);
                else atomicOr(err, (unsigned)kDevErrBadNode);
            }
            top -= take;
            const uint32_t nd = cls == 2 ? t.nnd[node] : 0u;
            uint32_t b = 0, size = 0;
            if (cls == 1 || (cls == 2 && nd == 0)) {
                b = t.nbeg[node];
                size = t.nend[node] - b;
            }
            // where the children and the points of short ranges go: two scans in one
            const uint32_t mine = nd | (size <= kWkSmall ? size << 16 : 0u);
            uint32_t incl = mine;
#pragma unroll
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(full, incl, d);
                if (lane >= (uint32_t)d) incl += o;
            }
            const uint32_t tot = __shfl_sync(full, incl, 31), at = incl - mine;
            if (top + (tot & 0xffffu) > kWkNodes) {  // a tree deeper than 32 levels
                if (lane == 0) atomicOr(err, (unsigned)kDevErrStackOverflow);
                return false;
            }
            __syncwarp();
            if (nd) {
                const uint32_t c0 = t.nfd[node];
                for (uint32_t c = 0; c < nd; ++c) s.node[top + (at & 0xffffu) + c] = c0 + c;
            }
            if (size <= kWkSmall)
                for (uint32_t c = 0; c < size; ++c) s.pts[(at >> 16) + c] = b + c;
            top += tot & 0xffffu;
            __syncwarp();
            const uint32_t np = tot >> 16;
            visited += np;
            for (uint32_t p0 = 0; p0 < np && !over; p0 += 32) {
                const bool have = p0 + lane < np;
                take_point(have ? s.pts[p0 + lane] : 0u, have);
            }
            for (unsigned m = __ballot_sync(full, size > kWkSmall); m && !over; m &= m - 1) {
                const int w = __ffs(m) - 1;
                const uint32_t bb = __shfl_sync(full, b, w), ss = __shfl_sync(full, size, w);
                visited += ss;
                for (uint32_t p0 = 0; p0 < ss && !over; p0 += 32) take_point(bb + p0 + lane, p0 + lane < ss);
            }
            if (over) return false;
        }
        if (visited >= k) return true;
    }
    if (lane == 0) atomicOr(err, (unsigned)kDevErrLoopLimit);
    return true;
}

// The exact k-set from the FP32 keys alone: the k smallest of the buffer are moved to its
// front, unless the (k+1)-th is too close to the k-th to tell (then false).
__device__ __forceinline__ bool wk_kset(WkBuf &s, uint32_t k, uint32_t n, uint32_t tau, Tol tol) {
    const uint32_t lane = threadIdx.x & 31;
    __syncwarp();
    if (n < k) return false;
    uint32_t count;
    const uint32_t T = wk_select(s.key, n, k, count);
    if (count != k) return false;
    uint32_t in = 0, out = tau;  // what was dropped lies above tau
    for (uint32_t j = lane; j < n; j += 32) {
        const uint32_t v = s.key[j];
        if (v <= T) in = max(in, v);
        else out = min(out, v);
    }
    in = __reduce_max_sync(0xffffffffu, in);
    out = __reduce_min_sync(0xffffffffu, out);
    if (!(f_hi(__uint_as_float(in), tol) < f_lo(__uint_as_float(out), tol))) return false;
    wk_filter(s.key, s.ix, n, T);
    return true;
}

// Ascending sort of (key, index) pairs [0, n) by one warp (bitonic, in shared memory; the
// entries up to the next power of two are padded, so C, a power of two, bounds n).
template <int C>
__device__ inline void warp_sort_pairs(unsigned long long *key, uint32_t *ix, uint32_t n, int lane) {
    uint32_t P = 1;
    while (P < n) P <<= 1;
    for (uint32_t j = n + lane; j < P; j += 32) {
        key[j] = ~0ull;
        ix[j] = 0xffffffffu;
    }
    __syncwarp();
    for (uint32_t size = 2; size <= P; size <<= 1)
        for (uint32_t stride = size >> 1; stride > 0; stride >>= 1) {
            for (uint32_t u = lane; u < P / 2; u += 32) {
                const uint32_t a = 2 * u - (u & (stride - 1)), b = a + stride;
                const bool up = (a & size) == 0;
                const unsigned long long ka = key[a], kb = key[b];
                const uint32_t ia = ix[a], ib = ix[b];
                const bool gt = ka > kb || (ka == kb && ia > ib);
                if (gt == up) {
                    key[a] = kb;
                    key[b] = ka;
                    ix[a] = ib;
                    ix[b] = ia;
                }
            }
            __syncwarp();
        }
}

// The exact k-set in ascending FP64 distance, in xkey (bits) and xix. False when two of its
// members, or the k-th and the next, are equally far: their order is the library heap's.
__device__ __forceinline__ bool wk_sorted(const KTree &t, const WkQuery &q, WkBuf &s, uint32_t k, uint32_t n, uint32_t tau, Tol tol) {
    const uint32_t lane = threadIdx.x & 31;
    wk_compact(s.key, s.ix, k, n, tau, tol);
    if (n < k || n > kWkExact) return false;
    __syncwarp();
    for (uint32_t j = lane; j < n; j += 32) {
        const uint32_t p = s.ix[j];
        s.xkey[j] = dbits(point_dr2(q.x, q.y, q.z, t.pos[p]));
        s.xix[j] = p;
    }
    __syncwarp();
    warp_sort_pairs<kWkExact>(s.xkey, s.xix, n, (int)lane);
    bool tie = false;
    for (uint32_t j = 1 + lane; j < min(k + 1, n); j += 32) tie = tie || s.xkey[j] == s.xkey[j - 1];
    return !__any_sync(0xffffffffu, tie);
}

}  // namespace plan
