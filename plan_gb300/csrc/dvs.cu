// --Density_Vs_Scale on the GPU: a warp takes a (cell centre, radius, sub-centre) query of
// BasicAnalysesWithTree at a time and walks the particle tree with the reference's sheared node
// tests in FP32, in FP64 where that cannot tell (dvs.cuh, the same code the CPU tests run); the
// largest count per radius is an atomic maximum, and queries that cannot exceed it stop early. The
// host sets up the grid with the reference's own arithmetic and turns the counts into densities.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <string>
#include <vector>

#include "dvs.cuh"
#include "pipeline.h"
#include "tree_walk.cuh"

namespace plan {

namespace {

struct DevTreeView {
    KTree t;
    __device__ uint32_t begin(uint32_t n) const { return t.nbeg[n]; }
    __device__ uint32_t end(uint32_t n) const { return t.nend[n]; }
    __device__ uint32_t first(uint32_t n) const { return t.nfd[n]; }
    __device__ uint32_t daughters(uint32_t n) const { return t.nnd[n]; }
};

// Query tid in the order they are taken: variant by variant, the largest radius first (the
// longest walks start first), the cells of a variant side by side (neighbours meet the same nodes).
__device__ __forceinline__ uint64_t dvs_order(const DvsGeom &g, uint64_t tid) {
    const uint64_t cells = (uint64_t)g.nx * g.ny * g.nz;
    const uint32_t v = (uint32_t)(tid / cells);
    return (tid % cells) * g.nvar + (v < (uint32_t)g.nlev ? g.nlev - 1 - v : v);
}

// A node's class in FP64: a call, so that no FP64 instruction is run under a predicate for nodes
// that FP32 decides.
static __device__ __noinline__ int dvs_class_call(const double4_32a *node, double x, double y, double z, int lev, const DvsGeom &g) {
    const double c[3] = {x, y, z}, nc[3] = {node->x, node->y, node->z};
    return dvs_class(c, nc, node->w, g.radius[lev], g.maxd[lev], g);
}

// A node's class in FP32, in FP64 where that cannot tell.
struct NodeClass {
    const DevTreeView &tv;
    const FTree &ft;
    const DvsGeom &g;
    const DvsGeomF &gf;
    double c[3];
    float cf[3];
    int lev;
    __device__ int operator()(uint32_t n) const {
        const float4 h = ft.nhi[n];
        const float nf[3] = {h.x, h.y, h.z};
        const int cls = dvs_class_f(cf, nf, h.w, lev, gf);
        if (cls >= 0) return cls;
        return dvs_class_call(tv.t.ncf + n, c[0], c[1], c[2], lev, g);
    }
};

struct DvsWarp {
    uint32_t at;
    __device__ uint32_t lane() const { return at; }
    __device__ uint32_t load(const uint32_t *word) const { return *(volatile const uint32_t *)word; }
    __device__ uint32_t first(uint32_t v) const { return __shfl_sync(0xffffffffu, v, 0); }
    __device__ uint32_t sum(uint32_t v) const { return __reduce_add_sync(0xffffffffu, v); }
};

// Only the largest count of each radius is wanted, so most queries end without a look at a
// point: the points of contained nodes bound a query's count from below, those of the met
// leaves on top bound it from above, and a query whose upper bound does not exceed the largest
// count known is done. k_dvs<0> finds the largest lower bound over the cell centres (a seed for
// k_dvs<1>, whose first queries would otherwise have nothing to compare with); k_dvs<1> bounds
// every query and counts the points of the met leaves, in FP32 with the exact FP64 test where
// that is too close, for those left, until the bound drops to the largest count.
//
// A warp takes one query: its lanes classify up to 32 nodes of a last-in first-out list at a
// time, append the children of the met ones, and later share the points of the met leaves.
// Measured with the tree's build, 150,000 particles, 32 cells a side, 1.2 M queries: 12.8 ms. A
// thread per query took 87 ms (the few thousand node tests and tens of thousands of points of
// each large ball one at a time), FP64 throughout with every point counted 1,075 ms. What
// bounds it: the node tests of the large radii, whose bounds are too loose to stop before the
// points.
constexpr uint32_t kDvsList = 1024;    // nodes to classify, per warp
constexpr uint32_t kDvsLeaves = 1024;  // met leaves, per warp
constexpr int kDvsWarps = 4;

template <int kCount>
__global__ void __launch_bounds__(32 * kDvsWarps) k_dvs(DevTreeView tv, FTree ft, const double *xs, const double *ys, const double *zs,
                                                        const __grid_constant__ DvsGeom g, const __grid_constant__ DvsGeomF gf, uint64_t n,
                                                        unsigned long long *next, uint32_t *maxc, unsigned *err) {
    __shared__ uint32_t s_list[kDvsWarps][kDvsList], s_leaf[kDvsWarps][kDvsLeaves];
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, below = (1u << lane) - 1u;
    const unsigned full = 0xffffffffu;
    uint32_t *list = s_list[w], *leaves = s_leaf[w];
    for (;;) {
        unsigned long long at = 0;
        if (lane == 0) at = atomicAdd(next, 1ull);
        at = __shfl_sync(full, at, 0);
        if (at >= n) return;
        double x, y, z;
        int lev;
        dvs_query(g, xs, ys, zs, dvs_order(g, at), x, y, z, lev);
        const NodeClass classify{tv, ft, g, gf, {x, y, z}, {(float)x, (float)y, (float)z}, lev};
        uint32_t inside = 0, partial = 0;  // of the whole warp, the same in every lane
        uint32_t top = 1, nleaf = 0;
        auto count_leaves = [&](const uint32_t *largest) {
            const double r = g.radius[lev], rr = r * r;
            const float rr32 = (float)rr;
            const float4 qh = make_float4(classify.cf[0], classify.cf[1], classify.cf[2], 0.f);
            const float4 ql = make_float4((float)(x - (double)qh.x), (float)(y - (double)qh.y), (float)(z - (double)qh.z), 0.f);
            dvs_count_leaves(DvsWarp{lane}, tv, leaves, nleaf, largest, inside, partial, [&](uint32_t p) {
                const float v = f_dr2(qh, ql, ft.phi[p], ft.plo[p]);
                if (f_hi(v, ft.tol) < rr32 * (1.f - kRel)) return true;
                if (f_lo(v, ft.tol) > rr32 * (1.f + kRel)) return false;
                return point_within(tv.t.pos + p, x, y, z, rr);
            });
        };
        if (lane == 0) list[0] = 0;
        __syncwarp();
        while (top) {
            // near the end of the list one node at a time: each of the tree's levels then adds at
            // most seven more
            const uint32_t take = min(top, top > kDvsList / 2 ? 1u : 32u);
            const bool mine = lane < take;
            const uint32_t node = mine ? list[top - 1 - lane] : 0u;
            const int cls = mine ? classify(node) : 0;
            top -= take;
            const uint32_t nd = cls == 2 ? tv.daughters(node) : 0u;
            const bool leaf = cls == 2 && nd == 0;
            const uint32_t size = cls == 1 || leaf ? tv.end(node) - tv.begin(node) : 0u;
            inside += __reduce_add_sync(full, cls == 1 ? size : 0u);
            const unsigned lm = __ballot_sync(full, leaf);
            uint32_t incl = nd;
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(full, incl, d);
                if (lane >= (uint32_t)d) incl += o;
            }
            const uint32_t add = __shfl_sync(full, incl, 31);
            if (top + add > kDvsList) {  // a tree deeper than an octree of 32 levels can be
                if (lane == 0) atomicOr(err, (unsigned)kDevErrCapacity);
                return;
            }
            __syncwarp();
            for (uint32_t c = 0; c < nd; ++c) list[top + incl - nd + c] = tv.first(node) + c;
            top += add;
            if (lm) {
                partial += __reduce_add_sync(full, leaf ? size : 0u);
                if (kCount) {
                    if (nleaf + __popc(lm) > kDvsLeaves) {
                        count_leaves(nullptr);
                        nleaf = 0;
                        __syncwarp();
                        // the leaves of this step stay in partial: they are listed now
                    }
                    if (leaf) leaves[nleaf + __popc(lm & below)] = node;
                    nleaf += __popc(lm);
                }
            }
            __syncwarp();
        }
        if (kCount) count_leaves(&maxc[lev]);
        // a query that stopped early is not above the largest count: what it counted is a lower bound
        if (lane == 0 && inside > *(volatile uint32_t *)&maxc[lev]) atomicMax(&maxc[lev], inside);
        __syncwarp();
    }
}

__global__ void k_z_extent(const double4_32a *pos, uint32_t n, unsigned long long *ext) {
    // ext[0] = min, ext[1] = max of z, as order-preserving keys of the doubles
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const long long b = __double_as_longlong(pos[i].z);
    const unsigned long long key = b < 0 ? ~(unsigned long long)b : (unsigned long long)b | 0x8000000000000000ull;
    atomicMin(&ext[0], key);
    atomicMax(&ext[1], key);
}

double key_to_double(unsigned long long key) {
    const unsigned long long b = (key & 0x8000000000000000ull) ? (key & 0x7fffffffffffffffull) : ~key;
    double d;
    std::memcpy(&d, &b, 8);
    return d;
}

}  // namespace

int density_vs_scale(Context &c, const plan_params &p, double time, std::vector<double> &radii, std::vector<double> &rho, cudaStream_t s) {
    const DevTree &tr = c.tree;
    if (!tr.Tu || !tr.pos) return kErrArgument;
    // z extent of the tree points (RecursiveFindExtreme finds the extreme values exactly)
    StreamBuf<unsigned long long> d_ext(s);
    PLAN_CUDA(d_ext.alloc(2));
    const unsigned long long init[2] = {~0ull, 0ull};
    PLAN_CUDA(cudaMemcpyAsync(d_ext.p, init, 16, cudaMemcpyHostToDevice, s));
    k_z_extent<<<grid_for(tr.Tu, 256), 256, 0, s>>>(tr.pos, tr.Tu, d_ext.p);
    c.launches++;
    PLAN_CUDA(cudaGetLastError());
    unsigned long long ext[2];
    PLAN_CUDA(cudaMemcpyAsync(ext, d_ext.p, 16, cudaMemcpyDeviceToHost, s));
    PLAN_CUDA(cudaStreamSynchronize(s));
    DvsParams dp;
    for (int d = 0; d < 3; ++d) {
        dp.box_length[d] = p.box_length[d];
        dp.box_min[d] = p.box_min[d];
        dp.box_max[d] = p.box_max[d];
        dp.box_center[d] = p.box_center[d];
        dp.cell_length[d] = p.cell_length[d];
    }
    dp.box_half_width0 = p.box_half_width[0];
    dp.max_half_width = p.max_half_width;
    dp.shear_speed = p.shear_speed;
    dp.mass_per_particle0 = p.mass_per_particle[0];
    DvsGeom g;
    std::vector<double> xs, ys, zs;
    const int src = dvs_setup(dp, time, key_to_double(ext[0]), key_to_double(ext[1]), g, xs, ys, zs);
    if (src) {
        c.last_error = src == -1   ? "density vs scale: the grid gives more radii than supported"
                       : src == -2 ? "density vs scale: the points or the box need more than 2^24 cell centres along an axis"
                                   : "density vs scale: the grid has more queries than one launch can take";
        return kErrUnsupported;
    }
    std::vector<uint32_t> maxc(g.nlev, 0);
    const uint64_t nthreads = (uint64_t)g.nx * g.ny * g.nz * g.nvar;
    if (nthreads) {
        StreamBuf<double> d_x(s), d_y(s), d_z(s);
        StreamBuf<uint32_t> d_max(s);
        PLAN_CUDA(d_x.alloc(xs.size()));
        PLAN_CUDA(d_y.alloc(ys.size()));
        PLAN_CUDA(d_z.alloc(zs.size()));
        PLAN_CUDA(d_max.alloc(g.nlev));
        PLAN_CUDA(cudaMemcpyAsync(d_x.p, xs.data(), xs.size() * 8, cudaMemcpyHostToDevice, s));
        PLAN_CUDA(cudaMemcpyAsync(d_y.p, ys.data(), ys.size() * 8, cudaMemcpyHostToDevice, s));
        PLAN_CUDA(cudaMemcpyAsync(d_z.p, zs.data(), zs.size() * 8, cudaMemcpyHostToDevice, s));
        PLAN_CUDA(cudaMemsetAsync(d_max.p, 0, (size_t)g.nlev * 4, s));
        // the largest magnitude of a coordinate: the root box holds every node, the centres are their own
        double coord = 0;
        for (int d = 0; d < 3; ++d) coord = std::fmax(coord, std::fabs(tr.box.root_center[d]) + tr.box.half_width);
        for (const std::vector<double> *v : {&xs, &ys, &zs})
            if (!v->empty()) coord = std::fmax(coord, std::fmax(std::fabs(v->front()), std::fabs(v->back())) + g.sub1[0] + g.sub1[1] + g.sub1[2]);
        const DvsGeomF gf = dvs_geom_f(g, coord);
        const FTree ft = ftree_of(tr);
        const DevTreeView tv{ktree_of(tr)};
        const uint64_t ncentre = (uint64_t)g.nx * g.ny * g.nz * g.nlev;
        int sms = 152;
        cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
        auto blocks = [&](uint64_t queries) { return (unsigned)std::min<uint64_t>((queries + kDvsWarps - 1) / kDvsWarps, (uint64_t)sms * 6); };
        StreamBuf<unsigned long long> d_next(s);
        PLAN_CUDA(d_next.alloc(2));
        PLAN_CUDA(cudaMemsetAsync(d_next.p, 0, 16, s));
        k_dvs<0><<<blocks(ncentre), 32 * kDvsWarps, 0, s>>>(tv, ft, d_x.p, d_y.p, d_z.p, g, gf, ncentre, d_next.p, d_max.p, c.d_err);
        k_dvs<1><<<blocks(nthreads), 32 * kDvsWarps, 0, s>>>(tv, ft, d_x.p, d_y.p, d_z.p, g, gf, nthreads, d_next.p + 1, d_max.p, c.d_err);
        c.launches += 2;
        PLAN_CUDA(cudaGetLastError());
        PLAN_CUDA(cudaMemcpyAsync(maxc.data(), d_max.p, (size_t)g.nlev * 4, cudaMemcpyDeviceToHost, s));
        PLAN_CUDA(cudaStreamSynchronize(s));
    }
    radii.assign(g.radius, g.radius + g.nlev);
    rho.resize(g.nlev);
    for (int i = 0; i < g.nlev; ++i) rho[i] = dvs_density(maxc[i], g.radius[i], dp.mass_per_particle0);
    return kOk;
}

}  // namespace plan
