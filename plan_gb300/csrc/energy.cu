// Batched boundness of particle groups: kinetic and pairwise potential energy of every group
// in one pass over all of them.
//
// For a group with centre of mass x_c and velocity v_c,
//   E_kin = 1/2 sum_i m_i |v_c - s (x_c,x - x_i,x) - v_i|^2   (s = (0, q Omega, 0): the shear
//           correction of the reference's boundness test, src/tree.hpp:4657-4659)
//   E_pot = -G sum_{i<j} m_i m_j / |x_i - x_j|                 (no softening, as the reference)
// and the group is bound when E_kin + E_pot < 0.
//
// Kinetic terms and centres are FP64 sums, one block per group. The potential is the O(n^2)
// part: every group is cut into w x w tiles of pairs (the upper triangle, diagonal tiles
// included), w by the group's size class (energy_tiles.h: 32-wide tiles for groups of tens of
// particles, up to 128 or 256 for large ones), and per class a persistent grid of blocks takes
// items (a row tile and one to four column tiles) from one queue across that class's groups, so
// groups from tens to millions of particles share the GPU without a launch per group. A block
// stages w column particles at a time in shared memory; each thread sums the m_j / r_ij of its
// rows in FP32 with compensated (Neumaier) addition and multiplies by their m_i in FP64; the
// block adds the threads' sums in FP64 into the item's own slot, and one block per group adds
// its items' slots in order: the result does not depend on which block ran which item.
// Coincident pairs (r = 0) are left out and counted. The particles arrive as three plain arrays
// and are packed on the device.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "energy.cuh"
#include "pipeline.h"

namespace plan {

namespace {

__device__ __forceinline__ float rsqrt_fast(float x) {
    float r;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

__global__ void __launch_bounds__(256) k_group_kinetic(const float4 *pm, const float4 *vel, const uint64_t *off, uint32_t ngroups,
                                                       double shear_y, double *e_kin, double4_32a *com) {
    __shared__ double s[256][7];
    const uint32_t g = blockIdx.x;
    if (g >= ngroups) return;
    const uint64_t b = off[g], e = off[g + 1];
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};  // M, M x, M y, M z, M vx, M vy, M vz
    for (uint64_t i = b + threadIdx.x; i < e; i += blockDim.x) {
        const float4 p = pm[i], v = vel[i];
        const double m = p.w;
        acc[0] += m;
        acc[1] += m * (double)p.x;
        acc[2] += m * (double)p.y;
        acc[3] += m * (double)p.z;
        acc[4] += m * (double)v.x;
        acc[5] += m * (double)v.y;
        acc[6] += m * (double)v.z;
    }
    for (int k = 0; k < 7; ++k) s[threadIdx.x][k] = acc[k];
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h)
            for (int k = 0; k < 7; ++k) s[threadIdx.x][k] += s[threadIdx.x + h][k];
        __syncthreads();
    }
    const double M = s[0][0];
    // an empty (or massless) group has no centre: zeros, and no kinetic energy below
    const double xc = M > 0.0 ? s[0][1] / M : 0.0, yc = M > 0.0 ? s[0][2] / M : 0.0, zc = M > 0.0 ? s[0][3] / M : 0.0;
    const double vx = M > 0.0 ? s[0][4] / M : 0.0, vy = M > 0.0 ? s[0][5] / M : 0.0, vz = M > 0.0 ? s[0][6] / M : 0.0;
    __syncthreads();
    double ek = 0;
    for (uint64_t i = b + threadIdx.x; i < e; i += blockDim.x) {
        const float4 p = pm[i], v = vel[i];
        const double dx = vx - (double)v.x;
        const double dy = vy - shear_y * (xc - (double)p.x) - (double)v.y;
        const double dz = vz - (double)v.z;
        ek += 0.5 * (double)p.w * (dx * dx + dy * dy + dz * dz);
    }
    s[threadIdx.x][0] = ek;
    __syncthreads();
    for (int h = blockDim.x / 2; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) s[threadIdx.x][0] += s[threadIdx.x + h][0];
        __syncthreads();
    }
    if (threadIdx.x == 0) {
        e_kin[g] = s[0][0];
        com[g] = make_double4_32a(xc, yc, zc, M);
    }
}

// *odd is set where a mass is negative or not a number (the pair sums then compare magnitudes).
__global__ void k_pack(const float *pos3, const float *vel3, const float *mass, uint64_t n, float4 *pm, float4 *vel, unsigned long long *odd) {
    const uint64_t i = (uint64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    if (!(mass[i] >= 0.f)) *odd = 1;
    pm[i] = make_float4(pos3[3 * i], pos3[3 * i + 1], pos3[3 * i + 2], mass[i]);
    vel[i] = make_float4(vel3[3 * i], vel3[3 * i + 1], vel3[3 * i + 2], 0.f);
}

// One row against W staged columns: m_q / r per column in FP32, added with the exact error of
// every addition kept (the larger of the two operands first, as Neumaier's branch does, by
// minimum and maximum). kDiag: the columns after the row's own only. A coincident pair makes the
// sum infinite or not a number, which the caller looks for once per row.
template <int W, int R, bool kDiag>
__device__ __forceinline__ void rows_against(const float4 *col, const float (&x)[R], const float (&y)[R], const float (&z)[R], float (&s)[R],
                                             float (&c)[R]) {
    constexpr int kThreads = W / R;
#pragma unroll 8
    for (int k = 0; k < W; ++k) {
        const float4 q = col[k];
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const float dx = x[j] - q.x, dy = y[j] - q.y, dz = z[j] - q.z;
            // (not fused: the squares' roundings and the reciprocal root's bias lean opposite ways)
            const float d2 = dx * dx + dy * dy + dz * dz;
            float term = q.w * rsqrt_fast(d2);
            if (kDiag) term = k > (int)threadIdx.x + j * kThreads ? term : 0.f;
            const float t = s[j] + term;
            c[j] += fminf(s[j], term) - (t - fmaxf(s[j], term));
            s[j] = t;
        }
    }
}

// The items of one size class: groups glist[0, ng), their queue items item_off (by list
// position); each item's FP64 sum goes to part[item]. W / R threads, R rows each (thread t: rows
// t, t + W/R, ...), so that a staged column is loaded once for R pairs.
//
// What bounds it: instructions per pair, 16 in FP32 with the compensated sum and one reciprocal
// root, at one instruction a cycle and scheduler. 5,000 groups of 32 to 20,000 particles, 7.8e10
// pairs, with the copies: 111 -> 43.7 ms against the loop of one row a thread with a branch for the
// larger operand and a test for coincident pairs. Fused squares: 40 ms, but the energies' error
// against FP64 grows from 5.6e-9 to 6.0e-9. Packed pairs of floats (f32x2) take two cycles an
// instruction and gain nothing.
template <int W, int R>
__global__ void __launch_bounds__(W / R) k_pair_tiles(const float4 *pm, const uint64_t *off, const uint32_t *glist, const uint64_t *item_off,
                                                      uint32_t ng, uint64_t nitems, unsigned long long *next, double *part,
                                                      unsigned long long *zero_pairs, const unsigned long long *odd) {
    constexpr int kThreads = W / R, kWarps = kThreads / 32;
    __shared__ float4 col[W];
    __shared__ double red[kWarps];
    __shared__ unsigned long long s_item;
    const int tid = threadIdx.x;
    const bool careful = *odd != 0;
    while (true) {
        if (tid == 0) s_item = atomicAdd(next, 1ull);
        __syncthreads();
        const uint64_t item = s_item;
        if (item >= nitems) return;
        // the group: last list position k with item_off[k] <= item
        uint32_t lo = 0, hi = ng;
        while (hi - lo > 1) {
            const uint32_t mid = (lo + hi) / 2;
            if (item_off[mid] <= item) lo = mid;
            else hi = mid;
        }
        const uint32_t g = glist[lo];
        const uint64_t b = off[g], n = off[g + 1] - b, T = (n + W - 1) / W;
        uint64_t ti, tj, te;
        strip_of_item(item - item_off[lo], T, ti, tj, te);
        float x[R], y[R], z[R], m[R], s[R], c[R];
        bool have[R];
#pragma unroll
        for (int j = 0; j < R; ++j) {
            const uint64_t r = ti * W + tid + j * kThreads;
            have[j] = r < n;
            const float4 q = have[j] ? pm[b + r] : make_float4(-1e18f, -1e18f, -1e18f, 0.f);
            x[j] = q.x; y[j] = q.y; z[j] = q.z; m[j] = q.w;
            s[j] = 0.f;
            c[j] = 0.f;
        }
        for (uint64_t t = tj; t < te; ++t) {
            __syncthreads();
#pragma unroll
            for (int j = 0; j < R; ++j) {
                const uint64_t k = t * W + tid + j * kThreads;  // past the end: far away, without mass
                col[tid + j * kThreads] = k < n ? pm[b + k] : make_float4(1e18f, 1e18f, 1e18f, 0.f);
            }
            __syncthreads();
            float s0[R], c0[R];
#pragma unroll
            for (int j = 0; j < R; ++j) {
                s0[j] = s[j];
                c0[j] = c[j];
            }
            if (careful) {
            } else if (t == ti) {
                rows_against<W, R, true>(col, x, y, z, s, c);
            } else {
                rows_against<W, R, false>(col, x, y, z, s, c);
            }
#pragma unroll
            for (int j = 0; j < R; ++j) {
                if (!have[j] || (!careful && s[j] < INFINITY && c[j] == c[j])) continue;
                // a coincident pair in this row: once more, leaving such pairs out and counting them
                const uint32_t cn = (uint32_t)(n - t * W < (uint64_t)W ? n - t * W : (uint64_t)W);
                uint32_t zeros = 0;
                s[j] = s0[j];
                c[j] = c0[j];
                pair_row_sum(PairParticle{x[j], y[j], z[j], m[j]}, reinterpret_cast<const PairParticle *>(col), cn,
                             t == ti ? tid + j * kThreads : -1, s[j], c[j], zeros);
                if (zeros) atomicAdd(zero_pairs, (unsigned long long)zeros);
            }
        }
        double sum = 0.0;
#pragma unroll
        for (int j = 0; j < R; ++j)
            if (have[j]) sum += (double)m[j] * ((double)s[j] + (double)c[j]);
#pragma unroll
        for (int d = 16; d > 0; d >>= 1) sum += __shfl_down_sync(0xffffffffu, sum, d);
        if (kWarps > 1) {
            if ((tid & 31) == 0) red[tid >> 5] = sum;
            __syncthreads();
            if (tid == 0)
                for (int w = 1; w < kWarps; ++w) sum += red[w];
        }
        if (tid == 0) part[item] = sum;
        __syncthreads();
    }
}

// One block per group: the sum of its tiles' slots part[base, base + count) in a fixed order
// (strided partial sums, then a tree of fixed shape).
__global__ void __launch_bounds__(256) k_group_pot(const double *part, const uint64_t *base, const uint64_t *count, uint32_t ngroups,
                                                   double *sum) {
    __shared__ double red[256];
    const uint32_t g = blockIdx.x;
    if (g >= ngroups) return;
    double a = 0.0;
    for (uint64_t k = threadIdx.x; k < count[g]; k += blockDim.x) a += part[base[g] + k];
    red[threadIdx.x] = a;
    __syncthreads();
    for (int h = 128; h > 0; h >>= 1) {
        if ((int)threadIdx.x < h) red[threadIdx.x] += red[threadIdx.x + h];
        __syncthreads();
    }
    if (threadIdx.x == 0) sum[g] = red[0];
}

template <int W, int R>
int launch_tiles(const float4 *pm, const uint64_t *off, const uint32_t *glist, const uint64_t *item_off, uint32_t ng, uint64_t nitems,
                 unsigned long long *next, double *part, unsigned long long *zeros, const unsigned long long *odd, int sms, cudaStream_t s) {
    int per = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per, k_pair_tiles<W, R>, W / R, 0);
    const unsigned grid = (unsigned)std::min<uint64_t>((uint64_t)sms * (per > 0 ? per : 1), nitems);
    k_pair_tiles<W, R><<<grid, W / R, 0, s>>>(pm, off, glist, item_off, ng, nitems, next, part, zeros, odd);
    return cudaGetLastError() == cudaSuccess ? kOk : kErrDevice;
}

}  // namespace

// The tile width of each size class: the measured table, or PLAN_ENERGY_TILES ("w0,w1,w2,w3").
static void energy_tiles(int w[kEnergyClasses]) {
    for (int k = 0; k < kEnergyClasses; ++k) w[k] = kEnergyTile[k];
    const char *e = std::getenv("PLAN_ENERGY_TILES");
    if (!e) return;
    int v[kEnergyClasses], k = 0;
    const char *p = e;
    while (k < kEnergyClasses && *p) {
        char *end = nullptr;
        const long x = std::strtol(p, &end, 10);
        if (end == p || !energy_tile_ok((int)x)) return;
        v[k++] = (int)x;
        p = *end == ',' ? end + 1 : end;
    }
    if (k == kEnergyClasses)
        for (int j = 0; j < kEnergyClasses; ++j) w[j] = v[j];
}

// A batch's workspace up to this size (17 million particles) stays in the context. An allocation of
// its own makes the first pass of a batch of 15 million 0.6 ms longer (43.8 -> 44.4 ms; 4 ms where it
// is the process's first) and the others no longer.
constexpr size_t kEnergyKept = 1u << 30;

int group_energies(Context &c, const float *pos3, const float *vel3, const float *mass, const uint64_t *offsets, uint32_t ngroups, double G,
                   double shear_y, double *e_kin, double *e_pot, uint64_t *zero_pairs, cudaStream_t s) {
    if (ngroups == 0) return kOk;
    for (uint32_t g = 0; g < ngroups; ++g)
        if (offsets[g + 1] < offsets[g]) return kErrArgument;
    const uint64_t n = offsets[ngroups];
    int w[kEnergyClasses];
    energy_tiles(w);
    // per class: its groups in order, their queue items; per group: where its tiles' slots are
    std::vector<uint32_t> glist[kEnergyClasses];
    for (uint32_t g = 0; g < ngroups; ++g) glist[energy_class(offsets[g + 1] - offsets[g])].push_back(g);
    std::vector<uint64_t> iofs[kEnergyClasses], gbase(ngroups, 0), gcount(ngroups, 0);
    uint64_t cbase[kEnergyClasses + 1] = {0};
    for (int k = 0; k < kEnergyClasses; ++k) {
        iofs[k].assign(glist[k].size() + 1, 0);
        for (size_t j = 0; j < glist[k].size(); ++j) {
            const uint32_t g = glist[k][j];
            const uint64_t T = (offsets[g + 1] - offsets[g] + w[k] - 1) / w[k];
            iofs[k][j + 1] = iofs[k][j] + strip_items(T);
            gbase[g] = cbase[k] + iofs[k][j];
            gcount[g] = iofs[k][j + 1] - iofs[k][j];
        }
        cbase[k + 1] = cbase[k] + iofs[k][glist[k].size()];
    }
    const uint64_t nitems = cbase[kEnergyClasses];
    // One workspace: the tables (and a small batch's particles) go up in one
    // copy, the results come back in one. Fifteen stream-ordered allocations and eight copies cost
    // a batch of 16 small groups two thirds of its 189 us.
    struct Layout {
        size_t at = 0;
        size_t take(size_t bytes) {
            const size_t o = at;
            at = (at + bytes + 255) & ~size_t(255);
            return o;
        }
    } lay;
    const size_t o_off = lay.take((ngroups + 1) * 8ull), o_items = lay.take((ngroups + kEnergyClasses) * 8ull), o_gbase = lay.take(ngroups * 8ull),
                 o_gcount = lay.take(ngroups * 8ull), o_gl = lay.take((ngroups + 1) * 4ull);
    const size_t o_next = lay.take((kEnergyClasses + 1) * 8);  // one queue per class, the odd-mass flag
    const size_t tables = lay.at;
    const size_t o_p3 = lay.take(12 * n), o_v3 = lay.take(12 * n), o_m = lay.take(4 * n), particles = lay.at;
    const size_t o_pm = lay.take(16 * n), o_v = lay.take(16 * n), o_part = lay.take(8 * nitems), o_com = lay.take(32ull * ngroups);
    const size_t o_ek = lay.take(8ull * ngroups), o_sum = lay.take(8ull * ngroups), o_zeros = lay.take(8), results = lay.at - o_ek;
    // the context's scratch, which stays with it, for small batches and wherever it is large enough
    // already; a larger batch gives its memory back
    StreamBuf<char> own(s);
    char *d;
    if (lay.at <= std::max(kEnergyKept, c.scratch.cap)) {
        if (c.ensure(c.scratch, lay.at)) return kErrOutOfMemory;
        d = c.scratch.base;
    } else {
        PLAN_CUDA(own.alloc(lay.at));
        d = own.p;
    }
    const bool together = particles - tables <= (1u << 20);
    std::vector<char> up(together ? particles : tables, 0);
    std::memcpy(up.data() + o_off, offsets, (ngroups + 1) * 8ull);
    std::memcpy(up.data() + o_gbase, gbase.data(), ngroups * 8ull);
    std::memcpy(up.data() + o_gcount, gcount.data(), ngroups * 8ull);
    size_t gl_at[kEnergyClasses], io_at[kEnergyClasses], gl_n = 0, io_n = 0;
    for (int k = 0; k < kEnergyClasses; ++k) {
        gl_at[k] = gl_n;
        io_at[k] = io_n;
        std::memcpy(up.data() + o_gl + 4 * gl_n, glist[k].data(), glist[k].size() * 4);
        std::memcpy(up.data() + o_items + 8 * io_n, iofs[k].data(), iofs[k].size() * 8);
        gl_n += glist[k].size();
        io_n += iofs[k].size();
    }
    if (together && n) {
        std::memcpy(up.data() + o_p3, pos3, 12 * n);
        std::memcpy(up.data() + o_v3, vel3, 12 * n);
        std::memcpy(up.data() + o_m, mass, 4 * n);
    }
    PLAN_CUDA(cudaMemcpyAsync(d, up.data(), up.size(), cudaMemcpyHostToDevice, s));
    if (!together) {
        PLAN_CUDA(cudaMemcpyAsync(d + o_p3, pos3, 12 * n, cudaMemcpyHostToDevice, s));
        PLAN_CUDA(cudaMemcpyAsync(d + o_v3, vel3, 12 * n, cudaMemcpyHostToDevice, s));
        PLAN_CUDA(cudaMemcpyAsync(d + o_m, mass, 4 * n, cudaMemcpyHostToDevice, s));
    }
    PLAN_CUDA(cudaMemsetAsync(d + o_zeros, 0, 8, s));
    const uint64_t *d_off = reinterpret_cast<const uint64_t *>(d + o_off), *d_items = reinterpret_cast<const uint64_t *>(d + o_items);
    const uint64_t *d_gbase = reinterpret_cast<const uint64_t *>(d + o_gbase), *d_gcount = reinterpret_cast<const uint64_t *>(d + o_gcount);
    const uint32_t *d_gl = reinterpret_cast<const uint32_t *>(d + o_gl);
    unsigned long long *d_next = reinterpret_cast<unsigned long long *>(d + o_next), *d_odd = d_next + kEnergyClasses;
    unsigned long long *d_zeros = reinterpret_cast<unsigned long long *>(d + o_zeros);
    float4 *d_pm = reinterpret_cast<float4 *>(d + o_pm), *d_v = reinterpret_cast<float4 *>(d + o_v);
    double *d_part = reinterpret_cast<double *>(d + o_part), *d_ek = reinterpret_cast<double *>(d + o_ek), *d_sum = reinterpret_cast<double *>(d + o_sum);
    if (n) {
        k_pack<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(reinterpret_cast<const float *>(d + o_p3), reinterpret_cast<const float *>(d + o_v3),
                                                           reinterpret_cast<const float *>(d + o_m), n, d_pm, d_v, d_odd);
        c.launches++;
    }
    k_group_kinetic<<<ngroups, 256, 0, s>>>(d_pm, d_v, d_off, ngroups, shear_y, d_ek, reinterpret_cast<double4_32a *>(d + o_com));
    c.launches++;
    int sms = 152;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, c.device);
    for (int k = 0; k < kEnergyClasses; ++k) {
        const uint64_t ni = cbase[k + 1] - cbase[k];
        if (!ni) continue;
        const uint32_t ng = (uint32_t)glist[k].size();
        const uint32_t *gl = d_gl + gl_at[k];
        const uint64_t *io = d_items + io_at[k];
        double *part = d_part + cbase[k];
        int rc = kErrArgument;
        switch (w[k]) {
            case 32: rc = launch_tiles<32, 1>(d_pm, d_off, gl, io, ng, ni, d_next + k, part, d_zeros, d_odd, sms, s); break;
            case 64: rc = launch_tiles<64, 2>(d_pm, d_off, gl, io, ng, ni, d_next + k, part, d_zeros, d_odd, sms, s); break;
            case 128: rc = launch_tiles<128, 2>(d_pm, d_off, gl, io, ng, ni, d_next + k, part, d_zeros, d_odd, sms, s); break;
            case 256: rc = launch_tiles<256, 4>(d_pm, d_off, gl, io, ng, ni, d_next + k, part, d_zeros, d_odd, sms, s); break;
        }
        if (rc) return rc;
        c.launches++;
    }
    k_group_pot<<<ngroups, 256, 0, s>>>(d_part, d_gbase, d_gcount, ngroups, d_sum);
    c.launches++;
    PLAN_CUDA(cudaGetLastError());
    std::vector<char> down(results);
    PLAN_CUDA(cudaMemcpyAsync(down.data(), d + o_ek, results, cudaMemcpyDeviceToHost, s));
    PLAN_CUDA(cudaStreamSynchronize(s));
    std::memcpy(e_kin, down.data(), ngroups * 8ull);
    const double *sum = reinterpret_cast<const double *>(down.data() + (o_sum - o_ek));
    unsigned long long zeros = 0;
    std::memcpy(&zeros, down.data() + (o_zeros - o_ek), 8);
    for (uint32_t g = 0; g < ngroups; ++g) e_pot[g] = -G * sum[g];
    if (zero_pairs) *zero_pairs = zeros;
    return kOk;
}

}  // namespace plan
