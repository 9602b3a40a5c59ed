// Stable LSD radix sort of 96-bit keys (three u32 words) with a u32 payload.
//
// One sort primitive serves three uses: Morton keys (src/tree.hpp:2831), the HOP group
// order (root, first-visit index, chain position) and per-clump distance orders
// (clump slot, distance bits). 8-bit digits, 12 passes at most; a pre-pass computes all
// twelve digit histograms in one read and passes whose digit is constant are skipped.
//
// A pass is bound by HBM: it reads and writes every 16-byte record once (and reads it once more
// for the tile counts). Each pass is reduce-then-scan over tiles of 4,096: per-tile digit counts,
// a per-digit scan over tiles, and a stable scatter that first orders the tile by digit in shared
// memory, so that a digit's records leave as one run (16 records on average: four separate words
// per key, scattered 32 lanes to 32 digits, took 0.38 ms per pass of 14 M keys; this 0.19 ms).
// Keys travel as records of three words and the payload; the first pass reads the separate
// arrays and the last writes them.
//
// Where the caller expects few keys with equal upper words (Morton keys, distances), large sorts
// leave the lowest word out (from kLowAt keys, where four passes cost more than the run kernel
// and its answer): an insertion sort per run of equal upper words finishes the order; a run
// longer than kLowRun sends the whole sort through all twelve digits instead.
// Up to one tile, one block sorts in shared memory (36 launches otherwise).
#include "sort.h"

#include <algorithm>
#include <cstdio>

namespace plan {

namespace {

constexpr int kThreads = 512;
constexpr int kWarps = kThreads / 32;
constexpr int kItems = 8;
constexpr int kTile = kThreads * kItems;  // keys per tile
constexpr int kRadix = 256;
constexpr size_t kLowAt = 1u << 18;       // keys from which the lowest word is left to the runs
constexpr uint32_t kLowRun = 16;

__device__ __forceinline__ uint32_t word_of(const uint4 &r, int word) { return word == 0 ? r.x : (word == 1 ? r.y : r.z); }

// Where the keys of a pass are: four arrays, or records (rec not null).
struct Keys {
    uint32_t *w0, *w1, *w2, *pay;
    uint4 *rec;
    __device__ __forceinline__ uint4 get(size_t i) const { return rec ? rec[i] : make_uint4(w0[i], w1[i], w2[i], pay[i]); }
    __device__ __forceinline__ uint32_t word(size_t i, int k) const {
        if (rec) return reinterpret_cast<const uint32_t *>(rec + i)[k];
        return k == 0 ? w0[i] : (k == 1 ? w1[i] : w2[i]);
    }
    __device__ __forceinline__ void put(size_t i, const uint4 &r) const {
        if (rec) {
            rec[i] = r;
        } else {
            w0[i] = r.x;
            w1[i] = r.y;
            w2[i] = r.z;
            pay[i] = r.w;
        }
    }
};

// All 12 digit histograms in one pass over the keys.
__global__ void k_hist_all(const uint32_t *w0, const uint32_t *w1, const uint32_t *w2, size_t n, unsigned long long *hist /*12*256*/) {
    __shared__ unsigned int s[12 * kRadix];
    for (int j = threadIdx.x; j < 12 * kRadix; j += blockDim.x) s[j] = 0;
    __syncthreads();
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) {
        uint32_t a = w0[i], b = w1[i], c = w2[i];
        for (int k = 0; k < 4; ++k) {
            atomicAdd(&s[(0 + k) * kRadix + ((a >> (8 * k)) & 0xff)], 1u);
            atomicAdd(&s[(4 + k) * kRadix + ((b >> (8 * k)) & 0xff)], 1u);
            atomicAdd(&s[(8 + k) * kRadix + ((c >> (8 * k)) & 0xff)], 1u);
        }
    }
    __syncthreads();
    for (int j = threadIdx.x; j < 12 * kRadix; j += blockDim.x)
        if (s[j]) atomicAdd(&hist[j], (unsigned long long)s[j]);
}

// Per-tile digit counts: counts[digit * ntiles + tile].
__global__ void __launch_bounds__(kThreads) k_tile_counts(Keys in, size_t n, int pass, uint32_t *counts, int ntiles) {
    __shared__ unsigned int s[kRadix];
    for (int j = threadIdx.x; j < kRadix; j += blockDim.x) s[j] = 0;
    __syncthreads();
    const size_t base = (size_t)blockIdx.x * kTile + threadIdx.x;
    uint32_t v[kItems];
#pragma unroll
    for (int r = 0; r < kItems; ++r) v[r] = base + r * kThreads < n ? in.word(base + r * kThreads, pass >> 2) : 0u;
#pragma unroll
    for (int r = 0; r < kItems; ++r)
        if (base + r * kThreads < n) atomicAdd(&s[(v[r] >> (8 * (pass & 3))) & 0xffu], 1u);
    __syncthreads();
    for (int j = threadIdx.x; j < kRadix; j += blockDim.x) counts[(size_t)j * ntiles + blockIdx.x] = s[j];
}

// Exclusive scan of counts[digit][*] over tiles plus the digit's global base.
// One block per digit.
__global__ void k_scan_tiles(uint32_t *counts, int ntiles, const unsigned long long *digit_base) {
    __shared__ uint32_t warp_sums[32];
    __shared__ uint32_t carry;
    int d = blockIdx.x;
    uint32_t *row = counts + (size_t)d * ntiles;
    if (threadIdx.x == 0) carry = (uint32_t)digit_base[d];
    __syncthreads();
    for (int start = 0; start < ntiles; start += blockDim.x) {
        int t = start + threadIdx.x;
        uint32_t v = t < ntiles ? row[t] : 0;
        // inclusive warp scan
        uint32_t x = v;
        int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
        for (int o = 1; o < 32; o <<= 1) {
            uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) warp_sums[warp] = x;
        __syncthreads();
        if (warp == 0) {
            int nw = blockDim.x / 32;
            uint32_t w = lane < nw ? warp_sums[lane] : 0;
            for (int o = 1; o < 32; o <<= 1) {
                uint32_t y = __shfl_up_sync(0xffffffffu, w, o);
                if (lane >= o) w += y;
            }
            if (lane < nw) warp_sums[lane] = w;
        }
        __syncthreads();
        uint32_t prefix = x - v + (warp > 0 ? warp_sums[warp - 1] : 0) + carry;
        if (t < ntiles) row[t] = prefix;
        __syncthreads();
        if (threadIdx.x == blockDim.x - 1) carry = prefix + v;
        __syncthreads();
    }
}

// Orders a tile's items (8 per thread in r, warp w holding items [256 w, 256 w + 256) round by
// round) by digit into shared memory, stably: a warp's counters rank its items as it reads them,
// a scan over (digit, warp) places them. start[d]: where digit d begins in the tile.
__device__ __forceinline__ void tile_order(const uint4 (&r)[kItems], int cnt, int pass, uint4 *stage, uint32_t (*wcnt)[kRadix], uint32_t *start,
                                           uint32_t *warp_sums) {
    const uint32_t lane = threadIdx.x & 31, w = threadIdx.x >> 5, full = 0xffffffffu;
    for (int j = threadIdx.x; j < kWarps * kRadix; j += kThreads) (&wcnt[0][0])[j] = 0;
    __syncthreads();
    uint32_t rank[kItems], dig[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const int i = (int)(w * (32 * kItems) + k * 32 + lane);
        const uint32_t d = i < cnt ? (word_of(r[k], pass >> 2) >> (8 * (pass & 3))) & 0xffu : (uint32_t)kRadix;
        const uint32_t peers = __match_any_sync(full, d), before = __popc(peers & ((1u << lane) - 1u));
        const uint32_t off = d < kRadix ? wcnt[w][d] : 0u;
        __syncwarp();
        if (d < kRadix && before == 0) wcnt[w][d] = off + __popc(peers);
        __syncwarp();
        rank[k] = off + before;
        dig[k] = d;
    }
    __syncthreads();
    uint32_t total = 0;
    if (threadIdx.x < kRadix) {
        for (int v = 0; v < kWarps; ++v) {
            const uint32_t c = wcnt[v][threadIdx.x];
            wcnt[v][threadIdx.x] = total;
            total += c;
        }
        uint32_t incl = total;
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(full, incl, o);
            if (lane >= (uint32_t)o) incl += y;
        }
        if (lane == 31) warp_sums[w] = incl;
        start[threadIdx.x] = incl - total;
    }
    __syncthreads();
    if (threadIdx.x < kRadix) {
        uint32_t add = 0;
        for (uint32_t v = 0; v < w; ++v) add += warp_sums[v];
        start[threadIdx.x] += add;
    }
    __syncthreads();
#pragma unroll
    for (int k = 0; k < kItems; ++k)
        if (dig[k] < kRadix) stage[start[dig[k]] + wcnt[w][dig[k]] + rank[k]] = r[k];
    __syncthreads();
}

constexpr size_t kTileSmem = (size_t)kTile * 16 + (size_t)kWarps * kRadix * 4 + kRadix * 4 + 64;

struct TileShared {
    uint4 *stage;
    uint32_t (*wcnt)[kRadix];
    uint32_t *start, *warp_sums;
    __device__ explicit TileShared(unsigned char *p, int stages = 1) {
        stage = reinterpret_cast<uint4 *>(p);
        wcnt = reinterpret_cast<uint32_t(*)[kRadix]>(p + (size_t)kTile * 16 * stages);
        start = &wcnt[0][0] + kWarps * kRadix;
        warp_sums = start + kRadix;
    }
};

// Stable scatter of one tile.
__global__ void __launch_bounds__(kThreads) k_scatter(Keys in, Keys out, size_t n, int pass, const uint32_t *counts, int ntiles) {
    extern __shared__ __align__(16) unsigned char dyn[];
    const TileShared sh(dyn);
    const size_t base = (size_t)blockIdx.x * kTile;
    const int cnt = (int)min((size_t)kTile, n - base);
    uint4 r[kItems];
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const int i = (int)((threadIdx.x >> 5) * (32 * kItems) + k * 32 + (threadIdx.x & 31));
        r[k] = i < cnt ? in.get(base + i) : make_uint4(0, 0, 0, 0);
    }
    tile_order(r, cnt, pass, sh.stage, sh.wcnt, sh.start, sh.warp_sums);
    // the counters are free: where a digit's run goes, less where it starts in the tile
    uint32_t *to = &sh.wcnt[0][0];
    if (threadIdx.x < kRadix) to[threadIdx.x] = counts[(size_t)threadIdx.x * ntiles + blockIdx.x] - sh.start[threadIdx.x];
    __syncthreads();
    for (int j = threadIdx.x; j < cnt; j += kThreads) {
        const uint4 v = sh.stage[j];
        out.put((size_t)(to[(word_of(v, pass >> 2) >> (8 * (pass & 3))) & 0xffu] + (uint32_t)j), v);
    }
}

// At most one tile: every pass in one block.
__global__ void __launch_bounds__(kThreads) k_sort_tile(Keys io, int n, unsigned pass_mask) {
    extern __shared__ __align__(16) unsigned char dyn[];
    const TileShared sh(dyn);
    __shared__ uint32_t s_or[3], s_and[3];
    if (threadIdx.x < 3) {
        s_or[threadIdx.x] = 0;
        s_and[threadIdx.x] = 0xffffffffu;
    }
    __syncthreads();
    uint4 r[kItems];
    uint32_t o[3] = {0, 0, 0}, a[3] = {0xffffffffu, 0xffffffffu, 0xffffffffu};
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const int i = (int)((threadIdx.x >> 5) * (32 * kItems) + k * 32 + (threadIdx.x & 31));
        r[k] = i < n ? io.get(i) : make_uint4(0, 0, 0, 0);
        if (i < n) {
            o[0] |= r[k].x; o[1] |= r[k].y; o[2] |= r[k].z;
            a[0] &= r[k].x; a[1] &= r[k].y; a[2] &= r[k].z;
        }
    }
    for (int k = 0; k < 3; ++k) {
        o[k] = __reduce_or_sync(0xffffffffu, o[k]);
        a[k] = __reduce_and_sync(0xffffffffu, a[k]);
        if ((threadIdx.x & 31) == 0) {
            atomicOr(&s_or[k], o[k]);
            atomicAnd(&s_and[k], a[k]);
        }
    }
    __syncthreads();
    for (int pass = 0; pass < 12; ++pass) {
        const uint32_t differ = (s_or[pass >> 2] ^ s_and[pass >> 2]) >> (8 * (pass & 3)) & 0xffu;
        if (!((pass_mask >> pass) & 1u) || !differ) continue;
        tile_order(r, n, pass, sh.stage, sh.wcnt, sh.start, sh.warp_sums);
#pragma unroll
        for (int k = 0; k < kItems; ++k) {
            const int i = (int)((threadIdx.x >> 5) * (32 * kItems) + k * 32 + (threadIdx.x & 31));
            if (i < n) r[k] = sh.stage[i];
        }
        __syncthreads();
    }
#pragma unroll
    for (int k = 0; k < kItems; ++k) {
        const int i = (int)((threadIdx.x >> 5) * (32 * kItems) + k * 32 + (threadIdx.x & 31));
        if (i < n) io.put(i, r[k]);
    }
}

// records back into the arrays
__global__ void k_unrecord(const uint4 *rec, size_t n, Keys out) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i < n) out.put(i, rec[i]);
}

// Runs of equal upper words ordered by the lowest (stable); *too_long where one has more than
// kLowRun keys (it is then left as it is).
__global__ void k_low_runs(uint32_t *w0, const uint32_t *w1, const uint32_t *w2, uint32_t *pay, size_t n, uint32_t *too_long) {
    const size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x;
    if (i + 1 >= n) return;
    const uint32_t a = w1[i], b = w2[i];
    if (w1[i + 1] != a || w2[i + 1] != b || (i > 0 && w1[i - 1] == a && w2[i - 1] == b)) return;
    size_t e = i + 2;
    while (e < n && e - i <= kLowRun && w1[e] == a && w2[e] == b) ++e;
    if (e - i > kLowRun) {
        *too_long = 1;
        return;
    }
    for (size_t j = i + 1; j < e; ++j) {
        const uint32_t v = w0[j], p = pay[j];
        size_t k = j;
        while (k > i && w0[k - 1] > v) {
            w0[k] = w0[k - 1];
            pay[k] = pay[k - 1];
            --k;
        }
        w0[k] = v;
        pay[k] = p;
    }
}

}  // namespace

size_t radix_sort96_scratch_bytes(size_t n) {
    const size_t ntiles = (n + kTile - 1) / kTile;
    return 2 * n * sizeof(uint4) +                         // ping-pong records
           (size_t)kRadix * ntiles * sizeof(uint32_t) +    // tile counts
           12 * kRadix * sizeof(unsigned long long) + 4096;  // histograms
}

static int sort_tile(uint32_t *w0, uint32_t *w1, uint32_t *w2, uint32_t *payload, size_t n, cudaStream_t stream, unsigned pass_mask) {
    PLAN_CUDA(cudaFuncSetAttribute(k_sort_tile, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmem));
    k_sort_tile<<<1, kThreads, kTileSmem, stream>>>(Keys{w0, w1, w2, payload, nullptr}, (int)n, pass_mask);
    PLAN_CUDA(cudaGetLastError());
    return kOk;
}

int radix_sort96(uint32_t *w0, uint32_t *w1, uint32_t *w2, uint32_t *payload, size_t n, void *scratch, size_t scratch_bytes,
                 cudaStream_t stream, unsigned pass_mask, bool few_low, uint64_t *launched) {
    uint64_t ignored = 0;
    uint64_t &count = launched ? *launched : ignored;
    if (n <= 1) return kOk;
    if (scratch_bytes < radix_sort96_scratch_bytes(n)) return kErrArgument;
    if (n <= (size_t)kTile) {
        ++count;
        return sort_tile(w0, w1, w2, payload, n, stream, pass_mask);
    }
    const size_t ntiles = (n + kTile - 1) / kTile;
    char *p = reinterpret_cast<char *>((reinterpret_cast<uintptr_t>(scratch) + 255) & ~uintptr_t(255));
    uint4 *rec[2];
    rec[0] = reinterpret_cast<uint4 *>(p); p += n * sizeof(uint4);
    rec[1] = reinterpret_cast<uint4 *>(p); p += n * sizeof(uint4);
    unsigned long long *hist = reinterpret_cast<unsigned long long *>((reinterpret_cast<uintptr_t>(p) + 255) & ~uintptr_t(255));
    uint32_t *counts = reinterpret_cast<uint32_t *>(hist + 12 * kRadix), *too_long = counts + (size_t)kRadix * ntiles;

    PLAN_CUDA(cudaFuncSetAttribute(k_scatter, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTileSmem));
    PLAN_CUDA(cudaMemsetAsync(hist, 0, 12 * kRadix * sizeof(unsigned long long), stream));
    const int hblocks = (int)std::min<size_t>((n + 255) / 256, 152 * 8);
    k_hist_all<<<hblocks, 256, 0, stream>>>(w0, w1, w2, n, hist);
    ++count;
    PLAN_CUDA(cudaGetLastError());
    unsigned long long h_hist[12 * kRadix];
    PLAN_CUDA(cudaMemcpyAsync(h_hist, hist, sizeof(h_hist), cudaMemcpyDeviceToHost, stream));
    PLAN_CUDA(cudaStreamSynchronize(stream));
    // digit bases (exclusive prefix per pass), uploaded in place of the histogram
    unsigned long long h_base[12 * kRadix];
    unsigned skip = ~pass_mask;
    for (int pass = 0; pass < 12; ++pass) {
        unsigned long long run = 0;
        for (int d = 0; d < kRadix; ++d) {
            const unsigned long long c = h_hist[pass * kRadix + d];
            if (c == n) skip |= 1u << pass;
            h_base[pass * kRadix + d] = run;
            run += c;
        }
    }
    PLAN_CUDA(cudaMemcpyAsync(hist, h_base, sizeof(h_base), cudaMemcpyHostToDevice, stream));
    auto passes = [&](unsigned left_out) -> int {
        const Keys arrays{w0, w1, w2, payload, nullptr};
        Keys src = arrays;
        int last = -1, side = 0;
        for (int pass = 0; pass < 12; ++pass)
            if (!((left_out >> pass) & 1u)) last = pass;
        bool first = true;
        for (int pass = 0; pass < 12; ++pass) {
            if ((left_out >> pass) & 1u) continue;
            // the only pass cannot write what it reads: through the records
            Keys dst{nullptr, nullptr, nullptr, nullptr, rec[side]};
            if (pass == last && !first) dst = arrays;
            k_tile_counts<<<(int)ntiles, kThreads, 0, stream>>>(src, n, pass, counts, (int)ntiles);
            k_scan_tiles<<<kRadix, 1024, 0, stream>>>(counts, (int)ntiles, hist + pass * kRadix);
            k_scatter<<<(int)ntiles, kThreads, kTileSmem, stream>>>(src, dst, n, pass, counts, (int)ntiles);
            PLAN_CUDA(cudaGetLastError());
            count += 3;
            src = dst;
            side ^= 1;
            first = false;
        }
        if (src.rec) {
            k_unrecord<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(src.rec, n, arrays);
            ++count;
            PLAN_CUDA(cudaGetLastError());
        }
        return kOk;
    };
    const bool runs = few_low && n >= kLowAt && (~skip & 0x00fu) && (~skip & 0xff0u);
    int rc = passes(skip | (runs ? 0x00fu : 0u));
    if (rc || !runs) return rc;
    PLAN_CUDA(cudaMemsetAsync(too_long, 0, 4, stream));
    k_low_runs<<<(unsigned)((n + 255) / 256), 256, 0, stream>>>(w0, w1, w2, payload, n, too_long);
    ++count;
    PLAN_CUDA(cudaGetLastError());
    uint32_t h_long = 0;
    PLAN_CUDA(cudaMemcpyAsync(&h_long, too_long, 4, cudaMemcpyDeviceToHost, stream));
    PLAN_CUDA(cudaStreamSynchronize(stream));
    return h_long ? passes(skip) : kOk;
}

}  // namespace plan
