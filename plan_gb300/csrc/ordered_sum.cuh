// Sequential FP64 sums, exactly as a loop would round them, 256 terms at a time.
//
// The reference accumulates member sums one term at a time (s = s + x[k], round to nearest
// even each time), and the clump catalogue must keep those bits. On this GPU a dependent FP64
// add waits 64 cycles (measured), so a loop over 100,000 members takes 3 ms. A warp evaluates
// the same recurrence in integers, without walking the terms one by one:
//
//  * Step k rounds s + x[k] onto the grid of the binade it lands in, u_k = 2^(e_k - 52). Which
//    binade that is follows from an unrounded prefix sum (64-bit integers, every term
//    truncated to a common unit): it is off by less than 2^16 units, so e_k is certain unless
//    the prefix comes that close to a power of two.
//  * Where the sum before the step lies on a grid at least as coarse (e_{k-1} >= e_k) and
//    x[k] / u_k is no tie, the step adds x[k] rounded to u_k, whatever the sum is. Such steps
//    are integer additions, and prefix sums give them all at once.
//  * A step into a higher binade, or a tie, also depends on the sum's low bits. Those steps
//    (one in seven where velocities hover around zero, one in a hundred or fewer where masses
//    and positions add up) are listed and walked in order: five dependent 32-bit operations
//    each, on the low 32 bits of the sum in units of a quarter of the finest grid. The terms
//    of these steps are rounded to odd there, which keeps every later rounding.
//  * The sum after the last term is known modulo 2^64 of those units from the additions and
//    the corrections of the listed steps, and its leading bits from the unrounded prefix.
//
// A chunk where a binade is uncertain (or the sum is exactly zero, tiny, huge or not finite, or
// spans more than 20 binades) is added term by term.
//
// What bounds it: instruction latency, of some 600 integer instructions per warp and chunk and
// two scans, then 34 cycles per listed step. Measured per chunk of 256 terms, seven sums in
// seven warps of one SM: 4,700 to 6,000 cycles (none to 67 listed steps) against 16,400 for the
// loop of FP64 adds. Eight terms per lane: fewer leave the scans' latency to fewer terms, more
// do not fit the registers.
#pragma once

#include <cstdint>

#include "exact64.cuh"

namespace plan {

constexpr int kSumK = 8;                          // consecutive terms per lane
constexpr uint32_t kSumChunk = 32 * kSumK;        // terms of a staged chunk
constexpr uint32_t kSumRow = kSumK + 2;           // a lane's terms, padded: 16-byte loads of 8 lanes meet no bank twice
constexpr uint32_t kSumStage = 32 * kSumRow;      // doubles per staged chunk
constexpr int kSumSpan = 20;                      // binades the sum may span in a chunk: 256 2^21 < 2^31

// where term k of a chunk is staged
__device__ __forceinline__ uint32_t sum_slot(uint32_t k) { return (k / kSumK) * kSumRow + k % kSumK; }

__device__ __forceinline__ void sum_load_row(const double *src, uint32_t row, double (&x)[kSumK]) {
    const double2 *p = reinterpret_cast<const double2 *>(src + row * kSumRow);
#pragma unroll
    for (int j = 0; j < kSumK / 2; ++j) {
        const double2 v = p[j];
        x[2 * j] = v.x;
        x[2 * j + 1] = v.y;
    }
}

__device__ __forceinline__ long long sum_scan(long long v, uint32_t lane) {  // inclusive, over the warp
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const long long o = __shfl_up_sync(0xffffffffu, v, d);
        if (lane >= (uint32_t)d) v += o;
    }
    return v;
}

// The sum after the chunk at src (terms at sum_slot(k)) is added to s, or false where that
// takes the term-by-term loop. src: on a 16-byte boundary. list: kSumChunk entries of this warp;
// their two-entry loads start on a 16-byte boundary wherever the list itself does.
__device__ __forceinline__ bool sum_chunk_int(const double *src, double &s, uint2 *list) {
    const uint32_t lane = threadIdx.x & 31;
    const unsigned full = 0xffffffffu;
    uint64_t x[kSumK];  // the terms' bits: no FP64 instruction here
    {
        const ulonglong2 *p = reinterpret_cast<const ulonglong2 *>(src + lane * kSumRow);
#pragma unroll
        for (int j = 0; j < kSumK / 2; ++j) {
            const ulonglong2 v = p[j];
            x[2 * j] = v.x;
            x[2 * j + 1] = v.y;
        }
    }
    const uint64_t sb = dbits(s);
    const uint32_t es = (uint32_t)(sb >> 52) & 0x7ffu;
    if (es == 0 && sb != 0) return false;
    // the largest exponent, and whether the lane has a term that is not zero
    uint32_t mx = 0, any = 0;
#pragma unroll
    for (int j = 0; j < kSumK; ++j) {
        const uint32_t hi = (uint32_t)(x[j] >> 32) & 0x7fffffffu;
        mx = max(mx, hi);
        any |= hi | (uint32_t)x[j];
    }
    const unsigned some = __ballot_sync(full, any != 0);
    if (!some) return true;  // adding zeros leaves s (which is never -0)
    mx = max(__reduce_max_sync(full, mx) >> 20, es);
    const uint32_t eb = mx + 9;  // |any partial sum| < 2^(eb - 1023): at most 257 terms below 2^(mx - 1022)
    if (eb > 2000 || mx < 100) return false;
    // terms before the first that is not zero do nothing to s = +0
    uint32_t start = 0, skip = 0;
    if (sb == 0) {
        uint32_t nz = kSumK;
#pragma unroll
        for (int j = kSumK - 1; j >= 0; --j)
            if ((((uint32_t)(x[j] >> 32) & 0x7fffffffu) | (uint32_t)x[j]) != 0) nz = j;
        start = (uint32_t)(__ffs(some) - 1);
        skip = lane < start ? (uint32_t)kSumK : lane == start ? nz : 0u;
    }
    // unrounded prefix sums in units of 2^(eb - 1084): a term's 53 bits shifted right
    auto unit = [&](uint64_t b) -> long long {
        const uint32_t e = (uint32_t)(b >> 52) & 0x7ffu;
        const uint32_t r = min(eb - 9 - e, 63u);
        const long long v = (long long)(((b & 0xfffffffffffffull) | (1ull << 52)) >> r);
        return (b >> 63) ? -v : v;
    };
    long long pre[kSumK];
    {
        long long run = 0;
#pragma unroll
        for (int j = 0; j < kSumK; ++j) {
            run += unit(x[j]);
            pre[j] = run;
        }
        const long long before = sum_scan(run, lane) - run + (es ? unit(sb) : 0ll);
#pragma unroll
        for (int j = 0; j < kSumK; ++j) pre[j] += before;
    }
    // the binade after each step, as its bit in units (biased exponent eb - 61 + bit)
    constexpr long long kTol = 1ll << 16;
    bool sure = true;
    uint32_t bit[kSumK], lo = 63, hi = 0;
#pragma unroll
    for (int j = 0; j < kSumK; ++j) {
        // |prefix| to one unit; below and above it by the tolerance, the leading bit is the same
        // where their difference stays below the smaller
        const uint64_t m = (uint64_t)(pre[j] ^ (pre[j] >> 63)), under = m - kTol, over = m + kTol;
        const uint32_t h = (uint32_t)(m >> 32);
        bit[j] = (h ? 63u : 31u) - (uint32_t)__clz((int)(h ? h : (uint32_t)m));
        const bool use = (uint32_t)j >= skip;
        sure = sure && (!use || (m > 2 * kTol && (under ^ over) < under));
        lo = min(lo, use ? bit[j] : 63u);
        hi = max(hi, use ? bit[j] : 0u);
    }
    lo = __reduce_min_sync(full, lo);
    hi = __reduce_max_sync(full, hi);
    const uint32_t sbit = es ? es + 61u - eb : 63u;  // s's own binade (wraps below the unit: refused)
    if (es) {
        lo = min(lo, sbit);
        hi = max(hi, sbit);
    }
    if (!__all_sync(full, sure) || hi > 62 || hi - lo > (uint32_t)kSumSpan || eb - 61 + lo <= 60) return false;
    // steps: additions in units of a quarter of the finest grid, 2^(emin - 1077). A term there
    // is rounded to odd where it has bits below the units; the low word then says how it
    // rounds to the grid of its step (bit d), and whether that is a tie.
    const int emin = (int)(eb - 61 + lo);
    uint32_t prev = __shfl_up_sync(full, bit[kSumK - 1], 1);
    if (lane == 0) prev = sbit;
    uint64_t q[kSumK];
    uint32_t listed = 0;
    {
        uint64_t run = 0;
#pragma unroll
        for (int j = 0; j < kSumK; ++j) {
            const uint64_t b = x[j];
            const uint32_t ex = (uint32_t)(b >> 52) & 0x7ffu;
            const uint64_t mant = (b & 0xfffffffffffffull) | (uint64_t)(ex ? 1u : 0u) << 52;
            const int sh = (int)max(ex, 1u) - emin + 2;  // the term's last bit in those units
            const uint32_t up = (uint32_t)min(max(sh, 0), 63), dn = (uint32_t)min(max(-sh, 0), 63);
            const uint64_t down = mant >> dn;
            uint64_t fine = (down << up) | (uint64_t)(down << dn != mant ? 1u : 0u);
            if (sh > 63) fine = 0;
            const uint32_t one = 1u << (bit[j] - lo + 2), low = (uint32_t)fine & (one - 1);  // its grid's bit
            const bool use = (uint32_t)j >= skip;
            const bool first = sb == 0 && lane == start && (uint32_t)j == skip;  // s = 0 before it: exact
            const bool special = use && ((bit[j] > prev && !first) || low == one >> 1);
            const uint64_t near = (fine + (one >> 1)) & ~(uint64_t)(one - 1);
            const uint64_t mag = use ? (special ? fine : near) : 0ull;
            listed |= special ? 1u << j : 0u;
            prev = use ? bit[j] : prev;
            run += (b >> 63) ? 0ull - mag : mag;
            q[j] = run;
        }
        const uint64_t incl = (uint64_t)sum_scan((long long)run, lane);
        // s is a multiple of its own grid, which is not finer than the units' grid
        const uint64_t smant = (sb & 0xfffffffffffffull) | (1ull << 52);
        const uint64_t s0 = es ? smant << (sbit - lo + 2) : 0ull;
        const uint64_t before = incl - run + ((sb >> 63) ? 0ull - s0 : s0);
#pragma unroll
        for (int j = 0; j < kSumK; ++j) q[j] += before;
    }
    // the listed steps in order: their place among them from ballots
    uint32_t place = 0, count = 0;
#pragma unroll
    for (int j = 0; j < kSumK; ++j) {
        const unsigned m = __ballot_sync(full, (listed >> j) & 1u);
        place += __popc(m & ((1u << lane) - 1u));
        count += __popc(m);
    }
    uint32_t c = 0;  // the listed steps' corrections so far: each at most half a grid bit, so below 2^30 in all
    if (count) {
#pragma unroll
        for (int j = 0; j < kSumK; ++j)
            if ((listed >> j) & 1u) {
                const uint32_t one = 1u << (bit[j] - lo + 2);
                list[place++] = make_uint2((uint32_t)q[j] + (one >> 1), one - 1);
            }
        __syncwarp();
        // round half to even at the grid's bit: with half of it added, clear below it, and on a
        // tie (nothing left below) the bit itself
        auto step = [&](uint32_t x, uint32_t m) {
            const uint32_t v = x + c, low = v & m;
            uint32_t w = v - low;
            if (low == 0) w &= ~(m + 1);
            c = w - (x - ((m >> 1) + 1));
        };
        uint32_t i = 0;
        if (reinterpret_cast<uintptr_t>(list) & 8) {
            step(list[0].x, list[0].y);
            i = 1;
        }
        for (; i + 4 <= count; i += 4) {
            const uint4 e0 = *reinterpret_cast<const uint4 *>(list + i), e1 = *reinterpret_cast<const uint4 *>(list + i + 2);
            step(e0.x, e0.y);
            step(e0.z, e0.w);
            step(e1.x, e1.y);
            step(e1.z, e1.w);
        }
        for (; i < count; ++i) step(list[i].x, list[i].y);
        __syncwarp();
    }
    const uint64_t n = __shfl_sync(full, q[kSumK - 1], 31) + (uint64_t)(long long)(int)c;
    const long long a = __shfl_sync(full, pre[kSumK - 1], 31);
    const uint32_t lb = __shfl_sync(full, bit[kSumK - 1], 31), d = lb - lo + 2;
    // s / u_last: its leading bits from the prefix (off by less than 2^(68 - lb) + 1), the others exactly
    if (lb < d + 7) return false;
    const long long lead = lb > 52 ? a >> (lb - 52) : a << (52 - lb);
    const long long diff = (long long)(((uint64_t)((long long)n >> d) - (uint64_t)lead) << d) >> d;
    s = grid_value(lead + diff, eb - 61 + lb);
    return true;
}

// Adds one staged chunk to the running sum of this warp (the same value in every lane; it
// starts at +0, and terms past the end of the members are staged as +0). loops counts the
// chunks taken term by term.
__device__ __forceinline__ void ordered_sum_chunk(const double *src, double &s, uint2 *list, uint32_t *loops = nullptr) {
    if (sum_chunk_int(src, s, list)) return;
    if (loops) ++*loops;
    double y[kSumK], z[kSumK];
    sum_load_row(src, 0, y);
    for (uint32_t k = 0; k < 32; ++k) {
        sum_load_row(src, k < 31 ? k + 1 : k, z);
#pragma unroll
        for (int j = 0; j < kSumK; ++j) s = s + y[j];
#pragma unroll
        for (int j = 0; j < kSumK; ++j) y[j] = z[j];
    }
}

}  // namespace plan
