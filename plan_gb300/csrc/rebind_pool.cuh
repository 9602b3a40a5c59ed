// Room in the member pool for the clumps of the rebinding loop. Included inside the namespace, after
// Pool and pool_try_alloc (the CPU tests bring their own).
#pragma once

// A clump's room in the member pool besides its members: the capacity of its present segment
// (0 where the host packed it), the segment it left last and the sort buffers. Calls go back and
// forth between two segments that grow by half, so a launch needs a few times the members
// instead of a segment per call, and the pool does not fill up: a launch that stops for a
// compaction costs the blocks that wait for one another their order.
struct RbSeg {
    uint32_t cap, spare, spare_cap, buf, buf_cap;
};

// room for n entries, half as many on top where the pool has them (cap: what was taken)
__device__ __forceinline__ uint32_t rb_alloc(const Pool &P, uint32_t n, uint32_t &cap) {
    cap = n + n / 2;
    uint32_t o = cap > n ? pool_try_alloc(P, cap) : kNone;
    if (o == kNone) {
        cap = n;
        o = pool_try_alloc(P, n);
    }
    return o;
}

// the segment a clump left last, or a new one in its place, with room for n entries
__device__ __forceinline__ uint32_t rb_spare(const Pool &P, RbSeg &g, uint32_t n) {
    if (g.spare_cap >= n) return g.spare;
    uint32_t cap;
    const uint32_t o = rb_alloc(P, n, cap);
    if (o != kNone) {
        g.spare = o;
        g.spare_cap = cap;
    }
    return o;
}

// the members moved from the present segment at o to the spare one
__device__ __forceinline__ void rb_switch(RbSeg &g, uint32_t o) {
    const uint32_t cap = g.cap;
    g.cap = g.spare_cap;
    g.spare = o;
    g.spare_cap = cap;
}

// room for the sort of m members: the spare segment for the sorted pairs and 2 m + 1 entries for the
// records. Where both are missing they are taken at once, so that the first of them never takes on
// top what the second needs: a sort whose bare needs fit always finds room.
__device__ __forceinline__ bool rb_sort_room(const Pool &P, RbSeg &g, uint32_t m) {
    const uint32_t records = 2 * m + 1;
    uint32_t cap;
    if (g.spare_cap < m && g.buf_cap < records) {
        const uint32_t o = rb_alloc(P, m + records, cap);
        if (o == kNone) return false;
        g.spare = o;
        g.spare_cap = m + (cap - m - records) / 3;
        g.buf = o + g.spare_cap;
        g.buf_cap = cap - g.spare_cap;
        return true;
    }
    if (rb_spare(P, g, m) == kNone) return false;
    if (g.buf_cap < records) {
        const uint32_t o = rb_alloc(P, records, cap);
        if (o == kNone) return false;
        g.buf = o;
        g.buf_cap = cap;
    }
    return true;
}
