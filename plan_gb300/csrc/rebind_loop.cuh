// Hill-sphere rebinding with every clump's calls on the device (src/tree.hpp:4196-4208).
//
// The reference runs, clump by clump in key order,
//     do { SearchBoundParticlesWithinHillRadius; CalculateHillRadius; } while (it grew)
// where a call that accepts anything ends with SortParticles (src/tree.hpp:4678-4711,
// 4446-4512, 4715-4717). k_rebind_loop runs that whole loop for a clump inside one block:
// a persistent grid (one 512-thread block per SM) takes clumps from a queue in key-rank
// order, so the host is involved once per pass, not once per call. Clumps of one launch run
// concurrently under the ordered-claim rule of the round kernel (owner / tent / defer
// records); a clump may first wait for the lower-ranked clumps it met in the previous pass
// (its blockers). Those were taken from the queue before it by running blocks, so every
// wait ends; each wait is bounded all the same and reports kDevErrLoopLimit if it runs out.
//
// On this GPU an FP64 instruction holds the SM's FP64 pipe for ~19 cycles whatever the
// number of active lanes, and a dependent one waits 36-55 cycles (a division ~590, a square
// root ~630), so the loop keeps FP64 work off its chains:
//  * ball search: the breadth-first frontier of the round kernel, then one block-wide pass
//    over the eligible points of every frontier entry (a contained node keeps all of them,
//    a boundary node keeps those in the ball), compacted in point order;
//  * acceptance: 512 candidates at a time, one per thread in registers (the next 512
//    prefetched meanwhile). Every thread tests its candidate against the current state in
//    FP32 (FP64 when too close to call), the block finds the first bound one, and warp 0
//    applies the reference's FP64 updates from it on, 32 candidates at a time: the updates of
//    those bound on entry back to back, then all tests at once. The division of an update is a
//    reciprocal product with Markstein's correction, the reciprocals taken off the chain;
//  * SortParticles: the seven member sums in member order (ordered_sum_chunk over per-point
//    products m, m x, ..., m vz formed once per snapshot, 256 members at a time, the next
//    ones staged meanwhile), the centre of mass and the Hill radius,
//    squared distances, and a stable sort by squared distance (a block radix sort on the
//    leading bits and an exact fix-up of equal keys; in shared memory up to kRbSmall members). Squared distances order members as distances do, except that two
//    squared distances may round to one distance: neighbours within a few ulps are compared
//    through their square roots, and a tie goes to the library-order replay exactly as in
//    the round kernels. The square roots of the last sort are taken when the loop ends.
#pragma once

constexpr int kRB = 512;                      // threads of a rebinding block
constexpr int kRbWarps = kRB / 32;
constexpr uint32_t kRbFront = 4096;           // frontier entries of the ball search
constexpr uint32_t kRbSmall = 2048;           // members sorted in shared memory
constexpr uint32_t kRbOnePass = 512;          // members sorted by one digit
// Updates of a window up to which the lanes share the splitting of its states: with 6 to a window
// (1,048,576 particles of the benchmark's mixture) a window takes 5,700 cycles instead of 7,200,
// with 27 (524,288) 1% more than with a lane splitting the seven values it needs.
constexpr uint32_t kRbFewStates = 12;
constexpr uint32_t kWaitLimit = 1u << 25;     // bounded waits on blockers: sleeps of 1 us per 2^24 points
constexpr uint32_t kCallLimit = 1u << 20;     // calls of one clump in one launch
constexpr int kRbStats = 40;                  // counters per slot
constexpr int kCk = 24;                       // checkpoints per clump and run
// digit of the member sort: two passes order 22 bits of the squared distances' range, which
// leaves runs of one or two members to the insertion sort
constexpr uint32_t kRbDigit = 11;
constexpr size_t kRbRadixBytes = ((size_t)kRbWarps << kRbDigit) * 4;  // a counter per digit and warp
// dynamic shared memory, reused by every phase: the frontier, the acceptance tile (per
// candidate: FP64 position and velocity, index, FP32 form), the stage of the sums, and the
// largest, the sort's counters with the records and sorted pairs of a small clump
constexpr size_t kRbTileBytes = (size_t)kRB * (64 + 4 + sizeof(CandF));
constexpr size_t kRbSmem = kRbRadixBytes + (size_t)kRbSmall * 28;
static_assert(kRbFront * 14 <= kRbSmem, "frontier");
static_assert(kRbTileBytes <= kRbSmem, "acceptance tile");

// Checkpoints of the clumps' runs, by key rank: after the calls ck_after() selects, the
// sorted member list (index, squared distance) and the state (M, centre, velocity, Hill
// radius). A rerun resumes from the last checkpoint before its first affected call.
struct Ckpt {
    uint32_t *n;          // per rank: checkpoints kept
    uint32_t *call, *off, *m;  // per rank x kCk: after which call, where in the store, members
    double *st;           // per rank x kCk: M, cx, cy, cz, vx, vy, vz, hill
    uint32_t *idx;        // the store (bump-allocated; a checkpoint that finds it full is not made)
    double *dist;
    uint32_t *top;
    uint32_t cap;
};

// calls 1, 2, 3, 4, 6, 8, 12, 16, 24, 32, ...: a rerun redoes at most a third of the calls
// before its first affected one
__host__ __device__ inline bool ck_after(uint32_t j) {
    if ((j & (j - 1)) == 0) return true;
    return j % 3 == 0 && ((j / 3) & (j / 3 - 1)) == 0;
}

#include "rebind_pool.cuh"

struct RbArgs {
    const uint32_t *list;  // clumps of this launch, in key-rank order
    uint32_t n;
    uint32_t *head;        // next queue position
    const uint32_t *blk_off, *blk;  // blockers of list[i]: blk[blk_off[i], blk_off[i+1]) (slots); null: none
    uint8_t *finished;     // per slot: its calls are done in this launch (or it is not in it)
    uint8_t *suspended;    // per slot: stopped because the member pool is full (state consistent)
    uint8_t *needsort;     // per slot: the last call grew the clump but its SortParticles is pending
    uint8_t *distsq;       // per slot: the segment's distances are still squared
    unsigned long long *stats;  // per slot, kRbStats counters (may be null)
    CT ct;
    Pool P;
    KTree t;
    FTree ft;
    const double4_32a *vel;
    const double4_32a *tm0, *tm1;  // per point: (m, m x, m y, m z), (m vx, m vy, m vz, 0)
    const uint32_t *E;
    const uint2 *enode;    // per node: its slice of the eligible points E
    uint32_t *owner;
    const uint32_t *rank_of, *slot_of_rank, *tent;
    uint32_t *dmax, *dset;
    uint8_t *dover;
    const double4_32a *com0;
    unsigned long long *reach;
    CP cp;
    unsigned *err;
    uint32_t wait_limit;   // sleeps a block waits for one blocker before it reports an error
    uint32_t *ccall;       // per slot: calls of the clump's run done (persists across launches)
    uint32_t *dcall, *dfirst;  // per deferral record / per slot: the earliest call that made it
    Ckpt ck;               // ck.n null: no checkpoints
    RbSeg *seg;            // per slot, zero at the start of a launch
    float xtop;            // the largest magnitude of a coordinate in the root box
    const uint32_t *vtop;  // of a velocity component: its upper 32 bits
};

// per-point products for the member sums (src/tree.hpp:4436-4440: mass, pos * mass,
// vel * mass, each component rounded once)
// *vtop (zero before): the upper 32 bits of the largest velocity component's magnitude.
__global__ void __launch_bounds__(256) k_member_terms(uint32_t Tu, const double4_32a *pos, const double4_32a *vel, double4_32a *tm0, double4_32a *tm1,
                                                      uint32_t *vtop) {
    __shared__ uint32_t s_top;
    if (threadIdx.x == 0) s_top = 0;
    __syncthreads();
    const uint32_t q = blockIdx.x * blockDim.x + threadIdx.x;
    uint32_t top = 0;
    if (q < Tu) {
        const double4_32a p = pos[q], v = vel[q];
        tm0[q] = make_double4_32a(p.w, p.x * p.w, p.y * p.w, p.z * p.w);
        tm1[q] = make_double4_32a(v.x * p.w, v.y * p.w, v.z * p.w, 0.0);
        top = max(max((uint32_t)(dbits(v.x) >> 32) & 0x7fffffffu, (uint32_t)(dbits(v.y) >> 32) & 0x7fffffffu),
                  (uint32_t)(dbits(v.z) >> 32) & 0x7fffffffu);
    }
    top = __reduce_max_sync(0xffffffffu, top);
    if ((threadIdx.x & 31) == 0) atomicMax(&s_top, top);
    __syncthreads();
    if (threadIdx.x == 0 && s_top > *(volatile uint32_t *)vtop) atomicMax(vtop, s_top);
}

// (calls, so that no FP64 instruction is run under a predicate where it is not needed)
static __device__ __noinline__ float2 split_call(double x) {
    float2 s;
    split_f(x, s.x, s.y);
    return s;
}

static __device__ __noinline__ bool equal_roots(double a, double b) { return sqrt(a) == sqrt(b); }

__device__ __forceinline__ void split_any(double x, float &h, float &l) {
    if (!split_hilo_bits(x, h, l)) {
        const float2 s = split_call(x);
        h = s.x;
        l = s.y;
    }
}

// block-wide compaction offset of this thread's flag; returns the block total
__device__ __forceinline__ uint32_t rb_block_rank(bool keep, uint32_t &rank, uint32_t *warp_tot) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const unsigned b = __ballot_sync(0xffffffffu, keep);
    if (lane == 0) warp_tot[wid] = __popc(b);
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (int w = 0; w < kRbWarps; ++w) {
        const uint32_t c = warp_tot[w];
        if (w < wid) before += c;
        total += c;
    }
    rank = before + __popc(b & ((1u << lane) - 1u));
    __syncthreads();
    return total;
}

// exclusive scan of a[0, n) in shared memory by the whole block; returns the total
__device__ uint32_t rb_scan_excl(uint32_t *a, uint32_t n, uint32_t *warp_tot) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const uint32_t per = (n + kRB - 1) / kRB;
    const uint32_t b = threadIdx.x * per, e = min(n, b + per);
    uint32_t sum = 0;
    for (uint32_t i = b; i < e; ++i) sum += a[i];
    uint32_t incl = sum;
    for (int d = 1; d < 32; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, incl, d);
        if (lane >= d) incl += v;
    }
    if (lane == 31) warp_tot[wid] = incl;
    __syncthreads();
    uint32_t before = 0, total = 0;
    for (int k = 0; k < kRbWarps; ++k) {
        if (k < wid) before += warp_tot[k];
        total += warp_tot[k];
    }
    uint32_t run = before + incl - sum;
    for (uint32_t i = b; i < e; ++i) {
        const uint32_t v = a[i];
        a[i] = run;
        run += v;
    }
    __syncthreads();
    return total;
}

// per node, its slice of the eligible points (epos: eligible points below a point)
__global__ void k_node_slices(uint32_t nodes, const uint32_t *nbeg, const uint32_t *nend, const uint32_t *epos, uint2 *enode) {
    const uint32_t n = blockIdx.x * blockDim.x + threadIdx.x;
    if (n < nodes) enode[n] = make_uint2(epos[nbeg[n]], epos[nend[n]]);
}

// ball_class with the node's slice at hand
__device__ __forceinline__ int rb_class(const KTree &t, const FTree &f, uint2 e, uint32_t node, const BallQ &b) {
    const float4 nh = f.nhi[node], nl = f.nlo[node];
    if (e.x == e.y) return 3;
    const int cont = f_contained(nh, nl, b.qh, b.ql, b.rf, f.tol);
    if (cont > 0) return 1;
    int inter = f_intersects(nh, nl, b.qh, b.ql, b.rf, f.tol);
    if (cont < 0 || inter < 0) {
        const int c = node_class(t.ncf + node, b.cx, b.cy, b.cz, b.r);
        if (c == 1) return 1;
        inter = c;
    }
    if (inter) return t.nnd[node] == 0 ? 2 : 4;
    return 3;
}

struct RbShared {
    unsigned char *buf;  // kRbSmem bytes, reused by every phase
    uint32_t *warp_tot;
    uint32_t *u;         // scalars
    double *st;          // M, com x y z, vcom x y z, hill (the call's starting state)
    double *sums;        // the member sums
    double *tk;          // a window's updates: per acceptance m x .. m vz, M', 1 / M'
    double *hist;        // the states of a window: x y z vx vy vz M, before it and after each update
    float *histf;        // the states of a window as float pairs: hi of the seven, lo of the seven
    float *sf;           // acceptance state for every thread: hi[6], lo[6], Mf
    double *sd;          // acceptance state in FP64: x y z vx vy vz M
};

// ------------------------------------------------------------------ one SearchBound call
// Returns the number of accepted particles, or kNone when the member pool is full (nothing
// changed).
__device__ uint32_t rb_call(const RbArgs &a, uint32_t slot, uint32_t myrank, RbShared &sh, unsigned long long *stat, uint32_t call) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint32_t *front = reinterpret_cast<uint32_t *>(sh.buf), *front2 = front + kRbFront, *fcnt = front2 + kRbFront;
    uint8_t *fcls = reinterpret_cast<uint8_t *>(fcnt + kRbFront), *fcls2 = fcls + kRbFront;
    uint32_t &s_nf = sh.u[0], &s_noff = sh.u[2], &s_nel = sh.u[3], &s_f = sh.u[4], &s_m0 = sh.u[5],
             &s_o = sh.u[6], &s_S = sh.u[7];
    uint32_t *s_cnt = sh.u + 20;  // per warp, four counts
    const long long t0 = clock64();
    if (tid == 0) {
        const double4_32a c = a.ct.com[slot], v = a.ct.vcom[slot];
        sh.st[0] = a.ct.M[slot];
        sh.st[1] = c.x; sh.st[2] = c.y; sh.st[3] = c.z;
        sh.st[4] = v.x; sh.st[5] = v.y; sh.st[6] = v.z;
        sh.st[7] = a.ct.hill[slot];
        s_m0 = a.ct.mn[slot];
        s_o = a.ct.moff[slot];
        s_nel = 0;
        const double4_32a c0 = a.com0[slot];  // how far this clump's balls reach from its centre before rebinding
        const double dx = c.x - c0.x, dy = c.y - c0.y, dz = c.z - c0.z;
        const double d = sqrt(dx * dx + dy * dy + dz * dz) + sh.st[7];
        if (d >= 0) atomicMax(&a.reach[slot], (unsigned long long)__double_as_longlong(d));
    }
    __syncthreads();
    const BallQ ball = make_ball(sh.st[1], sh.st[2], sh.st[3], sh.st[7]);
    const KTree &t = a.t;
    // 1) breadth-first frontier (classes 1..4; 0 = not yet classified): the levels of at most 32
    // entries by warp 0 alone, without block barriers; then 512 entries at a time, one per
    // thread, from one half of the buffer to the other. A level costs the latency of its node
    // loads, so a node's slice of eligible points is stored per node (enode).
    if (wid == 0) {
        uint32_t nf = 1, node = 0;
        int cls = 0;
        for (int level = 0; level < 40; ++level) {
            if ((uint32_t)lane < nf && cls == 0) {
                if (node >= t.nodes) {
                    atomicOr(a.err, (unsigned)kDevErrBadNode);
                    cls = 3;
                } else {
                    cls = rb_class(t, a.ft, a.enode[node], node, ball);
                }
            }
            const bool down = (uint32_t)lane < nf && cls == 4;
            if (!__any_sync(0xffffffffu, down)) break;
            const uint32_t c0 = down ? t.nfd[node] : 0u, n = (uint32_t)lane >= nf || cls == 3 ? 0u : (down ? t.nnd[node] : 1u);
            uint32_t incl = n;
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += o;
            }
            const uint32_t total = __shfl_sync(0xffffffffu, incl, 31);
            if (total > 32) break;
            for (uint32_t c = 0; c < n; ++c) {
                front2[incl - n + c] = down ? c0 + c : node;
                fcls2[incl - n + c] = down ? 0 : (uint8_t)cls;
            }
            __syncwarp();
            nf = total;
            if ((uint32_t)lane < nf) {
                node = front2[lane];
                cls = fcls2[lane];
            }
            __syncwarp();
        }
        if ((uint32_t)lane < nf) {
            front[lane] = node;
            fcls[lane] = (uint8_t)cls;
        }
        if (lane == 0) s_nf = nf;
    }
    __syncthreads();
    uint32_t nf = s_nf;
    for (int level = 0; level < 40; ++level) {
        uint32_t base = 0;
        bool expand = false, fits = true;
        for (uint32_t i0 = 0; i0 < nf; i0 += kRB) {
            const uint32_t i = i0 + tid, node = i < nf ? front[i] : 0u;
            int cls = i < nf ? fcls[i] : 3;
            if (cls == 0) {
                if (node >= t.nodes) {
                    atomicOr(a.err, (unsigned)kDevErrBadNode);
                    cls = 3;
                } else {
                    cls = rb_class(t, a.ft, a.enode[node], node, ball);
                }
                fcls[i] = (uint8_t)cls;
            }
            const uint32_t c0 = cls == 4 ? t.nfd[node] : 0u, n = cls == 4 ? t.nnd[node] : (cls == 3 ? 0u : 1u);
            uint32_t incl = n;
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(0xffffffffu, incl, d);
                if (lane >= d) incl += o;
            }
            if (lane == 31) sh.warp_tot[wid] = incl;
            expand = __syncthreads_or(cls == 4) || expand;
            uint32_t at = base + incl - n, total = 0;
            for (int w = 0; w < kRbWarps; ++w) {
                const uint32_t c = sh.warp_tot[w];
                if (w < wid) at += c;
                total += c;
            }
            base += total;
            fits = fits && base <= kRbFront;
            if (fits)
                for (uint32_t c = 0; c < n; ++c) {
                    front2[at + c] = cls == 4 ? c0 + c : node;
                    fcls2[at + c] = cls == 4 ? 0 : (uint8_t)cls;
                }
            __syncthreads();  // the totals are read, the next step's follow
        }
        if (!expand || !fits) break;  // the classes of this level are kept
        uint32_t *f = front; front = front2; front2 = f;
        uint8_t *g = fcls; fcls = fcls2; fcls2 = g;
        nf = base;
    }
    const long long tq1 = clock64();
    // 2) each entry's slice of eligible points: its start (front2) and length (fcnt), scanned
    for (uint32_t i = tid; i < nf; i += kRB) {
        uint2 e = make_uint2(0, 0);
        int cls = fcls[i];
        if (front[i] >= t.nodes) {
            cls = 3;
        } else {
            e = a.enode[front[i]];
            if (cls == 0) cls = rb_class(t, a.ft, e, front[i], ball);
        }
        fcls[i] = (uint8_t)cls;
        front2[i] = e.x;
        fcnt[i] = cls == 3 ? 0u : e.y - e.x;
    }
    __syncthreads();
    const uint32_t S = rb_scan_excl(fcnt, nf, sh.warp_tot);
    const long long tq2 = clock64();
    // 3) the new segment: the members, then room for every scanned point
    if (tid == 0) {
        s_S = S;
        s_noff = rb_spare(a.P, a.seg[slot], s_m0 + S);
    }
    __syncthreads();
    if (s_noff == kNone) return kNone;
    const uint32_t m0 = s_m0, o = s_o, no = s_noff;
    for (uint32_t k = tid; k < m0; k += kRB) a.P.idx[no + k] = a.P.idx[o + k];
    uint32_t *elig = a.P.idx + no + m0;
    // 2048 points a step, four per thread with their loads on the way together: a step costs the
    // latency of three dependent loads however many points it takes
    constexpr int kIn = 4;
    uint32_t found = 0;
    for (uint32_t base = 0; base < S; base += kIn * kRB) {
        uint32_t q[kIn], ow[kIn];
        float v[kIn];
        bool have[kIn], all[kIn], keep[kIn];
#pragma unroll
        for (int j = 0; j < kIn; ++j) {
            const uint32_t tt = base + j * kRB + tid;
            have[j] = tt < S;
            uint32_t lo = 0, hi = have[j] ? nf : 0;  // the last entry starting at or before tt
            while (hi - lo > 1) {
                const uint32_t mid = (lo + hi) >> 1;
                if (fcnt[mid] <= tt) lo = mid;
                else hi = mid;
            }
            q[j] = have[j] ? a.E[front2[lo] + (tt - fcnt[lo])] : 0u;
            all[j] = have[j] && fcls[lo] == 1;
        }
#pragma unroll
        for (int j = 0; j < kIn; ++j) {
            // this clump's own claims are its members: the acceptance would only skip them
            ow[j] = have[j] ? __ldcg(&a.owner[q[j]]) : myrank;
            v[j] = have[j] && !all[j] ? f_dr2(ball.qh, ball.ql, a.ft.phi[q[j]], a.ft.plo[q[j]]) : 0.f;
        }
#pragma unroll
        for (int j = 0; j < kIn; ++j) {
            keep[j] = have[j] && ow[j] != myrank;
            if (keep[j] && !all[j]) {
                if (f_lo(v[j], a.ft.tol) > ball.rr32 * (1.f + kRel)) keep[j] = false;
                else if (!(f_hi(v[j], a.ft.tol) < ball.rr32 * (1.f - kRel))) keep[j] = point_within(t.pos + q[j], ball.cx, ball.cy, ball.cz, ball.rr);
            }
        }
        unsigned m[kIn];
#pragma unroll
        for (int j = 0; j < kIn; ++j) {
            m[j] = __ballot_sync(0xffffffffu, keep[j]);
            if (lane == 0) s_cnt[j * kRbWarps + wid] = __popc(m[j]);
        }
        __syncthreads();
        uint32_t at[kIn], run = found;
#pragma unroll
        for (int j = 0; j < kIn; ++j) {
            for (int w = 0; w < kRbWarps; ++w) {
                if (w == wid) at[j] = run;
                run += s_cnt[j * kRbWarps + w];
            }
            if (keep[j]) elig[at[j] + __popc(m[j] & ((1u << lane) - 1u))] = q[j];
        }
        found = run;
        __syncthreads();
    }
    if (tid == 0) s_nel = found;
    __syncthreads();
    const uint32_t nel = s_nel;
    const long long t1 = clock64();
    // 4) the reference's sequential acceptance (src/tree.hpp:4686-4706), 512 candidates at a
    // time, those held by earlier clumps left out. Every thread holds one candidate (its FP32
    // form; the FP64 position and velocity, the index and the FP32 form are in shared memory).
    // The block finds the first bound candidate; warp 0 goes on from it alone, 32 candidates
    // (a window) at a time, until none of a window's is bound; the block search then resumes.
    //
    // An update depends on all before it (RN(RN(RN(c M') + RN(m q)) / M') for every component,
    // five dependent FP64 instructions of 64 cycles), the test of the next candidate on its
    // result. A window therefore supposes that exactly the candidates bound to the state on
    // entry (or too close to call) will be accepted: their masses M', the reciprocals and the
    // products m q are formed by all lanes at once, the updates run back to back, and then
    // every lane tests its candidate against the state just before it. What precedes the first
    // candidate that came out otherwise is as the reference has it; the window ends there.
    // Measured per accepted particle where they are dense: 550 cycles (27 to a window), against 1,790 with one
    // test and one update at a time.
    double4_32a *tpos = reinterpret_cast<double4_32a *>(sh.buf), *tvel = tpos + kRB;
    uint32_t *tq = reinterpret_cast<uint32_t *>(tvel + kRB);
    CandF *tf = reinterpret_cast<CandF *>(tq + kRB);
    uint32_t &s_pos = sh.u[8];
    const float G32 = (float)a.cp.G, shear32 = (float)a.cp.shear;
    // no candidate's limits are beyond those of the largest coordinate and velocity
    const BoundLimits limits = bound_limits(a.xtop, (float)dfrom((uint64_t)(*a.vtop + 1u) << 32), shear32);
    double comp = 0.0;      // warp 0, lane c < 6: component c of the state (x y z vx vy vz)
    double M = sh.st[0];    // warp 0: the mass
    uint32_t nacc = 0, rounds = 0;
    if (tid == 0) {
        sh.u[12] = 0;
        sh.u[13] = 0;
        sh.u[14] = 0;
        sh.u[15] = 0;
        sh.u[16] = 0;
        sh.u[17] = 0;
        sh.u[18] = 0;
    }
    if (tid < 32) {
        comp = lane < 6 ? sh.st[1 + lane] : 0.0;
        float h = 0.f, l = 0.f;
        split_any(comp, h, l);
        if (lane < 6) {
            sh.sf[lane] = h;
            sh.sf[6 + lane] = l;
            sh.sd[lane] = comp;
        }
        if (lane == 0) {
            float mh, ml;
            split_any(M, mh, ml);
            sh.sf[12] = mh;
            sh.sd[6] = M;
        }
    }
    // warp 0: candidate k against the state in FP32
    auto test = [&](const CandF &cf) { return bound_hilo_fast(cf, sh.sf[12], sh.sf, sh.sf + 6, G32, shear32, limits); };
    // warp 0 takes the window of the tile's candidates from at on; returns where the next one
    // starts, and whether any candidate was bound (or too close to call) on entry
    auto window = [&](uint32_t at, uint32_t tlen, bool &any) -> uint32_t {
        const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
        const uint32_t k = at + (uint32_t)lane;
        const bool has = k < tlen;
        CandF cf = tf[has ? k : at];
        const unsigned P = __ballot_sync(full, has && test(cf) != 0);
        any = P != 0;
        if (!any) return min(at + 32u, tlen);
        const long long tw0 = clock64();
        // the masses after each supposed acceptance: integers on the grid of M's binade, up to
        // the first lane where that does not hold (then one update with an ordinary addition)
        const double m = has ? tpos[k].w : 0.0;
        const bool sup = (P >> lane) & 1u;
        const uint64_t mb = dbits(M);
        const uint32_t ex = (uint32_t)(mb >> 52) & 0x7ffu;
        long long dn = 0;
        bool ok = true;
        if (sup) ok = (mb >> 63) == 0 && ex > 60u && ex < 2000u && grid_term(m, ex, dn) && dn > 0;
        long long nl = ok ? dn : 0;
        for (int d = 1; d < 32; d <<= 1) {
            const long long o = __shfl_up_sync(full, nl, d);
            if (lane >= d) nl += o;
        }
        nl += (long long)((mb & 0xfffffffffffffull) | (1ull << 52));
        ok = ok && (!sup || (nl > (1LL << 52) && nl < (1LL << 53)));
        const unsigned okm = __ballot_sync(full, ok);
        uint32_t lim = ~okm ? (uint32_t)__ffs(~okm) - 1u : 32u;  // lanes of this window
        unsigned use = lim < 32 ? P & ((1u << lim) - 1u) : P;
        double Ml = grid_value(nl, ex);
        if (!use) {
            const uint32_t j = (uint32_t)__ffs(P) - 1u;
            use = 1u << j;
            lim = j + 1;
            Ml = M + m;
        }
        const uint32_t rank = __popc(use & below), cnt = __popc(use);
        if ((use >> lane) & 1u) {
            const double4_32a p = tpos[k], v = tvel[k];
            double *t = sh.tk + 8 * rank;
            t[0] = m * p.x;
            t[1] = m * p.y;
            t[2] = m * p.z;
            t[3] = m * v.x;
            t[4] = m * v.y;
            t[5] = m * v.z;
            t[6] = Ml;
            t[7] = __drcp_rn(Ml);
        }
        if (lane < 6) sh.hist[lane] = comp;
        if (lane == 6) sh.hist[6] = M;
        __syncwarp();
        // the updates, lane c < 6 component c, the state after each one kept. With a correctly
        // rounded reciprocal Markstein's correction gives the correctly rounded quotient, but
        // makes +0 of a numerator -0, which only a component that is -0 already can lead to.
        auto updates = [&](auto zero) {
            const int c = lane < 6 ? lane : 6;
            double x = lane < 6 ? comp : 0.0;
            const double *t = sh.tk;
            double add = lane < 6 ? t[c] : 0.0, Mn = t[6], y = t[7];
            for (uint32_t a = 0; a < cnt; ++a) {
                t += a + 1 < cnt ? 8 : 0;
                const double add1 = lane < 6 ? t[c] : 0.0, Mn1 = t[6], y1 = t[7];
                const double num = x * Mn + add;
                const double q0 = num * y;
                x = fma(fma(-q0, Mn, num), y, q0);
                if constexpr (decltype(zero)::value)
                    if ((dbits(num) << 1) == 0) x = num;
                if (lane < 7) sh.hist[8 * (a + 1) + lane] = lane < 6 ? x : Mn;
                add = add1;
                Mn = Mn1;
                y = y1;
            }
        };
        if (__any_sync(full, dbits(comp) == 1ull << 63)) updates(std::true_type());
        else updates(std::false_type());
        __syncwarp();
        const long long tw1 = clock64();
        // every candidate against the state before it, in float pairs: those of a few states are
        // shared out over the lanes, of many each lane splits its own state's
        const bool few = cnt <= kRbFewStates;
        if (few) {
            for (uint32_t i = (uint32_t)lane; i < 7 * (cnt + 1); i += 32) {
                const uint32_t j = (i * 9363u) >> 16, c = i - 7 * j;  // i / 7
                float h, l;
                split_any(sh.hist[8 * j + c], h, l);
                sh.histf[14 * j + c] = h;
                sh.histf[14 * j + 7 + c] = l;
            }
            __syncwarp();
        }
        bool bound = false, unsure = false;
        const double *S = sh.hist + 8 * rank;
        if (has && (uint32_t)lane < lim) {
            int r;
            if (few) {
                const float *f = sh.histf + 14 * rank;
                r = bound_hilo_fast(cf, f[6], f, f + 7, G32, shear32, limits);
            } else {
                float h[6], l[6], mh, ml;
                for (int c = 0; c < 6; ++c) split_any(S[c], h[c], l[c]);
                split_any(S[6], mh, ml);
                r = bound_hilo_fast(cf, mh, h, l, G32, shear32, limits);
            }
            bound = r == 1;
            unsure = r < 0;
        }
        if (unsure) {
            bound = bound_fp64(tpos[k], tvel[k], S[6], S[0], S[1], S[2], S[3], S[4], S[5], a.cp);
            if (stat) atomicAdd(&sh.u[12], 1u);
        }
        const unsigned B = __ballot_sync(full, bound);
        unsigned diff = B ^ use;
        if (lim < 32) diff &= (1u << lim) - 1u;
        uint32_t end = diff ? (uint32_t)__ffs(diff) - 1u : lim;  // lanes before it came out as supposed
        const unsigned acc = end < 32 ? use & ((1u << end) - 1u) : use;
        if (diff && ((use >> end) & 1u)) ++end;  // supposed to be bound and is not: settled too
        const uint32_t n = __popc(acc);
        if ((acc >> lane) & 1u) {
            const uint32_t q2 = tq[k];
            // the lowest rank keeps the particle; who lost one is found after the pass
            atomicMin(&a.owner[q2], myrank);
            elig[nacc + rank] = q2;  // accepted ones overwrite candidates already consumed
        }
        nacc += n;
        comp = lane < 6 ? sh.hist[8 * n + lane] : 0.0;
        M = sh.hist[8 * n + 6];
        if (lane < 7) {  // the state for the next tests
            float h, l;
            if (few) {
                h = sh.histf[14 * n + lane];
                l = sh.histf[14 * n + 7 + lane];
            } else {
                split_any(sh.hist[8 * n + lane], h, l);
            }
            sh.sf[lane < 6 ? lane : 12] = h;
            if (lane < 6) sh.sf[6 + lane] = l;
            sh.sd[lane] = sh.hist[8 * n + lane];
        }
        __syncwarp();
        if (stat && lane == 0) {
            sh.u[13] += (uint32_t)(clock64() - tw0);
            sh.u[14] += 1;
            sh.u[15] += (uint32_t)(tw1 - tw0);
        }
        return min(at + end, tlen);
    };
    // the prefetched candidate of the next tile
    uint32_t nq = kNone, now_ = kNone, ntn = kNone;
    double4_32a np = make_double4_32a(0, 0, 0, 0), nv = make_double4_32a(0, 0, 0, 0);
    float4 nph = make_float4(0.f, 0.f, 0.f, 0.f), npl = nph;
    if ((uint32_t)tid < nel) {
        nq = elig[tid];
        now_ = __ldcg(&a.owner[nq]);
        ntn = a.tent[nq];
        np = t.pos[nq];
        nv = a.vel[nq];
        nph = a.ft.phi[nq];
        npl = a.ft.plo[nq];
    }
    long long t_setup = 0;
    uint32_t n_tiles = 0;
    for (uint32_t base = 0; base < nel; base += kRB) {
        const long long tt0 = clock64();
        const uint32_t q = nq;
        const bool valid = q != kNone;
        bool taken = true;
        CandF cf;
        if (valid) {
            uint32_t ow = now_, tn = ntn;
            if (tn != kNone && tn < myrank && *(volatile const uint8_t *)&a.finished[a.slot_of_rank[tn]]) {
                // that clump has finished its calls in this launch: its claims are its
                // holdings, and its prediction from the last pass no longer applies
                __threadfence();
                ow = __ldcg(&a.owner[q]);
                tn = kNone;
            }
            taken = (ow != kNone && ow <= myrank) || (tn != kNone && tn < myrank);
            if (stat) {
                if (tn != kNone && tn < myrank) atomicAdd(&sh.u[16], 1u);
                if (ow != kNone && ow < myrank) atomicAdd(&sh.u[17], 1u);
                if (taken) atomicAdd(&sh.u[18], 1u);
            }
            if (ow != kNone && ow < myrank)
                defer_add(a.dset, a.dover, a.dmax, slot, ow, *(volatile const uint8_t *)&a.finished[a.slot_of_rank[ow]] == 0, a.dcall,
                          a.dfirst, call);
            else if (tn != kNone && tn < myrank)
                defer_add(a.dset, a.dover, a.dmax, slot, tn, true, a.dcall, a.dfirst, call);
            cf.ph[0] = nph.x; cf.ph[1] = nph.y; cf.ph[2] = nph.z;
            cf.pl[0] = npl.x; cf.pl[1] = npl.y; cf.pl[2] = npl.z;
            split_any(nv.x, cf.vh[0], cf.vl[0]);
            split_any(nv.y, cf.vh[1], cf.vl[1]);
            split_any(nv.z, cf.vh[2], cf.vl[2]);
            float wl;
            split_any(np.w, cf.w, wl);
        }
        uint32_t place;  // the candidates left, side by side in the tile
        const uint32_t tlen = rb_block_rank(!taken, place, sh.warp_tot);
        if (!taken) {
            tpos[place] = np;
            tvel[place] = nv;
            tq[place] = q;
            tf[place] = cf;
        }
        nq = kNone;
        if (base + kRB + tid < nel) {  // prefetch (accepted ones are written below base + kRB only)
            nq = elig[base + kRB + tid];
            now_ = __ldcg(&a.owner[nq]);
            ntn = a.tent[nq];
            np = t.pos[nq];
            nv = a.vel[nq];
            nph = a.ft.phi[nq];
            npl = a.ft.plo[nq];
        }
        __syncthreads();
        t_setup += clock64() - tt0;
        ++n_tiles;
        if ((uint32_t)tid < tlen) cf = tf[tid];
        for (uint32_t pos = 0; pos < tlen;) {
            ++rounds;
            bool bound = false, unsure = false;
            if ((uint32_t)tid < tlen && (uint32_t)tid >= pos) {
                const int r = bound_hilo_fast(cf, sh.sf[12], sh.sf, sh.sf + 6, G32, shear32, limits);
                if (r >= 0) bound = r == 1;
                else unsure = true;
            }
            if (unsure) {
                bound = bound_fp64(tpos[tid], tvel[tid], sh.sd[6], sh.sd[0], sh.sd[1], sh.sd[2], sh.sd[3], sh.sd[4], sh.sd[5], a.cp);
                if (stat) atomicAdd(&sh.u[12], 1u);
            }
            const unsigned b = __ballot_sync(0xffffffffu, bound);
            if (lane == 0) sh.warp_tot[wid] = b ? (uint32_t)(wid * 32 + __ffs(b) - 1) : kNone;
            __syncthreads();
            uint32_t f = kNone;
            {
                uint32_t wv[kRbWarps];
                for (int w = 0; w < kRbWarps; ++w) wv[w] = sh.warp_tot[w];
                for (int w = kRbWarps - 1; w >= 0; --w) f = wv[w] != kNone ? wv[w] : f;
            }
            if (f == kNone) break;  // the rest of the tile is not bound
            if (tid < 32) {
                uint32_t at = f;
                for (bool any = true; any && at < tlen;) at = window(at, tlen, any);
                if (lane == 0) s_pos = at;
            }
            __syncthreads();
            pos = s_pos;
        }
        __syncthreads();
    }
    if (tid == 0) s_f = nacc;
    __syncthreads();
    nacc = s_f;
    const long long t2 = clock64();
    if (tid == 0) {
        if (stat) {
            stat[0] += 1;
            stat[1] += nel;
            stat[2] += nacc;
            stat[3] += (unsigned long long)(t1 - t0);
            stat[4] += (unsigned long long)(t2 - t1);
            stat[12] += rounds;
            stat[13] += S;
            stat[36] += (unsigned long long)(tq1 - t0);
            stat[37] += (unsigned long long)(tq2 - tq1);
            stat[38] += nf;
            stat[10] += sh.u[12];
            stat[14] += sh.u[13];  // warp 0's windows: cycles, number, and cycles up to the last update
            stat[15] += sh.u[14];
            stat[16] += sh.u[15];
            stat[31] += (unsigned long long)t_setup;  // tile set-up: loads arriving, filters, splits
            stat[32] += n_tiles;
            stat[33] += sh.u[16];  // candidates predicted for an earlier clump
            stat[34] += sh.u[17];  // held by an earlier clump
            stat[35] += sh.u[18];  // taken either way
        }
        if (nacc) {
            rb_switch(a.seg[slot], o);
            a.ct.moff[slot] = no;
            a.ct.mn[slot] = m0 + nacc;
        }
    }
    __syncthreads();
    return nacc;
}

// ------------------------------------------------------------------ SortParticles
// Stable block sort of n (squared distance, member) pairs by `bits` bits of key (the top 32 bits
// of the distance above kmin, without the lowest `drop`; bits <= 2 kRbDigit), by digits of
// kRbDigit bits: one pass goes from (dist, idx) to (od, oi), two go through rec. Every warp
// counts and then places a segment of its own with counters of its own, so a pass takes four
// block barriers however long the segments are.
//
// What bounds a pass is the placing: 32 lanes write to 32 lines, a wavefront each. The pair
// therefore travels as one 16-byte record in the first pass and goes straight to its place in
// the second (96 wavefronts per 32 members, where a key, a position and a gather of both arrays
// at the end took 192).
struct __align__(16) RbRec {
    double d;
    uint32_t i, pad;
};

__device__ void rb_radix(const double *dist, const uint32_t *idx, RbRec *rec, double *od, uint32_t *oi, uint32_t n, uint32_t kmin, uint32_t drop,
                         uint32_t bits, uint32_t *smem, uint32_t *warp_tot) {
    constexpr uint32_t kBins = 1u << kRbDigit, kPer = kBins / kRB;
    static_assert(kPer == 4, "a thread scans four digits");
    const uint32_t tid = threadIdx.x, lane = tid & 31, wid = tid >> 5, full = 0xffffffffu;
    const uint32_t seg = ((n + kRbWarps * 32 - 1) / (kRbWarps * 32)) * 32, b = min(n, wid * seg), e = min(n, b + seg);
    uint32_t *cnt = smem + wid * kBins;
    const uint32_t passes = bits > kRbDigit ? 2 : 1;
    for (uint32_t pass = 0; pass < passes; ++pass) {
        const uint32_t sh = pass * kRbDigit;
        auto digit = [&](double d) { return (((((uint32_t)(dbits(d) >> 32)) - kmin) >> drop) >> sh) & (kBins - 1); };
        uint4 *z = reinterpret_cast<uint4 *>(smem);
        for (uint32_t d = tid; d < kBins * kRbWarps / 4; d += kRB) z[d] = make_uint4(0, 0, 0, 0);
        __syncthreads();
        for (uint32_t i = b + lane; i < e; i += 128) {
            double k[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) k[j] = i + 32 * j < e ? (pass ? rec[i + 32 * j].d : dist[i + 32 * j]) : 0.0;
#pragma unroll
            for (int j = 0; j < 4; ++j)
                if (i + 32 * j < e) atomicAdd(&cnt[digit(k[j])], 1u);
        }
        __syncthreads();
        {  // exclusive prefix over (digit, warp): four digits per thread
            uint32_t s4[4] = {0, 0, 0, 0};
            for (int w = 0; w < kRbWarps; ++w) {
                const uint4 c = z[w * (kBins / 4) + tid];
                s4[0] += c.x;
                s4[1] += c.y;
                s4[2] += c.z;
                s4[3] += c.w;
            }
            const uint32_t mine = s4[0] + s4[1] + s4[2] + s4[3];
            uint32_t incl = mine;
            for (int d = 1; d < 32; d <<= 1) {
                const uint32_t o = __shfl_up_sync(full, incl, d);
                if ((int)lane >= d) incl += o;
            }
            if (lane == 31) warp_tot[wid] = incl;
            __syncthreads();
            uint32_t at = incl - mine;
            for (uint32_t w = 0; w < wid; ++w) at += warp_tot[w];
            uint4 run = make_uint4(at, at + s4[0], at + s4[0] + s4[1], at + s4[0] + s4[1] + s4[2]);
            for (int w = 0; w < kRbWarps; ++w) {
                const uint4 c = z[w * (kBins / 4) + tid];
                z[w * (kBins / 4) + tid] = run;
                run.x += c.x;
                run.y += c.y;
                run.z += c.z;
                run.w += c.w;
            }
        }
        __syncthreads();
        for (uint32_t i0 = b; i0 < e; i0 += 128) {
            double k[4];
            uint32_t v[4];
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const uint32_t i = i0 + 32 * j + lane;
                if (pass) {
                    const uint4 r = i < e ? *reinterpret_cast<const uint4 *>(&rec[i]) : make_uint4(0, 0, 0, 0);
                    k[j] = dfrom(((uint64_t)r.y << 32) | r.x);
                    v[j] = r.z;
                } else {
                    k[j] = i < e ? dist[i] : 0.0;
                    v[j] = i < e ? idx[i] : 0u;
                }
            }
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const bool some = i0 + 32 * j + lane < e;
                const uint32_t d = some ? digit(k[j]) : kBins;
                const uint32_t peers = __match_any_sync(full, d), rk = __popc(peers & ((1u << lane) - 1u));
                const uint32_t off = some ? cnt[d] : 0u;
                __syncwarp();
                if (some && rk == 0) cnt[d] = off + __popc(peers);
                __syncwarp();
                if (some) {
                    if (pass + 1 < passes) {
                        const uint64_t kb = dbits(k[j]);
                        *reinterpret_cast<uint4 *>(&rec[off + rk]) = make_uint4((uint32_t)kb, (uint32_t)(kb >> 32), v[j], 0);
                    } else {
                        od[off + rk] = k[j];
                        oi[off + rk] = v[j];
                    }
                }
            }
        }
        __syncthreads();
    }
}

// Runs of equal keys: insertion sort by the full squared distance (stable), a thread per run.
// Most runs are pairs, so every thread reads its entry's and the next two distances at once
// (coalesced), and a pair out of order changes places.
__device__ __forceinline__ void rb_fix_runs(double *dist, uint32_t *idx, uint32_t m, uint32_t kmin, uint32_t drop) {
    auto key = [&](double d) { return ((uint32_t)(dbits(d) >> 32) - kmin) >> drop; };
    // a run changes only within itself, and its keys are equal: what a thread reads of another
    // thread's run has the same key before and after
    for (uint32_t k = threadIdx.x; k + 1 < m; k += kRB) {
        const double d0 = dist[k], d1 = dist[k + 1];
        const uint32_t k1 = key(d0), k2 = key(d1), k0 = k ? key(dist[k - 1]) : ~k1, k3 = k + 2 < m ? key(dist[k + 2]) : ~k2;
        if (k0 == k1 || k1 != k2) continue;
        if (k2 != k3) {
            if (dbits(d0) > dbits(d1)) {
                const uint32_t i0 = idx[k], i1 = idx[k + 1];
                dist[k] = d1;
                dist[k + 1] = d0;
                idx[k] = i1;
                idx[k + 1] = i0;
            }
            continue;
        }
        uint32_t e = k + 3;
        while (e < m && key(dist[e]) == k1) ++e;
        for (uint32_t i = k + 1; i < e; ++i) {
            const double dv = dist[i];
            const uint32_t iv = idx[i];
            uint32_t j = i;
            while (j > k && dbits(dist[j - 1]) > dbits(dv)) {
                dist[j] = dist[j - 1];
                idx[j] = idx[j - 1];
                --j;
            }
            dist[j] = dv;
            idx[j] = iv;
        }
    }
}

// any two neighbours of a sorted run of squared distances whose square roots are equal
__device__ __forceinline__ bool rb_sqrt_tie(double s0, double s1) {
    const unsigned long long b0 = (unsigned long long)__double_as_longlong(s0), b1 = (unsigned long long)__double_as_longlong(s1);
    if (b1 - b0 > 64ull) return false;  // more than a few ulps apart: the roots differ
    return equal_roots(s0, s1);
}

// whether this thread's neighbours among m sorted squared distances tie
__device__ __forceinline__ int rb_ties(const double *dist, uint32_t m) {
    int tie = 0;
    for (uint32_t k0 = threadIdx.x + 1; k0 < m; k0 += 4 * kRB) {
        double x[4], y[4];
#pragma unroll
        for (int j = 0; j < 4; ++j) {
            const uint32_t k = k0 + j * kRB;
            x[j] = k < m ? dist[k - 1] : 0.0;
            y[j] = k < m ? dist[k] : 1.0;
        }
#pragma unroll
        for (int j = 0; j < 4; ++j) tie |= rb_sqrt_tie(x[j], y[j]);
    }
    return tie;
}

// SortParticles with the Hill radius after it (src/tree.hpp:4446-4512, 4715-4717). Returns
// false when the pool has no room for a large sort (the clump is then left with needsort).
__device__ bool rb_sort_particles(const RbArgs &a, uint32_t slot, RbShared &sh, unsigned long long *stat) {
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    uint32_t &s_o = sh.u[8], &s_m = sh.u[9], &s_tie = sh.u[10], &s_r = sh.u[11], &s_x = sh.u[12];
    uint32_t *s_kmin = sh.u + 20, *s_kmax = s_kmin + kRbWarps;
    const long long t0 = clock64();
    if (tid == 0) {
        s_o = a.ct.moff[slot];
        s_m = a.ct.mn[slot];
        s_tie = 0;
    }
    __syncthreads();
    const uint32_t o = s_o, m = s_m;
    uint32_t *idx = a.P.idx + o;
    double *dist = a.P.dist + o;
    // 1) the seven sums in member order (CalculateKinematicProperties): warp w < 7 runs sum w
    // over the per-point products from a shared-memory stage that the other nine warps fill:
    // 256 members at a time (one per loading thread), double-buffered, the products of a chunk
    // on their way to registers a whole chunk before they are staged, their indices one more
    double acc = 0.0;
    uint32_t its = 0;
    long long tsum = 0;
    {
        constexpr uint32_t kCh = kSumChunk;      // members per chunk
        constexpr uint32_t kLd = kRB - 7 * 32;   // loading threads (warps 7..15)
        constexpr uint32_t kBuf = 7 * kSumStage; // doubles per buffer
        static_assert(2 * kBuf * sizeof(double) + 7 * kSumChunk * sizeof(uint2) <= kRbSmem, "sum stage and lists");
        static_assert(kCh <= kLd, "sum chunk");
        double *stg = reinterpret_cast<double *>(sh.buf);  // [2][7][kSumStage]
        uint2 *list = reinterpret_cast<uint2 *>(stg + 2 * kBuf) + (size_t)kSumChunk * (wid < 7 ? wid : 0);
        const uint32_t nch = (m + kCh - 1) / kCh;
        const uint32_t k0 = (uint32_t)tid - 7u * 32u;  // loading threads: their member of a chunk
        const bool loads = wid >= 7 && k0 < kCh;
        const uint32_t at = sum_slot(k0 < kCh ? k0 : 0u);
        uint32_t qn = 0;  // a loading thread's member index, one chunk ahead of the products
        double4_32a p = make_double4_32a(0, 0, 0, 0), v = p;
        auto fetch = [&](uint32_t g) {  // the products of member g, whose index is in qn; then the next index
            p = v = make_double4_32a(0, 0, 0, 0);
            if (g < m) {
                p = a.tm0[qn];
                v = a.tm1[qn];
            }
            if (g + kCh < m) qn = idx[g + kCh];
        };
        auto put = [&](uint32_t b) {
            double *d = stg + (size_t)b * kBuf + at;
            d[0] = p.x;
            d[kSumStage] = p.y;
            d[2 * kSumStage] = p.z;
            d[3 * kSumStage] = p.w;
            d[4 * kSumStage] = v.x;
            d[5 * kSumStage] = v.y;
            d[6 * kSumStage] = v.z;
        };
        if (loads) {
            if (k0 < m) qn = idx[k0];
            fetch(k0);
            put(0);
            fetch(kCh + k0);
        }
        __syncthreads();
        const long long ts = clock64();
        for (uint32_t c = 0; c < nch; ++c) {
            const uint32_t b = c & 1u;
            if (wid < 7) {
                ordered_sum_chunk(stg + (size_t)b * kBuf + (size_t)wid * kSumStage, acc, list, &its);
            } else if (loads && c + 1 < nch) {
                put(b ^ 1u);
                fetch((c + 2) * kCh + k0);
            }
            __syncthreads();
        }
        tsum = clock64() - ts;
    }
    if (wid < 7 && lane == 0) sh.sums[wid] = acc;
    if (wid < 7 && lane == 0 && stat) {  // each sum: its time and the chunks it took term by term
        atomicAdd(&stat[17 + wid], (unsigned long long)its);
        atomicAdd(&stat[24 + wid], (unsigned long long)tsum);
    }
    __syncthreads();
    if (tid < 32) {
        const double Ms = sh.sums[0];
        double v = 0.0;
        if (lane >= 1 && lane <= 6) v = sh.sums[lane] / Ms;
        if (lane == 7) v = cr_pow_third(Ms * a.cp.G / 3. / a.cp.Omega / a.cp.Omega);  // src/tree.hpp:4715-4717
        if (lane >= 1 && lane <= 7) sh.st[lane] = v;
        if (lane == 0) sh.st[0] = Ms;
    }
    __syncthreads();
    const long long t_sum = clock64();
    if (tid == 0) {
        a.ct.M[slot] = sh.st[0];
        a.ct.com[slot] = make_double4_32a(sh.st[1], sh.st[2], sh.st[3], 0);
        a.ct.vcom[slot] = make_double4_32a(sh.st[4], sh.st[5], sh.st[6], 0);
        a.ct.hill[slot] = sh.st[7];
    }
    // 2) squared distances to the new centre (src/tree.hpp:4448-4450: (pos - com).Norm()), and
    // the range of their top 32 bits
    const double cx = sh.st[1], cy = sh.st[2], cz = sh.st[3];
    uint32_t kmin = kNone, kmax = 0;
    for (uint32_t k = tid; k < m; k += kRB) {
        const double4_32a p = a.t.pos[idx[k]];
        const double dx = p.x - cx, dy = p.y - cy, dz = p.z - cz;
        double s = dx * dx;
        s = s + dy * dy;
        s = s + dz * dz;
        dist[k] = s;
        const uint32_t hi = (uint32_t)(dbits(s) >> 32);
        kmin = min(kmin, hi);
        kmax = max(kmax, hi);
    }
    kmin = __reduce_min_sync(0xffffffffu, kmin);
    kmax = __reduce_max_sync(0xffffffffu, kmax);
    if (lane == 0) {
        s_kmin[wid] = kmin;
        s_kmax[wid] = kmax;
    }
    __syncthreads();
    for (int w = 0; w < kRbWarps; ++w) {
        kmin = min(kmin, s_kmin[w]);
        kmax = max(kmax, s_kmax[w]);
    }
    const long long t_dist = clock64();
    bool ok = true;
    // the keys of the sort: the leading bits of the range above the smallest
    const uint32_t range = 32u - (uint32_t)__clz((int)(kmax - kmin));
    if (m <= kRbSmall) {
        // 3a) in shared memory, behind the counters: the records and the sorted pairs. Up to
        // kRbOnePass members one digit is enough: over some 64 octaves it leaves runs of a few
        // equal keys to the insertion sort.
        const uint32_t most = m <= kRbOnePass && range <= 26 ? kRbDigit : 2 * kRbDigit, drop = range > most ? range - most : 0u;
        RbRec *rec = reinterpret_cast<RbRec *>(sh.buf + kRbRadixBytes);
        double *sd = reinterpret_cast<double *>(rec + kRbSmall);
        uint32_t *si = reinterpret_cast<uint32_t *>(sd + kRbSmall);
        rb_radix(dist, idx, rec, sd, si, m, kmin, drop, range - drop, reinterpret_cast<uint32_t *>(sh.buf), sh.warp_tot);
        rb_fix_runs(sd, si, m, kmin, drop);
        __syncthreads();
        // (every size: below 17 members the library's insertion sort is stable by distance,
        // which an order by squared distance only equals when no two roots tie)
        const int tie = rb_ties(sd, m);
        if (__syncthreads_or(tie)) {
            if (tid == 0) s_tie = 1;
        } else {
            for (uint32_t k = tid; k < m; k += kRB) {
                idx[k] = si[k];
                dist[k] = sd[k];
            }
        }
        __syncthreads();
    } else {
        // 3b) large: the records in the clump's sort buffer (16-byte aligned in the distances'
        // half of the pool), the sorted pairs in its spare segment
        if (tid == 0) {
            RbSeg &g = a.seg[slot];
            s_r = rb_sort_room(a.P, g, m) ? g.spare : kNone;
            s_x = g.buf;
        }
        __syncthreads();
        const uint32_t r = s_r;
        if (r == kNone) {
            ok = false;
        } else {
            const uint32_t drop = range > 2 * kRbDigit ? range - 2 * kRbDigit : 0u;
            RbRec *rec = reinterpret_cast<RbRec *>(a.P.dist + ((s_x + 1) & ~1u));
            uint32_t *didx = a.P.idx + r;
            double *ddist = a.P.dist + r;
            rb_radix(dist, idx, rec, ddist, didx, m, kmin, drop, range - drop, reinterpret_cast<uint32_t *>(sh.buf), sh.warp_tot);
            rb_fix_runs(ddist, didx, m, kmin, drop);
            __syncthreads();
            const int tie = rb_ties(ddist, m);
            if (__syncthreads_or(tie)) {
                if (tid == 0) s_tie = 1;  // the unsorted segment at o is intact
            } else if (tid == 0) {
                rb_switch(a.seg[slot], o);
                a.ct.moff[slot] = r;
            }
            __syncthreads();
        }
    }
    if (ok && s_tie) {
        // two members at the same distance: the library's std::sort order on the sequence
        // before the sort, with the distances themselves (lib_sort.cuh, one thread)
        for (uint32_t k = tid; k < m; k += kRB) dist[k] = sqrt(dist[k]);
        __syncthreads();
        if (tid == 0) lib_sort(dist, idx, m);
        __syncthreads();
    }
    if (tid == 0) {
        if (ok) {
            a.needsort[slot] = 0;
            a.distsq[slot] = s_tie ? 0 : 1;
        } else {
            a.needsort[slot] = 1;
        }
        if (stat) {
            const long long t3 = clock64();
            stat[5] += (unsigned long long)(t3 - t0);
            stat[6] += (unsigned long long)(t_sum - t0);
            stat[7] += 1;
            stat[8] += (unsigned long long)(t_dist - t_sum);
            stat[9] += (unsigned long long)(t3 - t_dist);
            stat[11] += m;
        }
    }
    __syncthreads();
    return ok;
}

// ------------------------------------------------------------------ checkpoints
__device__ uint32_t ck_try_alloc(const Ckpt &ck, uint32_t n) {
    uint32_t cur = *(volatile uint32_t *)ck.top;
    for (int it = 0; it < (1 << 22); ++it) {
        if ((uint64_t)cur + n > ck.cap) return kNone;
        const uint32_t prev = atomicCAS(ck.top, cur, cur + n);
        if (prev == cur) return cur;
        cur = prev;
    }
    return kNone;
}

// the clump's state after call j (its members just sorted): a checkpoint, if there is room
__device__ void rb_checkpoint(const RbArgs &a, uint32_t slot, uint32_t rank, uint32_t j, RbShared &sh) {
    const int tid = threadIdx.x;
    uint32_t &s_off = sh.u[19];
    const uint32_t o = a.ct.moff[slot], m = a.ct.mn[slot];
    if (tid == 0) {
        s_off = kNone;
        if (a.ck.n[rank] < (uint32_t)kCk) s_off = ck_try_alloc(a.ck, m);
    }
    __syncthreads();
    const uint32_t off = s_off;
    if (off != kNone) {
        for (uint32_t k = tid; k < m; k += kRB) {
            a.ck.idx[off + k] = a.P.idx[o + k];
            a.ck.dist[off + k] = a.P.dist[o + k];
        }
        if (tid == 0) {
            const uint32_t n = a.ck.n[rank];
            const size_t e = (size_t)rank * kCk + n;
            const double4_32a c = a.ct.com[slot], v = a.ct.vcom[slot];
            double *q = a.ck.st + e * 8;
            q[0] = a.ct.M[slot];
            q[1] = c.x; q[2] = c.y; q[3] = c.z;
            q[4] = v.x; q[5] = v.y; q[6] = v.z;
            q[7] = a.ct.hill[slot];
            a.ck.call[e] = j;
            a.ck.off[e] = off;
            a.ck.m[e] = m;
            a.ck.n[rank] = n + 1;
        }
    }
    __syncthreads();
}

// ------------------------------------------------------------------ the persistent loop
__global__ void __launch_bounds__(kRB, 1) k_rebind_loop(RbArgs a) {
    extern __shared__ __align__(16) unsigned char rb_dyn[];
    __shared__ uint32_t warp_tot[kRbWarps];
    __shared__ uint32_t u[20 + 4 * kRbWarps];
    __shared__ double st[8], sums[8], sd[8], tk[32 * 8], hist[33 * 8];
    __shared__ float sf[16], histf[(kRbFewStates + 1) * 14];
    __shared__ uint32_t s_item;
    RbShared sh{rb_dyn, warp_tot, u, st, sums, tk, hist, histf, sf, sd};
    const int tid = threadIdx.x;
    for (uint32_t guard = 0; guard <= a.n; ++guard) {
        if (tid == 0) s_item = atomicAdd(a.head, 1u);
        __syncthreads();
        const uint32_t item = s_item;
        __syncthreads();
        if (item >= a.n) return;
        const uint32_t slot = a.list[item];
        if (tid == 0 && a.blk_off) {
            for (uint32_t b = a.blk_off[item]; b < a.blk_off[item + 1]; ++b) {
                const uint32_t bs = a.blk[b];
                for (uint32_t it = 0; *(volatile uint8_t *)&a.finished[bs] == 0; ++it) {
                    if (it >= a.wait_limit) {
                        atomicOr(a.err, (unsigned)kDevErrLoopLimit);
                        break;
                    }
                    __nanosleep(1000);
                }
            }
            __threadfence();
        }
        __syncthreads();
        const uint32_t myrank = a.rank_of[slot];
        unsigned long long *stat = a.stats ? a.stats + kRbStats * (size_t)slot : nullptr;
        if (tid == 0) s_item = a.ccall ? a.ccall[slot] : 0u;
        __syncthreads();
        uint32_t done = s_item;  // calls of this clump's run so far
        __syncthreads();
        bool suspend = false;
        if (a.needsort[slot]) suspend = !rb_sort_particles(a, slot, sh, stat);
        for (uint32_t call = 0; !suspend; ++call) {
            if (call >= kCallLimit) {
                if (tid == 0) atomicOr(a.err, (unsigned)kDevErrLoopLimit);
                break;
            }
            const uint32_t j = done + 1;
            const uint32_t nacc = rb_call(a, slot, myrank, sh, stat, j);
            if (nacc == kNone) {
                suspend = true;
                break;
            }
            done = j;
            if (tid == 0 && a.ccall) a.ccall[slot] = j;
            if (nacc == 0) break;  // no growth: the Hill radius of the unchanged mass stays
            if (!rb_sort_particles(a, slot, sh, stat)) suspend = true;
            else if (a.ck.n && ck_after(j)) rb_checkpoint(a, slot, myrank, j, sh);
        }
        if (!suspend && a.distsq[slot]) {  // the distances of the last sort
            const uint32_t o = a.ct.moff[slot], m = a.ct.mn[slot];
            for (uint32_t k = tid; k < m; k += kRB) a.P.dist[o + k] = sqrt(a.P.dist[o + k]);
            __syncthreads();
            if (tid == 0) a.distsq[slot] = 0;
        }
        __syncthreads();
        if (tid == 0) {
            a.suspended[slot] = suspend ? 1 : 0;
            __threadfence();
            *(volatile uint8_t *)&a.finished[slot] = 1;
        }
        __syncthreads();
    }
}
