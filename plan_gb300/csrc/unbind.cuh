// RemoveUnboundParticles (src/tree.hpp:4615-4674): from the farthest member down, a member that
// is not bound to the others is taken out of the clump's mass, centre and velocity, and the next
// is tested against what remains.
//
// One block per clump, 256 members at a time, farthest first, one per thread. The test runs in
// FP32 on float pairs with an error bound, in FP64 where that cannot tell: FP64 for every member
// against every state cost 10,000 cycles per removal and per 256 bound members. The block finds
// the first unbound member; warp 0 goes on from it, 32 members (a window) at a time, supposing
// that those unbound on entry are removed: their masses, reciprocals and products are formed by
// all lanes, the updates run back to back (five dependent FP64 instructions each), and every lane
// then tests its member against the state just before it. What precedes the first member that
// came out otherwise is as the reference has it; the window ends there.
// What bounds it: the FP64 chain of the removals. Measured: 262,144 particles, 1,564
// clumps, with the sort after it: 9.6 -> 1.7 ms.
#pragma once

constexpr int kUb = 256;

struct UbShared {
    double4_32a pos[kUb], vel[kUb];  // pos.w: the mass
    UbCand f[kUb];
    uint32_t idx[kUb];
    double upd[32 * 9];   // a window's removals: m x .. m vz, the masses before and after, 1 / after
    double hist[33 * 8];  // its states: x y z vx vy vz M, before it and after each removal
    double sd[8];         // the state
    float sf[13];         // as float pairs: hi[6], lo[6]; M
    uint32_t first[kUb / 32];
    uint32_t at;
};

// The same as the reference writes it; S: x y z vx vy vz M.
__device__ __forceinline__ bool ub_exact(const double4_32a p, const double4_32a v, const double *S, const CP &cp) {
    const double M = S[6], Mr = M - p.w;  // > 0: at least two members remain
    const double y = __drcp_rn(Mr);
    const double cx = div_by_rcp(S[0] * M - p.x * p.w, Mr, y), cy = div_by_rcp(S[1] * M - p.y * p.w, Mr, y),
                 cz = div_by_rcp(S[2] * M - p.z * p.w, Mr, y);
    const double vx = div_by_rcp(S[3] * M - v.x * p.w, Mr, y), vy = div_by_rcp(S[4] * M - v.y * p.w, Mr, y),
                 vz = div_by_rcp(S[5] * M - v.z * p.w, Mr, y);
    const double dx = cx - p.x;
    const double ex = (vx - 0.0 * dx) - v.x, ey = (vy - cp.shear * dx) - v.y, ez = (vz - 0.0 * dx) - v.z;
    const double e = +0.5 / M * norm2_3(ex, ey, ez) - cp.G / norm3(cx - p.x, cy - p.y, cz - p.z);
    return e > 0;
}

__device__ __forceinline__ void ub_floats(const double *S, float *sf) {
#pragma unroll
    for (int c = 0; c < 6; ++c) split_any(S[c], sf[c], sf[6 + c]);
    float l;
    split_any(S[6], sf[12], l);
}

__global__ void __launch_bounds__(kUb) k_unbind(const uint32_t *list, CT ct, Pool P, const double4_32a *pos, const double4_32a *vel, FTree ft,
                                                CP cp) {
    extern __shared__ __align__(16) unsigned char ub_dyn[];
    UbShared &sh = *reinterpret_cast<UbShared *>(ub_dyn);
    const int tid = threadIdx.x, lane = tid & 31, wid = tid >> 5;
    const unsigned full = 0xffffffffu, below = (1u << lane) - 1u;
    const uint32_t s = list[blockIdx.x], o = ct.moff[s], m0 = ct.mn[s];
    const float G32 = (float)cp.G, shear32 = (float)cp.shear;
    double comp = 0.0, M = 0.0;  // warp 0: component `lane` < 6 of the state, the mass
    uint32_t back = m0 - 1;      // warp 0: the last member
    if (wid == 0) {
        const double4_32a c = ct.com[s], v = ct.vcom[s];
        M = ct.M[s];
        const double st[6] = {c.x, c.y, c.z, v.x, v.y, v.z};
        for (int k = 0; k < 6; ++k) comp = lane == k ? st[k] : comp;
        if (lane < 6) sh.sd[lane] = comp;
        if (lane == 6) sh.sd[6] = M;
        __syncwarp();
        if (lane == 0) ub_floats(sh.sd, sh.sf);
    }
    __syncthreads();
    // member i - k is the tile's entry k; member 0 is never tested
    for (int i = (int)m0 - 1; i >= 1; i -= kUb) {
        const int tlen = min(kUb, i);
        UbCand cf;
        if (tid < tlen) {
            const uint32_t q = P.idx[o + i - tid];
            const double4_32a p = pos[q], v = vel[q];
            const float4 ph = ft.phi[q], pl = ft.plo[q];
            cf.ph[0] = ph.x; cf.ph[1] = ph.y; cf.ph[2] = ph.z;
            cf.pl[0] = pl.x; cf.pl[1] = pl.y; cf.pl[2] = pl.z;
            split_any(v.x, cf.vh[0], cf.vl[0]);
            split_any(v.y, cf.vh[1], cf.vl[1]);
            split_any(v.z, cf.vh[2], cf.vl[2]);
            float l;
            split_any(p.w, cf.w, l);
            cf.lim = bound_limits(cf, shear32);
            sh.pos[tid] = p;
            sh.vel[tid] = v;
            sh.f[tid] = cf;
            sh.idx[tid] = q;
        }
        __syncthreads();
        for (int from = 0; from < tlen;) {
            bool un = false;
            if (tid >= from && tid < tlen) {
                const int r = ub_test(cf, sh.sf, G32, shear32);
                un = r == 1;
                if (r < 0) un = ub_exact(sh.pos[tid], sh.vel[tid], sh.sd, cp);
            }
            const unsigned b = __ballot_sync(full, un);
            if (lane == 0) sh.first[wid] = b ? (uint32_t)(wid * 32 + __ffs(b) - 1) : (uint32_t)kUb;
            __syncthreads();
            uint32_t f = kUb;
            for (int w = 0; w < kUb / 32; ++w) f = min(f, sh.first[w]);
            if (f == (uint32_t)kUb) break;  // the rest of the tile is bound
            if (wid == 0) {
                uint32_t at = f;
                for (bool any = true; any && at < (uint32_t)tlen;) {
                    const uint32_t k = at + lane;
                    const bool has = k < (uint32_t)tlen;
                    const UbCand c = sh.f[has ? k : at];
                    const unsigned U = __ballot_sync(full, has && ub_test(c, sh.sf, G32, shear32) != 0);
                    any = U != 0;
                    if (!any) {
                        at = min(at + 32u, (uint32_t)tlen);
                        break;
                    }
                    // the masses after each supposed removal: integers on the grid of M's binade, up
                    // to the first lane where that does not hold (then one ordinary subtraction)
                    const double m = has ? sh.pos[k].w : 0.0;
                    const bool sup = (U >> lane) & 1u;
                    const uint64_t mb = dbits(M);
                    const uint32_t ex = (uint32_t)(mb >> 52) & 0x7ffu;
                    long long dn = 0;
                    bool ok = true;
                    if (sup) ok = (mb >> 63) == 0 && ex > 60u && ex < 2000u && grid_term(m, ex, dn) && dn > 0;
                    const long long mine = ok ? dn : 0;
                    long long nl = mine;
                    for (int d = 1; d < 32; d <<= 1) {
                        const long long x = __shfl_up_sync(full, nl, d);
                        if (lane >= d) nl += x;
                    }
                    nl = (long long)((mb & 0xfffffffffffffull) | (1ull << 52)) - nl;
                    ok = ok && (!sup || (nl > (1LL << 52) && nl + mine <= (1LL << 53)));
                    const unsigned okm = __ballot_sync(full, ok);
                    uint32_t lim = ~okm ? (uint32_t)__ffs(~okm) - 1u : 32u;  // lanes of this window
                    unsigned use = lim < 32 ? U & ((1u << lim) - 1u) : U;
                    double Mo = grid_value(nl + mine, ex), Mn = grid_value(nl, ex);
                    if (!use) {
                        const uint32_t j = (uint32_t)__ffs(U) - 1u;
                        use = 1u << j;
                        lim = j + 1;
                        Mo = M;
                        Mn = M - m;
                    }
                    const uint32_t rank = __popc(use & below), cnt = __popc(use);
                    if ((use >> lane) & 1u) {
                        const double4_32a p = sh.pos[k], v = sh.vel[k];
                        double *t = sh.upd + 9 * rank;
                        t[0] = p.x * m;
                        t[1] = p.y * m;
                        t[2] = p.z * m;
                        t[3] = v.x * m;
                        t[4] = v.y * m;
                        t[5] = v.z * m;
                        t[6] = Mo;
                        t[7] = Mn;
                        t[8] = __drcp_rn(Mn);
                    }
                    if (lane < 6) sh.hist[lane] = comp;
                    if (lane == 6) sh.hist[6] = M;
                    __syncwarp();
                    // the updates: RN(RN(RN(c M) - RN(q m)) / M') per component, the state kept after each
                    {
                        const int cc = lane < 6 ? lane : 6;
                        double x = lane < 6 ? comp : 0.0;
                        for (uint32_t a = 0; a < cnt; ++a) {
                            const double *t = sh.upd + 9 * a;
                            const double sub = lane < 6 ? t[cc] : 0.0;
                            x = div_by_rcp(x * t[6] - sub, t[7], t[8]);
                            if (lane < 7) sh.hist[8 * (a + 1) + lane] = lane < 6 ? x : t[7];
                        }
                    }
                    __syncwarp();
                    // every member against the state before it
                    bool unb = false;
                    const double *S = sh.hist + 8 * rank;
                    if (has && (uint32_t)lane < lim) {
                        float sf[13];
                        ub_floats(S, sf);
                        const int r = ub_test(c, sf, G32, shear32);
                        unb = r < 0 ? ub_exact(sh.pos[k], sh.vel[k], S, cp) : r == 1;
                    }
                    const unsigned B = __ballot_sync(full, unb);
                    unsigned diff = B ^ use;
                    if (lim < 32) diff &= (1u << lim) - 1u;
                    uint32_t end = diff ? (uint32_t)__ffs(diff) - 1u : lim;  // lanes before it came out as supposed
                    const unsigned out = end < 32 ? use & ((1u << end) - 1u) : use;
                    if (diff && ((use >> end) & 1u)) ++end;  // supposed to be unbound and is bound: settled too
                    const uint32_t n = __popc(out);
                    // swap with the last member and drop it (src/tree.hpp:4660-4663), in order: at once
                    // where the last n members lie beyond this window
                    if (n) {
                        if (back - (n - 1) > (uint32_t)i - at) {
                            if ((out >> lane) & 1u) {
                                const uint32_t w = back - rank, last = P.idx[o + w];
                                P.idx[o + w] = sh.idx[k];
                                P.idx[o + i - k] = last;
                            }
                        } else if (lane == 0) {
                            uint32_t bk = back;
                            for (unsigned r = out; r; r &= r - 1, --bk) {
                                const uint32_t b = (uint32_t)i - (at + (uint32_t)__ffs(r) - 1u);
                                const uint32_t tmp = P.idx[o + b];
                                P.idx[o + b] = P.idx[o + bk];
                                P.idx[o + bk] = tmp;
                            }
                        }
                        back -= n;
                    }
                    comp = lane < 6 ? sh.hist[8 * n + lane] : 0.0;
                    M = sh.hist[8 * n + 6];
                    if (lane < 6) sh.sd[lane] = comp;
                    if (lane == 6) sh.sd[6] = M;
                    __syncwarp();
                    if (lane == 0) ub_floats(sh.sd, sh.sf);
                    __syncwarp();
                    at += end;
                }
                if (lane == 0) sh.at = at;
            }
            __syncthreads();
            from = (int)sh.at;
        }
        __syncthreads();
    }
    if (wid == 0) {
        if (lane == 0) {
            ct.mn[s] = back + 1;
            ct.M[s] = sh.sd[6];
            ct.com[s] = make_double4_32a(sh.sd[0], sh.sd[1], sh.sd[2], 0);
            ct.vcom[s] = make_double4_32a(sh.sd[3], sh.sd[4], sh.sd[5], 0);
        }
    }
}
