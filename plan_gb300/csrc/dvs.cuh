// The arithmetic of --Density_Vs_Scale, host+device (dvs.cu runs the set-up, the queries and the
// node classes on the GPU; the parity tests compile them for the CPU and run them, with the
// plain count dvs_count, on the oracle's tree).
//
// BasicAnalysesWithTree (src/analyses.hpp:196-333) counts the tree points within a ball
// around every cell centre of the grid (z from the cell centre at the box centre down past
// the lowest point, up to the highest point), for radii of half a cell times 1, 2, 4, ...
// up to the box, plus eight sub-centres (half a cell off along each orthant) for the three
// smallest radii and one more per orthant (a quarter cell further) for the smallest. Each
// count walks the tree with RecursiveBallSearchCountWithShear (src/tree.hpp:3306-3402): far
// nodes are compared through their shearing-periodic image (x and y faces; the x image moves
// in y by the shear), points in a reached leaf by their plain distance. The largest count per
// radius becomes a density, count * m / (4 pi / 3 r^3).
#pragma once

#include <cmath>
#include <cstdint>
#include <vector>

#ifdef __CUDACC__
#define PLAN_DVS_HD __host__ __device__
#else
#define PLAN_DVS_HD
#endif

namespace plan {

constexpr int kDvsMaxLevels = 24;
constexpr int kDvsDepth = 34;  // the root and 32 levels below it

struct DvsGeom {
    double box_length[3], box_min[3], box_max[3];
    double shear;    // shear_speed * time
    double diag;     // sqrt(3) (to_diagonal)
    double radius[kDvsMaxLevels];
    double maxd[kDvsMaxLevels][3];
    double sub1[3], sub2[3];  // half and quarter cell
    int nlev, nsub;           // levels; levels with sub-centres (at most 3)
    uint32_t nx, ny, nz, nvar;
};

// The parameters the analysis reads (after the first snapshot's box and the run's settings).
struct DvsParams {
    double box_length[3], box_min[3], box_max[3], box_center[3];
    double box_half_width0, max_half_width, cell_length[3], shear_speed, mass_per_particle0;
};

// Geometry and cell-centre coordinates, with the reference's host arithmetic (the centres are
// accumulated x += cell as its loops do). zlo, zhi: extreme z of the tree points. 0; -1 when
// the grid gives more radii than kDvsMaxLevels; -2 when an axis would need more than 2^24
// centres (coordinates far outside any box the parameters describe, where the reference's
// loops would run for ever); -3 when there are more than (2^31 - 1) x 128 queries (3 x 10^11: hours
// of device time).
inline int dvs_setup(const DvsParams &p, double time, double zlo, double zhi, DvsGeom &g, std::vector<double> &xs, std::vector<double> &ys,
                     std::vector<double> &zs) {
    g = DvsGeom{};
    for (int d = 0; d < 3; ++d) {
        g.box_length[d] = p.box_length[d];
        g.box_min[d] = p.box_min[d];
        g.box_max[d] = p.box_max[d];
        g.sub1[d] = p.cell_length[d] / 2.0;
        g.sub2[d] = p.cell_length[d] / 4.0;
    }
    g.shear = p.shear_speed * time;
    g.diag = std::sqrt(3);
    const double kMaxCentres = 16777216.0;
    if (!(p.cell_length[0] > 0 && p.cell_length[1] > 0 && p.cell_length[2] > 0)) return -2;
    for (int d = 0; d < 2; ++d)
        if (!((p.box_max[d] - p.box_min[d]) / p.cell_length[d] < kMaxCentres)) return -2;
    if (!((zhi - zlo) / p.cell_length[2] < kMaxCentres) || !(std::fabs(p.box_center[2] - zlo) / p.cell_length[2] < kMaxCentres)) return -2;
    double z_min = p.box_center[2] - p.cell_length[2] / 2.0;
    const double z_max = zhi;
    while (z_min - p.cell_length[2] > zlo) z_min -= p.cell_length[2];
    const int nlev = (int)std::round(std::log10(p.box_half_width0 * 2 / p.cell_length[0]) / std::log10(2.0)) + 1;
    if (nlev < 1 || nlev > kDvsMaxLevels) return -1;
    g.nlev = nlev;
    g.nsub = nlev < 3 ? nlev : 3;
    for (int i = 0; i < nlev; ++i) {
        g.radius[i] = p.cell_length[0] / 2.0;
        g.radius[i] *= std::pow(2.0, i);
        for (int d = 0; d < 3; ++d) g.maxd[i][d] = p.box_length[d] - g.radius[i];
        g.maxd[i][2] = 100 * p.max_half_width;  // no periodic search in z
    }
    g.nvar = (uint32_t)(nlev + 8 * g.nsub + 8);
    xs.clear();
    ys.clear();
    zs.clear();
    for (double z = z_min; z < z_max; z += p.cell_length[2]) zs.push_back(z);
    for (double y = p.box_min[1] + 0.5 * p.cell_length[1]; y < p.box_max[1]; y += p.cell_length[1]) ys.push_back(y);
    for (double x = p.box_min[0] + 0.5 * p.cell_length[0]; x < p.box_max[0]; x += p.cell_length[0]) xs.push_back(x);
    g.nx = (uint32_t)xs.size();
    g.ny = (uint32_t)ys.size();
    g.nz = (uint32_t)zs.size();
    // each axis is below 2^24, so the product is checked in double before it is formed in 64 bits
    if ((double)g.nx * g.ny * g.nz * g.nvar > 2147483647.0 * 128.0) return -3;
    return 0;
}

// Query `tid` of nx ny nz nvar: its point and radius level. Variant v < nlev is the centre at
// level v; then eight sub-centres per level below nsub; then the eight quarter-cell centres
// of level 0 (the reference's inner loop offsets by the outer orthant eight times over,
// src/analyses.hpp:296-305, so it adds one centre per orthant).
PLAN_DVS_HD inline void dvs_query(const DvsGeom &g, const double *xs, const double *ys, const double *zs, uint64_t tid, double &x, double &y,
                                  double &z, int &lev) {
    const int orth[8][3] = {{-1, -1, -1}, {1, -1, -1}, {-1, 1, -1}, {1, 1, -1}, {-1, -1, 1}, {1, -1, 1}, {-1, 1, 1}, {1, 1, 1}};
    const uint32_t v = (uint32_t)(tid % g.nvar);
    const uint64_t ci = tid / g.nvar;
    const uint32_t ix = (uint32_t)(ci % g.nx), iy = (uint32_t)((ci / g.nx) % g.ny), iz = (uint32_t)(ci / ((uint64_t)g.nx * g.ny));
    x = xs[ix];
    y = ys[iy];
    z = zs[iz];
    if (v < (uint32_t)g.nlev) {
        lev = (int)v;
        return;
    }
    int o;
    if (v < (uint32_t)(g.nlev + 8 * g.nsub)) {
        o = (int)(v - g.nlev) % 8;
        lev = (int)(v - g.nlev) / 8;
    } else {
        o = (int)(v - g.nlev - 8 * g.nsub);
        lev = 0;
    }
    x = x + g.sub1[0] * orth[o][0];
    y = y + g.sub1[1] * orth[o][1];
    z = z + g.sub1[2] * orth[o][2];
    if (v >= (uint32_t)(g.nlev + 8 * g.nsub)) {
        x = x + g.sub2[0] * orth[o][0];
        y = y + g.sub2[1] * orth[o][1];
        z = z + g.sub2[2] * orth[o][2];
    }
}

// Where a node lies for the ball of radius r around c: 0 outside, 1 contained, 2 met
// (src/tree.hpp:3308-3380). nc: the node's centre, hw its half width.
PLAN_DVS_HD inline int dvs_class(const double c[3], const double node[3], double hw, double r, const double *maxd, const DvsGeom &g) {
    double nc[3] = {node[0], node[1], node[2]}, c2c[3];
    // ShearedCenter2Center (src/tree.hpp:3308-3331)
    for (int i = 0; i < 3; ++i) {
        c2c[i] = c[i] - nc[i];
        if (std::fabs(c2c[i]) > maxd[i]) {
            if (c2c[i] > 0) c2c[i] -= g.box_length[i];
            else c2c[i] += g.box_length[i];
            if (i == 0) {
                if (c[0] < 0) {
                    nc[1] -= g.shear;
                    nc[1] += (double)(int)((g.box_max[1] - nc[1]) / g.box_length[1]) * g.box_length[1];
                } else {
                    nc[1] += g.shear;
                    nc[1] -= (double)(int)((nc[1] - g.box_min[1]) / g.box_length[1]) * g.box_length[1];
                }
            }
        }
    }
    // SphereContainNodeWithShear (src/tree.hpp:3335-3346)
    const double tmp = hw * g.diag;
    const double t0 = std::fabs(c2c[0]) + tmp, t1 = std::fabs(c2c[1]) + tmp, t2 = std::fabs(c2c[2]) + tmp;
    if (t0 * t0 + t1 * t1 + t2 * t2 < r * r) return 1;
    // SphereNodeIntersectWithShear (src/tree.hpp:3350-3380)
    const double cd = c2c[0] * c2c[0] + c2c[1] * c2c[1] + c2c[2] * c2c[2];
    const double tr = tmp + r;
    if (cd > tr * tr) return 0;
    if (cd < r || cd < hw) return 2;
    double m2 = 0;
    for (int d = 0; d < 3; ++d) {
        const double lo = (c[d] - c2c[d]) - hw, hi = (c[d] - c2c[d]) + hw;
        if (c[d] < lo) m2 += (c[d] - lo) * (c[d] - lo);
        else if (c[d] > hi) m2 += (c[d] - hi) * (c[d] - hi);
    }
    return m2 <= r * r ? 2 : 0;
}

// dvs_class in FP32: the same class, or -1 when a comparison is too close to call (or not
// finite). The single-precision geometry: every coordinate, length and shear rounded once, and
// eps, an absolute bound on the error of any difference formed from them: 2^-20 of the largest
// magnitude among them (their roundings and the few operations on them stay below half of it).
struct DvsGeomF {
    float box_length[3], box_min1, box_max1, shear, eps;
    float radius[kDvsMaxLevels];
    float maxd[kDvsMaxLevels][3];
};

// coord: the largest magnitude of a node's or a query's coordinate
inline DvsGeomF dvs_geom_f(const DvsGeom &g, double coord) {
    DvsGeomF f{};
    double big = coord + std::fabs(g.shear);
    for (int d = 0; d < 3; ++d) {
        f.box_length[d] = (float)g.box_length[d];
        big += std::fabs(g.box_length[d]) + std::fabs(g.box_min[d]) + std::fabs(g.box_max[d]);
    }
    f.box_min1 = (float)g.box_min[1];
    f.box_max1 = (float)g.box_max[1];
    f.shear = (float)g.shear;
    f.eps = (float)(big * 9.5367431640625e-07);
    for (int i = 0; i < g.nlev; ++i) {
        f.radius[i] = (float)g.radius[i];
        for (int d = 0; d < 3; ++d) f.maxd[i][d] = (float)g.maxd[i][d];
    }
    return f;
}

// a < b for values within ea and eb of the exact ones: 1 yes, 0 no, -1 too close or not finite
PLAN_DVS_HD inline int dvs_less(float a, float ea, float b, float eb) {
    if (a + ea < b - eb) return 1;
    if (a - ea > b + eb) return 0;
    return -1;
}

PLAN_DVS_HD inline int dvs_class_f(const float c[3], const float node[3], float hw, int lev, const DvsGeomF &g) {
    constexpr float kRel = 1.9073486328125e-06f;  // 2^-19: the roundings of the squares and sums below
    const float r = g.radius[lev];
    float n1 = node[1], d[3];
    for (int i = 0; i < 3; ++i) {
        d[i] = c[i] - (i == 1 ? n1 : node[i]);
        // z is never periodic: its limit is a hundred boxes (maxd[2]), which a tree inside it keeps
        const int far = dvs_less(g.maxd[lev][i], g.eps, std::fabs(d[i]), g.eps);
        if (far < 0) return -1;
        if (far) {
            d[i] = d[i] > 0 ? d[i] - g.box_length[i] : d[i] + g.box_length[i];
            if (i == 0) {
                if (std::fabs(c[0]) <= g.eps) return -1;
                float q;
                if (c[0] < 0) {
                    n1 = n1 - g.shear;
                    q = (g.box_max1 - n1) / g.box_length[1];
                } else {
                    n1 = n1 + g.shear;
                    q = (n1 - g.box_min1) / g.box_length[1];
                }
                const float k = std::trunc(q), e = 4.0f * g.eps / g.box_length[1];  // whole boxes moved
                const float f = std::fabs(q - k);
                if (!(e < 0.25f && std::fabs(q) < 4096.0f) || (f < e && std::fabs(q) > 0.5f) || f > 1.0f - e) return -1;
                n1 = c[0] < 0 ? n1 + k * g.box_length[1] : n1 - k * g.box_length[1];
            }
        }
    }
    const float e = 8.0f * g.eps + hw * kRel;  // of a difference, moved by boxes or not, and of what hw adds
    const float a0 = std::fabs(d[0]), a1 = std::fabs(d[1]), a2 = std::fabs(d[2]);
    const float tmp = hw * 1.7320508f, rr = r * r, erR = rr * kRel;
    const float t0 = a0 + tmp, t1 = a1 + tmp, t2 = a2 + tmp;
    const float s = t0 * t0 + t1 * t1 + t2 * t2;
    const int in = dvs_less(s, s * kRel + e * (2.0f * (t0 + t1 + t2) + 3.0f * e), rr, erR);
    if (in != 0) return in;
    const float cd = a0 * a0 + a1 * a1 + a2 * a2, ecd = cd * kRel + e * (2.0f * (a0 + a1 + a2) + 3.0f * e);
    const float tr = tmp + r, tt = tr * tr;
    const int out = dvs_less(tt, tt * kRel, cd, ecd);
    if (out != 0) return out < 0 ? -1 : 0;
    const int near_r = dvs_less(cd, ecd, r, r * kRel), near_h = dvs_less(cd, ecd, hw, hw * kRel);
    if (near_r == 1 || near_h == 1) return 2;
    if (near_r < 0 || near_h < 0) return -1;
    const float b0 = a0 > hw ? a0 - hw : 0.0f, b1 = a1 > hw ? a1 - hw : 0.0f, b2 = a2 > hw ? a2 - hw : 0.0f;
    const float m2 = b0 * b0 + b1 * b1 + b2 * b2;
    const int gap = dvs_less(rr, erR, m2, m2 * kRel + e * (2.0f * (b0 + b1 + b2) + 3.0f * e));
    return gap < 0 ? -1 : (gap ? 0 : 2);
}

// Walks the nodes the ball meets from the root, depth first: contained(n) for every contained
// node, leaf(n) for every leaf that is met. classify(n) gives dvs_class. The siblings still to
// visit are kept per level. *overflow is set (and the walk stops) if they would overrun the
// stack, which a 32-level octree cannot make happen.
template <class Tree, class Class, class Contained, class Leaf>
PLAN_DVS_HD inline void dvs_walk(const Tree &t, Class classify, Contained contained, Leaf leaf, bool *overflow) {
    uint32_t next[kDvsDepth], end[kDvsDepth];
    int top = 0;
    next[0] = 0;
    end[0] = 1;
    while (top >= 0) {
        if (next[top] == end[top]) {
            --top;
            continue;
        }
        const uint32_t n = next[top]++;
        const int cls = classify(n);
        if (cls == 1) {
            contained(n);
        } else if (cls == 2) {
            const uint32_t nd = t.daughters(n);
            if (nd == 0) {
                leaf(n);
            } else if (top + 1 == kDvsDepth) {
                *overflow = true;
                return;
            } else {
                ++top;
                next[top] = t.first(n);
                end[top] = next[top] + nd;
            }
        }
    }
}

// The points of the listed leaves, counted by a warp: inside grows by those within the ball, partial
// falls by all of a leaf's. Where largest is given, the warp stops once the count cannot exceed it.
// Other warps raise that word meanwhile, so the lanes must not each decide on a value of their
// own: one that leaves would be missing in the next sum. Warp: lane(), and first(v) and sum(v)
// over all lanes; load(word) reads what others write. near(p): whether point p lies within the ball.
template <class Warp, class Tree, class Near>
PLAN_DVS_HD inline void dvs_count_leaves(const Warp &w, const Tree &t, const uint32_t *leaves, uint32_t nleaf, const uint32_t *largest,
                                         uint32_t &inside, uint32_t &partial, Near near) {
    for (uint32_t k = 0; k < nleaf; ++k) {
        if (largest && inside + partial <= w.first(w.lane() == 0 ? w.load(largest) : 0u)) return;
        const uint32_t b = t.begin(leaves[k]), e = t.end(leaves[k]);
        uint32_t in = 0;
        for (uint32_t p = b + w.lane(); p < e; p += 32) in += near(p) ? 1u : 0u;
        inside += w.sum(in);
        partial -= e - b;
    }
}

// RecursiveBallSearchCountWithShear (src/tree.hpp:3382-3402): the points of the contained nodes
// and those of the met leaves within r, compared without the image. Tree provides node(n, cx,
// cy, cz, hw), begin(n), end(n), first(n), daughters(n) and point(q, x, y, z).
template <class Tree>
PLAN_DVS_HD inline uint32_t dvs_count(const Tree &t, double cx, double cy, double cz, double r, const double *maxd, const DvsGeom &g,
                                      bool *overflow) {
    uint32_t count = 0;
    const double c[3] = {cx, cy, cz};
    dvs_walk(
        t,
        [&](uint32_t n) {
            double nc[3], hw;
            t.node(n, nc[0], nc[1], nc[2], hw);
            return dvs_class(c, nc, hw, r, maxd, g);
        },
        [&](uint32_t n) { count += t.end(n) - t.begin(n); },
        [&](uint32_t n) {
            for (uint32_t q = t.begin(n); q != t.end(n); ++q) {
                double px, py, pz;
                t.point(q, px, py, pz);
                const double dx = c[0] - px, dy = c[1] - py, dz = c[2] - pz;
                if (dx * dx + dy * dy + dz * dz <= r * r) ++count;
            }
        },
        overflow);
    return count;
}

// The reported density of each radius from the largest count (src/analyses.hpp:325-328).
inline double dvs_density(uint32_t max_count, double radius, double mass_per_particle0) {
    double v = max_count;
    v *= (mass_per_particle0 / (4.1887902047863910 * std::pow(radius, 3)));
    return v;
}

}  // namespace plan
