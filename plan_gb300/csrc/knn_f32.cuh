// FP32-filtered KNN with the reference's exact results.
//
// On this GPU a dependent FP64 add takes ~63 cycles and FP64 issue is ~1/72 of FP32, so the
// reference's FP64 traversal is recast: points and node centres are held as exact float
// hi/lo pairs (every coordinate is a float32 or a float32 shifted by the box length, so two
// floats represent it exactly; node centres are dyadic), differences are formed as
// (a_hi - b_hi) + (a_lo - b_lo), and every comparison the reference makes in FP64 is
// decided in FP32 when the FP32 value is outside a proven error bound of the threshold.
// The bound used is relative 2^-17 plus a small absolute term, against a worst-case FP32
// error near 2^-20 relative, so a decided comparison always agrees with the FP64 one.
// Coordinates that are not float sums (ghost images shifted by the shear at t != 0, clump centres,
// a program's own positions) are held to 2^-48 relative, an absolute error below 1e-15 per
// difference for |x| < 0.25; squared distances then err by at most 2*sqrt(3)*d*1e-15, which
// 2^-17*d^2 + 1e-24 covers for every d. Larger coordinates scale the absolute terms (Tol).
// A node test inside its bound is decided in FP64. Where the order of two points matters and their
// distances are too close, the FP64 distances of the candidates are sorted; a tie among the k
// nearest or at their boundary sends the query to the exact heap path.
#pragma once

namespace plan {

// The absolute error terms of a squared distance and of a difference.
struct Tol {
    float sq, len;
};

// reach: the largest magnitude of a coordinate in the root box. Positions up to twice as far out
// are held as well as 2 reach; for one beyond, the distance to any point of the box is at least
// half its own magnitude, and the relative bound alone covers it.
inline Tol tol_of(double reach) {
    const double k = 8.0 * reach > 1.0 ? 8.0 * reach : 1.0;
    return Tol{(float)(1e-24 * k * k), (float)(1e-14 * k)};
}

struct FTree {
    const float4 *phi, *plo;  // points: x, y, z (hi / lo)
    const float4 *nhi, *nlo;  // nodes: cx, cy, cz, hw (hi / lo)
    Tol tol;
};

constexpr float kRel = 7.62939453125e-06f;  // 2^-17
constexpr float kAbs = 1e-30f;
constexpr float kSqrt3f = 1.7320508075688772f;

// a < b decided with relative/absolute error bounds on both sides (any signs): 1 true,
// 0 false, -1 unsure
__device__ __forceinline__ int f_less(float a, float b, float abs_a = kAbs) {
    float ea = fabsf(a) * kRel + abs_a, eb = fabsf(b) * kRel;
    if (a + ea < b - eb) return 1;
    if (a - ea > b + eb) return 0;
    return -1;
}

__device__ __forceinline__ float f_diff(float ah, float al, float bh, float bl) { return (ah - bh) + (al - bl); }

// SphereContainNode in FP32: 1 contained, 0 not, -1 unsure
__device__ __forceinline__ int f_contained(const float4 nh, const float4 nl, const float4 qh, const float4 ql, float r, Tol tol) {
    float t = nh.w * kSqrt3f;
    float a = fabsf(f_diff(nh.x, nl.x, qh.x, ql.x)) + t;
    float b = fabsf(f_diff(nh.y, nl.y, qh.y, ql.y)) + t;
    float c = fabsf(f_diff(nh.z, nl.z, qh.z, ql.z)) + t;
    float s = a * a + b * b + c * c;
    return f_less(s, r * r, tol.sq);
}

// SphereNodeIntersect in FP32: 1 intersects, 0 not, -1 unsure
__device__ __forceinline__ int f_intersects(const float4 nh, const float4 nl, const float4 qh, const float4 ql, float r, Tol tol) {
    float dx = f_diff(nh.x, nl.x, qh.x, ql.x), dy = f_diff(nh.y, nl.y, qh.y, ql.y), dz = f_diff(nh.z, nl.z, qh.z, ql.z);
    float c2c = dx * dx + dy * dy + dz * dz;
    float t = nh.w * kSqrt3f + r;
    int outside = f_less(t * t, c2c, tol.sq);  // c2c > t^2
    if (outside == 1) return 0;
    if (outside == -1) return -1;
    int a = f_less(c2c, r, tol.sq), b = f_less(c2c, nh.w, tol.sq);
    if (a == 1 || b == 1) return 1;
    if (a == -1 || b == -1) return -1;
    // exact box distance: q below, inside or above each face (differences q - c vs +-hw). What is
    // left beyond a face carries the roundings of the difference and of hw, 2^-22 (e + hw) at most,
    // whatever the sphere's size: in its square 2^-21 hw e on top of the relative bound.
    float m2 = 0.f, beyond = 0.f;
    float d3[3] = {-dx, -dy, -dz};  // q - c
    for (int k = 0; k < 3; ++k) {
        float u = d3[k];
        int below = f_less(u, -nh.w, tol.len), above = f_less(nh.w, u, tol.len);
        if (below == -1 || above == -1) return -1;
        if (below == 1) { float e = u + nh.w; m2 += e * e; beyond -= e; }
        else if (above == 1) { float e = u - nh.w; m2 += e * e; beyond += e; }
    }
    int in = f_less(r * r, m2, tol.sq + nh.w * beyond * 9.5367431640625e-07f);  // m2 > r^2 means no intersection
    if (in == -1) return -1;
    return in == 1 ? 0 : 1;
}

__device__ __forceinline__ float f_dr2(const float4 qh, const float4 ql, const float4 ph, const float4 pl) {
    float dx = f_diff(qh.x, ql.x, ph.x, pl.x), dy = f_diff(qh.y, ql.y, ph.y, pl.y), dz = f_diff(qh.z, ql.z, ph.z, pl.z);
    return dx * dx + dy * dy + dz * dz;
}

// Upper/lower bounds of the FP64 distance given the FP32 one.
__device__ __forceinline__ float f_hi(float v, Tol tol) { return v * (1.f + kRel) + tol.sq; }
__device__ __forceinline__ float f_lo(float v, Tol tol) { return v * (1.f - kRel) - tol.sq; }

}  // namespace plan
