// The boundness test of the rebinding (src/tree.hpp:4686-4694) in FP32, with the error bound that
// lets it decide.
#pragma once

namespace plan {

// A candidate as float hi/lo pairs (x = hi + lo to 2^-48): position, velocity, and its mass.
struct CandF {
    float ph[3], pl[3], vh[3], vl[3], w;
};

// What the pairs' absolute errors ask for: close, a squared distance below which positions of
// magnitude up to x cancel too far, and dv2, 2^22 times the square of the error that they and
// velocities of magnitude up to v leave in the sheared velocity.
struct BoundLimits {
    float close, dv2;
};

__device__ __forceinline__ BoundLimits bound_limits(float x, float v, float shear) {
    const float dv = (v + fabsf(shear) * x) * 2.910383045673e-11f;  // 2^-46 2^11
    return BoundLimits{fmaxf(x * x * 8.8817842e-16f, 1e-30f), dv * dv};  // 2^-50
}

// The limits of one candidate. Two pairs that nearly cancel have coordinates of one size, so the
// candidate's own stand for both.
__device__ __forceinline__ BoundLimits bound_limits(const CandF &c, float shear) {
    return bound_limits(fmaxf(fmaxf(fabsf(c.ph[0]), fabsf(c.ph[1])), fabsf(c.ph[2])),
                        fmaxf(fmaxf(fabsf(c.vh[0]), fabsf(c.vh[1])), fabsf(c.vh[2])), shear);
}

// The boundness test entirely in FP32 from hi/lo pairs of the state (sh, sl: x, y, z, vx,
// vy, vz) and of the candidate: 1 bound, 0 not, -1 too close to call (then bound_fp64).
// Differences of hi/lo pairs carry a relative error below 2^-22 and an absolute one of 2^-47 of
// the coordinates. For the distance the absolute one is below 2^-22 as well unless the pairs cancel
// to less than 2^-25 of the coordinates (refused). In the velocity every term errs by dv besides, and
// ey, a difference of two values, by d = 2^-20 (|t1| + |t2|). That is 2 |ey| d + 2 d^2 in K from d, and
// from dv 2 |e| dv <= 2^-21 e^2 + 2^21 dv^2 a term: a relative error, and 2^22 dv^2 in K / 2. With at
// most ten further FP32 roundings per term, A and B stay within their margins below; the
// reference's own FP64 rounding is far smaller.
__device__ __forceinline__ int bound_hilo(const CandF &c, float Mf, const float sh[6], const float sl[6], float G, float shear,
                                          const BoundLimits lim) {
    const float dx = (sh[0] - c.ph[0]) + (sl[0] - c.pl[0]);
    const float dy = (sh[1] - c.ph[1]) + (sl[1] - c.pl[1]);
    const float dz = (sh[2] - c.ph[2]) + (sl[2] - c.pl[2]);
    const float ex = (sh[3] - c.vh[0]) + (sl[3] - c.vl[0]);
    const float t1 = (sh[4] - c.vh[1]) + (sl[4] - c.vl[1]), t2 = shear * dx;
    const float ey = t1 - t2;
    const float ez = (sh[5] - c.vh[2]) + (sl[5] - c.vl[2]);
    const float K = ex * ex + ey * ey + ez * ez, D2 = dx * dx + dy * dy + dz * dz;
    const float M = Mf + c.w;
    if (!(K > 1e-30f && D2 > lim.close && K < 1e30f && D2 < 1e30f && M > 1e-30f && M < 1e30f)) return -1;
    const float A = 0.5f / M * K, B = G / sqrtf(D2);
    const float e = A - B;
    const float d = (fabsf(t1) + fabsf(t2)) * 9.5367431640625e-07f;   // 2^-20
    const float margin = (fabsf(A) + fabsf(B)) * 3.814697265625e-06f  // 2^-18
                         + (d * (fabsf(ey) + d) + lim.dv2) / M;
    if (e > margin) return 0;
    if (e < -margin) return 1;
    return -1;
}

// The same test with the FP32 quotient and square root taken by the fast intrinsics
// (__fdividef, rsqrtf: at most 2 ulp each for the argument ranges admitted above). With
// them A and B still carry a relative error below 2^-20, inside the margin.
__device__ __forceinline__ int bound_hilo_fast(const CandF &c, float Mf, const float sh[6], const float sl[6], float G, float shear,
                                          const BoundLimits lim) {
    const float dx = (sh[0] - c.ph[0]) + (sl[0] - c.pl[0]);
    const float dy = (sh[1] - c.ph[1]) + (sl[1] - c.pl[1]);
    const float dz = (sh[2] - c.ph[2]) + (sl[2] - c.pl[2]);
    const float ex = (sh[3] - c.vh[0]) + (sl[3] - c.vl[0]);
    const float t1 = (sh[4] - c.vh[1]) + (sl[4] - c.vl[1]), t2 = shear * dx;
    const float ey = t1 - t2;
    const float ez = (sh[5] - c.vh[2]) + (sl[5] - c.vl[2]);
    const float K = ex * ex + ey * ey + ez * ez, D2 = dx * dx + dy * dy + dz * dz;
    const float M = Mf + c.w;
    if (!(K > 1e-30f && D2 > lim.close && K < 1e30f && D2 < 1e30f && M > 1e-30f && M < 1e30f)) return -1;
    const float rM = __fdividef(1.0f, M);
    const float A = 0.5f * rM * K, B = G * rsqrtf(D2);
    const float e = A - B;
    const float d = (fabsf(t1) + fabsf(t2)) * 9.5367431640625e-07f;   // 2^-20
    const float margin = (fabsf(A) + fabsf(B)) * 3.814697265625e-06f  // 2^-18
                         + (d * (fabsf(ey) + d) + lim.dv2) * rM;
    if (e > margin) return 0;
    if (e < -margin) return 1;
    return -1;
}

}  // namespace plan
