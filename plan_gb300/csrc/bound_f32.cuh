// The boundness test of the rebinding (src/tree.hpp:4686-4694) in FP32, with the error bound that
// lets it decide.
#pragma once

namespace plan {

// A candidate as float hi/lo pairs (x = hi + lo to 2^-48): position, velocity, and its mass. close:
// a squared distance below which the pairs cancel too far; dv: the absolute error that the pairs
// leave in the sheared velocity. 15 words: odd, so that 32 candidates side by side meet no bank twice.
struct CandF {
    float ph[3], pl[3], vh[3], vl[3], w, close, dv;
};

// close and dv, once the pairs are there. Two pairs that nearly cancel have coordinates of one size,
// so the candidate's own stand for both.
__device__ __forceinline__ void cand_limits(CandF &c, float shear) {
    const float x = fmaxf(fmaxf(fabsf(c.ph[0]), fabsf(c.ph[1])), fabsf(c.ph[2]));
    const float v = fmaxf(fmaxf(fabsf(c.vh[0]), fabsf(c.vh[1])), fabsf(c.vh[2]));
    c.close = x * x * 8.8817842e-16f;                             // 2^-50
    c.dv = (v + fabsf(shear) * fabsf(c.ph[0])) * 1.4210855e-14f;  // 2^-46
}

// The boundness test entirely in FP32 from hi/lo pairs of the state (sh, sl: x, y, z, vx,
// vy, vz) and of the candidate: 1 bound, 0 not, -1 too close to call (then bound_fp64).
// Differences of hi/lo pairs carry a relative error below 2^-22 and an absolute one of 2^-47 of
// the coordinates. For the distance the absolute one is below 2^-22 as well unless the pairs cancel
// to less than 2^-25 of the coordinates (refused). In the velocity ex and ez err by dv besides, ey,
// a difference of two such values, by d = 2^-20 (|t1| + |t2|) + dv: 2 |e| d + d^2 per term in K. With
// at most ten further FP32 roundings per term, A and B stay within their margins below; the
// reference's own FP64 rounding is far smaller.
__device__ __forceinline__ int bound_hilo(const CandF &c, float Mf, const float sh[6], const float sl[6], float G, float shear) {
    const float dx = (sh[0] - c.ph[0]) + (sl[0] - c.pl[0]);
    const float dy = (sh[1] - c.ph[1]) + (sl[1] - c.pl[1]);
    const float dz = (sh[2] - c.ph[2]) + (sl[2] - c.pl[2]);
    const float ex = (sh[3] - c.vh[0]) + (sl[3] - c.vl[0]);
    const float t1 = (sh[4] - c.vh[1]) + (sl[4] - c.vl[1]), t2 = shear * dx;
    const float ey = t1 - t2;
    const float ez = (sh[5] - c.vh[2]) + (sl[5] - c.vl[2]);
    const float K = ex * ex + ey * ey + ez * ez, D2 = dx * dx + dy * dy + dz * dz;
    const float M = Mf + c.w;
    if (!(K > 1e-30f && D2 > 1e-30f && D2 > c.close && K < 1e30f && D2 < 1e30f && M > 1e-30f && M < 1e30f)) return -1;
    const float A = 0.5f / M * K, B = G / sqrtf(D2);
    const float e = A - B;
    const float d = (fabsf(t1) + fabsf(t2)) * 9.5367431640625e-07f + c.dv;  // 2^-20
    const float margin = (fabsf(A) + fabsf(B)) * 3.814697265625e-06f        // 2^-18
                         + (d * (fabsf(ey) + d) + c.dv * (fabsf(ex) + fabsf(ez) + c.dv)) / M;
    if (e > margin) return 0;
    if (e < -margin) return 1;
    return -1;
}

// The same test with the FP32 quotient and square root taken by the fast intrinsics
// (__fdividef, rsqrtf: at most 2 ulp each for the argument ranges admitted above). With
// them A and B still carry a relative error below 2^-20, inside the margin.
__device__ __forceinline__ int bound_hilo_fast(const CandF &c, float Mf, const float sh[6], const float sl[6], float G, float shear) {
    const float dx = (sh[0] - c.ph[0]) + (sl[0] - c.pl[0]);
    const float dy = (sh[1] - c.ph[1]) + (sl[1] - c.pl[1]);
    const float dz = (sh[2] - c.ph[2]) + (sl[2] - c.pl[2]);
    const float ex = (sh[3] - c.vh[0]) + (sl[3] - c.vl[0]);
    const float t1 = (sh[4] - c.vh[1]) + (sl[4] - c.vl[1]), t2 = shear * dx;
    const float ey = t1 - t2;
    const float ez = (sh[5] - c.vh[2]) + (sl[5] - c.vl[2]);
    const float K = ex * ex + ey * ey + ez * ez, D2 = dx * dx + dy * dy + dz * dz;
    const float M = Mf + c.w;
    if (!(K > 1e-30f && D2 > 1e-30f && D2 > c.close && K < 1e30f && D2 < 1e30f && M > 1e-30f && M < 1e30f)) return -1;
    const float rM = __fdividef(1.0f, M);
    const float A = 0.5f * rM * K, B = G * rsqrtf(D2);
    const float e = A - B;
    const float d = (fabsf(t1) + fabsf(t2)) * 9.5367431640625e-07f + c.dv;  // 2^-20
    const float margin = (fabsf(A) + fabsf(B)) * 3.814697265625e-06f        // 2^-18
                         + (d * (fabsf(ey) + d) + c.dv * (fabsf(ex) + fabsf(ez) + c.dv)) * rM;
    if (e > margin) return 0;
    if (e < -margin) return 1;
    return -1;
}

}  // namespace plan
