// The FP32 form of the unbinding test (unbind.cuh), with the error bound that lets it decide.
#pragma once

#include "bound_f32.cuh"

namespace plan {

// A member, with its own limits. 15 words: odd, so that 32 of them side by side meet no bank twice.
struct UbCand : CandF {
    BoundLimits lim;
};

// Whether the others bind the member: 1 unbound, 0 bound, -1 too close to call. With
// Mr = M - m, the centre of the others differs from the member's position by (com - p) M / Mr.
// The differences of float pairs carry the errors of bound_hilo. M and m are rounded by 2^-24 each
// and their difference is exact, so M / Mr errs by up to 2^-23 M / Mr: below 2^-20 while Mr > M / 8,
// and only there the test decides. It scales all differences alike, and the absolute errors with
// them; apart from that ey errs by less than d = 2^-19 (|t1| + |t2|). The FP64 form of
// the reference errs by 2^-50 of the coordinates, far less than the margin on the same terms.
__device__ __forceinline__ int ub_test(const UbCand &c, const float *sf, float G, float shear) {
    const float M = sf[12], Mr = M - c.w;
    if (!(Mr > M * 0.125f && M > 1e-30f && M < 1e30f)) return -1;
    const float rho = __fdividef(M, Mr);
    const float dx = ((sf[0] - c.ph[0]) + (sf[6] - c.pl[0])) * rho, dy = ((sf[1] - c.ph[1]) + (sf[7] - c.pl[1])) * rho;
    const float dz = ((sf[2] - c.ph[2]) + (sf[8] - c.pl[2])) * rho;
    const float ex = ((sf[3] - c.vh[0]) + (sf[9] - c.vl[0])) * rho, t1 = ((sf[4] - c.vh[1]) + (sf[10] - c.vl[1])) * rho, t2 = shear * dx;
    const float ey = t1 - t2, ez = ((sf[5] - c.vh[2]) + (sf[11] - c.vl[2])) * rho;
    const float K = ex * ex + ey * ey + ez * ez, D2 = dx * dx + dy * dy + dz * dz;
    if (!(K > 1e-30f && D2 > rho * rho * c.lim.close && K < 1e30f && D2 < 1e30f)) return -1;
    const float rM = __fdividef(1.0f, M);
    const float A = 0.5f * rM * K, B = G * rsqrtf(D2);
    const float e = A - B;
    const float d = (fabsf(t1) + fabsf(t2)) * 1.9073486328125e-06f;  // 2^-19
    const float margin = (fabsf(A) + fabsf(B)) * 7.62939453125e-06f  // 2^-17
                         + (d * (fabsf(ey) + d) + rho * rho * c.lim.dv2) * rM;
    if (e > margin) return 1;
    if (e < -margin) return 0;
    return -1;
}

}  // namespace plan
