// Several quotients by one divisor, each the bits of x / z (host and device).
//
// From the correctly rounded reciprocal r of z, q0 = fl(x r) is at most 1.5
// ulp from x / z, and q0 + (x - q0 z) r rounds to the quotient: P. Markstein's
// correction ("Computation of elementary functions on the IBM RISC System/6000
// processor", IBM J. Res. Dev. 34 (1990) 111-119).  The sum is within
// 3 * 2^-24 ulp of x / z before its rounding; the numerators whose quotients
// come nearer than 7 * 2^-24 ulp to a rounding boundary were enumerated for
// every 24-bit divisor, and all round as the division does.
// One reciprocal and three instructions per numerator instead of a division
// each.  It holds while nothing leaves the normal range: for z in
// [2^-24, 2^24] and |x| in [2^-100, 2^100] the quotient lies in [2^-124,
// 2^124] and the remainder's last bit at 2^-147 or above.  Zeros give x r,
// which has the quotient's sign; anything else (infinities, NaN, the ends of
// the range) is divided.
#pragma once

#include <cmath>

#ifdef __CUDACC__
#define CG_HOST_DEVICE __host__ __device__ __forceinline__
#else
#define CG_HOST_DEVICE inline
#endif

namespace cg {

struct Divisor {
    float z, r;
    bool plain;   // every numerator is divided
    CG_HOST_DEVICE explicit Divisor(float d) : z(d), r(1.f / d) {
        const float m = fabsf(d);
        plain = !(m >= 5.9604645e-8f && m <= 16777216.f);   // 2^-24, 2^24
    }
    // The quotient, or *divide set (never cleared) where it takes a division.  A
    // caller with several numerators tests once for all: a branch each cost a
    // gradient pass at 1024^2 26 us of 4120, one for three nothing.
    CG_HOST_DEVICE float quotient(float x, bool* divide) const {
        const float m = fabsf(x), q0 = x * r;
        // 2^-100, 2^100
        *divide |= plain || !((m >= 7.8886091e-31f || m == 0.f) && m <= 1.2676506e30f);
        return m == 0.f ? q0 : fmaf(fmaf(-q0, z, x), r, q0);
    }
};

}  // namespace cg
