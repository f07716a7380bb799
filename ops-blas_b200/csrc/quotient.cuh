// Correctly rounded quotients of many numerators by one divisor, from one reciprocal (P. W. Markstein,
// "Computation of elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34, 1990):
//   * y0 within one unit in the last place of 1 / b gives, by one Newton step in fused multiply-adds,
//     y = RN(1 / b), unless b's significand is all ones;
//   * with that y, one residual correction q + (a - q b) y of a rough quotient makes it faithful, a second
//     one makes it RN(a / b).
// No step may underflow or overflow: qt_usual(b) and qt_low <= |a| <= qt_high; a zero among the numerators
// would lose its sign. Plain C++, so that the steps are checked on the host for every significand and every
// y0 that the device's approximation is allowed to give.
#pragma once

#include <cstring>
#ifdef __CUDACC__
#include <cuda_runtime.h>
#define OPSBLAS_QT __host__ __device__ __forceinline__
#else
#include <cmath>
#define OPSBLAS_QT inline
#endif

namespace opsblas {

constexpr float qt_low = 0x1p-60f, qt_high = 0x1p60f;

// Whether the divisor's reciprocal serves: qt_low <= |b| <= qt_high and a significand that is not all ones.
OPSBLAS_QT bool qt_usual(float b)
{
    unsigned u;
    memcpy(&u, &b, 4);
    u &= 0x7fffffffu;
    return u - 0x21800000u <= 0x5d800000u - 0x21800000u && (u & 0x7fffffu) != 0x7fffffu;  // bits of qt_low, qt_high
}

OPSBLAS_QT float qt_newton(float b, float y0) { return fmaf(fmaf(-b, y0, 1.0f), y0, y0); }

OPSBLAS_QT float qt_quotient(float a, float b, float y)
{
    float q = a * y;
    q = fmaf(fmaf(-q, b, a), y, q);
    return fmaf(fmaf(-q, b, a), y, q);
}

#ifdef __CUDACC__
// RN(1 / b), qt_usual(b). rcp.approx is documented to err by one unit in the last place at most.
__device__ __forceinline__ float qt_reciprocal(float b)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(b));
    return qt_newton(b, y);
}

// l = a / b; y = RN(1 / b) if `usual` (qt_usual(b)), which is the same for the whole warp. BOUNDED: no a is
// larger than b in magnitude (NaN aside). Numerators out of range, and all of them for other divisors, take
// the division.
template <bool BOUNDED, int R>
__device__ __forceinline__ void qt_quotients(const float (&a)[R], float b, float y, bool usual, float (&l)[R])
{
    float least = fabsf(a[0]), most = least;
#pragma unroll
    for (int r = 0; r < R; r++) {
        if (r > 0) {
            least = fminf(least, fabsf(a[r]));
            if (!BOUNDED) most = fmaxf(most, fabsf(a[r]));
        }
        l[r] = qt_quotient(a[r], b, y);
    }
    if (!usual || least < qt_low || (!BOUNDED && most > qt_high)) {
#pragma unroll
        for (int r = 0; r < R; r++)
            if (!usual || fabsf(a[r]) < qt_low || (!BOUNDED && fabsf(a[r]) > qt_high)) l[r] = a[r] / b;
    }
}
#endif

}  // namespace opsblas
