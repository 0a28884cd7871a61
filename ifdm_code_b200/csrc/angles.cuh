// angles.cuh -- sine and cosine of the kick's phases, for the box kernels (and
// on the host, for their test).
#pragma once

#include <cuda_runtime.h>
#include <string.h>

#define IFDM_ANGLE __host__ __device__ __forceinline__

namespace ifdm {

IFDM_ANGLE int low_word(double m) {
#ifdef __CUDA_ARCH__
    return __double2loint(m);
#else
    long long b;
    memcpy(&b, &m, sizeof b);
    return (int)(b & 0xffffffffll);
#endif
}

// exp(-i p) and its pieces through sincospi: sincos(p) carries an out-of-line
// reduction for huge arguments, and the registers saved around that call
// (one per unrolled element) spilled kilobytes a thread.  p/pi = y + e with
// the product's rounding error and the constant's remainder in e, which turns
// the pair by the small angle pi e (to second order: 1.2e-14 of it at |p| =
// 1e9), so the argument keeps its full accuracy.
IFDM_ANGLE void sincos_pi(double p, double &s, double &c) {
    const double hi = 0.31830988618379067154, lo = -1.9678676675182486e-17, pi = 3.14159265358979323846;
    const double y = p * hi, e = pi * fma(p, lo, fma(p, hi, -y));
    double s0, c0;
    sincospi(y, &s0, &c0);
    const double h = -0.5 * e;
    s = fma(fma(h, s0, c0), e, s0);
    c = fma(fma(h, c0, -s0), e, c0);
}
// sin and cos of z = p - j pi/2, |z| <= pi/4, by their Taylor series; j from
// 2p/pi rounded by adding 1.5 2^52.  FULL: to z^15 and z^16 with the rounding
// error of p/pi in z, 2e-16; else to z^11 and z^12, 1e-11, a third of sincos's
// FP64 operations.
template <bool FULL = false> IFDM_ANGLE int sincos_quarter(double p, double &s, double &c) {
    const double big = 6755399441055744.0, inv_pi = 0.31830988618379067154;
    const double t = p * inv_pi, m = fma(t, 2.0, big);
    double z = fma(m - big, -0.5, t);
    if (FULL) z += fma(p, -1.9678676675182486e-17, fma(p, inv_pi, -t));
    z *= 3.14159265358979323846;
    const double z2 = z * z;
    if (FULL) {
        s = fma(z2, -1.0 / 1307674368000.0, 1.0 / 6227020800.0);
        c = fma(z2, 1.0 / 20922789888000.0, -1.0 / 87178291200.0);
        s = fma(s, z2, -1.0 / 39916800.0);
        c = fma(c, z2, 1.0 / 479001600.0);
        s = fma(s, z2, 1.0 / 362880.0);
        c = fma(c, z2, -1.0 / 3628800.0);
    } else {
        s = fma(z2, -1.0 / 39916800.0, 1.0 / 362880.0);
        c = fma(z2, 1.0 / 479001600.0, -1.0 / 3628800.0);
    }
    s = fma(s, z2, -1.0 / 5040.0);
    c = fma(c, z2, 1.0 / 40320.0);
    s = fma(s, z2, 1.0 / 120.0);
    c = fma(c, z2, -1.0 / 720.0);
    s = fma(s, z2, -1.0 / 6.0);
    c = fma(c, z2, 1.0 / 24.0);
    s = fma(s * z2, z, z);
    c = fma(c, z2, -0.5);
    c = fma(c, z2, 1.0);
    return low_word(m);  // p = z + j pi/2
}
// the same put together: sin and cos of p
template <bool FULL> IFDM_ANGLE void sincos_series(double p, double &s, double &c) {
    double s0, c0;
    const int j = sincos_quarter<FULL>(p, s0, c0);
    const double a = (j & 1) ? c0 : s0, b = (j & 1) ? -s0 : c0;
    s = (j & 2) ? -a : a;
    c = (j & 2) ? -b : b;
}

}  // namespace ifdm
