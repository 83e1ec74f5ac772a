// Reciprocal, square root, logarithm and first-quadrant arctangent for the
// closed forms of sa_front.cuh: inline, free of branches and of the special
// cases (zero, infinity, subnormal numbers) that their arguments never meet,
// so that the compiler interleaves the several independent ones of an
// evaluation.  The library's functions, one out-of-line copy each, left the
// level kernel waiting for instructions (3.0 stalled warps per issued
// instruction on the sphere of 320 triangles) and on fixed latencies (2.5).
//
// Methods: the hardware's approximate seed and one Newton-Raphson (Halley)
// correction for 1/x and sqrt(x); log x = e ln 2 + 2 atanh((m - 1)/(m + 1)),
// x = m 2^e with m in [sqrt(1/2), sqrt 2); arctangent by the half-angle
// breakpoints tan(pi/8), tan(3 pi/8).  The two series are interpolated at
// Chebyshev nodes over the reduced range (relative error 2.3e-18 and 3.1e-18
// before rounding; tests/test_front_cpu.py and, on the device,
// tests/test_math_gpu.py check the functions against the host's long double ones).
#pragma once

#include "sa_device.cuh"

#ifndef __CUDACC__
#include <cstdint>
#include <cstring>
#endif

namespace ebem {

EBEM_DI double q_rcp(double x) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
#else
    return 1.0 / x;
#endif
}

// sqrt(x), 0 for x <= 0.
EBEM_DI double q_sqrt(double x) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x * y, y, 1.0);
    y = fma(y * e, fma(0.375, e, 0.5), y);
    const double s = x * y;
    return x > 0.0 ? fma(fma(-s, s, x), 0.5 * y, s) : 0.0;
#else
    return x > 0.0 ? sqrt(x) : 0.0;
#endif
}

// log x, x > 0 and normal.
EBEM_DI double q_log(double x) {
#ifdef __CUDA_ARCH__
    const int hi = __double2hiint(x), e = (hi - 0x3fe6a09e) >> 20;
    const double m = __hiloint2double(hi - (e << 20), __double2loint(x));
#else
    uint64_t b;
    std::memcpy(&b, &x, 8);
    const int hi = (int)(b >> 32), e = (hi - 0x3fe6a09e) >> 20;
    b = ((uint64_t)(uint32_t)(hi - e * (1 << 20)) << 32) | (b & 0xffffffffu);
    double m;
    std::memcpy(&m, &b, 8);
#endif
    const double s = (m - 1.0) * q_rcp(m + 1.0), u = s * s;
    double p = 0.07405641283874514;
    p = fma(p, u, 0.0765618886791573);
    p = fma(p, u, 0.0909181864974045);
    p = fma(p, u, 0.11111098476681508);
    p = fma(p, u, 0.1428571438080474);
    p = fma(p, u, 0.19999999999649035);
    p = fma(p, u, 0.33333333333333826);
    const double s2 = s + s;
    return fma((double)e, 0.69314718055994530942, fma(s2 * u, p, s2));
}

// Angle of (x, y), x >= 0, y >= 0, not both zero.
EBEM_DI double q_atan2(double y, double x) {
    const bool hi = y > 2.41421356237309504880 * x, lo = !(y > 0.41421356237309504880 * x);
    const double num = hi ? -x : (lo ? y : y - x), den = hi ? y : (lo ? x : y + x);
    const double base = hi ? 0.5 * kPi : (lo ? 0.0 : 0.25 * kPi);
    const double t = num * q_rcp(den), u = t * t;
    double p = -0.017803896394812564;
    p = fma(p, u, 0.03796390316111083);
    p = fma(p, u, -0.05035049795312439);
    p = fma(p, u, 0.05846866752275139);
    p = fma(p, u, -0.06662950246036792);
    p = fma(p, u, 0.07692045194561481);
    p = fma(p, u, -0.09090896801472813);
    p = fma(p, u, 0.11111110744657099);
    p = fma(p, u, -0.14285714279244968);
    p = fma(p, u, 0.19999999999940837);
    p = fma(p, u, -0.3333333333333312);
    return base + fma(t * u, p, t);
}

}  // namespace ebem
