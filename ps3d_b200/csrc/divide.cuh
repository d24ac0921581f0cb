// divide.cuh — FP64 reciprocals and quotients by Newton-Raphson and residual
// steps, correctly rounded (Markstein, "Computation of elementary functions
// on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990).
#pragma once
#include <cmath>
#include "common.cuh"

namespace ps3d {

// The FP64 reciprocal of a normal number x from the hardware approximation
// (PTX rcp.approx.ftz.f64): each iteration y += y (1 - x y) squares the
// relative error, two take it far below the FP64 rounding unit, and a third,
// with the residual 1 - x y formed exactly by an FMA, rounds the result
// correctly; on a B200 it agreed bit for bit with the correctly rounded
// 1.0 / x on 2^30 random inputs over 81 binades, in fewer instructions.  The
// flush-to-zero approximation must not see a subnormal.
PS3D_HD double rcp_newton(double x) {
#ifdef __CUDA_ARCH__
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    double e = fma(-x, y, 1.0);
    y = fma(y, e, y);
    e = fma(-x, y, 1.0);
    y = fma(y, e, y);
    e = fma(-x, y, 1.0);
    return fma(y, e, y);
#else
    return 1.0 / x;
#endif
}

// v times -1/ks (pressure_solver.f90:59-69), zero where ks is not positive, by
// one reciprocal for both parts.
// FP64: the product with the reciprocal, then one residual step, which takes
// its up to 1.5 units of the last place to the division's half unit (equal to
// the division on 2^28 random operands); without a branch, an infinite or NaN
// product stays.
// FP32: to the quotient that an FP64 division of the part rounds to: one step
// brings q = d r within one unit of the FP64 quotient, the second, whose
// residual is exact, rounds it correctly.  Zeros, infinities and NaNs take the
// first product, and a ks so extreme that a step could leave the normal
// numbers is divided by.  With two divisions an element FP32 took longer than
// FP64: 512x256x64 47.2 us, now 33.
template <typename R>
PS3D_HD cpx<R> divide_neg(cpx<R> v, double ks) {
    if (!(ks > 0.0)) return mk<R>((R)0, (R)0);
    if constexpr (sizeof(R) == 8) {
        const double r = -1.0 / ks;
        auto quot = [&](double f) {
            const double q = f * r, s = fma(fma(q, ks, f), r, q);
            return fabs(q) <= 1.7976931348623157e308 ? s : q;
        };
        return mk<R>(quot(v.x), quot(v.y));
    } else {
        if (!(ks > 1e-200 && ks < 1e200)) return mk<R>((R)(-(double)v.x / ks), (R)(-(double)v.y / ks));
        const double r = rcp_newton(ks);
        auto quot = [&](float f) {
            const double d = -(double)f;
            double q = d * r;
            if (fabsf(f) > 0.0f && fabsf(f) <= 3.402823466e+38f) {
                q = fma(fma(-q, ks, d), r, q);
                q = fma(fma(-q, ks, d), r, q);
            }
            return (float)q;
        };
        return mk<R>(quot(v.x), quot(v.y));
    }
}

}  // namespace ps3d
