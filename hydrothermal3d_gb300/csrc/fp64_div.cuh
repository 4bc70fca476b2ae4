// FP64 quotients in few operations.
//
// GB300 issues an FP64 operation for one warp every 64 cycles per scheduler (2
// results per clock and SM), and an IEEE division costs nine or ten of them.
// The quotients here take an approximate reciprocal y of the divisor (refined by
// Newton's iteration, or rounded on the host for a divisor that a launch shares)
// and correct a y once by its exact remainder, r = a - b q with one fma, q' =
// fma(r, y, q) (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990).  Where y is the
// correctly rounded 1 / b (div_known, Divisor) q' is the operator's quotient
// (every pair of operands at 6 to 11 bits of significand checked).  Newton's y
// may be the neighbour of that.  It is for a divisor whose significand is all
// ones, which the operator takes; for others q' may then be the other one of the
// two doubles around a quotient that lies nearly in their middle (one pair in
// about 2^p at p bits, 10^16 for a double).  Operands outside the range in which
// nothing over- or underflows on the way (infinite, NaN, a zero divisor and -0,
// of which the remainder would lose the sign, among them) are divided by the
// operator.
#pragma once
#include <cuda_runtime.h>

// exponent test of the fast path: 2^-400 <= |x| < 2^400 (integer operations)
__device__ __forceinline__ bool mid_range(double x) {
    return ((unsigned)__double2hiint(x) & 0x7fffffffu) - 0x26f00000u < 0x32000000u;
}
// ... or +0, as a dividend
__device__ __forceinline__ bool mid_range0(double x) { return mid_range(x) || (__double2hiint(x) | __double2loint(x)) == 0; }
// 1/b to about an ulp: the hardware's approximation (20 bits or more), refined
// to third order: y (1 + e + e^2), e = 1 - b y
__device__ __forceinline__ double rcp_newton(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = __fma_rn(-b, y, 1.0);
    return __fma_rn(y, __fma_rn(e, e, e), y);
}
// a / b from y = 1/b to an ulp or so; a, b and a/b in the middle of the range
__device__ __forceinline__ double div_by(double a, double b, double y) {
    const double q = __dmul_rn(a, y);
    return __fma_rn(__fma_rn(-b, q, a), y, q);
}
__device__ __forceinline__ bool all_ones(double b) {
    return __double2loint(b) == -1 && (__double2hiint(b) & 0xfffff) == 0xfffff;
}
// a / b for any operands
__device__ __forceinline__ double div_any(double a, double b) {
    if (mid_range0(a) && mid_range(b) && !all_ones(b)) return div_by(a, b, rcp_newton(b));
    return __ddiv_rn(a, b);
}
// a / b where y = 1/b is at hand
__device__ __forceinline__ double div_known(double a, double b, double y) {
    if (mid_range0(a) && mid_range(b)) return div_by(a, b, y);
    return __ddiv_rn(a, b);
}
// A divisor that a launch shares, with its reciprocal rounded on the host.
struct Divisor {
    double b, y;
    Divisor() = default;
    __host__ explicit Divisor(double d) : b(d), y(1.0 / d) {}
};
__device__ __forceinline__ double operator/(double a, const Divisor& d) { return div_known(a, d.b, d.y); }

// v / 3, correctly rounded (but for subnormal results): 1/3 as the sum of two
// doubles; v/3 is at least a sixth of an ulp away from any middle between two
// doubles, and the sum errs by 2^-53 ulp.
__device__ __forceinline__ double third(double v) {
    return __fma_rn(v, 0x1.5555555555555p-2, __dmul_rn(v, 0x1.5555555555555p-56));
}

// One row of GershgorinPoisson!/GershgorinHydro!
// (Dimensional/kernels_HT3D_dimensional.jl:207-221): the sum of the magnitudes,
// and the diagonal.  Its thirteen divisors are the launch's: 45 operations
// instead of about 130.
struct GershSpacing {
    Divisor dt, dx, dy, dz, dx2, dy2, dz2;
    GershSpacing(double dt_, double x, double y, double z)
        : dt(dt_), dx(x), dy(y), dz(z), dx2(x * x), dy2(y * y), dz2(z * z) {}
};
__device__ __forceinline__ double gershgorin_row(double kW, double kE, double kS, double kN, double kB, double kF,
                                                 double rhoC, double transient, const GershSpacing& h, double& diag) {
    diag = ((kB / h.dz + kF / h.dz) / h.dz + (kN / h.dy + kS / h.dy) / h.dy + (kE / h.dx + kW / h.dx) / h.dx +
            rhoC * transient / h.dt);
    return fabs(kE / h.dx2) + fabs(kW / h.dx2) + fabs(kN / h.dy2) + fabs(kS / h.dy2) + fabs(kB / h.dz2) +
           fabs(kF / h.dz2) + fabs(diag);
}
