// Correctly rounded FP64 division with a shared reciprocal.
//
// The exact-form kernels divide by the same density several times per state (velocities, energy, heat flux), and every
// quotient has to be the correctly rounded one.  The compiler's division evaluates each of them on its own and ends in a
// branch to its slow path, which keeps the scheduler from overlapping neighbouring divisions; a cell update has 35 of
// them (2D Euler), so the sweeps were bound by those serial chains rather than by the FP64 pipe.  Here one reciprocal
// y of the divisor serves all quotients by it, each quotient takes three operations, nothing branches, and one flag per
// stage collects the operands outside the range for which the result is proven; a stage whose flag is set is evaluated
// again with the compiler's division.
//
// The algorithm is published: Newton-Raphson for the reciprocal from the hardware's reciprocal approximation, and
// Markstein's quotient correction with one multiplication and two fused multiply-adds (P. Markstein, "Computation of
// elementary functions on the IBM RISC System/6000 processor", IBM J. Res. Dev. 34(1), 1990; N. Brisebarre, J.-M. Muller,
// S. Raina, "Accelerating correctly rounded floating-point division when the divisor is known in advance", IEEE Trans.
// Computers 53(8), 2004):
//     q0 = RN(a y),  r = RN(b q0 - a),  q = RN(q0 - r y).
// Why q = RN(a / b) for p = 53, with a, b scaled into [1, 2) and |y - 1/b| <= 2^-(p+1) (1 + e):
//   * a / b differs from every midpoint of two neighbouring numbers by at least 2^(1-2p) / b (a >= b) or 2^-2p / b
//     (a < b), so q is right unless the argument of the last rounding is off by that much;
//   * near a midpoint q0 is half a unit from a / b (1.5 units would need a y - a / b of a whole unit, which with a < b < 2
//     forces a and b within a few units of 2, where a / b is next to a number and not to a midpoint), r is then exact, and
//     the argument is off by |r| |y - 1/b| <= b 2^-(2p+1) (1 + e) (half of that for a < b): a fraction b^2 (1 + e) / 4 of the
//     distance, below 1 for b <= 2 - e;
//   * away from midpoints the error of an inexact r (at most 2^(1-2p) / b) cannot reach one.
// The hardware's approximation is good to 2^-19.9, so the two Newton steps leave e < 2^-25.  For the divisors 2 - 2^-52 k above
// 2 - 2^-25 that this leaves out, 1/b is within 2^-80 of a midpoint only for odd k < 2^14; there y = RN(1/b), as for every k up
// to 2^24, for which the fraction is below 1 again.  Newton's second step multiplies the residual by y with its last bit set for
// the sake of k = 1: Newton ends below 1/b, which for a significand of all ones lies just above a midpoint, and would take the
// wrong neighbour.  Such densities are common (constant states with a rounding).  tests/test_division_device_gpu.py tries the
// approximation over every upper word of a binade, every one of those k, and 1e8 quotients of the whole range against IEEE
// division, a third of them next to midpoints or with divisors next to 2.
// Range: with b below 2^257 a dividend from 2^-764 on has a normal quotient, and a remainder whose last place is above 2^-1074;
// everything above is then the same for every exponent.  Operands outside fail the flag: a density or pressure far from 1, a
// velocity or heat flux between 0 and 2^-764.  What the second evaluation costs where every cell needs it (a component of 1e-310
// everywhere): 1024^2 Euler, 20 steps, 9.2 ms against 3.1, and 9.9 with the compiler's division throughout; 512^2 HPR with its
// forcing, 2 steps, 18.1 ms against 7.7, and 19.4.
#pragma once

#include <cuda_runtime.h>

namespace vg {

// Division policies.  Both give RN(a / b); a function template over them reads the same either way.
struct IeeeDiv {
    struct By {
        double b;
        __device__ __forceinline__ double operator()(double a) const { return a / b; }
        __device__ __forceinline__ double positive(double a) const { return a / b; }
    };
    __device__ __forceinline__ By by(double b) { return By{b}; }
    __device__ __forceinline__ double third(double a) { return a / 3.0; }
};

struct SharedDiv {
    // running extremes of the operands' upper words; ok() compares them once per stage
    unsigned pos = 0, low = 0xffffffffu, top = 0;

    // every operand so far was in the proven range
    __device__ __forceinline__ bool ok() const { return pos < 0x20000000u && low >= 0x205fffffu && top < 0xc0000000u; }

    // b in [2^-255, 2^257) and positive
    __device__ __forceinline__ void note_positive(double b) {
        pos = __viaddmax_u32((unsigned)__double2hiint(b), 0u - 0x30000000u, pos);
    }
    // |a| in [2^-764, 2^513) or a zero (whose quotient, sign included, comes out right for a positive divisor): t is the
    // upper word without its sign, its last bit set where the lower word holds something; a zero's t - 1 is the largest
    __device__ __forceinline__ void note_signed(double a) {
        const unsigned t = ((unsigned)__double2hiint(a) << 1) + min((unsigned)__double2loint(a), 1u);
        low = __viaddmin_u32(t, 0xffffffffu, low);
        top = max(top, t);
    }
    // |a| below 2^513, not a NaN
    __device__ __forceinline__ void note_below(double a) { top = max(top, (unsigned)__double2hiint(a) << 1); }

    __device__ __forceinline__ static double reciprocal(double b) {
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
        y = __fma_rn(y, __fma_rn(-b, y, 1.0), y);
        const double up = __hiloint2double(__double2hiint(y), __double2loint(y) | 1);
        return __fma_rn(up, __fma_rn(-b, y, 1.0), y);
    }
    __device__ __forceinline__ static double quotient(double a, double b, double y) {
        const double q = __dmul_rn(a, y);
        return __fma_rn(-__fma_rn(b, q, -a), y, q);
    }

    // quotients by one positive divisor: of a dividend of either sign or zero, and (pos) of one that is positive unless
    // the state is unphysical
    struct By {
        double b, y;
        SharedDiv* dv;
        __device__ __forceinline__ double operator()(double a) const {
            dv->note_signed(a);
            return quotient(a, b, y);
        }
        __device__ __forceinline__ double positive(double a) const {
            dv->note_positive(a);
            return quotient(a, b, y);
        }
    };
    __device__ __forceinline__ By by(double b) {
        note_positive(b);
        return By{b, reciprocal(b), this};
    }
    // a / b for operands whose range the caller knows
    __device__ __forceinline__ static double known(double a, double b) { return quotient(a, b, reciprocal(b)); }
    // a / 3 (RN(1/3) is within half a unit of 1/3, and 3 / 2 is far from 2)
    __device__ __forceinline__ double third(double a) {
        note_signed(a);
        return quotient(a, 3.0, 1.0 / 3.0);
    }
};

}  // namespace vg
