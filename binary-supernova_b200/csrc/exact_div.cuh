// exact_div.cuh -- correctly rounded FP64 quotients that share a reciprocal.
//
// The FP64 path's bits are IEEE division's, and a face of the reference
// scheme has some 85 of them: 12 per reconstructed field, several by the same
// density.  Here the reciprocal of a denominator is formed once and every
// quotient by it takes three more operations:
//   * recip_rn: the hardware's reciprocal approximation (PTX
//     rcp.approx.ftz.f64) refined by the geometric series of its residual e =
//     1 - b y, 1 / b = y (1 + e + e^2 + ...): first to e^2, then to e, each
//     in fused operations (Cornea-Hasegan, Golliver and Markstein, "Correctness
//     proofs outline for Newton-Raphson based floating-point divide and square
//     root algorithms", 14th IEEE Symposium on Computer Arithmetic, 1999; the
//     last step rounds correctly from a y within an ulp by Markstein, below,
//     unless b's significand is all ones, as in 0.1 + 0.6 + 0.3, the WENO
//     weights' sum in smooth flow).  The first step here is rounded upward:
//     the reciprocal of an all-ones significand lies just above a tie, and from
//     above the last step reaches its upper neighbour;
//   * quot: q = a y, then the remainder a - b q (exact in one fused
//     operation) times y added back.  This rounds correctly when y is the
//     rounded reciprocal and no intermediate leaves the normal range
//     (Markstein, "Computation of elementary functions on the IBM RISC
//     System/6000 processor", IBM J. Res. Dev. 34, 1990; Brisebarre, Muller
//     and Raina, "Accelerating correctly rounded floating-point division when
//     the divisor is known in advance", IEEE Trans. Comput. 53, 2004).
// The range is the caller's to keep: operands outside it take `a / b`.
// An FP64 step of a 256^3 blast wave: 53.1 ms with compiled division, 25.8 ms with
// these (B200, 1965 MHz).
#pragma once

#include <cuda_runtime.h>

namespace bsn {
namespace f64 {

// RN(1 / b) for b in [2^-340, 2^740]
__device__ __forceinline__ double recip_rn(double b) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    double e = fma(-b, y, 1.0);
    y = __fma_ru(y, fma(e, e, e), y);
    e = fma(-b, y, 1.0);
    return fma(y, e, y);
}

// a / b for y = RN(1 / b), b > 0 and a = +0 or positive, with a, a / b and
// a 2^-53 normal (a tiny a whose quotient only ever enters 1 + x^2 may round
// differently there).
__device__ __forceinline__ double quot_pos(double a, double b, double y) {
    const double q = a * y;
    return fma(fma(-b, q, a), y, q);
}

// a / b for y = RN(1 / |b|) and any signs, signed zeros included: the
// quotient of the magnitudes with the operands' sign.
__device__ __forceinline__ double quot(double a, double b, double y) {
    const double q = quot_pos(fabs(a), fabs(b), y);
    const int s = (__double2hiint(a) ^ __double2hiint(b)) & 0x80000000;
    return __hiloint2double(__double2hiint(q) | s, __double2loint(q));
}

// High words (sign off) of powers of two: the range checks are integer
// compares, which leave the FP64 pipe alone.
__host__ __device__ constexpr unsigned hi_pow2(int e) { return (unsigned)(1023 + e) << 20; }
__device__ __forceinline__ unsigned abs_hi(double x) { return (unsigned)__double2hiint(x) & 0x7fffffffu; }
// a numerator too small for quot (zero is fine)
__device__ __forceinline__ bool too_small(double a, unsigned lo) {
    const unsigned h = abs_hi(a);
    return h < lo && (h | (unsigned)__double2loint(a)) != 0u;
}
// a denominator outside [2^-340, 2^300)
__device__ __forceinline__ bool bad_denominator(double b) {
    return abs_hi(b) - hi_pow2(-340) >= hi_pow2(300) - hi_pow2(-340);
}

// Bounds of the ordinary range.  Cells below 2^116 in magnitude keep every
// WENO-Z ratio below 2^400 (their squares finite) and every HLLC density
// below 2^120; numerators over densities (at least 1e-30) need 2^-900, those
// over wave-speed differences (checked to lie in [2^-340, 2^300)) 2^-600.
constexpr unsigned kCellHi = hi_pow2(116), kNumRhoLo = hi_pow2(-900), kNumSpeedLo = hi_pow2(-600);

}  // namespace f64
}  // namespace bsn
