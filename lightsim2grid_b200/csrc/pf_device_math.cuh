// Device arithmetic shared by the batch kernels: complex helpers, the Jacobian entries of one
// Ybus entry, and the quotient used by the LU programs.
#pragma once

#include <cuda_runtime.h>

namespace l2g {
namespace {

__device__ __forceinline__ double2 cmul(double2 a, double2 b) {
    return make_double2(a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x);
}
__device__ __forceinline__ double2 cconj(double2 a) { return make_double2(a.x, -a.y); }
__device__ __forceinline__ double cabs2(double2 a) { return sqrt(a.x * a.x + a.y * a.y); }

constexpr double kPi = 3.141592653589793;

// Stands for t of an entry whose V_c is zero (hi word of a NaN that no operation gives).
constexpr int kZeroVoltage = 0x7ff8a5a5;

// t = conj(y V_c) V_r of a Ybus entry (r, c) from b = y V_c: its complex power at the row.  A V_c whose
// |V_c|^2 underflows to zero has no dS/d|V|: t is the mark that dsbus reads.
__device__ __forceinline__ double2 entry_power(double2 b, double2 vc, double2 vr) {
    const unsigned hi = (unsigned)(__double2hiint(vc.x) | __double2hiint(vc.y)) & 0x7fffffffu;
    const double2 t = cmul(cconj(b), vr);
    const double mark = __hiloint2double(kZeroVoltage, 0);
    return hi >= 0x1e500000u ? t : make_double2(mark, mark);  // either part at least 2^-538
}

// Jacobian values of Ybus entry (r, c) from t = conj(y V_c) V_r: dS/dVa = -j (t - d) and
// |V_c| dS/d|V_c| = t + d, with d = conj(I_r) V_r on the diagonal, else 0 (the dS/dVa and dS/dVm of
// BaseNRAlgo::_dSbus_dV, BaseNRAlgo.tpp:228-257, the latter's column c times |V_c|: the Newton
// unknown is dVm / |V|, which the voltage update multiplies by |V|).  The scaled columns need no
// |V| and no quotient: two complex products per entry in place of three, a square root and a division.
// A zero V_c gives the reference's dS/dVa = 0 and NaN dS/d|V|: a bus without a magnitude unknown then leaves
// the Jacobian singular (SolverReFactor), another one may also end in a step that is not finite.
__device__ __forceinline__ void dsbus(double2 t, double2 d, double &dvar, double &dvai, double2 &dvm) {
    const bool zero = __double2hiint(t.x) == kZeroVoltage;
    dvar = zero ? 0.0 : t.y - d.y;
    dvai = zero ? 0.0 : d.x - t.x;
    dvm = make_double2(t.x + d.x, t.y + d.y);
}

// a / b.  FP64: from the approximate reciprocal instruction, two Newton steps for the reciprocal, the
// product, and one correction by the exact remainder (Markstein, "IA-64 and Elementary Functions", ch. 8),
// without the special cases of the division operator (its range checks and their branch): the
// operator's quotient for finite operands in the normal range (a divisor whose significand is all ones, for which the
// reciprocal's last step does not round as the reciprocal, may round a quotient next to a tie the other way).  An
// infinite divisor gives zero, as the operator does (its reciprocal is zero, and the residuals are formed
// with a tiny value in its place); so does one above 2^1022 (the operator: at most 2^-1022 |a|).  A zero or
// subnormal divisor gives a value that is not finite.
// The quotient stands in every step of the elimination's serial chain, and the padding
// operations of a warp's phases (0 / 0) took the operator's slow branch: N-1 batches, 118 buses 0.126
// -> 0.100 ms, 1354 buses 3.14 -> 2.53 ms, 2848 buses FP64 16.9 -> 16.3 ms, DC 1.28 -> 1.09 ms, 6515
// buses FP64 66.2 -> 62.6 ms.
// FP32 (mixed form): the reciprocal-based quotient (within 2 ulp), whose error the FP64-residual
// refinement of the Newton step absorbs.
__device__ __forceinline__ double lu_div(double a, double b) {
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(b));
    const int hi = __double2hiint(b);
    b = __hiloint2double((hi & 0x7fffffff) >= 0x7ff00000 ? 0 : hi, __double2loint(b));
    r = fma(fma(-b, r, 1.0), r, r);
    r = fma(fma(-b, r, 1.0), r, r);
    const double q = a * r;
    return fma(fma(-b, q, a), r, q);
}
__device__ __forceinline__ float lu_div(float a, float b) { return __fdividef(a, b); }

// 1 / x for the dense tail's serial chain over the pivots.  FP32: the hardware's approximate reciprocal (subnormal
// results included) and one Newton step, its residual formed with zero in place of an infinite x; the rounded
// reciprocal took the 300-chord N-1 batch from 48.4 to 48.8 ms.
__device__ __forceinline__ float tail_reciprocal(float x) {
    float r;
    asm("rcp.approx.f32 %0, %1;" : "=f"(r) : "f"(x));
    const float y = fabsf(x) < INFINITY ? x : 0.0f;
    return fmaf(fmaf(-y, r, 1.0f), r, r);
}
__device__ __forceinline__ double tail_reciprocal(double x) { return 1.0 / x; }

// a / u from the pivot's reciprocal r: one product and one correction by the exact remainder (Markstein, as
// above), which rounds as the quotient does, without its branch on special operands.  An infinite pivot gives
// zero, as the operator does; a zero one, or one whose reciprocal overflows, a value that is not finite.
__device__ __forceinline__ float tail_quotient(float a, float u, float r) {
    const float q = a * r;
    return fmaf(fmaf(-q, fabsf(u) < INFINITY ? u : 0.0f, a), r, q);
}
__device__ __forceinline__ double tail_quotient(double a, double u, double r) {
    const double q = a * r;
    return fma(fma(-q, fabs(u) < (double)INFINITY ? u : 0.0, a), r, q);
}

}  // namespace
}  // namespace l2g
