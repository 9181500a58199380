// flash_div.cuh -- correctly rounded FP64 division written so that
// independent quotients overlap.
//
// The `/` operator's result, bit for bit (both are correctly rounded), from
// the reciprocal approximation rcp.approx.ftz.f64, y0 = (1 - e) / b with
// |e| < 2^-19, the first terms of 1 / b = y0 (1 + e + e^2 + ...), which leave
// a relative error of e^3, and P. Markstein's final correction (Computation of
// elementary functions on the IBM RISC System/6000 processor, IBM J. Res.
// Develop. 34(1), 1990; J.-M. Muller et al., Handbook of Floating-Point
// Arithmetic, 2nd ed., 2018, ch. 4): with y = RN(1/b) and q faithful the
// remainder r = a - b q is exact and RN(q + r y) is the correctly rounded
// quotient. The refinement gives RN(1/b) unless b's mantissa is all ones
// (1/b is then just above the middle of two numbers, and 1/(1 - 2^-53) would
// come out as 1). Such divisors, and operands outside 2^-450 .. 2^450 in
// magnitude (zeros, infinities and NaN among them), take the `/` operator.
//
// ocpf_check_division evaluates these functions and e on the device.
//
// Measured on B200, one warp: a dependent division 111 -> 72 cycles (81 with
// its range test); twelve independent ones 1,344 -> 602 cycles (each `/`
// brings a branch of its own, so that no two overlap).
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace ocpf {

// |x| in [2^-450, 2^450)
__device__ __forceinline__ bool div_mid(double x)
{
    const uint32_t h = (uint32_t)__double2hiint(x) & 0x7fffffffu;
    return h - (573u << 20) < (900u << 20);
}

// b's mantissa is all ones
__device__ __forceinline__ bool div_ones(double b)
{
    return (((uint32_t)__double2hiint(b) | 0xfff00000u) & (uint32_t)__double2loint(b)) == 0xffffffffu;
}

static __device__ __noinline__ double div_slow(double a, double b) { return a / b; }

// q = a / b where `bad`. One opaque statement: a branch in the source would
// split the block it stands in, and with it which products the compiler
// fuses into which sums around it.
__device__ __forceinline__ void div_redo(bool bad, double a, double b, double& q)
{
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %3, 0;\n\t@p div.rn.f64 %0, %1, %2;\n\t}"
        : "+d"(q)
        : "d"(a), "d"(b), "r"((uint32_t)bad));
}

// the start y0 of 1 / b
__device__ __forceinline__ double div_seed(double b)
{
    double y0;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y0) : "d"(b));
    return y0;
}

// a / b for operands with div_mid and not div_ones(b)
__device__ __forceinline__ double div_core(double a, double b)
{
    const double y0 = div_seed(b);
    const double e  = __fma_rn(-b, y0, 1.0);
    const double t  = __fma_rn(e, e, e);
    const double y1 = __fma_rn(y0, t, y0);               // 1/b but for the last bit
    const double q0 = __dmul_rn(a, y0);
    const double q1 = __fma_rn(q0, t, q0);
    const double y  = __fma_rn(y1, __fma_rn(-b, y1, 1.0), y1);  // RN(1/b)
    const double q2 = __fma_rn(__fma_rn(-b, q1, a), y1, q1);    // faithful
    return __fma_rn(__fma_rn(-b, q2, a), y, q2);
}

// a / b. The range test follows the quotient: a branch ahead of it would
// hold back the whole dependent sequence (110 cycles instead of 81).
__device__ __forceinline__ double div1(double a, double b)
{
    double q = div_core(a, b);
    div_redo(!(div_mid(a) & div_mid(b)) | div_ones(b), a, b, q);
    return q;
}

}  // namespace ocpf
