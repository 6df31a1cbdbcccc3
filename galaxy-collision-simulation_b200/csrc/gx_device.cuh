// gx_device.cuh -- device helpers shared by the sm_100a kernels of the engine.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

#include "precision.cuh"

namespace gx {

// ---------------------------------------------------------------------------------------
// FP64 reciprocal square root.  Seed: the hardware approximation rsqrt.approx.ftz.f64 (relative
// error below 2^-20: on B200 at most 2^-20.03 over every high word of two octaves, with all-zero and
// all-one low words, and over 4096 mantissas of every exponent from -894 to 896).  One Householder step of order 2 on the
// series (1 - e)^(-1/2) = 1 + e/2 + 3e^2/8 + O(e^3) with e = 1 - s*y^2 leaves a relative
// error of about (5/16) e^3 < 2^-57, i.e. at the level of the final rounding.
// 5 FP64 pipe operations after the MUFU seed.  s == 0 gives a non-finite result; callers
// with eps == 0 select it away.
// ---------------------------------------------------------------------------------------
__device__ __forceinline__ double rsqrt_f64(double s) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
    const double e = fma(-s, y * y, 1.0);
    const double p = fma(0.375, e, 0.5);
    return fma(y * e, p, y);
}

// m s^(-3/2), the weight of a softened pair.  From the same seed y, t = y^2 and e = 1 - s t,
// s^(-3/2) = y t (1 - e)^(-3/2) = y t (1 + 3e/2 + 15e^2/8 + O(e^3)), so the correction is
// applied to the product m y t itself: 7 FP64 pipe operations after the seed, where refining
// y first (5) and cubing it (3) took 8, and three roundings of the result instead of six.
// The truncated term is about (35/16) e^3 < 2^-55.  s > 0.
__device__ __forceinline__ double inv_cube_f64(double s, double m) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(s));
    const double t = y * y;
    const double e = fma(-s, t, 1.0);
    const double p = fma(1.875, e, 1.5);
    const double w = (m * y) * t;
    return fma(w * e, p, w);
}

// Sums without softening.  Where s^(-3/2) overflows (s below 3.1e-206; softened sums are always
// above) the reference's weight is infinite, but inv_cube_f64's correction can turn it into NaN.
// Testing every pair costs a fifth of the sum (N = 131,072: 21.7 ms with integer tests, 19.8 with a
// branch, against 18.2), so a target's share of the sum is looked at when it is complete: a term of
// such a pair is some 1e205 times the mass, beyond any sum of ordinary ones, and the share is then
// added up once more with the cube taken first, as the reference takes it.
__device__ __forceinline__ bool sum_overflowed(double fx, double fy, double fz) {
    return !(fabs(fx) < 1e180 && fabs(fy) < 1e180 && fabs(fz) < 1e180);  // NaN included
}
__device__ __forceinline__ double inv_cube_first(double s, double m) {
    if (s == 0.0 || m == 0.0) return 0.0;
    const double y = rsqrt_f64(s);
    return m * (y * y * y);
}

// RN(1 / RN(sqrt(s))), the value IEEE square root and division give, without their branches.
// The method is Markstein's (IBM J. Res. Dev. 34, 1990), the argument that of Cornea, Harrison
// and Tang: a bound, and a look at the exceptions.
//   y = s^-1/2 within 1.6 x 2^-53; g = s y; the residual r = s - g^2 makes g + r y/2 agree
//   with sqrt(s) to 10 x 2^-106 before its one rounding, so q could be wrong only for
//   s = M^2 - d with an odd 54-bit M and |d| <= 80.  These are the square roots of d modulo
//   2^54; q is right for all of them (|d| < 128; tests/test_exact_form_gpu.py meets each).
//   e = 1 - q y is exact and |e| <= 2.6 x 2^-53, so y + y e agrees with 1/q to 7 x 2^-106, and
//   inv could be wrong only where 1/q lies that close to the middle between two doubles.
//   Then the exact e1 = 1 - q inv is q times half an ulp of inv, a power of two, to 2^-51:
//   the mantissas of e1 and q agree, which the high words tell.  (Some sixty mantissas q,
//   divisors of 2^106 + d with small d, do round the wrong way and are caught so.)
// 12 FP64 operations and one MUFU; the checks are integer work.  A batch of arguments shares
// one ExactGuard: when it is not clean() -- an argument outside [2^-894, 2^897) (zero, infinity
// and NaN among them) or a rounding this cannot settle, about one argument in 2^18 -- the batch
// takes IEEE root and division instead.
struct ExactGuard {
    unsigned near = 0xffffffffu, range = 0u;
    __device__ __forceinline__ bool clean() const { return near > 2u && range < (1791u << 20); }
};
__device__ __forceinline__ double exact_inv(double s, ExactGuard& guard) {
    const double y = rsqrt_f64(s);
    const double g = __dmul_rn(s, y);
    const double r = __fma_rn(-g, g, s);
    const double q = __fma_rn(r, __dmul_rn(0.5, y), g);
    const double e = __fma_rn(-q, y, 1.0);
    const double inv = __fma_rn(e, y, y);
    const double e1 = __fma_rn(-q, inv, 1.0);
    guard.near = min(guard.near, (unsigned)(__double2hiint(e1) - __double2hiint(q) + 1) & 0xfffffu);
    guard.range = max(guard.range, (unsigned)__double2hiint(s) - (129u << 20));
    return inv;
}
__device__ __forceinline__ double ieee_inv(double s) { return __ddiv_rn(1.0, __dsqrt_rn(s)); }

__device__ __forceinline__ float rsqrt_f32(float s) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(s));
    return y;
}

// ---------------------------------------------------------------------------------------
// Packed FP32 pairs (PTX .f32x2, sm_100+).  One instruction applies the operation to two
// FP32 lanes held in a 64-bit register pair: the same FP32-pipe work as two scalar
// instructions but one issue slot, which leaves issue bandwidth for the MUFU rsqrt and the
// shared-memory loads of the pair kernel.
// ---------------------------------------------------------------------------------------
typedef unsigned long long f2;

__device__ __forceinline__ f2 pk2(float lo, float hi) {
    f2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(lo), "f"(hi));
    return r;
}
__device__ __forceinline__ void upk2(f2 v, float& lo, float& hi) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(lo), "=f"(hi) : "l"(v));
}
__device__ __forceinline__ f2 sub2(f2 a, f2 b) {
    f2 d;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 mul2(f2 a, f2 b) {
    f2 d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(a), "l"(b));
    return d;
}
__device__ __forceinline__ f2 fma2(f2 a, f2 b, f2 c) {
    f2 d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(a), "l"(b), "l"(c));
    return d;
}

// 16-byte shared-memory load of two packed pairs (p must be 16-byte aligned shared memory).
__device__ __forceinline__ void lds_v2b64(const float* p, f2& a, f2& b) {
    const unsigned addr = (unsigned)__cvta_generic_to_shared(p);
    asm volatile("ld.shared.v2.b64 {%0, %1}, [%2];" : "=l"(a), "=l"(b) : "r"(addr));
}

// Knuth's TwoSum: s + e == a + b exactly (round-to-nearest, no overflow).
__device__ __forceinline__ void two_sum(float a, float b, float& s, float& e) {
    s = __fadd_rn(a, b);
    const float bp = __fsub_rn(s, a);
    const float ap = __fsub_rn(s, bp);
    e = __fadd_rn(__fsub_rn(a, ap), __fsub_rn(b, bp));
}

// Compensated FP32 accumulator: value = hi + lo.
struct CompF {
    float hi, lo;
    __device__ __forceinline__ void init() { hi = 0.f; lo = 0.f; }
    __device__ __forceinline__ void add(float v) {
        float s, e;
        two_sum(hi, v, s, e);
        hi = s;
        lo = __fadd_rn(lo, e);
    }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// Reference-order FP64 helpers: no FMA contraction (the reference's x86-64 build has none).
__device__ __forceinline__ double dadd(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ double dmul(double a, double b) { return __dmul_rn(a, b); }
__device__ __forceinline__ double dsub(double a, double b) { return __dsub_rn(a, b); }

// Warp reductions.
__device__ __forceinline__ double warp_min(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmin(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_max(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}
__device__ __forceinline__ double warp_sum(double v) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

}  // namespace gx
