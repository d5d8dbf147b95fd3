// Device vector math for the PBF kernels.
//
// Bit-exact parity with the reference kernels needs every per-pair expression to round
// exactly as the reference's compiled kernels do.  nvcc contracts a*b+c into fused
// multiply-adds by default, and which product it fuses depends on the surrounding code,
// so the FP32 arithmetic here is written with explicit round-to-nearest intrinsics
// (__fmaf_rn, __fmul_rn, __fadd_rn, __fsub_rn, __fdiv_rn, __fsqrt_rn), which the compiler
// never re-contracts.  The fused forms were determined by comparing each pass against
// the reference kernels on identical inputs, e.g.
//   squared distance          fma(dz, dz, fma(dx, dx, dy * dy))
//   cross product component   fma(a.y, b.z, -(a.z * b.y))
//   accumulations             fma(factor, term, accumulator)
//   |S|^2 after the lambda loop and |eta| after the normal loop
//                             fma(z, z, fma(y, y, x * x))
// The FP64 helpers of the adjoint keep the operand order of the reference's
// domain/device.cuh:103-157 and pbf/pbf.cu:45-54.  Names and structure are this library's own.
#pragma once

#include <cstdint>
#include <cuda_runtime.h>

namespace pbf {

struct f3 { float x, y, z; };
struct d3 { double x, y, z; };

__device__ __forceinline__ f3 mk(float x, float y, float z) { return {x, y, z}; }
__device__ __forceinline__ f3 xyz(const float4 v) { return {v.x, v.y, v.z}; }

// ---------------------------------------------------------------- FP32, pinned rounding
__device__ __forceinline__ f3 add(const f3 a, const f3 b) {
    return {__fadd_rn(a.x, b.x), __fadd_rn(a.y, b.y), __fadd_rn(a.z, b.z)};
}
__device__ __forceinline__ f3 sub(const f3 a, const f3 b) {
    return {__fsub_rn(a.x, b.x), __fsub_rn(a.y, b.y), __fsub_rn(a.z, b.z)};
}
__device__ __forceinline__ f3 scale(const f3 v, const float s) {
    return {__fmul_rn(s, v.x), __fmul_rn(s, v.y), __fmul_rn(s, v.z)};
}
// acc + s * v, fused
__device__ __forceinline__ f3 fma3(const float s, const f3 v, const f3 acc) {
    return {__fmaf_rn(s, v.x, acc.x), __fmaf_rn(s, v.y, acc.y), __fmaf_rn(s, v.z, acc.z)};
}
// x*x + y*y + z*z as fma(z, z, fma(x, x, y*y))
__device__ __forceinline__ float sq_xfirst(const f3 d) {
    return __fmaf_rn(d.z, d.z, __fmaf_rn(d.x, d.x, __fmul_rn(d.y, d.y)));
}
// x*x + y*y + z*z as fma(z, z, fma(y, y, x*x))
__device__ __forceinline__ float sq_yfirst(const f3 d) {
    return __fmaf_rn(d.z, d.z, __fmaf_rn(d.y, d.y, __fmul_rn(d.x, d.x)));
}
// a x b with each component fma(p, q, -(r * s))
__device__ __forceinline__ f3 cross_f(const f3 a, const f3 b) {
    return {__fmaf_rn(a.y, b.z, -__fmul_rn(a.z, b.y)), __fmaf_rn(a.z, b.x, -__fmul_rn(a.x, b.z)),
            __fmaf_rn(a.x, b.y, -__fmul_rn(a.y, b.x))};
}

// ------------------------------------------------------------------- FP64 (adjoint)
__device__ __forceinline__ f3 operator+(const f3 a, const f3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ f3 operator-(const f3 a, const f3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }
__device__ __forceinline__ d3 operator+(const d3 a, const d3 b) { return {a.x + b.x, a.y + b.y, a.z + b.z}; }
__device__ __forceinline__ d3 operator-(const d3 a, const d3 b) { return {a.x - b.x, a.y - b.y, a.z - b.z}; }

// factor * component, factor on the left (as the reference's scale()).
__device__ __forceinline__ f3 times(const f3 v, const float s) { return {s * v.x, s * v.y, s * v.z}; }
__device__ __forceinline__ d3 times(const f3 v, const double s) { return {s * v.x, s * v.y, s * v.z}; }
__device__ __forceinline__ d3 times(const d3 v, const double s) { return {s * v.x, s * v.y, s * v.z}; }

__device__ __forceinline__ float dot(const f3 a, const f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ double dot(const d3 a, const f3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }
__device__ __forceinline__ double dot(const d3 a, const d3 b) { return a.x * b.x + a.y * b.y + a.z * b.z; }

__device__ __forceinline__ f3 cross(const f3 a, const f3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ d3 cross(const f3 a, const d3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ d3 cross(const d3 a, const f3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}
__device__ __forceinline__ d3 cross(const d3 a, const d3 b) {
    return {a.y * b.z - a.z * b.y, a.z * b.x - a.x * b.z, a.x * b.y - a.y * b.x};
}

// The float value of pi used by the reference kernels (density/device.cuh:8).
constexpr float kPi = 3.14159265358979323846F;

// Whether the packed pair arithmetic below covers support radius h.  Other radii evaluate every pair
// twice: at 262k particles a step of PBF / PCISPH / WCSPH takes 0.600 / 0.869 / 0.194 ms staged and 0.563 / 0.766 / 0.186 per
// lane.  With four lanes a particle the staged passes stay ahead: 0.148 against 0.197 ms at 5k.
__host__ __device__ __forceinline__ bool packed_radius(const float h) { return h >= 0x1p-10F && h <= 0x1p10F; }

// Per-scene constants, derived on the device once so they come from the same
// device powf / division the reference evaluates inline.
struct KernelConstants {
    float h;              // support radius
    float h2;             // h * h
    float poly6_denominator;   // 64 pi h2 h2 h2 h h h           (density/device.cuh:15)
    float poly6_grad_denominator; // 32 pi h2 h2 h2 h h h        (density/device.cuh:23)
    float spiky_coefficient;   // -45 / (pi powf(h, 6))          (pbf/pbf.cu:30)
    float spiky_threshold;     // smallest r2 with sqrtf(r2) >= h: spiky is non-zero iff 0 < r2 < this
    float union_threshold;     // max(h2, spiky_threshold)
    float hessian_threshold;   // smallest r2 with sqrt((double)r2) >= h: the FP64 spiky Hessian is non-zero iff 0 < r2 < this
    float adjoint_threshold;   // max(spiky_threshold, hessian_threshold)
    float list_threshold;      // max of all: every kernel term of every pass is zero at r2 >= this
    float poly6_radial_coefficient; // 315 / (64 pi powf(h, 9))  (pbf/pbf.cu:22)
    double spiky_coefficient_d;    // -45 / (pi pow(h, 6)) in FP64 (pbf/pbf.cu:52)
    float poly6_reciprocal;    // 1 / poly6_denominator, correctly rounded
    float poly6_grad_reciprocal;   // 1 / poly6_grad_denominator, correctly rounded
    float fast_min;            // smallest and largest non-zero r2 of the two-pair arithmetic below
    float fast_max;            // (largest < smallest where h is outside its range)
};

// The constants of support radius h.
__device__ inline KernelConstants kernel_constants(const float h) {
    const float squared_radius = __fmul_rn(h, h);
    KernelConstants k;
    k.h = h;
    k.h2 = squared_radius;
    k.poly6_denominator = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(64.0F * kPi, squared_radius), squared_radius),
                                                                     squared_radius), h), h), h);
    k.poly6_grad_denominator = __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(32.0F * kPi, squared_radius), squared_radius),
                                                                          squared_radius), h), h), h);
    k.spiky_coefficient = __fdiv_rn(-45.0F, __fmul_rn(kPi, powf(h, 6.0F)));
    // Smallest float r2 with sqrtf(r2) >= h; sqrtf is monotone, so bisect on the bit pattern.
    uint32_t lo = 0u, hi = 0x7f800000u;
    while (hi - lo > 1u) {
        const uint32_t mid = lo + (hi - lo) / 2u;
        if (sqrtf(__uint_as_float(mid)) >= h) hi = mid;
        else lo = mid;
    }
    k.spiky_threshold = __uint_as_float(hi);
    k.union_threshold = fmaxf(k.h2, k.spiky_threshold);
    // Smallest float r2 with sqrt((double)r2) >= h (the FP64 Hessian's support test).
    lo = 0u;
    hi = 0x7f800000u;
    while (hi - lo > 1u) {
        const uint32_t mid = lo + (hi - lo) / 2u;
        if (sqrt(static_cast<double>(__uint_as_float(mid))) >= static_cast<double>(h)) hi = mid;
        else lo = mid;
    }
    k.hessian_threshold = __uint_as_float(hi);
    k.adjoint_threshold = fmaxf(k.spiky_threshold, k.hessian_threshold);
    k.list_threshold = fmaxf(k.union_threshold, k.hessian_threshold);
    k.poly6_radial_coefficient = __fdiv_rn(315.0F, __fmul_rn(64.0F * kPi, powf(h, 9.0F)));
    k.spiky_coefficient_d = -45.0 / (static_cast<double>(kPi) * pow(static_cast<double>(h), 6.0));
    k.poly6_reciprocal = __frcp_rn(k.poly6_denominator);
    k.poly6_grad_reciprocal = __frcp_rn(k.poly6_grad_denominator);
    // The range of the packed arithmetic.  At its ends every intermediate of the packed arithmetic, and every last bit of
    // its residuals, is a normal float: r >= 2^-30 h, and a poly6 numerator 315 (h2 - r2)^3 >= 2^-100.
    k.fast_min = __fmul_rn(squared_radius, 0x1p-60F);
    k.fast_max = -1.0F;
    if (packed_radius(h)) {
        const float below = __uint_as_float(__float_as_uint(fminf(squared_radius, k.spiky_threshold)) - 1u);
        k.fast_max = fminf(below, __fsub_rn(squared_radius, 0x1p-36F));
    }
    return k;
}

// ------------------------------------------------------------ FP32 kernel functions
// Squared distance of a displacement, with the reference's rounding.
__device__ __forceinline__ float squared(const f3 d) { return sq_xfirst(d); }

// poly6 weight (density/device.cuh:10-16) for a squared distance already below h2.
__device__ __forceinline__ float poly6_inside(const float r2, const KernelConstants& k) {
    const float difference = __fsub_rn(k.h2, r2);
    return __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(315.0F, difference), difference), difference), k.poly6_denominator);
}

__device__ __forceinline__ float poly6(const f3 d, const KernelConstants& k) {
    const float r2 = squared(d);
    if (r2 >= k.h2) return 0.0F;
    return poly6_inside(r2, k);
}

// poly6 gradient (density/device.cuh:18-24).
__device__ __forceinline__ f3 poly6_gradient(const f3 d, const KernelConstants& k) {
    const float r2 = squared(d);
    if (r2 >= k.h2) return {0.0F, 0.0F, 0.0F};
    const float difference = __fsub_rn(k.h2, r2);
    return scale(d, __fdiv_rn(__fmul_rn(__fmul_rn(-945.0F, difference), difference), k.poly6_grad_denominator));
}

// Spiky gradient (pbf/pbf.cu:26-32) of a displacement of length `distance` (0 < distance < h).
__device__ __forceinline__ f3 spiky_gradient_at(const f3 d, const float distance, const KernelConstants& k) {
    const float difference = __fsub_rn(k.h, distance);
    return scale(d, __fdiv_rn(__fmul_rn(__fmul_rn(k.spiky_coefficient, difference), difference), distance));
}

// The same values out of line, for the pairs outside the range of the packed arithmetic below: a rare
// path, whose inlined root and divisions would cost the replay loops registers.
static __device__ __noinline__ float poly6_call(const float r2, const float h2, const float denominator) {
    const float difference = __fsub_rn(h2, r2);
    return __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(315.0F, difference), difference), difference), denominator);
}
static __device__ __noinline__ float sqrt_call(const float v) { return __fsqrt_rn(v); }
static __device__ __noinline__ float spiky_scale_call(const float distance, const float h, const float coefficient) {
    const float difference = __fsub_rn(h, distance);
    return __fdiv_rn(__fmul_rn(__fmul_rn(coefficient, difference), difference), distance);
}

__device__ __forceinline__ f3 spiky_gradient(const f3 d, const KernelConstants& k) {
    const float distance = __fsqrt_rn(squared(d));
    if (distance == 0.0F || distance >= k.h) return {0.0F, 0.0F, 0.0F};
    return spiky_gradient_at(d, distance, k);
}

// ------------------------------------------------- two pairs at a time, packed FP32
// The replay passes were bound by instruction issue, and most of a pair's instructions were its IEEE
// square root and divisions, each with range tests and a branch around a slow path.  Inside a
// range of r2 where nothing can overflow or turn subnormal (fast_min to fast_max) the same correctly rounded
// values follow from one reciprocal square root and fused residual corrections, without a branch,
// so two pairs share every instruction (packed FP32, each half rounded as the scalar intrinsic):
//   sqrt:  s0 = r2 y, s = s0 + (r2 - s0^2) y / 2 with y ~ 1 / sqrt(r2).  Equal to __fsqrt_rn for
//          every r2 of the range (all floats checked by tests/test_gpu_pair_math.py).
//   a / b: q0 = a R, q = q0 + (a - b q0) R with R = RN(1 / b), which is RN(a / b)
//          (P. Markstein, IBM J. Res. Dev. 34(1), 1990; M. Cornea, J. Harrison, P. Tang, Scientific
//          Computing on Itanium, 2002).  For b = s, R = y + y (e + 2^-44)
//          with e = 1 - s y: a Newton step that rounds up (|e| < 2^-22.2, so e^2 < 2^-44).  Without
//          the 2^-44, R is an ulp low for s = 2 - 2^-23 and 1 / s comes out wrong.  The same test
//          checks, for every s, the quotients that lie nearest a rounding boundary.
__device__ __forceinline__ float2 both(const float v) { return make_float2(v, v); }

// The negated squared distance, -squared(d), of displacement d.
__device__ __forceinline__ float negated_squared(const f3 d) {
    return __fmaf_rn(-d.z, d.z, __fmaf_rn(-d.x, d.x, -__fmul_rn(d.y, d.y)));
}

__device__ __forceinline__ float approximate_rsqrt(const float v) {
    float y;
    asm("rsqrt.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(v));
    return y;
}

// a / b of two pairs, given -b and the correctly rounded 1 / b.
__device__ __forceinline__ float2 quotient_pair(const float2 a, const float2 negated_b, const float2 reciprocal) {
    const float2 q = __fmul2_rn(a, reciprocal);
    return __ffma2_rn(__ffma2_rn(negated_b, q, a), reciprocal, q);
}

// -sqrt(r2) of two pairs from -r2, and the correctly rounded 1 / sqrt(r2) of that root.
__device__ __forceinline__ float2 negated_root_pair(const float2 nr2, float2& reciprocal) {
    const float2 y = make_float2(approximate_rsqrt(-nr2.x), approximate_rsqrt(-nr2.y));
    const float2 ns0 = __fmul2_rn(nr2, y);
    const float2 ns = __ffma2_rn(__ffma2_rn(ns0, ns0, nr2), __fmul2_rn(y, both(0.5F)), ns0);
    const float2 e = __ffma2_rn(ns, y, both(1.0F));
    reciprocal = __ffma2_rn(__fadd2_rn(e, both(0x1p-44F)), y, y);
    return ns;
}

// poly6_inside of two pairs from their negated squared distances.
__device__ __forceinline__ float2 poly6_pair(const float2 nr2, const KernelConstants& k) {
    const float2 difference = __fadd2_rn(both(k.h2), nr2);
    const float2 a = __fmul2_rn(__fmul2_rn(__fmul2_rn(both(315.0F), difference), difference), difference);
    return quotient_pair(a, both(-k.poly6_denominator), both(k.poly6_reciprocal));
}

// The scale of spiky_gradient_at, grad W = d * scale, of two pairs (undefined at r2 = 0).
__device__ __forceinline__ float2 spiky_scale_pair(const float2 nr2, const KernelConstants& k) {
    float2 reciprocal;
    const float2 ns = negated_root_pair(nr2, reciprocal);
    const float2 difference = __fadd2_rn(both(k.h), ns);
    const float2 a = __fmul2_rn(__fmul2_rn(both(k.spiky_coefficient), difference), difference);
    return quotient_pair(a, ns, reciprocal);
}

// ------------------------------------------------------------------ FP64 helpers of the adjoint
__device__ __forceinline__ d3 ld3(const double4 v) { return {v.x, v.y, v.z}; }
__device__ __forceinline__ double4 st3(const d3 v) { return make_double4(v.x, v.y, v.z, 0.0); }

// FP64 1 / sqrt(v) and 1 / v of a float: the FP32 approximation and one third-order step (relative
// error of the start e: 5/16 e^3 and e^3, below 2^-65), where rsqrt() and a division test their range
// and take two steps.
__device__ __forceinline__ double wide_rsqrt(const float v, const float approximation) {
    const double y = approximation;
    const double e = fma(-(static_cast<double>(v) * y), y, 1.0);
    return fma(y * e, fma(e, 0.375, 0.5), y);
}
__device__ __forceinline__ double wide_rsqrt(const float v) {
    if (v >= 0x1p-100F && v <= 0x1p100F) return wide_rsqrt(v, approximate_rsqrt(v));
    return rsqrt(static_cast<double>(v));
}
__device__ __forceinline__ double wide_reciprocal(const float v) {
    if (!(v >= 0x1p-100F && v <= 0x1p100F)) return 1.0 / static_cast<double>(v);
    float approximation;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(approximation) : "f"(v));
    const double y = approximation;
    const double e = fma(-static_cast<double>(v), y, 1.0);
    return fma(y, fma(e, e, e), y);
}

// One pair's kernel derivatives for the FP64 reverse passes: grad W = d * scale, rounded as
// spiky_gradient, and the Hessian as H(d) v = along v + across (d . v) d in FP64.  H is linear and
// H(-d) = H(d), so a pair's two directions need one product, of the difference of their vectors:
// half the FP64 work of a product each, and no unit direction is formed.  The FP64 reciprocal root
// starts from the FP32 one that the gradient needs anyway.
struct PairDerivatives {
    float scale;
    double along, across;
};
__device__ __forceinline__ PairDerivatives pair_derivatives(const float r2, const KernelConstants& k) {   // 0 < r2
    PairDerivatives p;
    const double r2d = r2;
    double inverse;
    if (r2 >= k.fast_min && r2 <= k.fast_max) {
        const float y = approximate_rsqrt(r2);
        const float s0 = r2 * y;
        const float s = __fmaf_rn(__fmaf_rn(-s0, s0, r2), 0.5F * y, s0);
        const float reciprocal = __fmaf_rn(__fadd_rn(__fmaf_rn(-s, y, 1.0F), 0x1p-44F), y, y);
        const float difference = __fsub_rn(k.h, s);
        const float a = __fmul_rn(__fmul_rn(k.spiky_coefficient, difference), difference);
        const float q = __fmul_rn(a, reciprocal);
        p.scale = __fmaf_rn(__fmaf_rn(-s, q, a), reciprocal, q);
        inverse = wide_rsqrt(r2, y);
    } else {
        p.scale = r2 < k.spiky_threshold ? spiky_scale_call(sqrt_call(r2), k.h, k.spiky_coefficient) : 0.0F;
        inverse = rsqrt(r2d);
    }
    const double difference = k.h - r2d * inverse;
    const double slope = k.spiky_coefficient_d * difference;
    p.along = slope * difference * inverse;
    p.across = -(slope + slope + p.along) * (inverse * inverse);
    if (r2 >= k.hessian_threshold) p.along = p.across = 0.0;   // sqrt((double)r2) >= h
    return p;
}
// H(d) v
__device__ __forceinline__ d3 hessian_product(const PairDerivatives& p, const d3 d, const d3 v) {
    const double across = p.across * (d.x * v.x + d.y * v.y + d.z * v.z);
    return {fma(across, d.x, p.along * v.x), fma(across, d.y, p.along * v.y), fma(across, d.z, p.along * v.z)};
}
__device__ __forceinline__ d3 wide(const f3 v) { return {v.x, v.y, v.z}; }

// The poly6 weight of poly6_inside without its division's range tests (r2 up to fast_max).
__device__ __forceinline__ float poly6_weight(const float r2, const KernelConstants& k) {
    if (r2 > k.fast_max) return r2 >= k.h2 ? 0.0F : poly6_call(r2, k.h2, k.poly6_denominator);
    const float difference = __fsub_rn(k.h2, r2);
    const float a = __fmul_rn(__fmul_rn(__fmul_rn(315.0F, difference), difference), difference);
    const float q = __fmul_rn(a, k.poly6_reciprocal);
    return __fmaf_rn(__fmaf_rn(-k.poly6_denominator, q, a), k.poly6_reciprocal, q);
}

// The scale of poly6_gradient, grad W = d * scale, likewise (r2 < h2).
__device__ __forceinline__ float poly6_gradient_scale(const float r2, const KernelConstants& k) {
    const float difference = __fsub_rn(k.h2, r2);
    const float a = __fmul_rn(__fmul_rn(-945.0F, difference), difference);
    if (r2 > k.fast_max) return __fdiv_rn(a, k.poly6_grad_denominator);
    const float q = __fmul_rn(a, k.poly6_grad_reciprocal);
    return __fmaf_rn(__fmaf_rn(-k.poly6_grad_denominator, q, a), k.poly6_grad_reciprocal, q);
}

// Spiky Hessian applied to a vector, in FP64 (pbf/pbf.cu:45-54 evaluation order).
// The adjoint is held to FP64 rounding against the reference, so the distance and its reciprocal
// come from one reciprocal square root rather than a square root and a division; the support test
// is the exact one on the squared distance.
__device__ __forceinline__ d3 spiky_hessian_product(const f3 d, const d3 v, const KernelConstants& k) {
    const float r2f = squared(d);
    if (r2f == 0.0F || r2f >= k.hessian_threshold) return {0.0, 0.0, 0.0};   // sqrt((double)r2) == 0 or >= h
    const double r2 = r2f;
    const double inverse = rsqrt(r2);
    const double distance = r2 * inverse;
    const d3 direction = times(d, inverse);
    const double projection = dot(direction, v);
    const d3 direction_tangent = times(v - times(direction, projection), inverse);
    const double difference = k.h - distance;
    return times(times(direction, -2.0 * difference * projection) + times(direction_tangent, difference * difference),
                 k.spiky_coefficient_d);
}

// d/dr of poly6 along a radius (pbf/pbf.cu:18-24).
__device__ __forceinline__ float poly6_radial_derivative(const float radius, const KernelConstants& k) {
    if (radius >= k.h) return 0.0F;
    const float difference = __fmaf_rn(-radius, radius, __fmul_rn(k.h, k.h));
    return __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(-6.0F, k.poly6_radial_coefficient), radius), difference), difference);
}

// Artificial pressure s_corr = -strength (W(d)/W(radius))^exponent and its derivatives (pbf/pbf.cu:56-71).
struct ArtificialPressure {
    float value, d_strength, d_exponent, d_radius;
    f3 gradient;
};

__device__ __forceinline__ ArtificialPressure artificial_pressure(const f3 d, const KernelConstants& k, const float strength,
                                                                  const float exponent, const float radius) {
    ArtificialPressure a;
    const float reference = poly6(mk(radius, 0.0F, 0.0F), k);
    const float kernel = poly6(d, k);
    if (kernel == 0.0F) {
        a.value = a.d_strength = a.d_exponent = a.d_radius = 0.0F;
        a.gradient = {0.0F, 0.0F, 0.0F};
        return a;
    }
    const float ratio = __fdiv_rn(kernel, reference);
    const float power = powf(ratio, exponent);
    a.value = __fmul_rn(-strength, power);
    a.d_strength = -power;
    a.d_exponent = __fmul_rn(a.value, logf(ratio));
    a.d_radius = __fdiv_rn(__fmul_rn(__fmul_rn(-a.value, exponent), poly6_radial_derivative(radius, k)), reference);
    a.gradient = scale(poly6_gradient(d, k),
                       __fdiv_rn(__fmul_rn(__fmul_rn(-strength, exponent), powf(ratio, exponent - 1.0F)), reference));
    return a;
}

}  // namespace pbf
