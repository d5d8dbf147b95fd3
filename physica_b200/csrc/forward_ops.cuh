// Per-pair operations of the forward passes and the packed candidate test, shared by the per-lane
// kernels (forward.cu) and the staged ones (staged.cu).
#pragma once

#include "gather.cuh"

namespace pbf {
namespace gather_detail {

// The same test over positions stored as three arrays, two candidates per packed FP32 instruction
// (__fadd2_rn, __fmul2_rn, __ffma2_rn round each half exactly as the scalar intrinsics do).  The
// difference is taken as candidate minus particle; it is the exact negation of the scalar form's
// particle minus candidate, so the squared distance has the same bits.  Groups of four slots are
// loaded as one aligned float4 per axis: a range is widened down to a multiple of four and the
// slots outside it are dropped from the mask.
struct PackedScan {
    float2 nx, ny, nz;   // the particle's negated coordinates, in both halves
    float threshold;
    uint32_t capacity;
    uint32_t* __restrict__ entries;
    uint32_t n;

    __device__ __forceinline__ uint32_t hits2(const float2 x, const float2 y, const float2 z) const {
        const float2 dx = __fadd2_rn(x, nx), dy = __fadd2_rn(y, ny), dz = __fadd2_rn(z, nz);
        const float2 r2 = __ffma2_rn(dz, dz, __ffma2_rn(dx, dx, __fmul2_rn(dy, dy)));
        return (r2.x < threshold ? 1u : 0u) | (r2.y < threshold ? 2u : 0u);
    }
    __device__ __forceinline__ uint32_t hits4(const float4 x, const float4 y, const float4 z) const {
        return hits2(make_float2(x.x, x.y), make_float2(y.x, y.y), make_float2(z.x, z.y)) |
               (hits2(make_float2(x.z, x.w), make_float2(y.z, y.w), make_float2(z.z, z.w)) << 2);
    }
    __device__ __forceinline__ void append(uint32_t mask, const uint32_t base) {
        while (mask) {
            const uint32_t k = static_cast<uint32_t>(__ffs(mask)) - 1u;
            if (n < capacity) entries[static_cast<size_t>(n) * 32u] = base + k;
            ++n;
            mask &= mask - 1u;
        }
    }
    // Hit mask of the 32-slot block at `base` (4-aligned) of the range [first, end).
    __device__ __forceinline__ uint32_t block_mask(const PackedPositions p, const uint32_t base, const uint32_t first,
                                                   const uint32_t end) const {
        const uint32_t stop = min(end, base + 32u);
        uint32_t mask = 0u;
        for (uint32_t k = 0u; base + k < stop; k += 4u) {
            const uint32_t t = base + k;
            mask |= hits4(*reinterpret_cast<const float4*>(p.x + t), *reinterpret_cast<const float4*>(p.y + t),
                          *reinterpret_cast<const float4*>(p.z + t))
                    << k;
        }
        if (base < first) mask &= ~0u << (first - base);
        if (end - base < 32u) mask &= (1u << (end - base)) - 1u;
        return mask;
    }
    __device__ __forceinline__ void run(const PackedPositions p, const uint32_t first, const uint32_t end) {
        if (first >= end) return;
        for (uint32_t base = first & ~3u; base < end; base += 32u) append(block_mask(p, base, first, end), base);
    }
    // The same as hit masks: one pair per block with a hit; `pairs` counts them, n the neighbours.
    __device__ __forceinline__ void run_masks(const PackedPositions p, const uint32_t first, const uint32_t end, uint2* row,
                                              const uint32_t pair_capacity, uint32_t& pairs) {
        if (first >= end) return;
        for (uint32_t base = first & ~3u; base < end; base += 32u) {
            const uint32_t mask = block_mask(p, base, first, end);
            if (mask) {
                if (pairs < pair_capacity) row[static_cast<size_t>(pairs) * 32u] = make_uint2(base, mask);
                ++pairs;
                n += static_cast<uint32_t>(__popc(mask));
            }
        }
    }
};

// density (density/density.cu:18-40) and lambda (pbf/pbf.cu:95-127) of one particle in one walk.
// m_j / rho0_i for a run of neighbours: most neighbours share a mass, so the last quotient is
// kept and reused while the mass bits repeat (same operands, same correctly rounded quotient).
struct MassRatio {
    uint32_t mass_bits;
    float quotient;
    __device__ __forceinline__ void reset(const float mass, const float rest_density) {
        mass_bits = __float_as_uint(mass);
        quotient = __fdiv_rn(mass, rest_density);
    }
    __device__ __forceinline__ float operator()(const float mass, const float rest_density) {
        const uint32_t bits = __float_as_uint(mass);
        if (bits != mass_bits) reset(mass, rest_density);
        return quotient;
    }
};

// WithBoundary: the scene has boundary particles (their entries carry kBoundaryBit); the plain
// instantiation, launched otherwise, carries no boundary test.
template <bool WithBoundary>
struct DensityLambdaOp {
    static constexpr bool kBoundary = WithBoundary;
    const float4* __restrict__ pos;
    const float4* __restrict__ boundary;
    f3 x;
    uint32_t self;
    float rest_density;
    KernelConstants k;
    float density;
    f3 gradient_sum;
    float denominator;
    uint32_t neighbors;
    MassRatio ratio;

    __device__ __forceinline__ float4 prefetch(const uint32_t t) const {
        if constexpr (WithBoundary) return (t & kBoundaryBit) ? boundary[t & ~kBoundaryBit] : pos[t];
        return pos[t];
    }
    __device__ __forceinline__ void apply(const uint32_t t, const float4 q) {
        const f3 d = sub(x, xyz(q));
        const float r2 = squared(d);
        if (WithBoundary && (t & kBoundaryBit)) {
            // boundary particle b: density += rho0_i V_b W (density/density.cu:34-37),
            // S += V_b grad W (pbf/pbf.cu:118-121); no denominator term
            if (r2 < k.h2) density = __fmaf_rn(__fmul_rn(rest_density, q.w), poly6_inside(r2, k), density);
            const float distance = __fsqrt_rn(r2);
            if (distance == 0.0F || distance >= k.h) return;
            gradient_sum = fma3(q.w, spiky_gradient_at(d, distance, k), gradient_sum);
            return;
        }
        if (r2 < k.h2) density = __fmaf_rn(q.w, poly6_inside(r2, k), density);
        if (t == self) return;
        if (r2 < k.h2) ++neighbors;
        const float distance = __fsqrt_rn(r2);
        if (distance == 0.0F || distance >= k.h) return;
        const f3 gradient = spiky_gradient_at(d, distance, k);
        const float coefficient = ratio(q.w, rest_density);
        gradient_sum = fma3(coefficient, gradient, gradient_sum);
        denominator = __fmaf_rn(__fmul_rn(coefficient, coefficient), sq_xfirst(gradient), denominator);
    }
    __device__ __forceinline__ void process(const uint32_t t) { apply(t, prefetch(t)); }
};

// -------------------------------------------------------------- correction
// correction (pbf/pbf.cu:254-288) and project (pbf/pbf.cu:417-431); on the last iteration
// also reconstruct (pbf/pbf.cu:456-460) and the write-back of next_state.positions.
struct PositionLambda {
    float4 q;
    float lambda;
};

template <bool WithBoundary>
struct CorrectionOp {
    static constexpr bool kBoundary = WithBoundary;
    const float4* __restrict__ pos;
    const float4* __restrict__ boundary;
    const float* __restrict__ lambda;
    f3 x;
    uint32_t self;
    float rest_density;
    float lambda_i;
    float strength, exponent, reference_weight;
    bool artificial_full;
    KernelConstants k;
    f3 correction;
    MassRatio ratio;

    __device__ __forceinline__ PositionLambda prefetch(const uint32_t t) const {
        if (WithBoundary && (t & kBoundaryBit)) return {boundary[t & ~kBoundaryBit], 0.0F};
        return {pos[t], lambda[t]};
    }
    __device__ __forceinline__ void apply(const uint32_t t, const PositionLambda in) {
        if (t == self) return;
        const f3 d = sub(x, xyz(in.q));
        const float r2 = squared(d);
        const float distance = __fsqrt_rn(r2);
        if (distance == 0.0F || distance >= k.h) return;
        // s_corr (pbf/pbf.cu:56-71).  With zero strength it is -strength * ratio^n, i.e. -0 inside
        // the poly6 support and 0 outside, which the fast branch yields without powf.
        float artificial;
        if (artificial_full) {
            const float weight = r2 >= k.h2 ? 0.0F : poly6_inside(r2, k);
            artificial = weight == 0.0F ? 0.0F : __fmul_rn(-strength, powf(__fdiv_rn(weight, reference_weight), exponent));
        } else {
            artificial = r2 < k.h2 ? -strength : 0.0F;
        }
        if (WithBoundary && (t & kBoundaryBit)) {
            // boundary particle b: V_b (lambda_i + s_corr) grad W (pbf/pbf.cu:278-285)
            const float factor = __fmul_rn(in.q.w, __fadd_rn(lambda_i, artificial));
            correction = fma3(factor, spiky_gradient_at(d, distance, k), correction);
            return;
        }
        const float coefficient = ratio(in.q.w, rest_density);
        const float factor = __fmul_rn(coefficient, __fadd_rn(__fadd_rn(lambda_i, in.lambda), artificial));
        correction = fma3(factor, spiky_gradient_at(d, distance, k), correction);
    }
    __device__ __forceinline__ void process(const uint32_t t) { apply(t, prefetch(t)); }
};

// -------------------------------------------------- vorticity, normal, XSPH
// vorticity (pbf/pbf.cu:476-497) and its magnitude (pbf/pbf.cu:565-569).
struct PositionVector {
    float4 q;
    float4 v;
};

struct VorticityOp {
    const float4* __restrict__ pos;
    const float4* __restrict__ velocity;
    f3 x, v;
    uint32_t self;
    KernelConstants k;
    f3 vorticity;

    __device__ __forceinline__ PositionVector prefetch(const uint32_t t) const { return {pos[t], velocity[t]}; }
    __device__ __forceinline__ void apply(const uint32_t t, const PositionVector in) {
        if (t == self) return;
        const f3 d = sub(x, xyz(in.q));
        const float distance = __fsqrt_rn(squared(d));
        if (distance == 0.0F || distance >= k.h) return;
        vorticity = add(vorticity, cross_f(sub(xyz(in.v), v), spiky_gradient_at(d, distance, k)));
    }
    __device__ __forceinline__ void process(const uint32_t t) { apply(t, prefetch(t)); }
};

// normal (pbf/pbf.cu:571-593) and confinement (pbf/pbf.cu:674-678).
struct PositionScalar {
    float4 q;
    float w;
};

struct NormalOp {
    const float4* __restrict__ pos;
    const float4* __restrict__ vorticity;
    f3 x;
    float magnitude;
    uint32_t self;
    KernelConstants k;
    f3 gradient;

    __device__ __forceinline__ PositionScalar prefetch(const uint32_t t) const { return {pos[t], vorticity[t].w}; }
    __device__ __forceinline__ void apply(const uint32_t t, const PositionScalar in) {
        if (t == self) return;
        const f3 d = sub(x, xyz(in.q));
        const float distance = __fsqrt_rn(squared(d));
        if (distance == 0.0F || distance >= k.h) return;
        gradient = fma3(__fsub_rn(in.w, magnitude), spiky_gradient_at(d, distance, k), gradient);
    }
    __device__ __forceinline__ void process(const uint32_t t) { apply(t, prefetch(t)); }
};

// XSPH (pbf/pbf.cu:700-721) and the write-back of next_state.velocities.
struct XsphOp {
    const float4* __restrict__ pos;
    const float4* __restrict__ confined;
    f3 x, v;
    uint32_t self;
    KernelConstants k;
    f3 smoothing;

    __device__ __forceinline__ PositionVector prefetch(const uint32_t t) const { return {pos[t], confined[t]}; }
    __device__ __forceinline__ void apply(const uint32_t t, const PositionVector in) {
        if (t == self) return;
        const f3 d = sub(x, xyz(in.q));
        const float r2 = squared(d);
        if (r2 >= k.h2) return;
        smoothing = fma3(poly6_inside(r2, k), sub(xyz(in.v), v), smoothing);
    }
    __device__ __forceinline__ void process(const uint32_t t) { apply(t, prefetch(t)); }
};

}  // namespace gather_detail
}  // namespace pbf
