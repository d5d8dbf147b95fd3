// Pair arithmetic and per-particle tails of the staged PBF passes (staged.cu, staged_group.cu).
#pragma once

#include "staged.cuh"

namespace pbf {
namespace staged_detail {

// ------------------------------------------------------------------- pair arithmetic
// Two pairs' displacements and negated squared distances.
struct TwoPairs {
    f3 d0, d1;
    float2 nr2;
};
__device__ __forceinline__ TwoPairs two_pairs(const f3 x, const f3 q0, const f3 q1) {
    TwoPairs t;
    t.d0 = sub(x, q0);
    t.d1 = sub(x, q1);
    t.nr2 = make_float2(negated_squared(t.d0), negated_squared(t.d1));
    return t;
}
__device__ __forceinline__ bool in_range(const float2 nr2, const KernelConstants& k) {
    return -nr2.x <= k.fast_max && -nr2.x >= k.fast_min && -nr2.y <= k.fast_max && -nr2.y >= k.fast_min;
}
// Any r2: the gradient scale, 0 where the pair has no gradient; the weight, 0 outside the support.
static __device__ __noinline__ float any_spiky_scale(const float r2, const float h, const float coefficient) {
    const float distance = __fsqrt_rn(r2);
    if (distance == 0.0F || distance >= h) return 0.0F;
    const float difference = __fsub_rn(h, distance);
    return __fdiv_rn(__fmul_rn(__fmul_rn(coefficient, difference), difference), distance);
}
static __device__ __noinline__ float any_poly6(const float r2, const float h2, const float denominator) {
    if (r2 >= h2) return 0.0F;
    const float difference = __fsub_rn(h2, r2);
    return __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(315.0F, difference), difference), difference), denominator);
}
__device__ __forceinline__ float2 any_spiky_scales(const float2 nr2, const KernelConstants& k) {
    return make_float2(any_spiky_scale(-nr2.x, k.h, k.spiky_coefficient), any_spiky_scale(-nr2.y, k.h, k.spiky_coefficient));
}
__device__ __forceinline__ float2 any_poly6s(const float2 nr2, const KernelConstants& k) {
    return make_float2(any_poly6(-nr2.x, k.h2, k.poly6_denominator), any_poly6(-nr2.y, k.h2, k.poly6_denominator));
}

// A pair whose kernel value is zero adds nothing, whatever its other factor is (it may be infinite).
// Called in the branch that such pairs take.  With one lane a particle the factors are formed before that branch (262k
// particles, three iterations: 0.500 against 0.504 ms a step), with four behind it, so that no call has them in flight (14k:
// normal 18.7 against 20.1 us, XSPH 18.2 against 19.5).
__device__ __forceinline__ void only_inside(const float2 kernel, float& f0, float& f1) {
    if (kernel.x == 0.0F) f0 = 0.0F;
    if (kernel.y == 0.0F) f1 = 0.0F;
}
__device__ __forceinline__ void only_inside(const float2 kernel, f3& f0, f3& f1) {
    if (kernel.x == 0.0F) f0 = mk(0.0F, 0.0F, 0.0F);
    if (kernel.y == 0.0F) f1 = mk(0.0F, 0.0F, 0.0F);
}

// The factors of two correction terms and the scales of their gradients.
struct PairFactors {
    TwoPairs t;
    float2 spiky;
    float first, second;
};
template <uint32_t S>
__device__ __forceinline__ PairFactors correction_factors(const KernelConstants& k, const f3 xi, const float mass,
                                                          const float rest_density, const float ratio, const float lambda,
                                                          const bool full, const float4 pb, const float reference,
                                                          const float (&field)[5][S], const uint32_t i0, const uint32_t i1) {
    const float m0 = field[3][i0], m1 = field[3][i1];
    PairFactors f;
    const TwoPairs t = two_pairs(xi, mk(field[0][i0], field[1][i0], field[2][i0]),
                                 mk(field[0][i1], field[1][i1], field[2][i1]));
    float2 spiky = spiky_scale_pair(t.nr2, k);
    // s_corr (pbf/pbf.cu:56-71): with zero strength -strength inside the poly6 support
    float a0 = -pb.x, a1 = -pb.x;
    float c0 = ratio, c1 = ratio;
    if (full) {
        const float2 weight = in_range(t.nr2, k) ? poly6_pair(t.nr2, k) : any_poly6s(t.nr2, k);
        a0 = weight.x == 0.0F ? 0.0F : __fmul_rn(-pb.x, powf(__fdiv_rn(weight.x, reference), pb.y));
        a1 = weight.y == 0.0F ? 0.0F : __fmul_rn(-pb.x, powf(__fdiv_rn(weight.y, reference), pb.y));
    }
    float s0 = __fadd_rn(lambda, field[4][i0]), s1 = __fadd_rn(lambda, field[4][i1]);
    if (!in_range(t.nr2, k) || m0 != mass || m1 != mass) {
        c0 = __fdiv_rn(m0, rest_density);
        c1 = __fdiv_rn(m1, rest_density);
        if (!in_range(t.nr2, k)) {
            spiky = any_spiky_scales(t.nr2, k);
            if (!full) {
                a0 = -t.nr2.x < k.h2 ? a0 : 0.0F;
                a1 = -t.nr2.y < k.h2 ? a1 : 0.0F;
            }
            if (spiky.x == 0.0F) c0 = s0 = a0 = 0.0F;   // no gradient: no term, whatever the factors are
            if (spiky.y == 0.0F) c1 = s1 = a1 = 0.0F;
        }
    }
    const float f0 = __fmul_rn(c0, __fadd_rn(s0, a0));
    const float f1 = __fmul_rn(c1, __fadd_rn(s1, a1));
    f.t = t;
    f.spiky = spiky;
    f.first = f0;
    f.second = f1;
    return f;
}

// The correction of a particle that replays slots or walks its stencil.
__device__ __forceinline__ f3 correction_alone(const StagedCorrectionArgs& a, const Particle& p, const f3 xi, const float mass,
                                               const float lambda) {
    const float4 pa = a.g.params_a[p.s];
    const float4 pb = a.g.params_b[p.s];
    CorrectionOp<false> op;
    op.pos = a.pos;
    op.boundary = nullptr;
    op.lambda = a.lambda;
    op.self = p.s;
    op.k = p.k;
    op.x = xi;
    op.rest_density = pa.x;
    op.ratio.reset(mass, pa.x);
    op.lambda_i = lambda;
    op.strength = pb.x;
    op.exponent = pb.y;
    op.artificial_full = pb.x != 0.0F;
    op.reference_weight = op.artificial_full ? poly6(mk(pb.z, 0.0F, 0.0F), p.k) : 1.0F;
    op.correction = mk(0.0F, 0.0F, 0.0F);
    replay_alone(op, p, a.g, a.list.list);
    return op.correction;
}

// Project (pbf/pbf.cu:417-431) and, on the last iteration, reconstruct (pbf/pbf.cu:456-460).
__device__ __forceinline__ void correction_tail(const StagedCorrectionArgs& a, const Particle& p, const f3 xi, const float mass,
                                                const f3 correction) {
    const uint32_t s = p.s;
    const Box& box = p.scene->box;
    const f3 candidate = add(xi, correction);
    const f3 projected = mk(fminf(box.max_x, fmaxf(box.min_x, candidate.x)), fminf(box.max_y, fmaxf(box.min_y, candidate.y)),
                            fminf(box.max_z, fmaxf(box.min_z, candidate.z)));
    a.pos_next[s] = make_float4(projected.x, projected.y, projected.z, mass);
    if (a.mask)
        a.mask[s] = static_cast<uint8_t>((candidate.x < box.min_x || candidate.x > box.max_x ? 1u : 0u) |
                                         (candidate.y < box.min_y || candidate.y > box.max_y ? 2u : 0u) |
                                         (candidate.z < box.min_z || candidate.z > box.max_z ? 4u : 0u));
    a.positions_next.x[s] = projected.x;
    a.positions_next.y[s] = projected.y;
    a.positions_next.z[s] = projected.z;
    if (a.last) {
        const uint32_t i = a.sorted_index[s];
        const f3 previous = mk(a.previous_positions.x[i], a.previous_positions.y[i], a.previous_positions.z[i]);
        const f3 velocity = scale(sub(projected, previous), p.scene->inverse_time_step);
        a.velocity[s] = make_float4(velocity.x, velocity.y, velocity.z, 0.0F);
        a.velocities.x[s] = velocity.x;
        a.velocities.y[s] = velocity.y;
        a.velocities.z[s] = velocity.z;
        a.out_positions.x[i] = projected.x;
        a.out_positions.y[i] = projected.y;
        a.out_positions.z[i] = projected.z;
    }
}

__device__ __forceinline__ f3 normal_alone(const StagedNormalArgs& a, const Particle& p, const f3 xi, const float magnitude) {
    NormalOp op;
    op.pos = a.pos;
    op.vorticity = a.vorticity;
    op.self = p.s;
    op.k = p.k;
    op.x = xi;
    op.magnitude = magnitude;
    op.gradient = mk(0.0F, 0.0F, 0.0F);
    replay_alone(op, p, a.g, a.list.list);
    return op.gradient;
}

// The normalised gradient and the confinement force (pbf/pbf.cu:674-678).
__device__ __forceinline__ void normal_tail(const StagedNormalArgs& a, const Particle& p, const float4 wi, const f3 gradient) {
    const uint32_t s = p.s;
    const float normalizer = __fsqrt_rn(sq_yfirst(gradient));
    const f3 normal = normalizer > 0.0F ? scale(gradient, __fdiv_rn(1.0F, normalizer)) : mk(0.0F, 0.0F, 0.0F);
    a.normal[s] = make_float4(normal.x, normal.y, normal.z, normalizer);
    const f3 v = xyz(a.velocity[s]);
    const f3 confined = fma3(__fmul_rn(p.scene->time_step, a.g.params_a[s].w), cross_f(normal, xyz(wi)), v);
    a.confined[s] = make_float4(confined.x, confined.y, confined.z, 0.0F);
    a.confined_soa.x[s] = confined.x;
    a.confined_soa.y[s] = confined.y;
    a.confined_soa.z[s] = confined.z;
}

__device__ __forceinline__ f3 xsph_alone(const StagedXsphArgs& a, const Particle& p, const f3 xi, const f3 vi) {
    XsphOp op;
    op.pos = a.pos;
    op.confined = a.confined;
    op.self = p.s;
    op.k = p.k;
    op.x = xi;
    op.v = vi;
    op.smoothing = mk(0.0F, 0.0F, 0.0F);
    replay_alone(op, p, a.g, a.list.list);
    return op.smoothing;
}

__device__ __forceinline__ void xsph_tail(const StagedXsphArgs& a, const Particle& p, const f3 vi, const f3 smoothing) {
    const uint32_t s = p.s;
    const f3 out = fma3(a.g.params_a[s].z, smoothing, vi);
    const uint32_t i = a.sorted_index[s];
    a.out_velocities.x[i] = out.x;
    a.out_velocities.y[i] = out.y;
    a.out_velocities.z[i] = out.z;
}

}  // namespace staged_detail
}  // namespace pbf
