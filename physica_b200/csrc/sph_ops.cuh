// Per-pair operations and per-particle tails of the SPH forward passes, shared by the per-lane kernels
// (sph.cu) and the staged ones (sph_staged.cu).
#pragma once

#include "sph_math.cuh"

namespace pbf {
namespace sph {
namespace detail {

// ------------------------------------------------------------------ density (+ Tait EOS)
template <bool WithBoundary>
struct DensityOp {
    static constexpr bool kBoundary = WithBoundary;
    const float4* __restrict__ pos;
    const float4* __restrict__ boundary;
    f3 x;
    float rest_density;
    SphConstants k;
    float density;

    __device__ __forceinline__ float4 prefetch(const uint32_t t) const {
        if constexpr (WithBoundary) return (t & kBoundaryBit) ? boundary[t & ~kBoundaryBit] : pos[t];
        return pos[t];
    }
    __device__ __forceinline__ void apply(const uint32_t t, const float4 q) {
        const float distance = __fsqrt_rn(sq_xfirst(sub(x, xyz(q))));
        if (distance >= k.h) return;
        const float w = cubic_inside(distance, k);
        // fluid: density += m_j W; boundary: density += rho0_i V_b W (density/density.cu:30-37)
        if (WithBoundary && (t & kBoundaryBit)) density = __fmaf_rn(__fmul_rn(rest_density, q.w), w, density);
        else density = __fmaf_rn(q.w, w, density);
    }
    __device__ __forceinline__ void process(const uint32_t t) { apply(t, prefetch(t)); }
};

// The density of a particle and what follows from it.
__device__ __forceinline__ void density_tail(const SphStep& st, const Own& o, const float rho, const uint32_t method,
                                             float* density_record, float* pressure, float* pressure_term, const float* warm) {
    const float4 pb = st.g.params_b[o.p.s];
    float p = 0.0F;
    if (method == kWcsph) {
        // p = rho0 c c ((rho / rho0)^gamma - 1) / gamma (sph/wcsph.cu:92-100)
        const float rest = o.pa.x, speed = o.pa.w, exponent = pb.x;
        const float ratio = __fdiv_rn(rho, rest);
        p = __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(rest, speed), speed), __fsub_rn(powf(ratio, exponent), 1.0F)), exponent);
        st.aux[o.p.s] = make_float4(rho, o.pa.y, speed, o.pa.z);
    } else {
        st.aux[o.p.s] = make_float4(rho, o.pa.y, 0.0F, 0.0F);
        if (warm) p = warm[st.sorted_index[o.p.s]];
    }
    if (density_record) density_record[o.p.s] = rho;
    if (pressure) pressure[o.p.s] = p;
    if (pressure_term) pressure_term[o.p.s] = __fdiv_rn(p, __fmul_rn(rho, rho));
}

// ------------------------------------------------------------------ WCSPH forces
struct ForceData {
    float4 q;    // (x, m) or boundary (x, V)
    float4 v;    // (v, -)
    float4 aux;  // (rho, viscosity, speed of sound, -)
    float pt;    // p / rho^2
};

template <bool WithBoundary>
struct WcsphForceOp {
    static constexpr bool kBoundary = WithBoundary;
    const float4* __restrict__ pos;
    const float4* __restrict__ vel;
    const float4* __restrict__ aux;
    const float* __restrict__ pt;
    const float4* __restrict__ boundary;
    const float4* __restrict__ boundary_velocity;
    uint32_t self;
    f3 x, v;
    float mass, rest, density, viscosity, speed, first_term, surface_tension, boundary_tension;
    float boundary_nu;   // viscosity_i h c_i / rho_i (sph/wcsph.cu:167)
    SphConstants k;
    f3 pressure, artificial, surface;

    __device__ __forceinline__ ForceData prefetch(const uint32_t t) const {
        ForceData d;
        if (WithBoundary && (t & kBoundaryBit)) {
            d.q = boundary[t & ~kBoundaryBit];
            d.v = boundary_velocity[t & ~kBoundaryBit];
            d.aux = make_float4(0.0F, 0.0F, 0.0F, 0.0F);
            d.pt = 0.0F;
            return d;
        }
        d.q = pos[t];
        d.v = vel[t];
        d.aux = aux[t];
        d.pt = pt[t];
        return d;
    }
    __device__ __forceinline__ void apply(const uint32_t t, const ForceData& d) {
        const bool is_boundary = WithBoundary && (t & kBoundaryBit);
        if (!is_boundary && t == self) return;
        const f3 disp = sub(x, xyz(d.q));
        const float r2 = sq_xfirst(disp);
        const float distance = __fsqrt_rn(r2);
        if (distance >= k.h) return;
        const bool has_gradient = distance != 0.0F;
        const float s = has_gradient ? cubic_gradient_scale(distance, k) : 0.0F;
        const f3 gradient = scale(disp, s);
        const f3 dv = sub(v, xyz(d.v));
        const float compression = dot_xfirst(dv, disp);
        const float weight = distance > k.diameter ? cubic_inside(distance, k) : k.contact_weight;
        if (is_boundary) {
            const float volume = d.q.w;
            const float rv = __fmul_rn(-rest, volume);
            // pressure: -rho0_i V_b p_i / rho_i^2 grad W (sph/common.cu:183-188)
            if (has_gradient) pressure = fma3(__fmul_rn(rv, first_term), gradient, pressure);
            // artificial viscosity against the boundary (sph/wcsph.cu:162-172)
            if (has_gradient && compression < 0.0F) {
                const float pi = __fdiv_rn(__fmul_rn(-boundary_nu, compression), __fmaf_rn(k.epsilon_factor, k.h, r2));
                artificial = fma3(__fmul_rn(rv, pi), gradient, artificial);
            }
            // boundary adhesion (sph/wcsph.cu:327-335)
            const float factor =
                __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(-boundary_tension, rest), volume), weight), mass);
            surface = fma3(factor, disp, surface);
            return;
        }
        const float mj = d.q.w;
        if (has_gradient) {
            // -m_j (p_i / rho_i^2 + p_j / rho_j^2) grad W (sph/common.cu:180-181)
            pressure = fma3(__fmul_rn(-mj, __fadd_rn(first_term, d.pt)), gradient, pressure);
            if (compression < 0.0F) {
                // Monaghan viscosity (sph/wcsph.cu:149-158)
                const float alpha = __fmul_rn(0.5F, __fadd_rn(viscosity, d.aux.y));
                const float c = __fmul_rn(0.5F, __fadd_rn(speed, d.aux.z));
                const float nu =
                    __fdiv_rn(__fmul_rn(__fmul_rn(__fmul_rn(2.0F, alpha), k.h), c), __fadd_rn(density, d.aux.x));
                // r2 + 0.01 h h with the last product fused into the sum
                const float pi = __fdiv_rn(__fmul_rn(-nu, compression), __fmaf_rn(k.epsilon_factor, k.h, r2));
                artificial = fma3(__fmul_rn(-mj, pi), gradient, artificial);
            }
        }
        // cohesion (sph/wcsph.cu:318-325)
        const float factor = __fdiv_rn(__fmul_rn(__fmul_rn(-surface_tension, mj), weight), mass);
        surface = fma3(factor, disp, surface);
    }
    __device__ __forceinline__ void process(const uint32_t t) { apply(t, prefetch(t)); }
};

// ------------------------------------------------------------------ predicted density
template <bool WithBoundary>
struct PredictedDensityOp {
    static constexpr bool kBoundary = WithBoundary;
    const float4* __restrict__ predicted;
    const float4* __restrict__ boundary;
    f3 x;
    float rest_density;
    SphConstants k;
    float density;

    __device__ __forceinline__ float4 prefetch(const uint32_t t) const {
        if (WithBoundary && (t & kBoundaryBit)) return boundary[t & ~kBoundaryBit];
        return predicted[t];
    }
    __device__ __forceinline__ void apply(const uint32_t t, const float4 q) {
        const bool is_boundary = WithBoundary && (t & kBoundaryBit);
        const float distance = __fsqrt_rn(sq_xfirst(sub(x, xyz(q))));
        if (distance >= k.h) return;
        const float w = cubic_inside(distance, k);
        if (is_boundary) density = __fmaf_rn(__fmul_rn(rest_density, q.w), w, density);
        else density = __fmaf_rn(q.w, w, density);
    }
    __device__ __forceinline__ void process(const uint32_t t) { apply(t, prefetch(t)); }
};

// The predicted density of a particle and the pressure update.
__device__ __forceinline__ void predicted_tail(const SphStep& st, const Own& o, const float predicted_density,
                                               const PressureUpdate& update, float* pressure, float* pressure_term, float* record) {
    const uint32_t s = o.p.s;
    if (record) record[s] = predicted_density;
    const float rho = st.aux[s].x;
    const float rest = o.pa.x;
    const float relaxation = update.relaxation == 0u ? o.pa.w : st.g.params_b[s].x;
    // PCISPH uses the rest volume m / rho0 (sph/pcisph.cu:107), IISPH and DFSPH m / rho (sph/iisph.cu:107)
    const float volume = __fdiv_rn(o.mass, update.method == kPcisph ? rest : rho);
    const float dt = o.p.scene->time_step;
    const float delta = __fdiv_rn(1.0F, __fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(__fmul_rn(2.0F, dt), dt), volume), volume),
                                                  o.k->reference_gradient_norm));
    const float target = update.target == 1u ? rho : rest;
    const float p = fmaxf(0.0F, __fmaf_rn(__fmul_rn(relaxation, delta), __fsub_rn(predicted_density, target), pressure[s]));
    pressure[s] = p;
    pressure_term[s] = __fdiv_rn(p, __fmul_rn(rho, rho));
}

// ------------------------------------------------------------------ pressure acceleration
template <bool WithBoundary>
struct PressureOp {
    static constexpr bool kBoundary = WithBoundary;
    const float4* __restrict__ pos;
    const float* __restrict__ pt;
    const float4* __restrict__ boundary;
    uint32_t self;
    f3 x;
    float rest, first_term;
    SphConstants k;
    f3 acceleration;

    struct Data {
        float4 q;   // (x, m) or boundary (x, V)
        float pt;   // p_j / rho_j^2
    };
    __device__ __forceinline__ Data prefetch(const uint32_t t) const {
        if (WithBoundary && (t & kBoundaryBit)) return {boundary[t & ~kBoundaryBit], 0.0F};
        return {pos[t], pt[t]};
    }
    __device__ __forceinline__ void apply(const uint32_t t, const Data& d) {
        const bool is_boundary = WithBoundary && (t & kBoundaryBit);
        if (!is_boundary && t == self) return;
        const f3 disp = sub(x, xyz(d.q));
        const float distance = __fsqrt_rn(sq_xfirst(disp));
        if (distance == 0.0F || distance >= k.h) return;
        const f3 gradient = scale(disp, cubic_gradient_scale(distance, k));
        // boundary: -rho0_i V_b p_i / rho_i^2 grad W; fluid: -m_j (p_i / rho_i^2 + p_j / rho_j^2) grad W
        // (sph/common.cu:180-188)
        const float factor = is_boundary ? __fmul_rn(__fmul_rn(-rest, d.q.w), first_term)
                                         : __fmul_rn(-d.q.w, __fadd_rn(first_term, d.pt));
        acceleration = fma3(factor, gradient, acceleration);
    }
    __device__ __forceinline__ void process(const uint32_t t) { apply(t, prefetch(t)); }
};

// The pressure acceleration of a particle and the next prediction.
__device__ __forceinline__ void pressure_tail(const SphStep& st, const Own& o, const f3 pressure_acceleration,
                                              const PressurePassArgs& p) {
    const uint32_t s = o.p.s;
    if (p.store_acceleration)
        p.store_acceleration[s] = make_float4(pressure_acceleration.x, pressure_acceleration.y, pressure_acceleration.z, 0.0F);
    // DFSPH's density phase predicts with divergence + density pressure accelerations (sph/sph.cpp:596)
    f3 total = pressure_acceleration;
    if (p.base) total = add(xyz(p.base[s]), pressure_acceleration);
    const float4 np = st.non_pressure[s];
    const SceneDesc& sc = *o.p.scene;
    f3 xo, vo;
    predict(o.x, xyz(st.velocity[s]), add(xyz(np), total), sc.time_step, sc.box, *o.k, xo, vo);
    const uint32_t i = st.sorted_index[s];
    if (p.warm_out) p.warm_out[i] = p.pressure[s];
    if (p.next_pressure) {
        const float pressure = p.next_warm ? p.next_warm[i] : 0.0F;
        const float rho = st.aux[s].x;
        p.next_pressure[s] = pressure;
        p.next_pressure_term[s] = __fdiv_rn(pressure, __fmul_rn(rho, rho));
    }
    if (!p.last) {
        st.predicted[s] = make_float4(xo.x, xo.y, xo.z, o.mass);
        record_displacement(st.displacement + p.displacement_slot, xo, o.x);
        return;
    }
    p.out_positions.x[i] = xo.x;
    p.out_positions.y[i] = xo.y;
    p.out_positions.z[i] = xo.z;
    p.out_velocities.x[i] = vo.x;
    p.out_velocities.y[i] = vo.y;
    p.out_velocities.z[i] = vo.z;
}

}  // namespace detail
}  // namespace sph
}  // namespace pbf
