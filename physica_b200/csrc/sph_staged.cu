// SPH forward passes over windows staged in shared memory (staged.cuh; scenes without boundary particles).
//
// One scan per substep, fused with the density, writes the list of sorted slots that the non-pressure,
// force, reverse and tangent passes replay and, for the iterative methods, the staged list that every
// predicted-density and pressure pass replays.  Those are most of a PCISPH, IISPH or DFSPH substep.
// Through L1 they waited on scattered loads and spent most of their instructions on IEEE roots and
// divisions, one pair at a time; from shared memory they take two pairs at a time with the packed
// arithmetic of sph_math.cuh.  Lists carry a skin (sph.cu); pairs in it are left out of the sums.  Every sum keeps the reference's order and rounding.
//
// A DFSPH substep at 270k particles (ten pressure iterations) went from 1.378 to 1.104 ms, a WCSPH substep at
// 1M, which uses the scan alone, from 0.665 to 0.634.  The force and non-pressure passes stay per lane: they
// run once a substep.  What bounds the replays is the shared-memory pipe, as in the PBF passes.
#include "dependent_launch.cuh"
#include "sph_ops.cuh"
#include "staged.cuh"

namespace pbf {
namespace sph {

namespace {

using namespace staged_detail;
using namespace detail;

__device__ __forceinline__ float2 negated_squares(const f3 d0, const f3 d1) {
    return make_float2(negated_squared(d0), negated_squared(d1));
}

// ------------------------------------------------------------------- scan + density
struct DensityPassArgs {
    GatherCommon g;
    SphStep st;
    SphStaged staged;
    uint32_t method;
    float* density_record;
    float* pressure;
    float* pressure_term;
    const float* warm;
};

template <bool Words>
__global__ void __launch_bounds__(kBlockParticles, 6) staged_sph_density_kernel(const DensityPassArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float field[4][kStage];
    __shared__ ColumnHits columns[9][kBlockParticles];
    const SphStep& st = a.st;
    const Own o = own(st);
    const uint32_t s = o.p.active ? o.p.s : 0u;
    const PackedPositions x = a.staged.positions;
    const f3 xi = mk(x.x[s], x.y[s], x.z[s]);
    const float* const fields[4] = {x.x, x.y, x.z, a.staged.mass};
    Hits hits;
    const bool staged = windows_and_hits<true>(w, a.staged.list, o.p, st.g, field, fields, xi, columns, hits);
    if (!o.p.active) return;
    const SphConstants& k = *o.k;
    float density = 0.0F;
    if (staged && fits<true>(hits, st.list)) {
        const float own_weight = cubic_inside(0.0F, k);
        replay_hits<Words, true>(w, a.staged.list.list, st.list, s, hits, columns,
                                 [&](const uint32_t i0, const uint32_t i1, const bool second, const uint32_t at) {
            const f3 d0 = sub(xi, mk(field[0][i0], field[1][i0], field[2][i0]));
            const f3 d1 = sub(xi, mk(field[0][i1], field[1][i1], field[2][i1]));
            const float2 nr2 = negated_squares(d0, d1);
            float2 weight = cubic_pair(nr2, k);
            if (!in_range(nr2, k)) weight = make_float2(any_cubic(-nr2.x, &k), any_cubic(-nr2.y, &k));
            // a zero mass beyond the support: 0.580 ms a WCSPH step of 1M, 0.582 where the term is left out
            const float m0 = inside(nr2.x, k) ? field[3][i0] : 0.0F, m1 = inside(nr2.y, k) ? field[3][i1] : 0.0F;
            if (at == hits.before) density = __fmaf_rn(o.mass, own_weight, density);
            density = __fmaf_rn(m0, weight.x, density);
            if (second) {
                if (at + 1u == hits.before) density = __fmaf_rn(o.mass, own_weight, density);
                density = __fmaf_rn(m1, weight.y, density);
            }
        });
        if (hits.before == hits.count) density = __fmaf_rn(o.mass, own_weight, density);
    } else {
        if constexpr (Words) a.staged.list.list.counts[s] = kOverflow;
        st.list.counts[s] = scan_global(o.p, st.g, x, xi, st.list);
        DensityOp<false> op;
        op.pos = st.topology;
        op.boundary = nullptr;
        op.x = xi;
        op.rest_density = o.pa.x;
        op.k = k;
        op.density = 0.0F;
        replay_written(op, o.p, st.g, st.list);
        density = op.density;
    }
    density_tail(st, o, density, a.method, a.density_record, a.pressure, a.pressure_term, a.warm);
}

// --------------------------------------------------------------- predicted density
struct PredictedPassArgs {
    GatherCommon g;
    SphStep st;
    StagedList list;
    PressureUpdate update;
    float* pressure;
    float* pressure_term;
    float* record;
};

__global__ void __launch_bounds__(kBlockParticles, 8) staged_predicted_density_kernel(const PredictedPassArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float4 positions[kStage];
    const SphStep& st = a.st;
    const Own o = own(st);
    load_windows(w, a.list.windows + static_cast<size_t>(first_particle(st.g) / kBlockParticles) * kWindowWords);
    // the pairs within h at the predicted positions are all listed while the skin covers the largest
    // displacement (the constants of an inactive thread's scene are not read: one scene per solver)
    const float displacement = __uint_as_float(st.displacement[a.update.displacement_slot]);
    const bool listed = __fmul_rn(2.0F, displacement) <= st.constants->skin_bound;
    if (w.staged && listed) {
        stage4(w, positions, st.predicted, st.g.count);
        copies_done();
    }
    if (!o.p.active) return;
    const uint32_t s = o.p.s;
    const SphConstants& k = *o.k;
    const f3 xi = xyz(st.predicted[s]);
    const uint32_t count = a.list.list.counts[s];
    float density = 0.0F;
    if (w.staged && listed && count != kOverflow) {
        const uint32_t n = entries_of(count), before = before_of(count);
        const float own_weight = cubic_inside(0.0F, k);
        uint32_t at = 0u;
        replay_words(a.list.list, s, n, [&](const uint32_t i0, const uint32_t i1, const bool second) {
            const float4 q0 = positions[i0], q1 = positions[i1];
            const float2 nr2 = negated_squares(sub(xi, xyz(q0)), sub(xi, xyz(q1)));
            float2 weight = cubic_pair(nr2, k);
            if (!in_range(nr2, k)) weight = make_float2(any_cubic(-nr2.x, &k), any_cubic(-nr2.y, &k));
            if (at == before) density = __fmaf_rn(o.mass, own_weight, density);
            if (inside(nr2.x, k)) density = __fmaf_rn(q0.w, weight.x, density);
            if (second) {
                if (at + 1u == before) density = __fmaf_rn(o.mass, own_weight, density);
                if (inside(nr2.y, k)) density = __fmaf_rn(q1.w, weight.y, density);
            }
            at += 2u;
        });
        if (before == n) density = __fmaf_rn(o.mass, own_weight, density);
    } else {
        PredictedDensityOp<false> op;
        op.predicted = st.predicted;
        op.boundary = nullptr;
        op.x = xi;
        op.rest_density = o.pa.x;
        op.k = k;
        op.density = 0.0F;
        if (listed) replay(op, o.p, st.g, st.list);
        else walk(op, o.p, st.g);
        density = op.density;
    }
    predicted_tail(st, o, density, a.update, a.pressure, a.pressure_term, a.record);
}

// ------------------------------------------------------- pressure acceleration + predict
struct PressurePass {
    GatherCommon g;
    SphStep st;
    StagedList list;
    PressurePassArgs p;
};

__global__ void __launch_bounds__(kBlockParticles, 7) staged_pressure_kernel(const PressurePass a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float4 positions[kStage];
    __shared__ __align__(16) float term[1][kStage];
    const SphStep& st = a.st;
    const Own o = own(st);
    load_windows(w, a.list.windows + static_cast<size_t>(first_particle(st.g) / kBlockParticles) * kWindowWords);
    if (w.staged) {
        stage4(w, positions, st.topology, st.g.count);
        const float* const fields[1] = {a.p.pressure_term};
        stage(w, term, fields);
    }
    if (!o.p.active) return;
    const uint32_t s = o.p.s;
    const SphConstants& k = *o.k;
    const float first = a.p.pressure_term[s];
    const uint32_t count = a.list.list.counts[s];
    f3 acceleration = mk(0.0F, 0.0F, 0.0F);
    if (w.staged && count != kOverflow) {
        replay_words(a.list.list, s, entries_of(count), [&](const uint32_t i0, const uint32_t i1, const bool second) {
            const float4 q0 = positions[i0], q1 = positions[i1];
            const f3 d0 = sub(o.x, xyz(q0)), d1 = sub(o.x, xyz(q1));
            const float2 nr2 = negated_squares(d0, d1);
            float f0 = __fmul_rn(-q0.w, __fadd_rn(first, term[0][i0]));
            float f1 = __fmul_rn(-q1.w, __fadd_rn(first, term[0][i1]));
            float2 slope = cubic_gradient_pair(nr2, k);
            if (!in_range(nr2, k)) {
                slope = make_float2(any_cubic_gradient(-nr2.x, &k), any_cubic_gradient(-nr2.y, &k));
                if (nr2.x == 0.0F) f0 = 0.0F;   // coincident particles: no gradient, whatever the pressures
                if (nr2.y == 0.0F) f1 = 0.0F;
            }
            if (inside(nr2.x, k)) acceleration = fma3(f0, scale(d0, slope.x), acceleration);
            if (second && inside(nr2.y, k)) acceleration = fma3(f1, scale(d1, slope.y), acceleration);
        });
    } else {
        PressureOp<false> op;
        op.pos = st.topology;
        op.pt = a.p.pressure_term;
        op.boundary = nullptr;
        op.self = s;
        op.x = o.x;
        op.rest = o.pa.x;
        op.first_term = first;
        op.k = k;
        op.acceleration = acceleration;
        replay(op, o.p, st.g, st.list);
        acceleration = op.acceleration;
    }
    pressure_tail(st, o, acceleration, a.p);
}

template <class Args>
cudaError_t launch(void (*kernel)(Args), cudaStream_t stream, const Args& a) {
    if (a.g.count == 0) return cudaSuccess;
    launch_after(stream, kernel, (a.g.count + kBlockParticles - 1u) / kBlockParticles, kBlockParticles, a);
    count_launch();
    return cudaGetLastError();
}

}  // namespace

cudaError_t staged_sph_wave(uint32_t& particles) { return one_wave(staged_sph_density_kernel<false>, kBlockParticles, particles); }

cudaError_t launch_staged_sph_density(cudaStream_t stream, const SphStep& st, const SphStaged& staged, const uint32_t method,
                                      float* density_record, float* pressure, float* pressure_term, const float* warm) {
    const DensityPassArgs a{st.g, st, staged, method, density_record, pressure, pressure_term, warm};
    return launch(method == kWcsph ? staged_sph_density_kernel<false> : staged_sph_density_kernel<true>, stream, a);
}

cudaError_t launch_staged_predicted_density(cudaStream_t stream, const SphStep& st, const StagedList& list,
                                            const PressureUpdate update, float* pressure, float* pressure_term,
                                            float* predicted_density_record) {
    return launch(staged_predicted_density_kernel, stream,
                  PredictedPassArgs{st.g, st, list, update, pressure, pressure_term, predicted_density_record});
}

cudaError_t launch_staged_pressure(cudaStream_t stream, const SphStep& st, const StagedList& list, const PressurePassArgs& a) {
    return launch(staged_pressure_kernel, stream, PressurePass{st.g, st, list, a});
}

}  // namespace sph
}  // namespace pbf
