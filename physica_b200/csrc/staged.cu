// Forward gather passes over windows staged in shared memory (scenes without boundary particles).
//
// A block owns 128 consecutive sorted particles.  Its particles' home cells are a run of the sort
// order, so for each of the nine stencil columns the slots they may touch are one contiguous window:
// about 150 slots each, 1,350 in all, 10.6 per particle.  The block copies the nine windows of every
// field a pass reads into shared memory with 16-byte asynchronous copies, and both the candidate
// tests and the pair terms read them there.  List entries are 16-bit positions in the staged windows,
// so a list is half as long, and its entries are drained two at a time with the packed pair
// arithmetic (pbf_math.cuh).
//
// Reading neighbours through L1 instead (lists of sorted slots or of hit masks, one pair at a time), a
// pass waited on scattered loads and issued 70 instructions per pair, half of them for the IEEE root and
// divisions.  At 1M particles, ms per launch before and now: scan + density/lambda 0.293 -> 0.262,
// correction 0.155 -> 0.107, normal 0.151 -> 0.096, XSPH 0.157 -> 0.120; the post-loop scan and the vorticity,
// 0.143 + 0.158 before and 0.305 in one kernel now, save a launch and no time.  What bounds them now: the scan issues 70 % of its cycles, and the replays keep
// the shared-memory pipe 70-78 % busy.
//
// Blocks of 64 or 32 particles stage 12.4 and 15.9 slots per particle and were slower (0.264 and 0.298 ms
// against 0.252 for the scan + density kernel as it was then, 0.150 and 0.176 for the correction).
//
// The first kernel of a list (scan) finds the windows and records them per block; passes that replay
// the list read the record.  Where that does not fit, the particle keeps a list of hit masks over sorted
// slots in its own words and replays it from global memory, in the same kernels: all particles of a block
// whose windows exceed the stage (sparse spray whose neighbour columns are dense, 1-2 % of a dam break's
// blocks), and a particle with a column of more candidates than its hit record covers (clumps).  In the
// late, splashing state of a 1M-particle dam break plain walks of the stencil in their place cost 5.6 ms
// a step instead of 4.7.
//
// Every sum keeps the reference's order and rounding (gather.cuh): the lists hold the same neighbours
// in the same order, without the particle itself, whose only term is its own density.
#include "dependent_launch.cuh"
#include "staged_ops.cuh"

namespace pbf {

namespace {

using namespace staged_detail;

// ------------------------------------------------------------------- density + lambda
// Slots: also store the list of sorted slots that the reverse and tangent passes read.
template <bool Slots>
__global__ void __launch_bounds__(kBlockParticles, 6) staged_density_kernel(const StagedDensityArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float field[4][kStage];
    __shared__ ColumnHits columns[9][kBlockParticles];
    const Particle p = locate(a.g);
    const uint32_t s = p.active ? p.s : 0u;
    const f3 xi = mk(a.positions.x[s], a.positions.y[s], a.positions.z[s]);
    const float mass = a.mass[s];
    const float4 pa = a.g.params_a[s];
    const float* const fields[4] = {a.positions.x, a.positions.y, a.positions.z, a.mass};
    Hits hits;
    const bool staged = windows_and_hits<Slots>(w, a.list, p, a.g, field, fields, xi, columns, hits);
    if (!p.active) return;
    const StoredList& list = a.list.list;
    float density = 0.0F, denominator = pa.y;   // relaxation
    f3 gradient_sum = mk(0.0F, 0.0F, 0.0F);
    uint32_t neighbors = 0u;
    if (staged && fits<Slots>(hits, list)) {
        const uint32_t n = hits.count;
        neighbors = n;
        const float own = any_poly6(0.0F, p.k.h2, p.k.poly6_denominator);   // W(0)
        const float ratio = __fdiv_rn(mass, pa.x);
        replay_hits<true, Slots>(w, list, a.slots, s, hits, columns,
                                 [&](const uint32_t i0, const uint32_t i1, const bool second, const uint32_t k) {
            float m0 = field[3][i0], m1 = field[3][i1];
            const TwoPairs t = two_pairs(xi, mk(field[0][i0], field[1][i0], field[2][i0]),
                                         mk(field[0][i1], field[1][i1], field[2][i1]));
            float2 weight = poly6_pair(t.nr2, p.k), spiky = spiky_scale_pair(t.nr2, p.k);
            float c0 = ratio, c1 = ratio;   // m_j / rho0_i
            if (!in_range(t.nr2, p.k) || m0 != mass || m1 != mass) {
                c0 = __fdiv_rn(m0, pa.x);
                c1 = __fdiv_rn(m1, pa.x);
                if (!in_range(t.nr2, p.k)) {
                    weight = any_poly6s(t.nr2, p.k);
                    spiky = any_spiky_scales(t.nr2, p.k);
                    // no kernel: no term, whatever the factors are
                    if (spiky.x == 0.0F) c0 = 0.0F;
                    if (spiky.y == 0.0F) c1 = 0.0F;
                    if (-t.nr2.x >= p.k.h2) m0 = 0.0F;
                    if (-t.nr2.y >= p.k.h2) m1 = 0.0F;
                    neighbors -= -t.nr2.x >= p.k.h2 ? 1u : 0u;
                    neighbors -= second && -t.nr2.y >= p.k.h2 ? 1u : 0u;
                }
            }
            const f3 g0 = scale(t.d0, spiky.x), g1 = scale(t.d1, spiky.y);
            if (k == hits.before) density = __fmaf_rn(mass, own, density);
            density = __fmaf_rn(m0, weight.x, density);
            gradient_sum = fma3(c0, g0, gradient_sum);
            denominator = __fmaf_rn(__fmul_rn(c0, c0), sq_xfirst(g0), denominator);
            if (second) {
                if (k + 1u == hits.before) density = __fmaf_rn(mass, own, density);
                density = __fmaf_rn(m1, weight.y, density);
                gradient_sum = fma3(c1, g1, gradient_sum);
                denominator = __fmaf_rn(__fmul_rn(c1, c1), sq_xfirst(g1), denominator);
            }
        });
        if (hits.before == n) density = __fmaf_rn(mass, own, density);
    } else {
        DensityLambdaOp<false> op;
        op.pos = a.pos;
        op.boundary = nullptr;
        op.self = s;
        op.k = p.k;
        op.x = xi;
        op.rest_density = pa.x;
        op.density = 0.0F;
        op.gradient_sum = mk(0.0F, 0.0F, 0.0F);
        op.denominator = pa.y;
        op.neighbors = 0;
        op.ratio.reset(mass, pa.x);
        fallback_lists<Slots>(p, a.g, a.positions, xi, list, a.slots);
        replay_alone(op, p, a.g, list);
        density = op.density;
        gradient_sum = op.gradient_sum;
        denominator = op.denominator;
        neighbors = op.neighbors;
    }
    const float total = __fadd_rn(denominator, sq_yfirst(gradient_sum));
    a.lambda[s] = __fdiv_rn(-__fsub_rn(__fdiv_rn(density, pa.x), 1.0F), total);
    if (a.density) a.density[s] = density;
    if (a.gsum_denom) a.gsum_denom[s] = make_float4(gradient_sum.x, gradient_sum.y, gradient_sum.z, total);
    if (a.neighbor_count) a.neighbor_count[s] = neighbors;
}

// ----------------------------------------------------------------- correction + project
__global__ void __launch_bounds__(kBlockParticles, 7) staged_correction_kernel(const StagedCorrectionArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float field[5][kStage];
    const Particle p = locate(a.g);
    load_windows(w, a.list.windows + static_cast<size_t>(first_particle(a.g) / kBlockParticles) * kWindowWords);
    const float* const fields[5] = {a.positions.x, a.positions.y, a.positions.z, a.mass, a.lambda};
    if (w.staged) stage(w, field, fields);
    if (!p.active) return;
    const uint32_t s = p.s;
    const StoredList& list = a.list.list;
    const f3 xi = mk(a.positions.x[s], a.positions.y[s], a.positions.z[s]);
    const float mass = a.mass[s], lambda = a.lambda[s];
    const float4 pa = a.g.params_a[s];
    const float4 pb = a.g.params_b[s];
    const bool full = pb.x != 0.0F;   // s_corr has a strength
    const uint32_t n = list.counts[s];
    f3 correction = mk(0.0F, 0.0F, 0.0F);
    if (w.staged && is_staged(n)) {
        const float ratio = __fdiv_rn(mass, pa.x);
        const float reference = full ? poly6(mk(pb.z, 0.0F, 0.0F), p.k) : 1.0F;
        replay_words(list, s, entries_of(n), [&](const uint32_t i0, const uint32_t i1, const bool second) {
            const PairFactors f = correction_factors(p.k, xi, mass, pa.x, ratio, lambda, full, pb, reference, field, i0, i1);
            correction = fma3(f.first, scale(f.t.d0, f.spiky.x), correction);
            if (second) correction = fma3(f.second, scale(f.t.d1, f.spiky.y), correction);
        });
    } else {
        correction = correction_alone(a, p, xi, mass, lambda);
    }
    correction_tail(a, p, xi, mass, correction);
}

// ----------------------------------------------------------- post-loop scan + vorticity
template <bool Slots>
__global__ void __launch_bounds__(kBlockParticles, 4) staged_vorticity_kernel(const StagedVorticityArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float field[6][kStage];
    __shared__ ColumnHits columns[9][kBlockParticles];
    const Particle p = locate(a.g);
    const uint32_t s = p.active ? p.s : 0u;
    const f3 xi = mk(a.positions.x[s], a.positions.y[s], a.positions.z[s]);
    const f3 vi = mk(a.velocities.x[s], a.velocities.y[s], a.velocities.z[s]);
    const float* const fields[6] = {a.positions.x, a.positions.y, a.positions.z, a.velocities.x, a.velocities.y, a.velocities.z};
    Hits hits;
    const bool staged = windows_and_hits<Slots>(w, a.list, p, a.g, field, fields, xi, columns, hits);
    if (!p.active) return;
    const StoredList& list = a.list.list;
    f3 vorticity = mk(0.0F, 0.0F, 0.0F);
    if (staged && fits<Slots>(hits, list)) {
        replay_hits<true, Slots>(w, list, a.slots, s, hits, columns,
                                 [&](const uint32_t i0, const uint32_t i1, const bool second, uint32_t) {
            const TwoPairs t = two_pairs(xi, mk(field[0][i0], field[1][i0], field[2][i0]),
                                         mk(field[0][i1], field[1][i1], field[2][i1]));
            f3 v0 = sub(mk(field[3][i0], field[4][i0], field[5][i0]), vi);
            f3 v1 = sub(mk(field[3][i1], field[4][i1], field[5][i1]), vi);
            float2 spiky = spiky_scale_pair(t.nr2, p.k);
            if (!in_range(t.nr2, p.k)) {
                spiky = any_spiky_scales(t.nr2, p.k);
                only_inside(spiky, v0, v1);
            }
            vorticity = add(vorticity, cross_f(v0, scale(t.d0, spiky.x)));
            if (second) vorticity = add(vorticity, cross_f(v1, scale(t.d1, spiky.y)));
        });
    } else {
        VorticityOp op;
        op.pos = a.pos;
        op.velocity = a.velocity;
        op.self = s;
        op.k = p.k;
        op.x = xi;
        op.v = vi;
        op.vorticity = vorticity;
        fallback_lists<Slots>(p, a.g, a.positions, xi, list, a.slots);
        replay_alone(op, p, a.g, list);
        vorticity = op.vorticity;
    }
    const float magnitude = __fsqrt_rn(sq_xfirst(vorticity));
    a.vorticity[s] = make_float4(vorticity.x, vorticity.y, vorticity.z, magnitude);
    a.magnitude[s] = magnitude;
}

// ------------------------------------------------------------------ normal + confinement
__global__ void __launch_bounds__(kBlockParticles, 8) staged_normal_kernel(const StagedNormalArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float field[4][kStage];
    const Particle p = locate(a.g);
    load_windows(w, a.list.windows + static_cast<size_t>(first_particle(a.g) / kBlockParticles) * kWindowWords);
    const float* const fields[4] = {a.positions.x, a.positions.y, a.positions.z, a.magnitude};
    if (w.staged) stage(w, field, fields);
    if (!p.active) return;
    const uint32_t s = p.s;
    const StoredList& list = a.list.list;
    const f3 xi = mk(a.positions.x[s], a.positions.y[s], a.positions.z[s]);
    const float4 wi = a.vorticity[s];
    const uint32_t n = list.counts[s];
    f3 gradient = mk(0.0F, 0.0F, 0.0F);
    if (w.staged && is_staged(n)) {
        replay_words(list, s, entries_of(n), [&](const uint32_t i0, const uint32_t i1, const bool second) {
            const TwoPairs t = two_pairs(xi, mk(field[0][i0], field[1][i0], field[2][i0]),
                                         mk(field[0][i1], field[1][i1], field[2][i1]));
            float f0 = __fsub_rn(field[3][i0], wi.w), f1 = __fsub_rn(field[3][i1], wi.w);
            float2 spiky = spiky_scale_pair(t.nr2, p.k);
            if (!in_range(t.nr2, p.k)) {
                spiky = any_spiky_scales(t.nr2, p.k);
                only_inside(spiky, f0, f1);
            }
            gradient = fma3(f0, scale(t.d0, spiky.x), gradient);
            if (second) gradient = fma3(f1, scale(t.d1, spiky.y), gradient);
        });
    } else {
        gradient = normal_alone(a, p, xi, wi.w);
    }
    normal_tail(a, p, wi, gradient);
}

// -------------------------------------------------------------------------------- XSPH
__global__ void __launch_bounds__(kBlockParticles, 5) staged_xsph_kernel(const StagedXsphArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float field[6][kStage];
    const Particle p = locate(a.g);
    load_windows(w, a.list.windows + static_cast<size_t>(first_particle(a.g) / kBlockParticles) * kWindowWords);
    const float* const fields[6] = {a.positions.x, a.positions.y, a.positions.z, a.confined_soa.x, a.confined_soa.y,
                                    a.confined_soa.z};
    if (w.staged) stage(w, field, fields);
    if (!p.active) return;
    const uint32_t s = p.s;
    const StoredList& list = a.list.list;
    const f3 xi = mk(a.positions.x[s], a.positions.y[s], a.positions.z[s]);
    const f3 vi = mk(a.confined_soa.x[s], a.confined_soa.y[s], a.confined_soa.z[s]);
    const uint32_t n = list.counts[s];
    f3 smoothing = mk(0.0F, 0.0F, 0.0F);
    if (w.staged && is_staged(n)) {
        replay_words(list, s, entries_of(n), [&](const uint32_t i0, const uint32_t i1, const bool second) {
            const TwoPairs t = two_pairs(xi, mk(field[0][i0], field[1][i0], field[2][i0]),
                                         mk(field[0][i1], field[1][i1], field[2][i1]));
            f3 v0 = sub(mk(field[3][i0], field[4][i0], field[5][i0]), vi);
            f3 v1 = sub(mk(field[3][i1], field[4][i1], field[5][i1]), vi);
            float2 weight = poly6_pair(t.nr2, p.k);
            if (!in_range(t.nr2, p.k)) {
                weight = any_poly6s(t.nr2, p.k);
                only_inside(weight, v0, v1);
            }
            smoothing = fma3(weight.x, v0, smoothing);
            if (second) smoothing = fma3(weight.y, v1, smoothing);
        });
    } else {
        smoothing = xsph_alone(a, p, xi, vi);
    }
    xsph_tail(a, p, vi, smoothing);
}

inline unsigned blocks_of(const uint32_t n) { return (n + kBlockParticles - 1u) / kBlockParticles; }

template <class Args>
cudaError_t launch(void (*kernel)(Args), cudaStream_t stream, const Args& a) {
    if (a.g.count == 0) return cudaSuccess;
    launch_after(stream, kernel, blocks_of(a.g.count), kBlockParticles, a);
    count_launch();
    return cudaGetLastError();
}

}  // namespace

size_t window_words(const uint32_t count) { return (static_cast<size_t>(count) + 31u) / 32u * kWindowWords; }

cudaError_t launch_staged_density(cudaStream_t stream, const StagedDensityArgs& a) {
    return launch(a.slots.entries ? staged_density_kernel<true> : staged_density_kernel<false>, stream, a);
}
cudaError_t launch_staged_correction(cudaStream_t stream, const StagedCorrectionArgs& a) {
    return launch(staged_correction_kernel, stream, a);
}
cudaError_t launch_staged_vorticity(cudaStream_t stream, const StagedVorticityArgs& a) {
    return launch(a.slots.entries ? staged_vorticity_kernel<true> : staged_vorticity_kernel<false>, stream, a);
}
cudaError_t launch_staged_normal(cudaStream_t stream, const StagedNormalArgs& a) { return launch(staged_normal_kernel, stream, a); }
cudaError_t launch_staged_xsph(cudaStream_t stream, const StagedXsphArgs& a) { return launch(staged_xsph_kernel, stream, a); }

}  // namespace pbf
