// The staged forward passes (staged.cu) with four lanes per particle, for scenes that do not fill the GPU
// with one: a block of 128 threads owns 32 particles.
//
// Such scenes wait on the serial chain of a particle's 30 to 40 pairs.  Here each lane scans its share of
// the nine stencil columns and evaluates two of every eight entries of the list; the pairs' terms go through
// shared memory to the lanes that own the sums (lane c % 4 owns component c), which add them one by one in
// list order.  The sums are the same sums in the same order, so the results are those of the other passes
// bit for bit.  A forward step of 5k particles, four iterations, in a graph: 0.240 ms with one lane, 0.164
// with four; of those the two passes of an iteration take 23 us in place of 39.
#include "dependent_launch.cuh"
#include "staged_ops.cuh"

namespace pbf {

namespace {

using namespace staged_detail;

constexpr uint32_t kThreads = kBlockParticles;
constexpr int L = 4;   // lanes per particle
constexpr uint32_t kParticles = kThreads / L;
static_assert(kParticles == kGroupParticles, "a block's windows");
// A longer list walks the stencil.
constexpr uint32_t kGroupList = 96;

// One particle's terms of 2 L consecutive entries: (factor, value) of each of C components.
template <int C>
struct Exchange {
    float2 term[C][2u * L];
};

struct Member {
    Particle p;
    uint32_t lane, local;   // lane of the group, particle of the block
};

__device__ __forceinline__ Member member(const GatherCommon& g) {
    Member m;
    m.lane = threadIdx.x % L;
    m.local = threadIdx.x / L;
    m.p.s = blockIdx.x * kParticles + m.local;
    m.p.active = m.p.s < g.count;
    m.p.c = m.p.active ? g.cell[m.p.s] : make_int4(0, 0, 0, 0);
    m.p.scene = g.scenes + m.p.c.w;
    m.p.k = g.constants[m.p.scene->constants];
    return m;
}

__device__ __forceinline__ uint32_t* record_of(const StagedList& list) {
    return list.windows + static_cast<size_t>(blockIdx.x) * kWindowWords;
}

// A scan's hits, and in their place, once they are lists, the exchange.
template <int C>
union ScanOrExchange {
    ColumnHits columns[9][kThreads];
    Exchange<C> exchange[kParticles];
};

// Adds the terms of n entries in order.  words(j): entries 2 j and 2 j + 1; step(i0, i1, a, b): the terms
// of two entries; add(c, k, term, sum): the sum of component c with entry k's term.  sums[j] is the sum of
// component lane + L j.  Every lane of the warp calls it (n = 0: no entries).
template <int C, class Words, class Step, class Add>
__device__ __forceinline__ void group_replay(Exchange<C>& x, const uint32_t lane, const uint32_t n,
                                             float (&sums)[(C + L - 1) / L], Words words,
                                             Step step, Add add) {
    const uint32_t longest = __reduce_max_sync(kFull, n);
#pragma unroll 1
    for (uint32_t k0 = 0; k0 < longest; k0 += 2u * L) {
        const uint32_t k = k0 + 2u * lane;
        if (k < n) {
            const uint32_t word = words(k / 2u);
            float2 a[C], b[C];
            step(word & 0xffffu, word >> 16, a, b);
#pragma unroll
            for (int c = 0; c < C; ++c)
                *reinterpret_cast<float4*>(&x.term[c][2u * lane]) = make_float4(a[c].x, a[c].y, b[c].x, b[c].y);
        }
        __syncwarp();
#pragma unroll
        for (int j = 0; j < (C + L - 1) / L; ++j) {
            const uint32_t c = lane + L * static_cast<uint32_t>(j);
            if (c < static_cast<uint32_t>(C)) {
#pragma unroll
                for (uint32_t e = 0; e < 2u * L; ++e)
                    if (k0 + e < n) sums[j] = add(c, k0 + e, x.term[c][e], sums[j]);
            }
        }
        __syncwarp();
    }
}

// Component c of the sums, in every lane of the group.
template <int N>
__device__ __forceinline__ float component(const float (&sums)[N], const uint32_t c) {
    return __shfl_sync(kFull, sums[c / L], static_cast<int>(c % L), static_cast<int>(L));
}
__device__ __forceinline__ uint32_t group_mask() {
    return ((1u << L) - 1u) << (threadIdx.x & 31u & ~(L - 1u));
}
struct FusedAdd {
    __device__ __forceinline__ float operator()(uint32_t, uint32_t, const float2 t, const float sum) const {
        return __fmaf_rn(t.x, t.y, sum);
    }
};

// The scan of a particle by its group: the entries of its staged list in `entries` (a last odd entry
// repeated) and, as list words, in global memory; returns their number, or kOverflow (no list written).  Every thread of the
// block calls it; `before` as Hits::before.
__device__ __forceinline__ uint32_t group_scan(Windows& w, const StagedList& list, const Member& m, const GatherCommon& g,
                                               float (*shared)[kGroupStage], const f3 xi, ColumnHits (*columns)[kThreads],
                                               uint16_t (*entries)[kGroupList], uint32_t& before) {
    Hits hits{0u, 0u, ~0u, true, true};
    // Columns 0..2, 3..4, 5..6, 7..8.
    const int from = m.lane == 0u ? 0 : 2 * static_cast<int>(m.lane) + 1;
    const int to = 2 * static_cast<int>(m.lane) + 3;
    if (w.staged) {
        if (m.p.active) hits = scan<false>(w, m.p, g, shared[0], shared[1], shared[2], xi, columns, from, to);
        if (__syncthreads_or(!hits.inside) && threadIdx.x == 0u) w.staged = 0u;
        __syncthreads();
    }
    store_windows(w, record_of(list));
    if (!w.staged) return kOverflow;
    uint32_t end = hits.count;
#pragma unroll
    for (int o = 1; o < L; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, end, o, L);
        if (static_cast<int>(m.lane) >= o) end += v;
    }
    const uint32_t first = end - hits.count;
    const uint32_t n = __shfl_sync(kFull, end, L - 1u, L);
    before = __reduce_min_sync(group_mask(), hits.before == ~0u ? ~0u : first + hits.before);   // one lane found it
    const bool fits = __reduce_min_sync(group_mask(), hits.covered ? 1u : 0u) != 0u && n < kGroupList;
    if (fits && hits.count > 0u) {
        HitCursor cursor(w, columns);
        for (uint32_t j = first; j < end; ++j) entries[m.local][j] = static_cast<uint16_t>(cursor.take());
        if (end == n && n % 2u == 1u) entries[m.local][n] = entries[m.local][n - 1u];
    }
    __syncthreads();   // the hits' memory becomes the exchange
    if (!fits) return kOverflow;
    if (m.p.active) {
        const uint32_t* __restrict__ words = reinterpret_cast<const uint32_t*>(entries[m.local]);
        for (uint32_t j = m.lane; 2u * j < n; j += L) *word_of(list.list, m.p.s, j) = words[j];
        if (m.lane == 0u) list.list.counts[m.p.s] = n | (before << 16);
    }
    return n;
}

// The list words of a stored list, for group_replay.
struct StoredWords {
    const uint32_t* __restrict__ row;
    __device__ __forceinline__ uint32_t operator()(const uint32_t j) const { return row[static_cast<size_t>(j / 4u) * 128u + j % 4u]; }
};
__device__ __forceinline__ StoredWords stored_words(const StoredList& list, const uint32_t s) {
    return {reinterpret_cast<const uint32_t*>(quad_row(list, s))};
}

// ------------------------------------------------------------------- density + lambda
__global__ void __launch_bounds__(kThreads) group_density_kernel(const StagedDensityArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float field[4][kGroupStage];
    __shared__ __align__(16) uint16_t entries[kParticles][kGroupList];
    __shared__ __align__(16) ScanOrExchange<5> scratch;
    const Member m = member(a.g);
    const Particle& p = m.p;
    const uint32_t s = p.active ? p.s : 0u;
    const uint32_t block_first = blockIdx.x * kParticles;
    const f3 xi = mk(a.positions.x[s], a.positions.y[s], a.positions.z[s]);
    const float mass = a.mass[s];
    const float4 pa = a.g.params_a[s];
    const float* const fields[4] = {a.positions.x, a.positions.y, a.positions.z, a.mass};
    find_windows(w, a.g, block_first, min(block_first + kParticles, a.g.count) - 1u, kGroupStage);
    __syncthreads();
    if (w.staged) stage(w, field, fields);
    uint32_t before = ~0u;
    const uint32_t listed = group_scan(w, a.list, m, a.g, field, xi, scratch.columns, entries, before);
    const uint32_t n = p.active && listed != kOverflow ? listed : 0u;
    const float own = any_poly6(0.0F, p.k.h2, p.k.poly6_denominator);   // W(0)
    const float ratio = __fdiv_rn(mass, pa.x);
    uint32_t misses = 0u;
    // components: density, gradient sum (3), denominator
    float sums[2] = {};
    if (m.lane == 0u) sums[1] = pa.y;   // relaxation
    group_replay<5>(scratch.exchange[m.local], m.lane, n, sums,
        [&](const uint32_t j) { return reinterpret_cast<const uint32_t*>(entries[m.local])[j]; },
        [&](const uint32_t i0, const uint32_t i1, float2 (&t0)[5], float2 (&t1)[5]) {
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
                    misses += -t.nr2.x >= p.k.h2 ? 1u : 0u;
                    misses += i1 != i0 && -t.nr2.y >= p.k.h2 ? 1u : 0u;   // i1 = i0: a last odd entry repeated
                }
            }
            const f3 g0 = scale(t.d0, spiky.x), g1 = scale(t.d1, spiky.y);
            t0[0] = make_float2(m0, weight.x);
            t0[1] = make_float2(c0, g0.x);
            t0[2] = make_float2(c0, g0.y);
            t0[3] = make_float2(c0, g0.z);
            t0[4] = make_float2(__fmul_rn(c0, c0), sq_xfirst(g0));
            t1[0] = make_float2(m1, weight.y);
            t1[1] = make_float2(c1, g1.x);
            t1[2] = make_float2(c1, g1.y);
            t1[3] = make_float2(c1, g1.z);
            t1[4] = make_float2(__fmul_rn(c1, c1), sq_xfirst(g1));
        },
        [&](const uint32_t c, const uint32_t k, const float2 t, float sum) {
            if (c == 0u && k == before) sum = __fmaf_rn(mass, own, sum);
            return __fmaf_rn(t.x, t.y, sum);
        });
    if (m.lane == 0u && before == n) sums[0] = __fmaf_rn(mass, own, sums[0]);
    f3 gradient_sum = mk(component(sums, 1u), component(sums, 2u), component(sums, 3u));
    float denominator = component(sums, 4u);
    misses = __reduce_add_sync(group_mask(), misses);
    if (!p.active || m.lane != 0u) return;
    float density = sums[0];
    uint32_t neighbors = n - misses;
    if (listed == kOverflow) {
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
        fallback_lists<false>(p, a.g, a.positions, xi, a.list.list, a.slots);
        replay_alone(op, p, a.g, a.list.list);
        density = op.density;
        gradient_sum = op.gradient_sum;
        denominator = op.denominator;
        neighbors = op.neighbors;
    }
    const float total = __fadd_rn(denominator, sq_yfirst(gradient_sum));
    a.lambda[s] = __fdiv_rn(-__fsub_rn(__fdiv_rn(density, pa.x), 1.0F), total);
    if (a.density) a.density[s] = density;
    if (a.neighbor_count) a.neighbor_count[s] = neighbors;
}

// ----------------------------------------------------------------- correction + project
__global__ void __launch_bounds__(kThreads) group_correction_kernel(const StagedCorrectionArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float field[5][kGroupStage];
    __shared__ __align__(16) Exchange<3> exchange[kParticles];
    const Member m = member(a.g);
    const Particle& p = m.p;
    load_windows(w, record_of(a.list));
    const float* const fields[5] = {a.positions.x, a.positions.y, a.positions.z, a.mass, a.lambda};
    if (w.staged) stage(w, field, fields);
    const uint32_t s = p.active ? p.s : 0u;
    const StoredList& list = a.list.list;
    const f3 xi = mk(a.positions.x[s], a.positions.y[s], a.positions.z[s]);
    const float mass = a.mass[s], lambda = a.lambda[s];
    const float4 pa = a.g.params_a[s];
    const float4 pb = a.g.params_b[s];
    const bool full = pb.x != 0.0F;   // s_corr has a strength
    const uint32_t count = p.active ? list.counts[s] : 0u;
    const bool grouped = w.staged && is_staged(count);
    const float ratio = __fdiv_rn(mass, pa.x);
    const float reference = full ? poly6(mk(pb.z, 0.0F, 0.0F), p.k) : 1.0F;
    float sums[1] = {};
    group_replay<3>(exchange[m.local], m.lane, grouped ? entries_of(count) : 0u, sums, stored_words(list, s),
        [&](const uint32_t i0, const uint32_t i1, float2 (&t0)[3], float2 (&t1)[3]) {
            const PairFactors f = correction_factors(p.k, xi, mass, pa.x, ratio, lambda, full, pb, reference, field, i0, i1);
            const f3 g0 = scale(f.t.d0, f.spiky.x), g1 = scale(f.t.d1, f.spiky.y);
            t0[0] = make_float2(f.first, g0.x);
            t0[1] = make_float2(f.first, g0.y);
            t0[2] = make_float2(f.first, g0.z);
            t1[0] = make_float2(f.second, g1.x);
            t1[1] = make_float2(f.second, g1.y);
            t1[2] = make_float2(f.second, g1.z);
        },
        FusedAdd{});
    f3 correction = mk(component(sums, 0u), component(sums, 1u), component(sums, 2u));
    if (!p.active || m.lane != 0u) return;
    if (!grouped) correction = correction_alone(a, p, xi, mass, lambda);
    correction_tail(a, p, xi, mass, correction);
}

// ----------------------------------------------------------- post-loop scan + vorticity
__global__ void __launch_bounds__(kThreads) group_vorticity_kernel(const StagedVorticityArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float field[6][kGroupStage];
    __shared__ __align__(16) uint16_t entries[kParticles][kGroupList];
    __shared__ __align__(16) ScanOrExchange<3> scratch;
    const Member m = member(a.g);
    const Particle& p = m.p;
    const uint32_t s = p.active ? p.s : 0u;
    const uint32_t block_first = blockIdx.x * kParticles;
    const f3 xi = mk(a.positions.x[s], a.positions.y[s], a.positions.z[s]);
    const f3 vi = mk(a.velocities.x[s], a.velocities.y[s], a.velocities.z[s]);
    const float* const fields[6] = {a.positions.x, a.positions.y, a.positions.z, a.velocities.x, a.velocities.y, a.velocities.z};
    find_windows(w, a.g, block_first, min(block_first + kParticles, a.g.count) - 1u, kGroupStage);
    __syncthreads();
    if (w.staged) stage(w, field, fields);
    uint32_t before = ~0u;
    const uint32_t listed = group_scan(w, a.list, m, a.g, field, xi, scratch.columns, entries, before);
    float sums[1] = {};
    group_replay<3>(scratch.exchange[m.local], m.lane, p.active && listed != kOverflow ? listed : 0u, sums,
        [&](const uint32_t j) { return reinterpret_cast<const uint32_t*>(entries[m.local])[j]; },
        [&](const uint32_t i0, const uint32_t i1, float2 (&t0)[3], float2 (&t1)[3]) {
            const TwoPairs t = two_pairs(xi, mk(field[0][i0], field[1][i0], field[2][i0]),
                                         mk(field[0][i1], field[1][i1], field[2][i1]));
            float2 spiky = spiky_scale_pair(t.nr2, p.k);
            const bool rare = !in_range(t.nr2, p.k);
            if (rare) spiky = any_spiky_scales(t.nr2, p.k);
            f3 v0 = sub(mk(field[3][i0], field[4][i0], field[5][i0]), vi);
            f3 v1 = sub(mk(field[3][i1], field[4][i1], field[5][i1]), vi);
            if (rare) only_inside(spiky, v0, v1);
            const f3 c0 = cross_f(v0, scale(t.d0, spiky.x));
            const f3 c1 = cross_f(v1, scale(t.d1, spiky.y));
            t0[0] = make_float2(0.0F, c0.x);
            t0[1] = make_float2(0.0F, c0.y);
            t0[2] = make_float2(0.0F, c0.z);
            t1[0] = make_float2(0.0F, c1.x);
            t1[1] = make_float2(0.0F, c1.y);
            t1[2] = make_float2(0.0F, c1.z);
        },
        [&](uint32_t, uint32_t, const float2 t, const float sum) { return __fadd_rn(sum, t.y); });
    f3 vorticity = mk(component(sums, 0u), component(sums, 1u), component(sums, 2u));
    if (!p.active || m.lane != 0u) return;
    if (listed == kOverflow) {
        VorticityOp op;
        op.pos = a.pos;
        op.velocity = a.velocity;
        op.self = s;
        op.k = p.k;
        op.x = xi;
        op.v = vi;
        op.vorticity = mk(0.0F, 0.0F, 0.0F);
        fallback_lists<false>(p, a.g, a.positions, xi, a.list.list, a.slots);
        replay_alone(op, p, a.g, a.list.list);
        vorticity = op.vorticity;
    }
    const float magnitude = __fsqrt_rn(sq_xfirst(vorticity));
    a.vorticity[s] = make_float4(vorticity.x, vorticity.y, vorticity.z, magnitude);
    a.magnitude[s] = magnitude;
}

// ------------------------------------------------------------------ normal + confinement
__global__ void __launch_bounds__(kThreads) group_normal_kernel(const StagedNormalArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float field[4][kGroupStage];
    __shared__ __align__(16) Exchange<3> exchange[kParticles];
    const Member m = member(a.g);
    const Particle& p = m.p;
    load_windows(w, record_of(a.list));
    const float* const fields[4] = {a.positions.x, a.positions.y, a.positions.z, a.magnitude};
    if (w.staged) stage(w, field, fields);
    const uint32_t s = p.active ? p.s : 0u;
    const StoredList& list = a.list.list;
    const f3 xi = mk(a.positions.x[s], a.positions.y[s], a.positions.z[s]);
    const float4 wi = a.vorticity[s];
    const uint32_t count = p.active ? list.counts[s] : 0u;
    const bool grouped = w.staged && is_staged(count);
    float sums[1] = {};
    group_replay<3>(exchange[m.local], m.lane, grouped ? entries_of(count) : 0u, sums, stored_words(list, s),
        [&](const uint32_t i0, const uint32_t i1, float2 (&t0)[3], float2 (&t1)[3]) {
            const TwoPairs t = two_pairs(xi, mk(field[0][i0], field[1][i0], field[2][i0]),
                                         mk(field[0][i1], field[1][i1], field[2][i1]));
            float2 spiky = spiky_scale_pair(t.nr2, p.k);
            const bool rare = !in_range(t.nr2, p.k);
            if (rare) spiky = any_spiky_scales(t.nr2, p.k);
            float f0 = __fsub_rn(field[3][i0], wi.w), f1 = __fsub_rn(field[3][i1], wi.w);
            if (rare) only_inside(spiky, f0, f1);
            const f3 g0 = scale(t.d0, spiky.x), g1 = scale(t.d1, spiky.y);
            t0[0] = make_float2(f0, g0.x);
            t0[1] = make_float2(f0, g0.y);
            t0[2] = make_float2(f0, g0.z);
            t1[0] = make_float2(f1, g1.x);
            t1[1] = make_float2(f1, g1.y);
            t1[2] = make_float2(f1, g1.z);
        },
        FusedAdd{});
    f3 gradient = mk(component(sums, 0u), component(sums, 1u), component(sums, 2u));
    if (!p.active || m.lane != 0u) return;
    if (!grouped) gradient = normal_alone(a, p, xi, wi.w);
    normal_tail(a, p, wi, gradient);
}

// -------------------------------------------------------------------------------- XSPH
__global__ void __launch_bounds__(kThreads) group_xsph_kernel(const StagedXsphArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ __align__(16) float field[6][kGroupStage];
    __shared__ __align__(16) Exchange<3> exchange[kParticles];
    const Member m = member(a.g);
    const Particle& p = m.p;
    load_windows(w, record_of(a.list));
    const float* const fields[6] = {a.positions.x, a.positions.y, a.positions.z, a.confined_soa.x, a.confined_soa.y,
                                    a.confined_soa.z};
    if (w.staged) stage(w, field, fields);
    const uint32_t s = p.active ? p.s : 0u;
    const StoredList& list = a.list.list;
    const f3 xi = mk(a.positions.x[s], a.positions.y[s], a.positions.z[s]);
    const f3 vi = mk(a.confined_soa.x[s], a.confined_soa.y[s], a.confined_soa.z[s]);
    const uint32_t count = p.active ? list.counts[s] : 0u;
    const bool grouped = w.staged && is_staged(count);
    float sums[1] = {};
    group_replay<3>(exchange[m.local], m.lane, grouped ? entries_of(count) : 0u, sums, stored_words(list, s),
        [&](const uint32_t i0, const uint32_t i1, float2 (&t0)[3], float2 (&t1)[3]) {
            const TwoPairs t = two_pairs(xi, mk(field[0][i0], field[1][i0], field[2][i0]),
                                         mk(field[0][i1], field[1][i1], field[2][i1]));
            float2 weight = poly6_pair(t.nr2, p.k);
            const bool rare = !in_range(t.nr2, p.k);
            if (rare) weight = any_poly6s(t.nr2, p.k);
            f3 v0 = sub(mk(field[3][i0], field[4][i0], field[5][i0]), vi);
            f3 v1 = sub(mk(field[3][i1], field[4][i1], field[5][i1]), vi);
            if (rare) only_inside(weight, v0, v1);
            t0[0] = make_float2(weight.x, v0.x);
            t0[1] = make_float2(weight.x, v0.y);
            t0[2] = make_float2(weight.x, v0.z);
            t1[0] = make_float2(weight.y, v1.x);
            t1[1] = make_float2(weight.y, v1.y);
            t1[2] = make_float2(weight.y, v1.z);
        },
        FusedAdd{});
    f3 smoothing = mk(component(sums, 0u), component(sums, 1u), component(sums, 2u));
    if (!p.active || m.lane != 0u) return;
    if (!grouped) smoothing = xsph_alone(a, p, xi, vi);
    xsph_tail(a, p, vi, smoothing);
}

template <class Args>
cudaError_t launch(void (*kernel)(Args), cudaStream_t stream, const Args& a) {
    if (a.g.count == 0) return cudaSuccess;
    launch_after(stream, kernel, (a.g.count + kParticles - 1u) / kParticles, kThreads, a);
    count_launch();
    return cudaGetLastError();
}

}  // namespace

cudaError_t launch_group_density(cudaStream_t stream, const StagedDensityArgs& a) { return launch(group_density_kernel, stream, a); }
cudaError_t launch_group_correction(cudaStream_t stream, const StagedCorrectionArgs& a) { return launch(group_correction_kernel, stream, a); }
cudaError_t launch_group_vorticity(cudaStream_t stream, const StagedVorticityArgs& a) { return launch(group_vorticity_kernel, stream, a); }
cudaError_t launch_group_normal(cudaStream_t stream, const StagedNormalArgs& a) { return launch(group_normal_kernel, stream, a); }
cudaError_t launch_group_xsph(cudaStream_t stream, const StagedXsphArgs& a) { return launch(group_xsph_kernel, stream, a); }

}  // namespace pbf
