// Forward gather passes over windows staged in shared memory (forward mode, no boundary particles).
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
// divisions.  At 1M particles, ms per launch before and now: scan + density/lambda 0.293 -> 0.252,
// correction 0.155 -> 0.108, post-loop scan and vorticity 0.143 + 0.158 -> 0.291, normal 0.151 -> 0.094,
// XSPH 0.157 -> 0.117.  What bounds them now: the scan issues 70 % of its cycles, and the replays keep
// the shared-memory pipe 70-78 % busy.
//
// Blocks of 64 or 32 particles stage 12.4 and 15.9 slots per particle and were slower (0.264 and 0.298 ms
// for the scan + density kernel, 0.150 and 0.176 ms for the correction).
//
// The first kernel of a list (scan) finds the windows and records them per block; passes that replay
// the list read the record.  A block whose windows exceed the stage (sparse spray whose neighbour
// columns are dense, 1-2 % of a dam break's blocks) keeps 32-bit slots in its lists and replays them
// from global memory, in the same kernels.
//
// Every sum keeps the reference's order and rounding (gather.cuh): the lists hold the same neighbours
// in the same order, without the particle itself, whose only term is its own density.
#include "forward_ops.cuh"

namespace pbf {

namespace {

using namespace gather_detail;

constexpr uint32_t kBlockParticles = 128;
// Staged slots: 2 % of the blocks of a 1M-particle dam break need more.  Six fields and the hit masks
// then fit 48 KB.
constexpr uint32_t kStage = 1600;
// Hit masks a particle may hold (one per 32 candidates of a column: nine at rest density).
constexpr uint32_t kMasks = 12;

struct Windows {
    uint32_t base[9];     // first sorted slot of each window, a multiple of four
    uint32_t start[10];   // its first staged position; start[9] is the total
    uint32_t staged;      // 0: the windows do not fit, the block works on global memory
};
static_assert(sizeof(Windows) <= kWindowWords * sizeof(uint32_t), "a block's record");

__device__ __forceinline__ void copy16(float* shared, const float* global) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(shared))),
                 "l"(global)
                 : "memory");
}
__device__ __forceinline__ void copies_done() {
    asm volatile("cp.async.commit_group;\ncp.async.wait_group 0;" ::: "memory");
    __syncthreads();
}

// The nine windows of the block's particles first .. last (warp 0; the caller synchronises).  A window
// runs from the cell before the first particle's stencil column to the cell after the last one's, both
// clamped to their scenes' cells.
__device__ __forceinline__ void find_windows(Windows& w, const GatherCommon& g, const uint32_t first, const uint32_t last) {
    if (threadIdx.x >= 32u) return;
    const uint32_t lane = lane_id();
    uint32_t base = 0u, length = 0u;
    if (lane < 9u) {
        const int4 a = g.cell[first], b = g.cell[last];
        const Grid& ga = g.scenes[a.w].grid;
        const Grid& gb = g.scenes[b.w].grid;
        const int dx = static_cast<int>(lane) / 3 - 1, dy = static_cast<int>(lane) % 3 - 1;
        const int64_t low = static_cast<int64_t>(cell_index(ga, a.x, a.y, a.z)) +
                            (static_cast<int64_t>(dx) * ga.cells_y + dy) * ga.cells_z - 1;
        const int64_t high = static_cast<int64_t>(cell_index(gb, b.x, b.y, b.z)) +
                             (static_cast<int64_t>(dx) * gb.cells_y + dy) * gb.cells_z + 1;
        const int64_t end_a = static_cast<int64_t>(ga.cell_base) + static_cast<int64_t>(ga.cells_x) * ga.cells_y * ga.cells_z - 1;
        const int64_t end_b = static_cast<int64_t>(gb.cell_base) + static_cast<int64_t>(gb.cells_x) * gb.cells_y * gb.cells_z - 1;
        const uint32_t begin = g.cell_offsets[min(max(low, static_cast<int64_t>(ga.cell_base)), end_a)];
        const uint32_t end = g.cell_offsets[min(max(high, static_cast<int64_t>(gb.cell_base)), end_b) + 1];
        base = begin & ~3u;
        if (end > base) length = min((end - base + 3u) & ~3u, kStage + 4u);
    }
    uint32_t inclusive = length;
#pragma unroll
    for (int o = 1; o < 16; o <<= 1) {
        const uint32_t v = __shfl_up_sync(kFull, inclusive, o);
        if (lane >= static_cast<uint32_t>(o)) inclusive += v;
    }
    if (lane < 9u) {
        w.base[lane] = base;
        w.start[lane] = inclusive - length;
    }
    if (lane == 8u) {
        w.start[9] = inclusive;
        w.staged = inclusive <= kStage ? 1u : 0u;
    }
}

__device__ __forceinline__ void store_windows(const Windows& w, uint32_t* __restrict__ record) {
    if (threadIdx.x < sizeof(Windows) / sizeof(uint32_t)) record[threadIdx.x] = reinterpret_cast<const uint32_t*>(&w)[threadIdx.x];
}
__device__ __forceinline__ void load_windows(Windows& w, const uint32_t* __restrict__ record) {
    if (threadIdx.x < sizeof(Windows) / sizeof(uint32_t)) reinterpret_cast<uint32_t*>(&w)[threadIdx.x] = record[threadIdx.x];
    __syncthreads();
}

// Copies the windows of N fields into shared memory (16 bytes a copy; the fields are readable up to
// three floats past their last slot) and waits for them.
template <int N>
__device__ __forceinline__ void stage(const Windows& w, float (*shared)[kStage], const float* const (&fields)[N]) {
    for (uint32_t u = threadIdx.x * 4u; u < w.start[9]; u += kBlockParticles * 4u) {
        uint32_t o = 0u;
#pragma unroll
        for (int q = 1; q < 9; ++q) o += u >= w.start[q] ? 1u : 0u;
        const uint32_t at = w.base[o] + (u - w.start[o]);
#pragma unroll
        for (int f = 0; f < N; ++f) copy16(&shared[f][u], fields[f] + at);
    }
    copies_done();
}

// ------------------------------------------------------------------------------ the scan
// Hit masks of this thread's particle over its nine stencil columns, in shared memory: bit 31 - j of
// masks[m][thread] is candidate bases[m][thread] + j.  A hit is a squared distance below the list
// threshold, widened by a few ulps so that the sign of (dx^2 + dy^2 + dz^2 - threshold), evaluated in
// any order, decides it; one funnel shift per candidate collects the sign (comparisons and selects
// instead: the scan + density kernel 0.268 against 0.252 ms at 1M particles).  The extra entries at the
// support's edge contribute nothing.
struct Hits {
    uint32_t count;    // neighbours, the particle itself excluded
    uint32_t masks;    // masks stored
    uint32_t before;   // neighbours listed before the particle itself (~0: it is not in its own stencil)
    bool inside;       // every column range lay inside the block's windows
};

__device__ __forceinline__ Hits scan(const Windows& w, const Particle& p, const GatherCommon& g, const float* __restrict__ x,
                                     const float* __restrict__ y, const float* __restrict__ z, const f3 xi,
                                     uint32_t (*masks)[kBlockParticles], uint16_t (*bases)[kBlockParticles]) {
    Hits hits{0u, 0u, ~0u, true};
    const Grid& grid = p.scene->grid;
    const int cx = static_cast<int>(grid.cells_x), cy = static_cast<int>(grid.cells_y), cz = static_cast<int>(grid.cells_z);
    const uint32_t z_lo = static_cast<uint32_t>(p.c.z > 0 ? p.c.z - 1 : 0);
    const uint32_t z_hi = static_cast<uint32_t>(p.c.z + 1 < cz ? p.c.z + 1 : cz - 1);
    const float2 nx = both(-xi.x), ny = both(-xi.y), nz = both(-xi.z);
    const float2 nt = both(-__fmul_rn(p.k.list_threshold, 1.0F + 0x1p-20F));
    const uint32_t* __restrict__ offsets = g.cell_offsets;
#pragma unroll 1
    for (int o = 0; o < 9; ++o) {
        const int cellx = p.c.x + o / 3 - 1, celly = p.c.y + o % 3 - 1;
        if (cellx < 0 || cellx >= cx || celly < 0 || celly >= cy) continue;
        const uint32_t first = offsets[cell_index(grid, cellx, celly, z_lo)];
        const uint32_t end = offsets[cell_index(grid, cellx, celly, z_hi) + 1u];
        if (first >= end) continue;
        const uint32_t base = w.base[o], start = w.start[o], next = w.start[o + 1];
        if (first < base || end - base > next - start) {
            hits.inside = false;
            break;
        }
        const uint32_t a = start + (first - base), b = start + (end - base);
        const uint32_t self = start + (p.s - base);   // meaningful in the particle's own column
        for (uint32_t block = a & ~3u; block < b; block += 32u) {
            const uint32_t stop = min(b, block + 32u);
            uint32_t mask = 0u, k = block;
            for (; k < stop; k += 4u) {
                const float4 qx = *reinterpret_cast<const float4*>(x + k);
                const float4 qy = *reinterpret_cast<const float4*>(y + k);
                const float4 qz = *reinterpret_cast<const float4*>(z + k);
                auto test = [&](const float2 ax, const float2 ay, const float2 az) {
                    const float2 dx = __fadd2_rn(ax, nx), dy = __fadd2_rn(ay, ny), dz = __fadd2_rn(az, nz);
                    const float2 r = __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, nt)));
                    mask = __funnelshift_l(__float_as_uint(r.x), mask, 1);
                    mask = __funnelshift_l(__float_as_uint(r.y), mask, 1);
                };
                test(make_float2(qx.x, qx.y), make_float2(qy.x, qy.y), make_float2(qz.x, qz.y));
                test(make_float2(qx.z, qx.w), make_float2(qy.z, qy.w), make_float2(qz.z, qz.w));
            }
            mask <<= 32u - (k - block);
            if (block < a) mask &= 0xffffffffu >> (a - block);
            if (b - block < 32u) mask &= ~(0xffffffffu >> (b - block));
            if (o == 4 && self - block < 32u) {
                const uint32_t bit = 0x80000000u >> (self - block);
                if (mask & bit) {
                    mask ^= bit;
                    hits.before = hits.count + static_cast<uint32_t>(__popc(mask & ~(bit | (bit - 1u))));
                }
            }
            if (mask) {
                if (hits.masks < kMasks) {
                    masks[hits.masks][threadIdx.x] = mask;
                    bases[hits.masks][threadIdx.x] = static_cast<uint16_t>(block);
                }
                ++hits.masks;
                hits.count += static_cast<uint32_t>(__popc(mask));
            }
        }
    }
    return hits;
}

// Yields the staged positions of a particle's hits in order.
struct HitCursor {
    const uint32_t (*masks)[kBlockParticles];
    const uint16_t (*bases)[kBlockParticles];
    uint32_t mask, base, next_mask, next_base, next;
    __device__ __forceinline__ void load() {
        const uint32_t m = min(next, kMasks - 1u);
        next_mask = masks[m][threadIdx.x];
        next_base = bases[m][threadIdx.x];
        ++next;
    }
    __device__ __forceinline__ void start() {
        next = 0u;
        load();
        mask = next_mask;
        base = next_base;
        load();
    }
    __device__ __forceinline__ uint32_t take() {
        if (mask == 0u) {
            mask = next_mask;
            base = next_base;
            load();
        }
        const uint32_t j = static_cast<uint32_t>(__clz(static_cast<int>(mask)));
        mask &= ~(0x80000000u >> j);
        return base + j;
    }
};

// A staged list's row: word w (entries 2w and 2w + 1) of a particle is component w % 4 of quad w / 4,
// and a warp's quads are interleaved, so eight entries are one 16-byte load.
__device__ __forceinline__ uint4* quad_row(const StoredList& list, const uint32_t s) {
    return reinterpret_cast<uint4*>(list.entries) + static_cast<size_t>(s >> 5) * (list.capacity / 4u) * 32u + (s & 31u);
}

// Calls step(i0, i1, second) for each pair of entries of a stored list of n, in order (`second`: the
// second entry exists; otherwise i1 repeats i0).  The next quad is loaded a whole quad ahead: copying
// a register that a load has not filled yet would wait for the load.
template <class Step>
__device__ __forceinline__ void replay_words(const StoredList& list, const uint32_t s, const uint32_t n, Step step) {
    const uint4* __restrict__ row = quad_row(list, s);
    if (n == 0u) return;
    uint4 quad = row[0];
#pragma unroll 1
    for (uint32_t k = 0; k < n; k += 8u) {
        uint4 ahead = quad;
        if (k + 8u < n) ahead = row[static_cast<size_t>(k / 8u + 1u) * 32u];
        step(quad.x & 0xffffu, quad.x >> 16, k + 1u < n);
        if (k + 2u < n) step(quad.y & 0xffffu, quad.y >> 16, k + 3u < n);
        if (k + 4u < n) step(quad.z & 0xffffu, quad.z >> 16, k + 5u < n);
        if (k + 6u < n) step(quad.w & 0xffffu, quad.w >> 16, k + 7u < n);
        quad = ahead;
    }
}

// The same over the hits of a scan, which it stores as the list.
template <class Step>
__device__ __forceinline__ void replay_hits(const StoredList& list, const uint32_t s, const uint32_t n,
                                            const uint32_t (*masks)[kBlockParticles], const uint16_t (*bases)[kBlockParticles],
                                            Step step) {
    uint4* __restrict__ row = quad_row(list, s);
    if (n == 0u) return;
    HitCursor cursor{masks, bases};
    cursor.start();
    auto pair = [&](const uint32_t k) -> uint32_t {
        const uint32_t i0 = cursor.take();
        const bool second = k + 1u < n;
        const uint32_t i1 = second ? cursor.take() : i0;
        step(i0, i1, second, k);
        return i0 | (i1 << 16);
    };
#pragma unroll 1
    for (uint32_t k = 0; k < n; k += 8u) {
        uint4 quad = make_uint4(0u, 0u, 0u, 0u);
        quad.x = pair(k);
        if (k + 2u < n) quad.y = pair(k + 2u);
        if (k + 4u < n) quad.z = pair(k + 4u);
        if (k + 6u < n) quad.w = pair(k + 6u);
        row[static_cast<size_t>(k / 8u) * 32u] = quad;
    }
}

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
__device__ __noinline__ float any_spiky_scale(const float r2, const float h, const float coefficient) {
    const float distance = __fsqrt_rn(r2);
    if (distance == 0.0F || distance >= h) return 0.0F;
    const float difference = __fsub_rn(h, distance);
    return __fdiv_rn(__fmul_rn(__fmul_rn(coefficient, difference), difference), distance);
}
__device__ __noinline__ float any_poly6(const float r2, const float h2, const float denominator) {
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

// A global-memory block's scan: sorted slots, the particle itself included (as launch_list_scan).
__device__ __forceinline__ uint32_t scan_global(const Particle& p, const GatherCommon& g, const PackedPositions packed, const f3 xi,
                                                const StoredList& list) {
    const Grid& grid = p.scene->grid;
    const int cx = static_cast<int>(grid.cells_x), cy = static_cast<int>(grid.cells_y), cz = static_cast<int>(grid.cells_z);
    const uint32_t z_lo = static_cast<uint32_t>(p.c.z > 0 ? p.c.z - 1 : 0);
    const uint32_t z_hi = static_cast<uint32_t>(p.c.z + 1 < cz ? p.c.z + 1 : cz - 1);
    PackedScan s;
    s.nx = both(-xi.x);
    s.ny = both(-xi.y);
    s.nz = both(-xi.z);
    s.threshold = p.k.list_threshold;
    s.n = 0u;
    s.capacity = list.capacity;
    s.entries = list.entries + list_row(p.s, list.capacity);
#pragma unroll 1
    for (int o = 0; o < 9; ++o) {
        const int x = p.c.x + o / 3 - 1, y = p.c.y + o % 3 - 1;
        if (x < 0 || x >= cx || y < 0 || y >= cy) continue;
        s.run(packed, g.cell_offsets[cell_index(grid, x, y, z_lo)], g.cell_offsets[cell_index(grid, x, y, z_hi) + 1u]);
    }
    return s.n <= list.capacity ? s.n : kOverflow;
}

__device__ __forceinline__ uint32_t first_particle(const GatherCommon& g) {
    return (g.reverse ? gridDim.x - 1u - blockIdx.x : blockIdx.x) * kBlockParticles;
}

// Windows and hits of the block's particles at the staged positions (fields 0..2 of `shared`); false:
// the block works on global memory.  Every thread of the block calls it.
template <int N>
__device__ __forceinline__ bool windows_and_hits(Windows& w, const StagedList& list, const Particle& p, const GatherCommon& g,
                                                 float (*shared)[kStage], const float* const (&fields)[N], const f3 xi,
                                                 uint32_t (*masks)[kBlockParticles], uint16_t (*bases)[kBlockParticles],
                                                 Hits& hits) {
    const uint32_t first = first_particle(g);
    find_windows(w, g, first, min(first + kBlockParticles, g.count) - 1u);
    __syncthreads();
    hits = Hits{0u, 0u, ~0u, true};
    if (w.staged) {
        stage(w, shared, fields);
        if (p.active) hits = scan(w, p, g, shared[0], shared[1], shared[2], xi, masks, bases);
        // a gather cell beyond the window of its neighbours' sort cells (the two cell formulas round
        // differently): the whole block takes global memory
        if (__syncthreads_or(!hits.inside) && threadIdx.x == 0u) w.staged = 0u;
        __syncthreads();
    }
    store_windows(w, list.windows + static_cast<size_t>(first / kBlockParticles) * kWindowWords);
    return w.staged != 0u;
}

// ------------------------------------------------------------------- density + lambda
__global__ void __launch_bounds__(kBlockParticles, 6) staged_density_kernel(const StagedDensityArgs a) {
    __shared__ Windows w;
    __shared__ __align__(16) float field[4][kStage];
    __shared__ uint32_t masks[kMasks][kBlockParticles];
    __shared__ uint16_t bases[kMasks][kBlockParticles];
    const Particle p = locate(a.g);
    const uint32_t s = p.active ? p.s : 0u;
    const f3 xi = mk(a.positions.x[s], a.positions.y[s], a.positions.z[s]);
    const float mass = a.mass[s];
    const float4 pa = a.g.params_a[s];
    const float* const fields[4] = {a.positions.x, a.positions.y, a.positions.z, a.mass};
    Hits hits;
    const bool staged = windows_and_hits(w, a.list, p, a.g, field, fields, xi, masks, bases, hits);
    if (!p.active) return;
    const StoredList& list = a.list.list;
    float density = 0.0F, denominator = pa.y;   // relaxation
    f3 gradient_sum = mk(0.0F, 0.0F, 0.0F);
    uint32_t neighbors = 0u;
    if (staged && hits.masks <= kMasks && hits.count <= 2u * list.capacity) {
        const uint32_t n = hits.count;
        list.counts[s] = n;
        neighbors = n;
        const float own = any_poly6(0.0F, p.k.h2, p.k.poly6_denominator);   // W(0)
        const float ratio = __fdiv_rn(mass, pa.x);
        replay_hits(list, s, n, masks, bases, [&](const uint32_t i0, const uint32_t i1, const bool second, const uint32_t k) {
            const float m0 = field[3][i0], m1 = field[3][i1];
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
        list.counts[s] = staged ? kOverflow : scan_global(p, a.g, a.positions, xi, list);
        replay(op, p, a.g, list);
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
__global__ void __launch_bounds__(kBlockParticles, 7) staged_correction_kernel(const StagedCorrectionArgs a) {
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
    if (w.staged && n != kOverflow) {
        const float ratio = __fdiv_rn(mass, pa.x);
        const float reference = full ? poly6(mk(pb.z, 0.0F, 0.0F), p.k) : 1.0F;
        replay_words(list, s, n, [&](const uint32_t i0, const uint32_t i1, const bool second) {
            const float m0 = field[3][i0], m1 = field[3][i1];
            const TwoPairs t = two_pairs(xi, mk(field[0][i0], field[1][i0], field[2][i0]),
                                         mk(field[0][i1], field[1][i1], field[2][i1]));
            float2 spiky = spiky_scale_pair(t.nr2, p.k);
            // s_corr (pbf/pbf.cu:56-71): with zero strength -strength inside the poly6 support
            float a0 = -pb.x, a1 = -pb.x;
            float c0 = ratio, c1 = ratio;
            if (full) {
                const float2 weight = in_range(t.nr2, p.k) ? poly6_pair(t.nr2, p.k) : any_poly6s(t.nr2, p.k);
                a0 = weight.x == 0.0F ? 0.0F : __fmul_rn(-pb.x, powf(__fdiv_rn(weight.x, reference), pb.y));
                a1 = weight.y == 0.0F ? 0.0F : __fmul_rn(-pb.x, powf(__fdiv_rn(weight.y, reference), pb.y));
            }
            float s0 = __fadd_rn(lambda, field[4][i0]), s1 = __fadd_rn(lambda, field[4][i1]);
            if (!in_range(t.nr2, p.k) || m0 != mass || m1 != mass) {
                c0 = __fdiv_rn(m0, pa.x);
                c1 = __fdiv_rn(m1, pa.x);
                if (!in_range(t.nr2, p.k)) {
                    spiky = any_spiky_scales(t.nr2, p.k);
                    if (!full) {
                        a0 = -t.nr2.x < p.k.h2 ? a0 : 0.0F;
                        a1 = -t.nr2.y < p.k.h2 ? a1 : 0.0F;
                    }
                    if (spiky.x == 0.0F) s0 = a0 = 0.0F;   // no gradient: no term, whatever lambda is
                    if (spiky.y == 0.0F) s1 = a1 = 0.0F;
                }
            }
            const float f0 = __fmul_rn(c0, __fadd_rn(s0, a0));
            const float f1 = __fmul_rn(c1, __fadd_rn(s1, a1));
            correction = fma3(f0, scale(t.d0, spiky.x), correction);
            if (second) correction = fma3(f1, scale(t.d1, spiky.y), correction);
        });
    } else {
        CorrectionOp<false> op;
        op.pos = a.pos;
        op.boundary = nullptr;
        op.lambda = a.lambda;
        op.self = s;
        op.k = p.k;
        op.x = xi;
        op.rest_density = pa.x;
        op.ratio.reset(mass, pa.x);
        op.lambda_i = lambda;
        op.strength = pb.x;
        op.exponent = pb.y;
        op.artificial_full = full;
        op.reference_weight = full ? poly6(mk(pb.z, 0.0F, 0.0F), p.k) : 1.0F;
        op.correction = correction;
        replay(op, p, a.g, list);
        correction = op.correction;
    }
    const Box& box = p.scene->box;
    const f3 candidate = add(xi, correction);
    const f3 projected = mk(fminf(box.max_x, fmaxf(box.min_x, candidate.x)), fminf(box.max_y, fmaxf(box.min_y, candidate.y)),
                            fminf(box.max_z, fmaxf(box.min_z, candidate.z)));
    a.pos_next[s] = make_float4(projected.x, projected.y, projected.z, mass);
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

// ----------------------------------------------------------- post-loop scan + vorticity
__global__ void __launch_bounds__(kBlockParticles, 4) staged_vorticity_kernel(const StagedVorticityArgs a) {
    __shared__ Windows w;
    __shared__ __align__(16) float field[6][kStage];
    __shared__ uint32_t masks[kMasks][kBlockParticles];
    __shared__ uint16_t bases[kMasks][kBlockParticles];
    const Particle p = locate(a.g);
    const uint32_t s = p.active ? p.s : 0u;
    const f3 xi = mk(a.positions.x[s], a.positions.y[s], a.positions.z[s]);
    const f3 vi = mk(a.velocities.x[s], a.velocities.y[s], a.velocities.z[s]);
    const float* const fields[6] = {a.positions.x, a.positions.y, a.positions.z, a.velocities.x, a.velocities.y, a.velocities.z};
    Hits hits;
    const bool staged = windows_and_hits(w, a.list, p, a.g, field, fields, xi, masks, bases, hits);
    if (!p.active) return;
    const StoredList& list = a.list.list;
    f3 vorticity = mk(0.0F, 0.0F, 0.0F);
    if (staged && hits.masks <= kMasks && hits.count <= 2u * list.capacity) {
        const uint32_t n = hits.count;
        list.counts[s] = n;
        replay_hits(list, s, n, masks, bases, [&](const uint32_t i0, const uint32_t i1, const bool second, uint32_t) {
            const TwoPairs t = two_pairs(xi, mk(field[0][i0], field[1][i0], field[2][i0]),
                                         mk(field[0][i1], field[1][i1], field[2][i1]));
            const f3 v0 = mk(field[3][i0], field[4][i0], field[5][i0]), v1 = mk(field[3][i1], field[4][i1], field[5][i1]);
            float2 spiky = spiky_scale_pair(t.nr2, p.k);
            if (!in_range(t.nr2, p.k)) spiky = any_spiky_scales(t.nr2, p.k);
            vorticity = add(vorticity, cross_f(sub(v0, vi), scale(t.d0, spiky.x)));
            if (second) vorticity = add(vorticity, cross_f(sub(v1, vi), scale(t.d1, spiky.y)));
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
        list.counts[s] = staged ? kOverflow : scan_global(p, a.g, a.positions, xi, list);
        replay(op, p, a.g, list);
        vorticity = op.vorticity;
    }
    const float magnitude = __fsqrt_rn(sq_xfirst(vorticity));
    a.vorticity[s] = make_float4(vorticity.x, vorticity.y, vorticity.z, magnitude);
    a.magnitude[s] = magnitude;
}

// ------------------------------------------------------------------ normal + confinement
__global__ void __launch_bounds__(kBlockParticles, 8) staged_normal_kernel(const StagedNormalArgs a) {
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
    if (w.staged && n != kOverflow) {
        replay_words(list, s, n, [&](const uint32_t i0, const uint32_t i1, const bool second) {
            const TwoPairs t = two_pairs(xi, mk(field[0][i0], field[1][i0], field[2][i0]),
                                         mk(field[0][i1], field[1][i1], field[2][i1]));
            float2 spiky = spiky_scale_pair(t.nr2, p.k);
            if (!in_range(t.nr2, p.k)) spiky = any_spiky_scales(t.nr2, p.k);
            gradient = fma3(__fsub_rn(field[3][i0], wi.w), scale(t.d0, spiky.x), gradient);
            if (second) gradient = fma3(__fsub_rn(field[3][i1], wi.w), scale(t.d1, spiky.y), gradient);
        });
    } else {
        NormalOp op;
        op.pos = a.pos;
        op.vorticity = a.vorticity;
        op.self = s;
        op.k = p.k;
        op.x = xi;
        op.magnitude = wi.w;
        op.gradient = gradient;
        replay(op, p, a.g, list);
        gradient = op.gradient;
    }
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

// -------------------------------------------------------------------------------- XSPH
__global__ void __launch_bounds__(kBlockParticles, 5) staged_xsph_kernel(const StagedXsphArgs a) {
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
    if (w.staged && n != kOverflow) {
        replay_words(list, s, n, [&](const uint32_t i0, const uint32_t i1, const bool second) {
            const TwoPairs t = two_pairs(xi, mk(field[0][i0], field[1][i0], field[2][i0]),
                                         mk(field[0][i1], field[1][i1], field[2][i1]));
            const f3 v0 = mk(field[3][i0], field[4][i0], field[5][i0]), v1 = mk(field[3][i1], field[4][i1], field[5][i1]);
            float2 weight = poly6_pair(t.nr2, p.k);
            if (!in_range(t.nr2, p.k)) weight = any_poly6s(t.nr2, p.k);
            smoothing = fma3(weight.x, sub(v0, vi), smoothing);
            if (second) smoothing = fma3(weight.y, sub(v1, vi), smoothing);
        });
    } else {
        XsphOp op;
        op.pos = a.pos;
        op.confined = a.confined;
        op.self = s;
        op.k = p.k;
        op.x = xi;
        op.v = vi;
        op.smoothing = smoothing;
        replay(op, p, a.g, list);
        smoothing = op.smoothing;
    }
    const f3 out = fma3(a.g.params_a[s].z, smoothing, vi);
    const uint32_t i = a.sorted_index[s];
    a.out_velocities.x[i] = out.x;
    a.out_velocities.y[i] = out.y;
    a.out_velocities.z[i] = out.z;
}

inline unsigned blocks_of(const uint32_t n) { return (n + kBlockParticles - 1u) / kBlockParticles; }

template <class Args>
cudaError_t launch(void (*kernel)(Args), cudaStream_t stream, const Args& a) {
    if (a.g.count == 0) return cudaSuccess;
    kernel<<<blocks_of(a.g.count), kBlockParticles, 0, stream>>>(a);
    count_launch();
    return cudaGetLastError();
}

}  // namespace

size_t window_words(const uint32_t count) { return static_cast<size_t>(blocks_of(count)) * kWindowWords; }

cudaError_t launch_staged_density(cudaStream_t stream, const StagedDensityArgs& a) { return launch(staged_density_kernel, stream, a); }
cudaError_t launch_staged_correction(cudaStream_t stream, const StagedCorrectionArgs& a) {
    return launch(staged_correction_kernel, stream, a);
}
cudaError_t launch_staged_vorticity(cudaStream_t stream, const StagedVorticityArgs& a) {
    return launch(staged_vorticity_kernel, stream, a);
}
cudaError_t launch_staged_normal(cudaStream_t stream, const StagedNormalArgs& a) { return launch(staged_normal_kernel, stream, a); }
cudaError_t launch_staged_xsph(cudaStream_t stream, const StagedXsphArgs& a) { return launch(staged_xsph_kernel, stream, a); }

}  // namespace pbf
