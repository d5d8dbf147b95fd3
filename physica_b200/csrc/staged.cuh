// Windows of the sorted particles staged in shared memory, the candidate scan over them and the lists
// of 16-bit staged positions it leaves: the machinery of the staged passes (staged.cu, sph_staged.cu).
#pragma once

#include "forward_ops.cuh"

namespace pbf {
namespace staged_detail {

using namespace gather_detail;

constexpr uint32_t kBlockParticles = 128;   // and threads
// Staged slots: 2 % of the blocks of a 1M-particle dam break need more.  Six fields and the hit masks
// then fit 48 KB.
constexpr uint32_t kStage = 1600;
// The same with four lanes per particle (staged_group.cu): 0.6 % of the blocks of a dam break of 5k to 20k
// particles have more in their windows.
constexpr uint32_t kGroupParticles = 32;
constexpr uint32_t kGroupStage = 704;
// Candidates of one stencil column that its hit record covers (26 on average in a dam break at its
// densest, 24 at rest).
constexpr uint32_t kColumn = 48;

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
__device__ __forceinline__ void find_windows(Windows& w, const GatherCommon& g, const uint32_t first, const uint32_t last,
                                             const uint32_t capacity) {
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
        if (end > base) length = min((end - base + 3u) & ~3u, capacity + 4u);
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
        w.staged = inclusive <= capacity ? 1u : 0u;
    }
}

__device__ __forceinline__ void store_windows(const Windows& w, uint32_t* __restrict__ record) {
    if (threadIdx.x < sizeof(Windows) / sizeof(uint32_t)) record[threadIdx.x] = reinterpret_cast<const uint32_t*>(&w)[threadIdx.x];
}
__device__ __forceinline__ void load_windows(Windows& w, const uint32_t* __restrict__ record) {
    if (threadIdx.x < sizeof(Windows) / sizeof(uint32_t)) reinterpret_cast<uint32_t*>(&w)[threadIdx.x] = record[threadIdx.x];
    __syncthreads();
}

// Copies the windows of one field of float4.
__device__ __forceinline__ void stage4(const Windows& w, float4* shared, const float4* field, const uint32_t count) {
    for (uint32_t u = threadIdx.x; u < w.start[9]; u += kBlockParticles) {
        uint32_t o = 0u;
#pragma unroll
        for (int q = 1; q < 9; ++q) o += u >= w.start[q] ? 1u : 0u;
        const uint32_t at = min(w.base[o] + (u - w.start[o]), count - 1u);   // a window ends on a multiple of four
        copy16(reinterpret_cast<float*>(shared + u), reinterpret_cast<const float*>(field + at));
    }
}

// Copies the windows of N fields into shared memory (16 bytes a copy; the fields are readable up to
// three floats past their last slot) and waits for them.
template <int N, uint32_t S>
__device__ __forceinline__ void stage(const Windows& w, float (*shared)[S], const float* const (&fields)[N]) {
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
// The hits of one stencil column that has some: bit 31 - j of `low` is the candidate at staged position
// base + j, bit 15 - j of the lower half of `rest` the one at base + 32 + j.  The upper half of `rest` is
// the base and, above its 11 bits, the column's window.
struct ColumnHits {
    uint32_t low, rest;
};

// Hits of this thread's particle over its nine stencil columns, columns[0 .. columns - 1][thread] in shared
// memory.  A hit is a squared distance below the list threshold.  Exact: the squared distance and comparison
// of the per-lane scan (PackedScan), so that lists of slots are the same whatever scan wrote them.
// Otherwise the threshold is widened by a few ulps so that the sign of (dx^2 + dy^2 + dz^2 - threshold),
// evaluated in any order, decides it, and the extra entries at the support's edge contribute nothing.  One
// funnel shift per candidate collects the sign (comparisons and selects instead: the scan + density kernel
// 0.268 against 0.252 ms at 1M particles).  A column has at most 48 candidates: one block of 32 and half a
// one, unrolled (a loop over the halves: 0.269 against 0.262 ms).
struct Hits {
    uint32_t count;    // neighbours, the particle itself excluded
    uint32_t columns;  // columns with some
    uint32_t before;   // neighbours listed before the particle itself (~0: it is not in its own stencil)
    bool inside;       // every column range lay inside the block's windows
    bool covered;      // every column fitted its record
};

template <bool Exact>
__device__ __forceinline__ Hits scan(const Windows& w, const Particle& p, const GatherCommon& g, const float* __restrict__ x,
                                     const float* __restrict__ y, const float* __restrict__ z, const f3 xi,
                                     ColumnHits (*columns)[kBlockParticles], const int first_column = 0,
                                     const int end_column = 9) {
    Hits hits{0u, 0u, ~0u, true, true};
    const Grid& grid = p.scene->grid;
    const int cx = static_cast<int>(grid.cells_x), cy = static_cast<int>(grid.cells_y), cz = static_cast<int>(grid.cells_z);
    const uint32_t z_lo = static_cast<uint32_t>(p.c.z > 0 ? p.c.z - 1 : 0);
    const uint32_t z_hi = static_cast<uint32_t>(p.c.z + 1 < cz ? p.c.z + 1 : cz - 1);
    const float2 nx = both(-xi.x), ny = both(-xi.y), nz = both(-xi.z);
    const float2 nt = both(Exact ? -p.k.list_threshold : -__fmul_rn(p.k.list_threshold, 1.0F + 0x1p-20F));
    const uint32_t* __restrict__ offsets = g.cell_offsets;
#pragma unroll 1
    for (int o = first_column; o < end_column; ++o) {
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
        const uint32_t begin = a & ~3u;
        hits.covered = hits.covered && b - begin <= kColumn;
        // the particle's place, in the column that holds its slot: its sort cell's, which is not always its
        // gather cell's column (the two cell formulas round differently)
        uint32_t self = p.s - first < end - first ? start + (p.s - base) - begin : ~0u;
        auto test_block = [&](const uint32_t block, const uint32_t stop, const uint32_t valid) -> uint32_t {
            uint32_t mask = 0u, k = block;
            for (; k < stop; k += 4u) {
                const float4 qx = *reinterpret_cast<const float4*>(x + k);
                const float4 qy = *reinterpret_cast<const float4*>(y + k);
                const float4 qz = *reinterpret_cast<const float4*>(z + k);
                auto test = [&](const float2 ax, const float2 ay, const float2 az) {
                    const float2 dx = __fadd2_rn(ax, nx), dy = __fadd2_rn(ay, ny), dz = __fadd2_rn(az, nz);
                    const float2 r = Exact ? __fadd2_rn(__ffma2_rn(dz, dz, __ffma2_rn(dx, dx, __fmul2_rn(dy, dy))), nt)
                                           : __ffma2_rn(dz, dz, __ffma2_rn(dy, dy, __ffma2_rn(dx, dx, nt)));
                    mask = __funnelshift_l(__float_as_uint(r.x), mask, 1);
                    mask = __funnelshift_l(__float_as_uint(r.y), mask, 1);
                };
                test(make_float2(qx.x, qx.y), make_float2(qy.x, qy.y), make_float2(qz.x, qz.y));
                test(make_float2(qx.z, qx.w), make_float2(qy.z, qy.w), make_float2(qz.z, qz.w));
            }
            mask = (mask << (32u - (k - block))) & valid;
            if (b - block < 32u) mask &= ~(0xffffffffu >> (b - block));
            if (self < 32u) {
                const uint32_t bit = 0x80000000u >> self;
                if (mask & bit) {
                    mask ^= bit;
                    hits.before = hits.count + static_cast<uint32_t>(__popc(mask & ~(bit | (bit - 1u))));
                }
            }
            return mask;
        };
        uint32_t low = test_block(begin, min(b, begin + 32u), 0xffffffffu >> (a - begin));
        hits.count += static_cast<uint32_t>(__popc(low));
        uint32_t high = 0u, placed = begin;
        if (b - begin > 32u) {
            self -= 32u;
            high = test_block(begin + 32u, min(b, begin + kColumn), ~0u) >> 16;
            hits.count += static_cast<uint32_t>(__popc(high));
            if (low == 0u) {   // a record's low half has hits
                low = high << 16;
                high = 0u;
                placed += 32u;
            }
        }
        if (low) {
            columns[hits.columns][threadIdx.x] = {low, high | (placed << 16) | (static_cast<uint32_t>(o) << 27)};
            ++hits.columns;
        }
    }
    return hits;
}

// Yields the staged positions of a particle's hits in order; position + shift is the sorted slot.
struct HitCursor {
    const Windows& w;
    const ColumnHits (*columns)[kBlockParticles];
    uint32_t mask, base, shift, high;   // of the current column
    ColumnHits ahead;                   // the column after it
    uint32_t next;
    __device__ __forceinline__ HitCursor(const Windows& windows, const ColumnHits (*c)[kBlockParticles])
        : w(windows), columns(c), ahead(c[0][threadIdx.x]), next(1u) {
        advance();
    }
    __device__ __forceinline__ void advance() {
        mask = ahead.low;
        high = ahead.rest & 0xffffu;
        base = (ahead.rest >> 16) & 0x7ffu;
        const uint32_t o = min(ahead.rest >> 27, 8u);
        shift = w.base[o] - w.start[o];
        ahead = columns[min(next, 8u)][threadIdx.x];
        ++next;
    }
    // Call while entries are left.
    __device__ __forceinline__ uint32_t take() {
        if (mask == 0u) {
            if (high != 0u) {
                mask = high << 16;
                base += 32u;
                high = 0u;
            } else {
                advance();
            }
        }
        const uint32_t j = static_cast<uint32_t>(__clz(static_cast<int>(mask)));
        mask &= ~(0x80000000u >> j);
        return base + j;
    }
};

// A staged list's count word: entries in its lower half, entries before the particle itself (0xffff: it
// is not in its own stencil) in the upper one.  0xfffe there marks a list of hit masks over sorted slots
// (below), kOverflow a particle without a list.
constexpr uint32_t kMaskList = 0xfffeu;
__device__ __forceinline__ uint32_t entries_of(const uint32_t count) { return count & 0xffffu; }
__device__ __forceinline__ uint32_t before_of(const uint32_t count) { return count >> 16; }
__device__ __forceinline__ bool is_staged(const uint32_t count) { return count < (kMaskList << 16) || (count >> 16 == 0xffffu && count != kOverflow); }

// A staged list's row: word w (entries 2w and 2w + 1) of a particle is component w % 4 of quad w / 4,
// and a warp's quads are interleaved, so eight entries are one 16-byte load.
__device__ __forceinline__ uint4* quad_row(const StoredList& list, const uint32_t s) {
    return reinterpret_cast<uint4*>(list.entries) + static_cast<size_t>(s >> 5) * (list.capacity / 4u) * 32u + (s & 31u);
}
// Word w of the row as one 32-bit value.
__device__ __forceinline__ uint32_t* word_of(const StoredList& list, const uint32_t s, const uint32_t w) {
    return reinterpret_cast<uint32_t*>(quad_row(list, s)) + static_cast<size_t>(w / 4u) * 128u + w % 4u;
}

// Pair j of a hit-mask list, in the words 2 j and 2 j + 1 of the particle's row: the rows of a warp's staged
// lists and hit-mask lists share their memory, so both keep to their own particle's words.
__device__ __forceinline__ uint2* pair_of(const StoredList& list, const uint32_t s, const uint32_t j) {
    return reinterpret_cast<uint2*>(quad_row(list, s) + static_cast<size_t>(j / 2u) * 32u) + j % 2u;
}

// Yields the slots of a hit-mask list in order: the set bits of each (base, mask) pair, ascending.
// The next pair is loaded while the current one is drained.
struct MaskCursor {
    const StoredList& list;
    uint32_t s, next;
    uint2 current, upcoming;
    __device__ __forceinline__ MaskCursor(const StoredList& l, const uint32_t particle)
        : list(l), s(particle), next(2u), current(*pair_of(l, particle, 0u)), upcoming(*pair_of(l, particle, 1u)) {}
    // The next slot; call at most as many times as the list has neighbours.
    __device__ __forceinline__ uint32_t take() {
        if (current.y == 0u) {
            current = upcoming;
            upcoming = 2u * next < list.capacity ? *pair_of(list, s, next) : make_uint2(0u, 0u);
            ++next;
        }
        const uint32_t k = static_cast<uint32_t>(__ffs(static_cast<int>(current.y))) - 1u;
        current.y &= current.y - 1u;
        return current.x + k;
    }
};

// Drains a hit-mask list of n neighbours in order.
template <class Op>
__device__ __forceinline__ void replay_masks(Op& op, const Particle& p, const StoredList& list, const uint32_t n) {
    if (n == 0) return;
    MaskCursor cursor(list, p.s);
    uint32_t t = cursor.take();
    auto data = op.prefetch(t);
    for (uint32_t k = 1; k < n; ++k) {
        const uint32_t tn = cursor.take();
        const auto next = op.prefetch(tn);
        op.apply(t, data);
        t = tn;
        data = next;
    }
    op.apply(t, data);
}

// Builds the hit-mask list of a particle from global memory, the particle itself included: one (slot of
// bit 0, 32-bit mask) pair per 32 candidates of a column with a hit, any number of neighbours in
// capacity / 2 pairs.  For blocks whose windows do not fit the stage and particles whose hits do not fit
// their records: the surface spray of a dam break, and its clumps, where a particle has hundreds of
// neighbours.
__device__ __forceinline__ void scan_masks(const Particle& p, const GatherCommon& g, const PackedPositions packed, const f3 xi,
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
    const uint32_t capacity = list.capacity / 2u;
    uint32_t n = 0u, pairs = 0u;
#pragma unroll 1
    for (int o = 0; o < 9; ++o) {
        const int x = p.c.x + o / 3 - 1, y = p.c.y + o % 3 - 1;
        if (x < 0 || x >= cx || y < 0 || y >= cy) continue;
        const uint32_t first = g.cell_offsets[cell_index(grid, x, y, z_lo)];
        const uint32_t end = g.cell_offsets[cell_index(grid, x, y, z_hi) + 1u];
        if (first >= end) continue;
        for (uint32_t base = first & ~3u; base < end; base += 32u) {
            const uint32_t mask = s.block_mask(packed, base, first, end);
            if (mask) {
                if (pairs < capacity) *pair_of(list, p.s, pairs) = make_uint2(base, mask);
                ++pairs;
                n += static_cast<uint32_t>(__popc(mask));
            }
        }
    }
    list.counts[p.s] = pairs <= capacity && n < 0xffffu ? (kMaskList << 16) | n : kOverflow;
    __threadfence_block();   // read back by this thread
}

// The replay of a list of slots that this kernel wrote.  replay() may read a list through the read-only
// path, which does not see them.
template <class Op>
__device__ __forceinline__ void replay_written(Op& op, const Particle& p, const GatherCommon& g, const StoredList& list) {
    const uint32_t n = list.counts[p.s];
    if (n == kOverflow) {
        walk(op, p, g);
        return;
    }
    const uint32_t* entries = list.entries + list_row(p.s, list.capacity);
    for (uint32_t k = 0; k < n; ++k) op.process(entries[static_cast<size_t>(k) * 32u]);
}

// The replay of a particle without a staged list.
template <class Op>
__device__ __forceinline__ void replay_alone(Op& op, const Particle& p, const GatherCommon& g, const StoredList& list) {
    const uint32_t count = list.counts[p.s];
    if (count == kOverflow) walk(op, p, g);
    else replay_masks(op, p, list, entries_of(count));
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

// The same over the hits of a scan, step(i0, i1, second, k), storing them as a list of staged positions
// (Words) and as one of sorted slots (Slots; the particle itself among them, as every list of slots
// holds it, at its place `before`).
template <bool Words, bool Slots, class Step>
__device__ __forceinline__ void replay_hits(const Windows& w, const StoredList& words, const StoredList& slots, const uint32_t s,
                                            const Hits& hits, const ColumnHits (*columns)[kBlockParticles], Step step) {
    const uint32_t n = hits.count, before = hits.before;
    uint32_t* __restrict__ slot_row = nullptr;
    if constexpr (Slots) slot_row = slots.entries + list_row(s, slots.capacity);
    auto store = [&](const uint32_t slot) {
        *slot_row = slot;
        slot_row += 32;
    };
    if (n > 0u) {
        HitCursor cursor(w, columns);
        auto take = [&](const uint32_t k) -> uint32_t {
            const uint32_t i = cursor.take();
            if constexpr (Slots) {
                if (k == before) store(s);
                store(i + cursor.shift);
            }
            return i;
        };
        auto pair = [&](const uint32_t k) -> uint32_t {
            const uint32_t i0 = take(k);
            const bool second = k + 1u < n;
            const uint32_t i1 = second ? take(k + 1u) : i0;
            step(i0, i1, second, k);
            return i0 | (i1 << 16);
        };
        uint4* __restrict__ row = nullptr;
        if constexpr (Words) row = quad_row(words, s);
#pragma unroll 1
        for (uint32_t k = 0; k < n; k += 8u) {
            uint4 quad = make_uint4(0u, 0u, 0u, 0u);
            quad.x = pair(k);
            if (k + 2u < n) quad.y = pair(k + 2u);
            if (k + 4u < n) quad.z = pair(k + 4u);
            if (k + 6u < n) quad.w = pair(k + 6u);
            if constexpr (Words) row[static_cast<size_t>(k / 8u) * 32u] = quad;
        }
    }
    if constexpr (Words) words.counts[s] = n | (before << 16);
    if constexpr (Slots) {
        if (before == n) store(s);
        slots.counts[s] = n + (before != ~0u ? 1u : 0u);
    }
}

// A block that works on global memory: its particle's list of sorted slots, the particle itself
// included (as launch_list_scan).
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
    __threadfence_block();   // read back by this thread
    return s.n <= list.capacity ? s.n : kOverflow;
}

// Whether a particle's hits fit its lists.
template <bool Slots>
__device__ __forceinline__ bool fits(const Hits& hits, const StoredList& list) {
    return hits.covered && hits.count < (Slots ? list.capacity : 2u * list.capacity);
}

// The lists of a particle without a staged one.
template <bool Slots>
__device__ __forceinline__ void fallback_lists(const Particle& p, const GatherCommon& g, const PackedPositions positions, const f3 xi,
                                               const StoredList& list, const StoredList& slots) {
    scan_masks(p, g, positions, xi, list);
    if constexpr (Slots) slots.counts[p.s] = scan_global(p, g, positions, xi, slots);
}

__device__ __forceinline__ uint32_t first_particle(const GatherCommon& g) {
    return (g.reverse ? gridDim.x - 1u - blockIdx.x : blockIdx.x) * kBlockParticles;
}

// Windows and hits of the block's particles at the staged positions (fields 0..2 of `shared`); false:
// the block works on global memory.  Every thread of the block calls it.
template <bool Exact, int N>
__device__ __forceinline__ bool windows_and_hits(Windows& w, const StagedList& list, const Particle& p, const GatherCommon& g,
                                                 float (*shared)[kStage], const float* const (&fields)[N], const f3 xi,
                                                 ColumnHits (*columns)[kBlockParticles], Hits& hits) {
    const uint32_t first = first_particle(g);
    find_windows(w, g, first, min(first + kBlockParticles, g.count) - 1u, kStage);
    __syncthreads();
    hits = Hits{0u, 0u, ~0u, true, true};
    if (w.staged) {
        stage(w, shared, fields);
        if (p.active) hits = scan<Exact>(w, p, g, shared[0], shared[1], shared[2], xi, columns);
        // a gather cell beyond the window of its neighbours' sort cells (the two cell formulas round
        // differently): the whole block takes global memory
        if (__syncthreads_or(!hits.inside) && threadIdx.x == 0u) w.staged = 0u;
        __syncthreads();
    }
    store_windows(w, list.windows + static_cast<size_t>(first / kBlockParticles) * kWindowWords);
    return w.staged != 0u;
}

}  // namespace staged_detail
}  // namespace pbf
