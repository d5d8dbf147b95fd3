// The measurement behind staged_fit.h.
#include <algorithm>
#include <mutex>
#include <vector>

#include "dependent_launch.cuh"
#include "engine.h"
#include "staged.cuh"
#include "staged_fit.h"

namespace pbf {

namespace {

using namespace staged_detail;

constexpr uint32_t kEvery = 16;            // steps
constexpr uint32_t kSampledBlocks = 1024;  // blocks looked at, evenly spread

// The staged passes pay while at most `unfit` of the warps hold a particle without room, or, where the per-lane
// passes would overflow their lists, once more than `crowded` of them hold one with more than `candidates`.
// A sphere of the support radius holds 4 pi / 3 / 27 of its stencil's particles, so 598 candidates fill a list
// of kListCapacity at an even density.
// Staged / per lane, ms a step, at the shares on either side of each line:
//   forward, 262k: unfit 0.02 0.551 / 0.612, 0.18 0.731 / 0.668; crowded 0.01 1.920 / 1.799, 0.53 1.992 / 2.211
//   grouped, 14k: unfit 0.002 0.176 / 0.215, 0.07 0.275 / 0.232; more than 500 candidates (smaller scenes wait for
//     the few lists that the later iterations overflow): 0.12 0.428 / 0.391, 0.59 0.459 / 0.761
//   differentiable, 600k, which write both lists: unfit 0.02 1.089 / 1.144, 0.05 1.239 / 1.222; crowded 0.59
//     5.744 / 3.942, 0.82 6.276 / 9.115
//   SPH (PCISPH), 262k: unfit 0.02 0.890 / 0.931, 0.18 1.090 / 1.032; crowded ones fall back to the per-lane lists
struct Limits {
    uint32_t candidates;
    float unfit, crowded;
};
constexpr Limits kLimits[4] = {{598u, 1.0F / 16.0F, 0.5F}, {500u, 1.0F / 16.0F, 0.25F}, {598u, 1.0F / 32.0F, 0.7F},
                               {~0u, 1.0F / 16.0F, 1.0F}};

struct FitArgs {
    GatherCommon g;
    uint32_t particles, capacity, candidates, stride, tag;
    uint32_t* counts;   // unfit warps, crowded warps, warps, blocks done; zero before and after
    uint64_t* result;   // the tag and both shares, in units of 1 / 65535
};

__global__ void __launch_bounds__(kBlockParticles) staged_fit_kernel(const FitArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ uint32_t unfit_warps, crowded_warps;
    const uint32_t first = blockIdx.x * a.stride * a.particles;
    const uint32_t last = min(first + a.particles, a.g.count) - 1u;
    if (threadIdx.x == 0u) unfit_warps = crowded_warps = 0u;
    find_windows(w, a.g, first, last, a.capacity);
    __syncthreads();
    const uint32_t s = first + threadIdx.x;
    uint32_t longest = 0u, candidates = 0u;
    if (s <= last) {
        const int4 c = a.g.cell[s];
        const Grid& grid = a.g.scenes[c.w].grid;
        const int cx = static_cast<int>(grid.cells_x), cy = static_cast<int>(grid.cells_y), cz = static_cast<int>(grid.cells_z);
        const uint32_t z_lo = static_cast<uint32_t>(c.z > 0 ? c.z - 1 : 0);
        const uint32_t z_hi = static_cast<uint32_t>(c.z + 1 < cz ? c.z + 1 : cz - 1);
        for (int o = 0; o < 9; ++o) {
            const int x = c.x + o / 3 - 1, y = c.y + o % 3 - 1;
            if (x < 0 || x >= cx || y < 0 || y >= cy) continue;
            const uint32_t begin = a.g.cell_offsets[cell_index(grid, x, y, z_lo)];
            const uint32_t end = a.g.cell_offsets[cell_index(grid, x, y, z_hi) + 1u];
            if (begin >= end) continue;
            longest = max(longest, end - (begin & ~3u));
            candidates += end - begin;
        }
    }
    const bool unfit = __any_sync(kFull, s <= last && (w.staged == 0u || longest > kColumn));
    const bool crowded = __any_sync(kFull, candidates > a.candidates);
    if (lane_id() == 0u) {
        if (unfit) atomicAdd(&unfit_warps, 1u);
        if (crowded) atomicAdd(&crowded_warps, 1u);
    }
    __syncthreads();
    if (threadIdx.x != 0u) return;
    if (unfit_warps) atomicAdd(a.counts, unfit_warps);
    if (crowded_warps) atomicAdd(a.counts + 1, crowded_warps);
    atomicAdd(a.counts + 2, (last - first) / 32u + 1u);
    __threadfence();
    if (atomicAdd(a.counts + 3, 1u) != gridDim.x - 1u) return;
    __threadfence();
    const uint32_t total_unfit = atomicExch(a.counts, 0u), total_crowded = atomicExch(a.counts + 1, 0u);
    const uint32_t warps = atomicExch(a.counts + 2, 0u);
    atomicExch(a.counts + 3, 0u);
    *a.result = (static_cast<uint64_t>(a.tag) << 32) | ((total_unfit * 65535u / warps) << 16) | (total_crowded * 65535u / warps);
}

// Pinned words, one a solver, of one page that lives as long as the process; a solver beyond them measures
// nothing.
class PinnedWords {
public:
    uint64_t* take(uint32_t& tag) {
        const std::lock_guard<std::mutex> lock(mutex_);
        if (!tried_) {
            tried_ = true;
            void* page = nullptr;
            if (cudaHostAlloc(&page, kWords * sizeof(uint64_t), cudaHostAllocPortable | cudaHostAllocMapped) == cudaSuccess) {
                free_.reserve(kWords);
                for (uint32_t k = 0; k < kWords; ++k) {
                    static_cast<uint64_t*>(page)[k] = 0u;
                    free_.push_back(static_cast<uint64_t*>(page) + k);
                }
            } else {
                cudaGetLastError();
            }
        }
        if (free_.empty()) return nullptr;
        uint64_t* word = free_.back();
        free_.pop_back();
        if (++tag_ == 0u) ++tag_;
        tag = tag_;
        return word;
    }
    void give(uint64_t* word) {
        const std::lock_guard<std::mutex> lock(mutex_);
        free_.push_back(word);
    }

private:
    static constexpr uint32_t kWords = 512;
    std::mutex mutex_;
    std::vector<uint64_t*> free_;
    uint32_t tag_ = 0;
    bool tried_ = false;
};
PinnedWords& pinned_words() {
    static PinnedWords* words = new PinnedWords;   // outlives every solver
    return *words;
}

}  // namespace

StagedFit::~StagedFit() {
    if (word_) pinned_words().give(word_);
}

cudaError_t StagedFit::init(DeviceArena& arena, cudaStream_t stream, const Kind kind) {
    kind_ = kind;
    cudaError_t e = cudaSuccess;
    counts_ = arena.alloc<uint32_t>(4, e);
    if (e == cudaSuccess) e = cudaMemsetAsync(counts_, 0, 4 * sizeof(uint32_t), stream);
    if (e == cudaSuccess) word_ = pinned_words().take(tag_);
    return e;
}

cudaError_t StagedFit::measure(cudaStream_t stream, const GatherCommon& g) {
    if (!word_ || g.count == 0) return cudaSuccess;
    if (calls_ % kEvery != 0u) {
        ++calls_;
        return cudaSuccess;
    }
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(stream, &capture) != cudaSuccess || capture != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return cudaSuccess;   // at a later step
    }
    ++calls_;
    const uint32_t particles = kind_ == kGrouped ? kGroupParticles : kBlockParticles;
    const uint32_t blocks = (g.count + particles - 1u) / particles;
    const uint32_t stride = std::max(1u, blocks / kSampledBlocks);
    launch_after(stream, staged_fit_kernel, (blocks + stride - 1u) / stride, particles,
                 FitArgs{g, particles, kind_ == kGrouped ? kGroupStage : kStage, kLimits[kind_].candidates, stride, tag_, counts_, word_});
    count_launch();
    return cudaGetLastError();
}

bool StagedFit::pays() const {
    if (!word_) return true;
    const uint64_t word = *static_cast<const volatile uint64_t*>(word_);
    if (static_cast<uint32_t>(word >> 32) != tag_) return true;   // not measured yet
    const float unfit = static_cast<float>((word >> 16) & 0xffffu) / 65535.0F;
    const float crowded = static_cast<float>(word & 0xffffu) / 65535.0F;
    return unfit <= kLimits[kind_].unfit || crowded > kLimits[kind_].crowded;
}

}  // namespace pbf
