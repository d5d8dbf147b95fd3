// The measurement behind staged_fit.h.
#include <algorithm>
#include <bitset>
#include <cstdlib>
#include <cstring>
#include <mutex>

#include "dependent_launch.cuh"
#include "engine.h"
#include "staged.cuh"
#include "staged_fit.h"

namespace pbf {

namespace {

using namespace staged_detail;

// Blocks of the measurement's kernel: about as many as are resident at once, since each ends with an atomic on one word.
constexpr uint32_t kMaxBlocks = 2048;
// Steps from one measurement to the next.  A measurement takes 8 us at 5k particles and 10 at 262k, a step 0.09 and 0.5 ms; a
// differentiable one (2^19 particles or more) 24 us at 1M, a step 1 ms and up.
constexpr uint32_t kEvery[5] = {8, 16, 4, 16, 16};

// The staged passes pay while few of the warps hold a particle without room: at most `columns` of them one whose
// stencil columns outgrow its hit record, which leaves its warp waiting in every pass, and at most `unfit` one
// of either kind (a block whose windows outgrow the stage costs its own time only).  Where the per-lane passes keep
// lists of slots (grouped and differentiable steps) the staged ones also pay, up to half of the warps, if any
// particle has more than `candidates`: it overflows its list, and its stencil walk takes as long as the rest of its
// scene; and above, once `crowded` of the warps hold one.  A sphere of the support radius holds 4 pi / 3 / 27 of its stencil's
// particles, so 598 candidates fill a list of kListCapacity at an even density; small scenes wait for the few lists that
// later iterations overflow, and count from 500 (480) on.
// Staged / per lane, ms a step (lattices by the spacings in a radius; dam breaks by the step; shares of columns, all):
//   forward: 262k 2.1 (0.02, 0.02) 0.547 / 0.596, 2.15 (0.18, 0.18) 0.730 / 0.651, step 20 (0.08, 0.12) 0.929 / 0.864; 1M step 30
//     (0.11, 0.14) 4.90 / 5.04, step 100 (0.04, 0.14) 4.37 / 4.32; 256 scenes step 20 (0.01, 0.09) 8.62 / 9.91, 40 (0.10, 0.26) 10.73 / 9.88
//   grouped, 14k: 2.1 (0, 0) 0.176 / 0.215, 2.15 (0.07, 0.07) 0.275 / 0.232; step 100 (0, 0.14) 0.235 / 0.251; crowded 0.12
//     0.428 / 0.391, 0.59 0.459 / 0.761
//   differentiable, which write both lists: 32 scenes step 20 (0.02, 0.07) 5.74 / 5.96, step 2 (0, 0.22) 5.61 / 4.93; 600k
//     2.1 (0.05, 0.05) 1.239 / 1.222, 2.15 (0.2, 0.2) 1.634 / 1.327; crowded 0.59 5.744 / 3.942, 0.82 6.276 / 9.115
//   SPH (PCISPH), 262k: 2.1 (0.02, 0.02) 0.890 / 0.931, 2.15 (0.18, 0.18) 1.090 / 1.032; crowded ones fall back to the
//     per-lane lists
// In between, hit masks / lists of slots: 60k 2.6 (crowded 0.2) 0.487 / 0.471, 2.7 (0.6) 0.511 / 0.696, 3 0.669 / 2.116.
struct Limits {
    uint32_t candidates;
    float columns, unfit, crowded;
};
constexpr Limits kLimits[5] = {{~0u, 0.1F, 0.13F, 1.0F}, {500u, 0.03F, 0.2F, 0.25F}, {598u, 0.1F, 0.1F, 0.7F},
                               {~0u, 0.06F, 0.15F, 1.0F}, {480u, 0.0F, 0.0F, 1.0F}};
constexpr float kCrowdedUnfit = 0.5F;

enum Share { kColumns, kUnfit, kCrowded, kShares };

struct FitArgs {
    GatherCommon g;
    uint32_t blocks, stride, capacity, candidates, tag;   // every stride-th block
    uint32_t* counts;   // warps of each share, then blocks done; zero before and after
    uint64_t* result;   // the tag and the shares, 16 bits each, in units of 1 / 65535, rounded up
};

__global__ void __launch_bounds__(kBlockParticles) staged_fit_kernel(const FitArgs a) {
    after_predecessor();
    __shared__ Windows w;
    __shared__ uint32_t warps[kShares];
    if (threadIdx.x < kShares) warps[threadIdx.x] = 0u;
    for (uint32_t block = blockIdx.x; block < a.blocks; block += gridDim.x) {
        const uint32_t first = block * a.stride * blockDim.x;
        const uint32_t last = min(first + blockDim.x, a.g.count) - 1u;
        __syncthreads();
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
        const bool columns = __any_sync(kFull, longest > kColumn);
        const bool unfit = __any_sync(kFull, s <= last && (w.staged == 0u || longest > kColumn));
        const bool crowded = __any_sync(kFull, candidates > a.candidates);
        if (lane_id() == 0u) {
            if (columns) atomicAdd(&warps[kColumns], 1u);
            if (unfit) atomicAdd(&warps[kUnfit], 1u);
            if (crowded) atomicAdd(&warps[kCrowded], 1u);
        }
    }
    __syncthreads();
    if (threadIdx.x != 0u) return;
    for (int k = 0; k < kShares; ++k)
        if (warps[k]) atomicAdd(a.counts + k, warps[k]);
    __threadfence();
    if (atomicAdd(a.counts + kShares, 1u) != gridDim.x - 1u) return;
    __threadfence();
    const float unit = 65535.0F * static_cast<float>(a.stride) / static_cast<float>((a.g.count + 31u) / 32u);
    uint64_t result = static_cast<uint64_t>(a.tag) << 48;
    for (int k = 0; k < kShares; ++k)
        result |= static_cast<uint64_t>(min(__float2uint_ru(static_cast<float>(atomicExch(a.counts + k, 0u)) * unit), 65535u)) << (16 * k);
    atomicExch(a.counts + kShares, 0u);
    *a.result = result;
}

// Pinned words, one a solver, in one page a CUDA context.  A page is host memory that is registered with its context and
// kept, so a solver may read its word even after that context is gone (cudaDeviceReset).  A solver beyond
// the words or pages there are measures nothing.
class PinnedWords {
public:
    struct Word {
        uint64_t* host = nullptr;
        uint64_t* device = nullptr;
        uint32_t slot = 0, tag = 0;
    };
    Word take() {
        unsigned long long context = 0;
        if (current_context_id(&context) || context == 0) return {};
        const std::lock_guard<std::mutex> lock(mutex_);
        uint32_t p = 0;
        while (p < used_ && pages_[p].context != context) ++p;
        if (p == used_ && !add_page(context)) return {};
        Page& page = pages_[p];
        for (uint32_t k = 0; k < kWords; ++k) {
            if (page.taken[k]) continue;
            page.taken[k] = true;
            if (++tag_ == 0x10000u) tag_ = 1u;
            return {page.host + k, page.device + k, p * kWords + k, tag_};
        }
        return {};
    }
    void give(const uint32_t slot) {
        const std::lock_guard<std::mutex> lock(mutex_);
        pages_[slot / kWords].taken[slot % kWords] = false;
    }

private:
    static constexpr uint32_t kWords = 512, kPages = 16;
    struct Page {
        unsigned long long context = 0;
        uint64_t* host = nullptr;
        uint64_t* device = nullptr;
        std::bitset<kWords> taken;
    };
    bool add_page(const unsigned long long context) {
        if (used_ == kPages) return false;
        void* host = std::aligned_alloc(4096, kWords * sizeof(uint64_t));
        if (!host) return false;
        std::memset(host, 0, kWords * sizeof(uint64_t));
        // another thread may be capturing
        cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
        cudaThreadExchangeStreamCaptureMode(&mode);
        void* device = nullptr;
        cudaError_t e = cudaHostRegister(host, kWords * sizeof(uint64_t), cudaHostRegisterMapped);
        if (e == cudaSuccess && (e = cudaHostGetDevicePointer(&device, host, 0)) != cudaSuccess) cudaHostUnregister(host);
        cudaThreadExchangeStreamCaptureMode(&mode);
        if (e != cudaSuccess) {
            cudaGetLastError();
            std::free(host);
            return false;
        }
        pages_[used_].context = context;
        pages_[used_].host = static_cast<uint64_t*>(host);
        pages_[used_].device = static_cast<uint64_t*>(device);
        ++used_;
        return true;
    }
    std::mutex mutex_;
    Page pages_[kPages];
    uint32_t used_ = 0, tag_ = 0;
};
PinnedWords& pinned_words() {
    static PinnedWords* words = new PinnedWords;   // outlives every solver
    return *words;
}

}  // namespace

StagedFit::~StagedFit() {
    if (word_) pinned_words().give(slot_);
}

cudaError_t StagedFit::init(DeviceArena& arena, cudaStream_t stream, const Kind kind) {
    kind_ = kind;
    cudaError_t e = cudaSuccess;
    counts_ = arena.alloc<uint32_t>(kShares + 1, e);
    if (e == cudaSuccess) e = cudaMemsetAsync(counts_, 0, (kShares + 1) * sizeof(uint32_t), stream);
    if (e != cudaSuccess) return e;
    const PinnedWords::Word word = pinned_words().take();
    word_ = word.host;
    device_word_ = word.device;
    slot_ = word.slot;
    tag_ = word.tag;
    return cudaSuccess;
}

cudaError_t StagedFit::measure(cudaStream_t stream, const GatherCommon& g) {
    if (!word_ || g.count == 0) return cudaSuccess;
    if (calls_ % kEvery[kind_] != 0u) {
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
    // every block where one crowded particle decides, a sample otherwise
    const uint32_t all = (g.count + particles - 1u) / particles;
    const uint32_t stride = kLimits[kind_].candidates == ~0u ? std::max(1u, all / 1024u) : 1u;
    const uint32_t blocks = (all + stride - 1u) / stride;
    launch_after(stream, staged_fit_kernel, std::min(blocks, kMaxBlocks), particles,
                 FitArgs{g, blocks, stride, kind_ == kGrouped ? kGroupStage : kStage, kLimits[kind_].candidates, tag_, counts_, device_word_});
    count_launch();
    return cudaGetLastError();
}

uint64_t StagedFit::measured() const {
    if (!word_) return 0u;
    const uint64_t word = *static_cast<const volatile uint64_t*>(word_);
    return static_cast<uint32_t>(word >> 48) == tag_ ? word : 0u;   // otherwise another solver's
}

namespace {
float share_of(const uint64_t word, const Share k) { return static_cast<float>((word >> (16 * k)) & 0xffffu) / 65535.0F; }
}  // namespace

bool StagedFit::pays() const {
    const uint64_t word = measured();
    if (word == 0u) return true;
    const Limits& limits = kLimits[kind_];
    const float unfit = share_of(word, kUnfit), crowded = share_of(word, kCrowded);
    return (share_of(word, kColumns) <= limits.columns && unfit <= limits.unfit) || (crowded > 0.0F && unfit <= kCrowdedUnfit) ||
           crowded > limits.crowded;
}

bool StagedFit::crowded() const { return share_of(measured(), kCrowded) > 0.0F; }

}  // namespace pbf
