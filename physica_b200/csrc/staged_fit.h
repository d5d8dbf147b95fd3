// Whether a scene's particles fit the staged passes (staged.cuh), measured on the device now and then.
//
// The windows and hit records of the staged passes have room for about 10 particles a cell, support radii of
// 2.15 spacings.  A particle or block without room falls back inside the staged kernels, and where many do,
// scanning in vain and warps that wait for their slowest lane cost more than the per-lane passes take
// altogether: staged / per lane at 262k particles, ms a step of three iterations, 0.502 / 0.569 at a radius of 2
// spacings, 0.551 / 0.612 at 2.1, 0.731 / 0.668 at 2.15, 0.840 / 0.722 at 2.2, 1.531 / 1.031 at 2.4, 1.820 / 1.245 at 2.6.
// From 2.8 spacings on the per-lane lists overflow (1.992 / 2.211, and 2.445 / 4.766 at 3).  How dense the particles are
// is known on the device only, so every 4th to 16th step ends with a small kernel that looks at its cell offsets and
// leaves three shares in pinned host memory, and later steps are routed by them: nothing waits, and both routes
// give the same bits.  Until a first measurement has arrived a solver takes the staged passes.
#pragma once

#include <cstdint>

#include "pbf_launch.h"

namespace pbf {

class DeviceArena;

class StagedFit {
public:
    // kGrouped: four lanes a particle; kMiddle: sizes that never run staged passes
    enum Kind { kForward, kGrouped, kDifferentiable, kSph, kMiddle };

    StagedFit() = default;
    StagedFit(const StagedFit&) = delete;
    StagedFit& operator=(const StagedFit&) = delete;
    ~StagedFit();
    // Without pinned memory nothing is ever measured.
    cudaError_t init(DeviceArena& arena, cudaStream_t stream, Kind kind);
    // Call after each step that may run staged passes.  Launches nothing into a capture.
    cudaError_t measure(cudaStream_t stream, const GatherCommon& g);
    // Whether the staged passes are the faster ones.
    bool pays() const;
    // Whether particles are so crowded that the per-lane passes' lists of slots overflow.
    bool crowded() const;

private:
    uint64_t measured() const;          // 0: nothing yet
    uint32_t* counts_ = nullptr;        // device scratch
    const uint64_t* word_ = nullptr;    // pinned: a tag and the shares measured
    uint64_t* device_word_ = nullptr;   // the same for the device
    uint32_t slot_ = 0;                 // its place among the pinned words
    uint32_t tag_ = 0;                  // of this object: a word is used again after its solver is gone
    uint32_t calls_ = 0;
    Kind kind_ = kForward;
};

}  // namespace pbf
