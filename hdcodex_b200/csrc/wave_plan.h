// wave_plan.h - device memory of a wave's path state. Host-only and free of
// CUDA, so that the rule is unit-tested on the CPU (tests/cpp/wave_plan_tests.cpp).
#pragma once

#include <algorithm>
#include <cstdint>

namespace hdcx {

// Device bytes of path state per path (PathStore::allocate): records of a
// group of three lanes (light, state, spectrum); ray, medium and hit; six
// queues of 32-bit entries, one of them for half the paths; the deferred
// subsurface walks; the ray cone; per shadow slot a ray, its factors and its
// description.
constexpr uint64_t kShadowSlots = 3;
constexpr uint64_t kPathStateBytes =
    (48 + 48 + 64 + 2) / 3 + (32 + 16 + 16) + (5 * 4 + 2) + 3 * 16 + 8 + kShadowSlots * (32 + 16 + 4);

// Smallest wave an automatic wave is shrunk to when device memory is short.
constexpr uint64_t kMinimumAutomaticWave = 1ull << 16;

// An automatic wave of `wave` paths, bounded so that its path state takes at
// most three quarters of the free memory and what `heldPaths` paths of path
// state hold already. Held buffers serve as they are.
inline uint64_t boundedWave(uint64_t wave, uint64_t freeBytes, uint64_t heldPaths)
{
    const uint64_t fit = std::max((freeBytes + heldPaths * kPathStateBytes) / 4 * 3 / kPathStateBytes, heldPaths);
    return std::min(wave, std::max(fit, std::min(wave, kMinimumAutomaticWave)));
}

}  // namespace hdcx
