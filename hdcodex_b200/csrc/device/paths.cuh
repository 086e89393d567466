// paths.cuh - path groups: the device view of a wave's queues and path state.
//
// A wave holds the paths of whole samples, so path slots come in threes: slot
// 3 g + lane is wavelength lane `lane` of group g (one sample of one pixel).
// The lanes of a group that are still on the same path (same ray, same random
// state) travel as one queue entry: (g << 3) | lane mask. What they share (ray,
// random state, flags, hit, ray cone) is kept at the slot of the entry's first
// lane, its leader; what depends on the wavelength (throughput, radiance,
// previous pdfs, light samples, spectrum) in records of the group, the medium
// at each lane's own slot. Where lanes part, the entry becomes several, each
// with its own leader.
#pragma once

#include "../integrator.h"
#include "common.cuh"

namespace hdcx {

constexpr uint32_t kFlagEnvironmentOnMiss = 1u;
constexpr uint32_t kFlagPreviousWasDelta = 2u;
constexpr uint32_t kFlagInsideMedium = 4u;
constexpr uint32_t kFlagTraining = 8u;  // radiance-cache mode: a full-length training path

enum ShadowKind : uint32_t {
    kShadowAnalytic = 0,
    kShadowSun = 1,
    kShadowSky = 2,
    kShadowMesh = 3,
};
// PathBuffers::shadowInfo: kind | light-sample slot << 2 | kShadowGeneral | light << 8.
// kShadowGeneral: what a blocked ray leaves is not plainly zero (a shadow
// colour, a falloff, a factor that is not finite); the factors are stored.
constexpr uint32_t kShadowGeneral = 16u;

HDCX_D uint32_t firstLane(uint32_t mask) { return static_cast<uint32_t>(__ffs(mask)) - 1u; }
HDCX_D uint32_t entryLeader(uint32_t entry) { return (entry >> 3) * 3u + firstLane(entry & 7u); }

// Warp-aggregated appends: one atomic for the threads that arrive together.
// Written with the warp intrinsics: cooperative_groups' coalesced group packs
// ballots and searches set bits in software, which was a fifth of the shade
// kernel's code (144 KB of instructions with it, see shade.cuh).
HDCX_D uint32_t appendIndex(uint32_t* counter)
{
    const uint32_t together = __activemask();
    const uint32_t leader = firstLane(together);
    uint32_t lane;
    asm("mov.u32 %0, %%laneid;" : "=r"(lane));
    uint32_t base = 0;
    if (lane == leader) base = atomicAdd(counter, static_cast<uint32_t>(__popc(together)));
    base = __shfl_sync(together, base, static_cast<int>(leader));
    return base + static_cast<uint32_t>(__popc(together & ((1u << lane) - 1u)));
}

// Appends an entry of the lanes in `mask`: entries are counted in the
// counter's low half, lanes (the rays of the statistics) in the high half.
HDCX_D uint32_t appendEntry(unsigned long long* counter, uint32_t mask)
{
    const uint32_t together = __activemask();
    const uint32_t leader = firstLane(together);
    uint32_t lane;
    asm("mov.u32 %0, %%laneid;" : "=r"(lane));
    const uint32_t lanes = __popc(__ballot_sync(together, (mask & 1u) != 0u)) + __popc(__ballot_sync(together, (mask & 2u) != 0u)) +
                           __popc(__ballot_sync(together, (mask & 4u) != 0u));
    uint32_t base = 0;
    if (lane == leader)
        base = static_cast<uint32_t>(atomicAdd(counter, static_cast<unsigned long long>(__popc(together)) | (static_cast<unsigned long long>(lanes) << 32)));
    base = __shfl_sync(together, base, static_cast<int>(leader));
    return base + static_cast<uint32_t>(__popc(together & ((1u << lane) - 1u)));
}

// PathBuffers::laneLight and laneState: the per-lane state of a group in
// records of three lanes to a field, so that an entry scattered anywhere in
// the wave costs few memory sectors, and vector accesses when it holds all
// lanes. What the light sample completes (laneLight) is written before what
// the BSDF sample does.
enum : uint32_t {
    kLaneRadiance = 0,    // laneLight
    kLaneLight = 3,       // + 3 j: light-sample slot j: the value it adds at the next vertex, zero where there is none
    kLaneThroughput = 0,  // laneState
    kLaneBsdfPdf = 3,     // previousBsdfPdf
    kLaneLightPdf = 6,    // previousEnvironmentLightPdf
};
// A scene whose light samples use one slot takes two float4, others three
// (with slots 1 and 2 in an array of their own, the shade stage of a 301x199
// 8 spp box with a mesh light took 0.80 ms instead of 0.56).
HDCX_D float* lightRecord(const PathBuffers& p, uint32_t group)
{
    return reinterpret_cast<float*>(p.laneLight + (p.lightSlots > 1u ? 3u : 2u) * static_cast<size_t>(group));
}
HDCX_D float* laneRecord(const PathBuffers& p, uint32_t group) { return reinterpret_cast<float*>(p.laneState + 3u * static_cast<size_t>(group)); }
HDCX_D const float* spectrumRecord(const PathBuffers& p, uint32_t group)
{
    return reinterpret_cast<const float*>(p.laneSpectrum + 4u * static_cast<size_t>(group));
}

}  // namespace hdcx
