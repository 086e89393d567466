// shade.h - launches of the shade kernel's variants (device/shade.cuh), which
// are compiled in translation units of their own (shade_*.cu).
#pragma once

#include "integrator.h"

namespace hdcx {

struct ShadeVariant {
    bool full;   // DeviceScene::fullShading
    bool lit;    // analytic or dome lights and no emissive triangles
    bool cache;  // radiance-cache mode
    bool defer;  // subsurface walks go to walkKernel
};

struct ShadeLaunch {
    const DeviceScene& scene;
    const FrameConst& frame;
    const PathBuffers& paths;
    uint32_t bounce;
    const uint32_t* queue;
    const uint32_t* count;
    uint32_t* nextQueue;
    unsigned long long* nextCount;
    bool misses;  // this launch also shades the bounce's miss queue
    int grid;
    cudaStream_t stream;
};

// Entries of several lanes (never in cache mode), entries of one lane, and
// re-shading of failed deferred walks.
void launchShadeGroups(const ShadeVariant& v, const ShadeLaunch& l);
void launchShadeSingles(const ShadeVariant& v, const ShadeLaunch& l);
void launchShadeReplays(const ShadeVariant& v, const ShadeLaunch& l);

// By translation unit.
void shadePlainGroups(bool lit, const ShadeLaunch& l);
void shadePlainSingles(bool lit, bool cache, const ShadeLaunch& l);
void shadeFullGroups(bool lit, const ShadeLaunch& l);
void shadeFullSinglesLit(bool cache, bool defer, const ShadeLaunch& l);
void shadeFullSinglesUnlit(bool cache, bool defer, const ShadeLaunch& l);
void shadeFullReplaysLit(bool cache, const ShadeLaunch& l);
void shadeFullReplaysUnlit(bool cache, const ShadeLaunch& l);

}  // namespace hdcx
