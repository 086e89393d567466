// shade_plain_singles.cu - shade variants of scenes without textures and layered lobes, entries of one lane.
#include "device/shade.cuh"
#include "shade.h"

namespace hdcx {

namespace {

template <int kLanes, bool kFull, bool kLit, bool kCache, int kWalk>
void launch(const ShadeLaunch& l)
{
    constexpr int kThreads = shadeThreads<kLanes, kFull>();
    const int grid = (l.grid * 128 + kThreads - 1) / kThreads;
    shadeKernel<kLanes, kFull, kLit, kCache, kWalk><<<grid, kThreads, 0, l.stream>>>(l.scene, l.frame, l.paths, l.bounce, l.queue,
                                                                                  l.count, l.nextQueue, l.nextCount, l.misses);
}

}  // namespace

void shadePlainSingles(bool lit, bool cache, const ShadeLaunch& l)
{
    if (cache) {
        if (lit) launch<1, false, true, true, kWalkInline>(l);
        else launch<1, false, false, true, kWalkInline>(l);
    } else if (lit) {
        launch<1, false, true, false, kWalkInline>(l);
    } else {
        launch<1, false, false, false, kWalkInline>(l);
    }
}

}  // namespace hdcx
