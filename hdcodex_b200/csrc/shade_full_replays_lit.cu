// shade_full_replays_lit.cu - shade variants that re-shade failed subsurface walks (lit scenes).
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

void shadeFullReplaysLit(bool cache, const ShadeLaunch& l)
{
    if (cache) launch<1, true, true, true, kWalkReplay>(l);
    else launch<1, true, true, false, kWalkReplay>(l);
}

}  // namespace hdcx
