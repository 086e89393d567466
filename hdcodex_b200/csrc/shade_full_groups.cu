// shade_full_groups.cu - shade variants of the whole closure, entries of several lanes.
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

void shadeFullGroups(bool lit, const ShadeLaunch& l)
{
    if (lit) launch<3, true, true, false, kWalkDefer>(l);
    else launch<3, true, false, false, kWalkDefer>(l);
}

}  // namespace hdcx
