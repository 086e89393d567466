// shade_full_replays_lit.cu - shade variants that re-shade failed subsurface walks (lit scenes).
#include "device/shade.cuh"
#include "shade.h"

namespace hdcx {

namespace {

template <int kLanes, bool kFull, bool kLit, bool kCache, int kWalk>
void launch(const ShadeLaunch& l)
{
    shadeKernel<kLanes, kFull, kLit, kCache, kWalk><<<l.grid, 128, 0, l.stream>>>(l.scene, l.frame, l.paths, l.bounce, l.queue,
                                                                                  l.count, l.nextQueue, l.nextCount);
}

}  // namespace

void shadeFullReplaysLit(bool cache, const ShadeLaunch& l)
{
    if (cache) launch<1, true, true, true, kWalkReplay>(l);
    else launch<1, true, true, false, kWalkReplay>(l);
}

}  // namespace hdcx
