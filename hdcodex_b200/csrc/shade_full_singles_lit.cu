// shade_full_singles_lit.cu - shade variants of the whole closure, entries of one lane (lit scenes).
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

void shadeFullSinglesLit(bool cache, bool defer, const ShadeLaunch& l)
{
    if (cache) {
        if (defer) launch<1, true, true, true, kWalkDefer>(l);
        else launch<1, true, true, true, kWalkInline>(l);
    } else if (defer) {
        launch<1, true, true, false, kWalkDefer>(l);
    } else {
        launch<1, true, true, false, kWalkInline>(l);
    }
}

}  // namespace hdcx
