// shade_full_singles_unlit.cu - shade variants of the whole closure, entries of one lane (unlit scenes).
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

void shadeFullSinglesUnlit(bool cache, bool defer, const ShadeLaunch& l)
{
    if (cache) {
        if (defer) launch<1, true, false, true, kWalkDefer>(l);
        else launch<1, true, false, true, kWalkInline>(l);
    } else if (defer) {
        launch<1, true, false, false, kWalkDefer>(l);
    } else {
        launch<1, true, false, false, kWalkInline>(l);
    }
}

}  // namespace hdcx
