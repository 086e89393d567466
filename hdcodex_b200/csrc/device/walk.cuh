// walk.cuh - the subsurface random walk (vulkan_path_tracer.cpp:1130-1186).
#pragma once

#include "paths.cuh"
#include "shading.cuh"
#include "traverse.cuh"

namespace hdcx {
namespace {

// A walk under way: one boundary ray per step, at most kWalkSteps of them.
constexpr int kWalkSteps = 8;
struct SubsurfaceWalk {
    float3 origin, direction;
    float sigmaS, sigmaA, anisotropy;
    float attenuation;
    uint32_t rng;
    int step;
};

enum : int { kWalkContinues = 0, kWalkExits = 1, kWalkFails = 2 };

HDCX_D SubsurfaceWalk beginWalk(float3 entry, float3 outwardNormal, float meanFreePath, float albedo, float anisotropy, uint32_t rng)
{
    // :1153-1160
    SubsurfaceWalk w;
    const float radius = gmax(meanFreePath, 0.001f);
    w.sigmaS = 1.0f / radius;
    w.sigmaA = -glog(clampf(albedo, 0.001f, 0.9999f)) / radius;
    w.origin = entry - outwardNormal * 0.003f;
    w.rng = rng;
    w.direction = cosineHemisphere(-outwardNormal, w.rng);
    w.anisotropy = anisotropy;
    w.attenuation = 1.0f;
    w.step = 0;
    return w;
}

// One step (:1161-1186): the boundary ray (:1130-1151; an escaping one ends
// the walk), then a scattering event or the exit, whose ray is left in
// origin and direction.
template <int kInst = -1>
__device__ __forceinline__ int stepWalk(const DeviceScene& s, SubsurfaceWalk& w, uint32_t& fault)
{
    HitRecord h;
    uint32_t rng = w.rng;
    const float scatterDistance = -glog(gmax(1.0f - randomFloat(rng), 1e-6f)) / w.sigmaS;
    const bool forceExit = w.step == kWalkSteps - 1;
    // The boundary's distance counts only up to the scattering event's: beyond
    // it, that there is a boundary is enough (shading stage of a 1280x720 8 spp
    // scene with subsurface objects: 23.4 -> 22.6 ms).
    if (!traceRay<Accept::Boundary, false, false, kInst>(s, w.origin, w.direction, 0.001f, 10000.0f, 0u, h, fault, nullptr,
                                                        forceExit ? INFINITY : scatterDistance))
        return kWalkFails;
    w.rng = rng;
    const float boundaryDistance = h.t;
    const float travel = forceExit ? boundaryDistance : gmin(scatterDistance, boundaryDistance);
    w.attenuation = w.attenuation * gexp(-w.sigmaA * travel);
    if (forceExit || scatterDistance >= boundaryDistance) {
        w.origin = (w.origin + w.direction * boundaryDistance) + w.direction * 0.003f;
        return kWalkExits;
    }
    w.origin = w.origin + w.direction * scatterDistance;
    w.direction = sampleHenyeyGreenstein(w.direction, w.anisotropy, w.rng);
    ++w.step;
    return kWalkContinues;
}

// A whole walk in one call, for renders without walk buffers.
__device__ inline bool randomWalkSubsurface(const DeviceScene& s, PathBuffers& p, float3 entry, float3 outwardNormal,
                                            float meanFreePath, float albedo, float anisotropy, uint32_t& state,
                                            float3& exitOrigin, float3& exitDirection, float& attenuation)
{
    SubsurfaceWalk w = beginWalk(entry, outwardNormal, meanFreePath, albedo, anisotropy, state);
    uint32_t fault = 0u;
    int result;
    do {
        result = stepWalk(s, w, fault);
    } while (result == kWalkContinues);
    atomicAdd(p.stats + 2, static_cast<unsigned long long>(w.step + 1));
    if (fault != 0u) atomicOr(reinterpret_cast<unsigned int*>(p.stats + 7), fault);
    state = w.rng;
    exitOrigin = w.origin;
    exitDirection = w.direction;
    attenuation = w.attenuation;
    return result == kWalkExits;
}

}  // namespace
}  // namespace hdcx
