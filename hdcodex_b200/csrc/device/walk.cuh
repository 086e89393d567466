// walk.cuh - the subsurface random walk (vulkan_path_tracer.cpp:1130-1186).
#pragma once

#include "paths.cuh"
#include "shading.cuh"
#include "traverse.cuh"

namespace hdcx {
namespace {

template <int kInst = -1>
__device__ bool traceOpaqueBoundary(const DeviceScene& s, PathBuffers& p, float3 origin, float3 direction,
                                    float3& boundary, float3& boundaryNormal, float& boundaryDistance)
{
    // :1130-1151
    atomicAdd(p.stats + 2, 1ull);
    HitRecord h;
    uint32_t fault = 0u;
    const bool found = traceRay<Accept::Opaque, false, false, kInst>(s, origin, direction, 0.001f, 10000.0f, 0u, h, fault);
    if (fault != 0u) atomicOr(reinterpret_cast<unsigned int*>(p.stats + 7), fault);
    if (!found) return false;
    const uint32_t primitive = h.primitive;
    const float3 p0 = xyz(__ldg(s.vertices + __ldg(s.indices + primitive * 3u + 0u)));
    const float3 p1 = xyz(__ldg(s.vertices + __ldg(s.indices + primitive * 3u + 1u)));
    const float3 p2 = xyz(__ldg(s.vertices + __ldg(s.indices + primitive * 3u + 2u)));
    boundaryDistance = h.t;
    boundary = origin + direction * boundaryDistance;
    boundaryNormal = normalize(cross(p1 - p0, p2 - p0));
    if (dot(boundaryNormal, direction) > 0.0f) boundaryNormal = -boundaryNormal;
    return true;
}

template <int kInst = -1>
__device__ bool randomWalkSubsurface(const DeviceScene& s, PathBuffers& p, float3 entry, float3 outwardNormal,
                                     float meanFreePath, float albedo, float anisotropy, uint32_t& state,
                                     float3& exitOrigin, float3& exitDirection, float& attenuation)
{
    // :1153-1186
    const float radius = gmax(meanFreePath, 0.001f);
    const float sigmaS = 1.0f / radius;
    const float sigmaA = -glog(clampf(albedo, 0.001f, 0.9999f)) / radius;
    float3 origin = entry - outwardNormal * 0.003f;
    float3 direction = cosineHemisphere(-outwardNormal, state);
    attenuation = 1.0f;
    for (int step = 0; step < 8; ++step) {
        float3 boundary, boundaryNormal;
        float boundaryDistance;
        if (!traceOpaqueBoundary<kInst>(s, p, origin, direction, boundary, boundaryNormal, boundaryDistance)) return false;
        const float scatterDistance = -glog(gmax(1.0f - randomFloat(state), 1e-6f)) / sigmaS;
        const bool forceExit = step == 7;
        const float travel = forceExit ? boundaryDistance : gmin(scatterDistance, boundaryDistance);
        attenuation = attenuation * gexp(-sigmaA * travel);
        if (forceExit || scatterDistance >= boundaryDistance) {
            exitDirection = direction;
            exitOrigin = boundary + direction * 0.003f;
            return true;
        }
        origin = origin + direction * scatterDistance;
        direction = sampleHenyeyGreenstein(direction, anisotropy, state);
    }
    return false;
}

}  // namespace
}  // namespace hdcx
