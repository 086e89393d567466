// shade.cuh - the shade kernel: one bounce of every path whose ray hit
// (emission, medium, material, light samples, BSDF sample, roulette;
// vulkan_path_tracer.cpp:1245-1879). Included by one translation unit per
// group of variants (shade_*.cu).
#pragma once

#include "paths.cuh"
#include "shading.cuh"
#include "walk.cuh"

#include <type_traits>

namespace hdcx {
namespace {

// ---------------------------------------------------------------------------
// shadeKernel<kLanes, kFull, kLit, kCache, kWalk>
//
// kLanes: 1 shades entries of one lane; 3 entries of several lanes, one
// thread per entry: geometry, textures, light and BSDF directions are computed
// once for the lanes, spectral values per lane (Lanes3). Where a decision
// parts the lanes, the rest of the bounce runs once per part. An entry this
// form does not take (a scattering medium, whose flight distances differ by
// lane) is split into single-lane hits, which the one-lane kernel shades
// after it.
//   Shading was bound by memory latency and instruction issue with one thread
//   per lane; see the measurements beside the launch bounds.
//
// kFull = false serves scenes whose materials bind no textures and have no
// coat, sheen, transmission, subsurface or diffuse-transmission weight and use
// the Lambert diffuse model (DeviceScene::fullShading == 0): there those
// quantities are the constants the general kernel computes for them (fallback
// values, zero weights), so both kernels return the same bits and the
// specialised one carries far less code and state.
// ---------------------------------------------------------------------------
template <bool kFull>
HDCX_D float4 materialTexture(float lodBase, const DeviceScene& s, uint32_t index, float2 uv, float4 fallback)
{
    if (!kFull) return fallback;
    return sampleMaterialTexture(s, index, uv, fallback, lodBase);
}

// Light-sample visibility that needs no ray: shadowVisibility's early returns
// (vulkan_path_tracer.cpp:858-861) give vec3(1.0).
HDCX_D bool analyticNeedsRay(const GpuLight& light, float maximumDistance, float& traceDistance)
{
    if (light.shadow.x < 0.5f) return false;
    traceDistance = maximumDistance;
    if (light.shadow.y >= 0.0f) traceDistance = gmin(traceDistance, light.shadow.y);
    return !(traceDistance <= 0.001f);
}

// Analytic/sun/sky sample: value = contribution with visibility sv.
template <class V>
HDCX_D V combineShadow(uint32_t kind, V a, V sv, V g1, V g2, V g3)
{
    if (kind == kShadowAnalytic) return overLikelyOne(a * sv * g1 * g2, g3);
    if (kind == kShadowSun) return a * sv;
    return a * sv * g1;  // sky
}

// Appends the shadow ray that lanes `lanes` of `group` share for light-sample
// slot j.
HDCX_D void emitShadow(PathBuffers& p, uint32_t group, uint32_t lanes, uint32_t info, float3 origin, float3 direction, float tmax)
{
    const uint32_t i = appendEntry(reinterpret_cast<unsigned long long*>(p.counters + kCountShadow), lanes);
    p.shadowRay[2u * i] = make_float4(origin.x, origin.y, origin.z, tmax);
    p.shadowRay[2u * i + 1u] = make_float4(direction.x, direction.y, direction.z, __uint_as_float((group << 3) | lanes));
    p.shadowInfo[i] = info;
}

// Environment on a miss (vulkan_path_tracer.cpp:1245-1255) of an entry's lanes,
// looked up once. All loads come before the stores: lanes that loaded after a
// neighbour's store to the same sector took ten times as long.
HDCX_D void shadeMiss(const DeviceScene& s, const FrameConst& f, const PathBuffers& p, uint32_t entry, uint32_t lightSlots)
{
    const float4 d = p.ray[2u * entryLeader(entry) + 1u];
    const uint32_t flags = __float_as_uint(d.w);
    const bool lit = (flags & kFlagEnvironmentOnMiss) != 0u;
    const float3 sky = lit ? environment(s, f, xyz(d)) : f3(0.0f);
    const uint32_t group = entry >> 3;
    const float4* light = reinterpret_cast<const float4*>(lightRecord(p, group));
    const float4* state = reinterpret_cast<const float4*>(laneRecord(p, group));
    const float4* spectra = p.laneSpectrum + 4u * static_cast<size_t>(group);
    const float4 l0 = light[0], l1 = light[1], a = state[0], b = state[1], c = state[2];
    const float4 basis[3] = {spectra[0], spectra[1], spectra[2]}, w = spectra[3];
    // Light samples of the previous bounce, in slot order.
    float radiance[3] = {l0.x + l0.w, l0.y + l1.x, l0.z + l1.y};
    if (lightSlots > 1u) {
        const float4 l2 = light[2];
        radiance[0] = radiance[0] + l1.z + l2.y;
        radiance[1] = radiance[1] + l1.w + l2.z;
        radiance[2] = radiance[2] + l2.x + l2.w;
    }
    const float throughput[3] = {a.x, a.y, a.z}, bsdfPdf[3] = {a.w, b.x, b.y}, lightPdf[3] = {b.z, b.w, c.x};
    const float wavelength[3] = {w.x, w.y, w.z};
#pragma unroll
    for (uint32_t lane = 0; lane < 3u; ++lane) {
        if (lit) {
            const Spectrum spec = spectrumFromBasis(wavelength[lane], basis[lane]);
            const float misWeight = (flags & kFlagPreviousWasDelta) != 0u ? 1.0f : powerHeuristic(bsdfPdf[lane], lightPdf[lane]);
            radiance[lane] += throughput[lane] * misWeight * illuminantSpectrum(sky, spec);
        }
    }
    float* out = lightRecord(p, group);
    if ((entry & 7u) == 7u) {
        reinterpret_cast<float4*>(out)[0] = make_float4(radiance[0], radiance[1], radiance[2], 0.0f);
        reinterpret_cast<float4*>(out)[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        if (lightSlots > 1u) reinterpret_cast<float4*>(out)[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        return;
    }
#pragma unroll
    for (uint32_t lane = 0; lane < 3u; ++lane) {
        if (!(entry >> lane & 1u)) continue;
        out[kLaneRadiance + lane] = radiance[lane];
        for (uint32_t j = 0; j < lightSlots; ++j) out[kLaneLight + 3u * j + lane] = 0.0f;
    }
}

// kLit: the scene has analytic or dome lights and no emissive triangles, so
// neither the fallback sun and sky (:1593-1668) nor emissive-triangle
// sampling (:1670-1731) can run; both are compiled out.
// kCache: radiance-cache mode (PathBuffers::cache): queries and training
// records at surface vertices; the plain kernels compile without it.
//
// kWalk: how a subsurface random walk (:1153-1186) runs.
//   kWalkInline - inside this kernel, nested in shading (renders without
//                 walk buffers);
//   kWalkDefer  - the walk's start (entry, normal, mean free path, albedo,
//                 anisotropy, RNG state, throughput) is recorded per lane and
//                 the path handed to walkKernel, a traversal kernel;
//                 everything before it in the bounce (emission, the light
//                 sample, the radiance so far) is done;
//   kWalkReplay - re-shades a path whose deferred walk failed (a boundary ray
//                 escaped): the same bounce from its stored start, with the
//                 light sample and radiance writes of the first pass
//                 suppressed, taking the walk's RNG state after the failed
//                 walk at the walk's place and continuing with the diffuse
//                 lobe as the inline form does.
// All three give the same bits. On the last bounce nothing after the light
// sample can change the image, and it is not run.
enum : int { kWalkInline = 0, kWalkDefer = 1, kWalkReplay = 2 };

// Light records a shade block copies into shared memory (3.5 KB).
constexpr uint32_t kStagedLights = 16;

// One random decision with lane probabilities `p`, taken where the first lane
// `f` of `sub` has a positive probability (kGuard) and drawn once: lanes that
// decide otherwise, or whose guard differs, leave `sub`.
template <bool kGuard, class V>
HDCX_D bool decide(V p, int f, uint32_t& sub, uint32_t& rng)
{
    if (kGuard) {
        const uint32_t positive = maskGreater(p, V(0.0f));
        const bool taken = (positive >> f & 1u) != 0u;
        sub &= taken ? positive : ~positive;
        if (!taken) return false;
    }
    const uint32_t less = maskLess(V(randomFloat(rng)), p);
    const bool yes = (less >> f & 1u) != 0u;
    sub &= yes ? less : ~less;
    return yes;
}

// Threads per block and resident blocks per SM of a variant.
//
// The kernels are 120-220 KB of instructions, more than an SM's instruction
// cache holds, and a warp runs most of them once per entry: warps at different
// places of the code evict each other's instructions (ncu: 27.7 cycles of
// `no_instruction` stall per issue on a textured scene, 0.08 issued per cycle
// and scheduler). So the warps of an SM are kept together: one block of 16
// warps per SM shades several lanes at 128 registers, with a barrier at the
// top of each iteration and one before the BSDF sample. Shade time per frame
// (800x450 4 spp textured / 639x361 8 spp, seven lights / 1920x1080 16 spp,
// 1M triangles): blocks of 128 without barriers 8.2 / 2.7 / 29.3 ms; with a
// barrier per iteration 6.0 / 2.4 / 25.2; one block of 512 with both barriers
// 2.7 / 1.5 / 23.3. Blocks of 768 (80 registers) 2.7 / 1.7 / 25.5, of 640
// 2.9 / 1.6 / 27.1; two barriers more change nothing. Entries of one lane are
// few and scattered: smaller blocks (glass scene 27.5 ms; 28.8 in one block
// of 384).
template <int kLanes, bool kFull>
constexpr int shadeThreads()
{
    return kLanes == 3 ? 512 : (kFull ? 128 : 256);
}
template <int kLanes, bool kFull, bool kLit>
constexpr int shadeMinBlocks()
{
    if (kLanes == 3) return 1;
    return kFull ? (kLit ? 4 : 1) : (kLit ? 3 : 1);
}

template <int kLanes, bool kFull, bool kLit, bool kCache, int kWalk>
__global__ void __launch_bounds__((shadeThreads<kLanes, kFull>()), (shadeMinBlocks<kLanes, kFull, kLit>()))
    shadeKernel(DeviceScene s, FrameConst f, PathBuffers p, uint32_t bounce, const uint32_t* queue,
                const uint32_t* count, uint32_t* nextQueue, unsigned long long* nextCount, bool misses)
{
    using V = std::conditional_t<kLanes == 3, Lanes3, float>;
    using U = typename LaneTraits<V>::U;
    constexpr bool kReplay = kWalk == kWalkReplay;
    static_assert(kWalk == kWalkInline || kFull, "deferred walks are for the full kernels");
    static_assert(kLanes == 1 || (!kCache && !kReplay), "cache renders and replays take single lanes");
    const uint32_t n = *count;
    const bool lastBounce = bounce + 1u >= f.maxBounces;
    const uint32_t lightSlots = kLit ? 1u : p.lightSlots;
    // Closure staging: with hits sorted by material (tuning sort_hits) a
    // block's consecutive hits mostly share one material. Its 368-byte
    // record is copied once per block iteration into shared memory, 16 bytes
    // per thread, and every thread whose hit uses it reads it from there;
    // other hits read theirs from global memory. Every thread of the block
    // runs the same iterations (the loop steps by block, not by thread).
    constexpr bool kStageable = kFull && !kReplay;
    const bool stage = kStageable && p.sortHits != 0u;
    __shared__ __align__(16) GpuMaterial stagedMaterial;
    __shared__ uint32_t stagedIndex;
    // The scene's light records, read two to three times over per shade
    // event by light selection and the environment pdf: copied once per
    // block into shared memory when there are at most kStagedLights of them.
    __shared__ __align__(16) GpuLight stagedLights[kStagedLights];
    const bool lightsStaged = s.lightCount <= kStagedLights;
    if (lightsStaged) {
        const uint32_t words = s.lightCount * static_cast<uint32_t>(sizeof(GpuLight) / sizeof(uint4));
        for (uint32_t w = threadIdx.x; w < words; w += blockDim.x)
            reinterpret_cast<uint4*>(stagedLights)[w] = __ldg(reinterpret_cast<const uint4*>(s.lights) + w);
    }
    __shared__ float3 stagedAxes[kStagedLights];  // normalize(basisZ) of each
    if (lightsStaged && threadIdx.x < s.lightCount) stagedAxes[threadIdx.x] = normalize(xyz(s.lights[threadIdx.x].basisZ));
    __syncthreads();
    const GpuLight* lights = lightsStaged ? stagedLights : s.lights;
    const float3* lightAxes = lightsStaged ? stagedAxes : nullptr;
    for (uint32_t blockBase = blockIdx.x * blockDim.x; blockBase < n; blockBase += gridDim.x * blockDim.x) {
        if (stage) {
            __syncthreads();  // the previous iteration's reads of the staged record are done
            if (threadIdx.x == 0)
                stagedIndex = __ldg(s.triangleMaterials + __float_as_uint(p.hit[entryLeader(queue[blockBase])].y));
            __syncthreads();
            if (threadIdx.x < sizeof(GpuMaterial) / sizeof(uint4)) {
                reinterpret_cast<uint4*>(&stagedMaterial)[threadIdx.x] =
                    __ldg(reinterpret_cast<const uint4*>(s.materials + stagedIndex) + threadIdx.x);
            }
            __syncthreads();
        }
        __syncthreads();  // the block's warps together (see shadeThreads)
        // A thread without an entry follows another's, with no lane of its own:
        // every thread of the block reaches every barrier.
        const uint32_t i = min(blockBase + threadIdx.x, n - 1u);
        const uint32_t entry = queue[i];
        const uint32_t group = entry >> 3;
        const uint32_t slot = entryLeader(entry);  // the leader's
        // Component k of a V is lane k of the group, or the one lane there is.
        uint32_t mask = blockBase + threadIdx.x >= n ? 0u : (kLanes == 3 ? entry & 7u : 1u);
        const uint32_t first = kLanes == 3 ? group * 3u : slot;
        const float4 ray0 = p.ray[2u * slot], ray1 = p.ray[2u * slot + 1u];
        float3 rayOrigin = xyz(ray0);
        float3 rayDirection = xyz(ray1);
        uint32_t rng = __float_as_uint(ray0.w);
        const uint32_t flags = __float_as_uint(ray1.w);
        const bool previousWasDelta = (flags & kFlagPreviousWasDelta) != 0u;
        const bool insideMedium = (flags & kFlagInsideMedium) != 0u;
        const float4 hitRec = p.hit[slot];
        const uint32_t primitive = __float_as_uint(hitRec.y);
        // The medium coefficients matter only inside a medium (entering one
        // sets all three), so paths outside one neither read nor write them.
        V mediumAbsorption = V(0.0f), mediumScattering = V(0.0f), mediumAnisotropy = V(0.0f);
        if (insideMedium) {
#pragma unroll
            for (int k = 0; k < kLanes; ++k) {
                if (!(mask >> k & 1u)) continue;
                const float4 medium = p.medium[first + k];
                put(mediumAbsorption, k, medium.x);
                put(mediumScattering, k, medium.y);
                put(mediumAnisotropy, k, medium.z);
            }
            if (kLanes == 3 && (maskGreater(mediumScattering, V(0.0f)) & mask) != 0u) {
                // Flight distances differ by lane: single lanes, shaded next.
#pragma unroll
                for (int k = 0; k < kLanes; ++k) {
                    if (!(mask >> k & 1u)) continue;
                    const uint32_t own = first + k;
                    if (own != slot) {
                        p.ray[2u * own] = ray0;
                        p.ray[2u * own + 1u] = ray1;
                        p.hit[own] = hitRec;
                        if (p.cone != nullptr) p.cone[own] = p.cone[slot];
                    }
                    p.hitQueue[appendIndex(p.counters + kCountHits)] = (group << 3) | (1u << k);
                }
                mask = 0u;
            }
        }
        // The lanes' state and spectra. Light samples of the previous bounce are
        // added in slot order; a slot without one holds zero. (A replay finds
        // this bounce's own samples in the slots: they stay.)
        V radiance, throughput, previousBsdfPdf, previousEnvironmentLightPdf;
        SpectrumOf<V> spec;
        float* record = laneRecord(p, group);
        float* lightOf = lightRecord(p, group);
        const uint32_t onlyLane = firstLane(entry & 7u);  // kLanes = 1
        if constexpr (kLanes == 3) {
            const float4* l = reinterpret_cast<const float4*>(lightOf);
            const float4* r = reinterpret_cast<const float4*>(record);
            const float4 l0 = l[0], l1 = l[1], a = r[0], b = r[1], c = r[2];
            radiance = Lanes3(l0.x, l0.y, l0.z) + Lanes3(l0.w, l1.x, l1.y);
            if (!kLit && lightSlots > 1u) {
                const float4 l2 = l[2];
                radiance = radiance + Lanes3(l1.z, l1.w, l2.x) + Lanes3(l2.y, l2.z, l2.w);
            }
            throughput = Lanes3(a.x, a.y, a.z);
            previousBsdfPdf = Lanes3(a.w, b.x, b.y);
            previousEnvironmentLightPdf = Lanes3(b.z, b.w, c.x);
            const float4* q = p.laneSpectrum + 4u * static_cast<size_t>(group);
            const float4 s0 = q[0], s1 = q[1], s2 = q[2], w = q[3];
            spec.wavelength = Lanes3(w.x, w.y, w.z);
            spec.br = Lanes3(s0.x, s1.x, s2.x);
            spec.bg = Lanes3(s0.y, s1.y, s2.y);
            spec.bb = Lanes3(s0.z, s1.z, s2.z);
            spec.planck = Lanes3(s0.w, s1.w, s2.w);
            spec.denominator = gmax(spec.br + spec.bg + spec.bb, Lanes3(1e-5f));
        } else {
            throughput = record[kLaneThroughput + onlyLane];
            radiance = lightOf[kLaneRadiance + onlyLane];
            if (!kReplay) radiance += lightOf[kLaneLight + onlyLane];
            if (!kReplay && !kLit && lightSlots > 1u) {
                radiance += lightOf[kLaneLight + 3u + onlyLane];
                radiance += lightOf[kLaneLight + 6u + onlyLane];
            }
            previousBsdfPdf = record[kLaneBsdfPdf + onlyLane];
            previousEnvironmentLightPdf = record[kLaneLightPdf + onlyLane];
            const float* q = spectrumRecord(p, group);
            spec = spectrumFromBasis(q[12u + onlyLane], reinterpret_cast<const float4*>(q)[onlyLane]);
        }
        // This bounce's light-sample slots.
        V lightValue = V(0.0f), secondValue = V(0.0f), thirdValue = V(0.0f);
        // Ray cone (width, spread) of texture LOD; spread <= 0: level 0.
        const bool lodOn = kFull && f.pixelSpread > 0.0f && p.cone != nullptr;
        const float2 cone = lodOn ? p.cone[slot] : make_float2(0.0f, -1.0f);
        float coneWidth = 0.0f;
        // Writes the state of lanes `alive` after this bounce and queues them.
        auto advance = [&](uint32_t alive, float3 origin, float3 direction, uint32_t state, uint32_t newFlags, bool coneKept,
                           V newThroughput, V bsdfPdf, V lightPdf) {
            const uint32_t lead = first + firstLane(alive);
            p.ray[2u * lead] = make_float4(origin.x, origin.y, origin.z, __uint_as_float(state));
            p.ray[2u * lead + 1u] = make_float4(direction.x, direction.y, direction.z,
                                                __uint_as_float(newFlags | (kCache ? (flags & kFlagTraining) : 0u)));
            if (lodOn) p.cone[lead] = coneKept ? make_float2(coneWidth, cone.y) : make_float2(0.0f, -1.0f);
            if (kLanes == 3 && alive == 7u) {
                float4* r = reinterpret_cast<float4*>(record);
                r[0] = make_float4(at(newThroughput, 0), at(newThroughput, 1), at(newThroughput, 2), at(bsdfPdf, 0));
                r[1] = make_float4(at(bsdfPdf, 1), at(bsdfPdf, 2), at(lightPdf, 0), at(lightPdf, 1));
                r[2] = make_float4(at(lightPdf, 2), 0.0f, 0.0f, 0.0f);
            } else {
#pragma unroll
                for (int k = 0; k < kLanes; ++k) {
                    if (!(alive >> k & 1u)) continue;
                    const uint32_t lane = kLanes == 3 ? static_cast<uint32_t>(k) : onlyLane;
                    record[kLaneThroughput + lane] = at(newThroughput, k);
                    record[kLaneBsdfPdf + lane] = at(bsdfPdf, k);
                    record[kLaneLightPdf + lane] = at(lightPdf, k);
                }
            }
            if ((newFlags & kFlagInsideMedium) != 0u) {
#pragma unroll
                for (int k = 0; k < kLanes; ++k)
                    if (alive >> k & 1u)
                        p.medium[first + k] = make_float4(at(mediumAbsorption, k), at(mediumScattering, k), at(mediumAnisotropy, k), 0.0f);
            }
            const uint32_t lanes = kLanes == 3 ? alive : entry & 7u;
            nextQueue[appendEntry(nextCount, lanes)] = (group << 3) | lanes;
        };
        // Writes radiance and light sample of the lanes of `mask`.
        auto storeLight = [&] {
            if (kReplay) return;
            if (kLanes == 3 && mask == 7u) {
                float4* l = reinterpret_cast<float4*>(lightOf);
                l[0] = make_float4(at(radiance, 0), at(radiance, 1), at(radiance, 2), at(lightValue, 0));
                l[1] = make_float4(at(lightValue, 1), at(lightValue, 2), at(secondValue, 0), at(secondValue, 1));
                if (!kLit && lightSlots > 1u)
                    l[2] = make_float4(at(secondValue, 2), at(thirdValue, 0), at(thirdValue, 1), at(thirdValue, 2));
                return;
            }
#pragma unroll
            for (int k = 0; k < kLanes; ++k) {
                if (!(mask >> k & 1u)) continue;
                const uint32_t lane = kLanes == 3 ? static_cast<uint32_t>(k) : onlyLane;
                lightOf[kLaneRadiance + lane] = at(radiance, k);
                lightOf[kLaneLight + lane] = at(lightValue, k);
                if (!kLit && lightSlots > 1u) {
                    lightOf[kLaneLight + 3u + lane] = at(secondValue, k);
                    lightOf[kLaneLight + 6u + lane] = at(thirdValue, k);
                }
            }
        };

            const uint32_t i0 = __ldg(s.indices + primitive * 3u + 0u);
            const uint32_t i1 = __ldg(s.indices + primitive * 3u + 1u);
            const uint32_t i2 = __ldg(s.indices + primitive * 3u + 2u);
            const float3 p0 = xyz(__ldg(s.vertices + i0));
            const float3 p1 = xyz(__ldg(s.vertices + i1));
            const float3 p2 = xyz(__ldg(s.vertices + i2));
            const float3 geometricNormal = normalize(cross(p1 - p0, p2 - p0));
            const bool frontFace = dot(geometricNormal, rayDirection) < 0.0f;
            const float3 orientedGeometricNormal = frontFace ? geometricNormal : -geometricNormal;
            const float b1 = hitRec.z, b2 = hitRec.w;
            const float3 authoredNormal = surfaceShadingNormal(s, primitive, b1, b2, geometricNormal);
            float3 normal = frontFace ? authoredNormal : -authoredNormal;
            const float2 uv0 = __ldg(s.texcoords + primitive * 3u + 0u);
            const float2 uv1 = __ldg(s.texcoords + primitive * 3u + 1u);
            const float2 uv2 = __ldg(s.texcoords + primitive * 3u + 2u);
            const float2 surfaceUv = surfaceTextureCoordinates(s, primitive, b1, b2);
            const float distance = hitRec.x;
            // Texture LOD by ray cones (hdcx_set_texture_lod; Akenine-Moller et
            // al., "Texture Level of Detail Strategies for Real-Time Ray
            // Tracing", 2019): the cone's width at the hit, the triangle's
            // texel-to-world area ratio and the incidence give the
            // texture-independent part of the level; -inf samples level 0.
            float lodBase = -INFINITY;
            if (kFull && lodOn && cone.y > 0.0f) {
                coneWidth = cone.x + cone.y * distance;
                const float2 du = uv1 - uv0, dv = uv2 - uv0;
                const float uvArea = fabsf(du.x * dv.y - du.y * dv.x);
                const float3 c = cross(p1 - p0, p2 - p0);
                const float worldArea = sqrtf(dot(c, c));
                const float incidence = fmaxf(fabsf(dot(geometricNormal, rayDirection)), 1e-4f);
                if (uvArea > 0.0f && worldArea > 0.0f && coneWidth > 0.0f)
                    lodBase = 0.5f * log2f(uvArea / worldArea) + log2f(coneWidth / incidence);
            }
            const float3 hit = rayOrigin + rayDirection * distance;
            if (insideMedium) {
                // :1279-1295
                if (kLanes == 1 && mask != 0u && at(mediumScattering, 0) > 0.0f) {
                    const float scatterDistance = -glog(gmax(1.0f - randomFloat(rng), 1e-6f)) / at(mediumScattering, 0);
                    if (scatterDistance < distance) {
                        throughput = throughput * V(gexp(-at(mediumAbsorption, 0) * scatterDistance));
                        rayOrigin = rayOrigin + rayDirection * scatterDistance;
                        rayDirection = sampleHenyeyGreenstein(rayDirection, at(mediumAnisotropy, 0), rng);
                        storeLight();
                        if (!lastBounce)
                            advance(mask, rayOrigin, rayDirection, rng,
                                    kFlagEnvironmentOnMiss | kFlagPreviousWasDelta | kFlagInsideMedium, false, throughput,
                                    V(0.0f), previousEnvironmentLightPdf);
                        mask = 0u;
                    }
                }
#pragma unroll
                for (int k = 0; k < kLanes; ++k)
                    if (mask >> k & 1u) put(throughput, k, at(throughput, k) * gexp(-at(mediumAbsorption, k) * distance));
            }
            const uint32_t materialIndex = __ldg(s.triangleMaterials + primitive);
            const GpuMaterial* material =
                (stage && materialIndex == stagedIndex) ? &stagedMaterial : s.materials + materialIndex;
            float3 baseColorRgb = xyz(material->baseColorMetalness);
            if (kFull && material->textureIndices0.x != kMissingTexture) {
                const float4 sample = materialTexture<kFull>(lodBase, s, material->textureIndices0.x, surfaceUv, f4(baseColorRgb, 1.0f));
                const float scaleW = material->baseColorTextureScale.w;
                const int channel = static_cast<int>(roundf(scaleW));
                float3 sourceColor;
                if (channel < 0) {
                    sourceColor = f3(sample.x, sample.y, sample.z);
                } else {
                    const int c = min(channel, 3);
                    sourceColor = f3(c == 0 ? sample.x : (c == 1 ? sample.y : (c == 2 ? sample.z : sample.w)));
                }
                baseColorRgb = xyz(material->baseColorTextureBias) + xyz(material->baseColorTextureScale) * sourceColor;
            }
            const V baseColor = reflectanceSpectrum(baseColorRgb, spec);
            const float metalness = clampf(
                materialTexture<kFull>(lodBase, s, material->textureIndices0.y, surfaceUv, f4(material->baseColorMetalness.w)).x, 0.0f, 1.0f);
            const float4 roughnessSample = materialTexture<kFull>(
                lodBase, s, material->textureIndices0.z, surfaceUv,
                make_float4(material->emissionRoughness.w, material->subsurfaceColor.w, 0.0f, 1.0f));
            const float2 roughness = make_float2(clampf(roughnessSample.x, 0.02f, 1.0f), clampf(roughnessSample.y, 0.02f, 1.0f));
            const float diffuseRoughness = clampf(
                materialTexture<kFull>(lodBase, s, material->textureIndices4.z, surfaceUv, f4(material->diffuseProperties.x)).x, 0.0f, 1.0f);
            const float diffuseWeight = clampf(
                materialTexture<kFull>(lodBase, s, material->textureIndices4.w, surfaceUv, f4(material->diffuseProperties.z)).x, 0.0f, 1.0f);
            const uint32_t diffuseModel = kFull ? static_cast<uint32_t>(material->diffuseProperties.y + 0.5f) : 0u;
            if (kFull) normal = applyNormalMap(s, material->textureIndices1.y, material->coatWeightRoughnessIor.w > 0.5f,
                                    material->subsurfaceWeightScale.w, surfaceUv, normal, p0, p1, p2, uv0, uv1, uv2);
            const float3 tangent = surfaceTangent(normal, p0, p1, p2, uv0, uv1, uv2);
            // (A replay re-shades a bounce whose first pass went past this
            // point without ending the path and has recorded its vertex.)
            if constexpr (kCache && !kReplay) if (mask != 0u) {
                const bool training = (flags & kFlagTraining) != 0u;
                bool terminate = bounce >= p.cache.prefixBounces;
                if (p.cache.spreadFactor > 0.0f) {
                    // Path spread (Mueller, Rousselle, Keller and Novak, "Real-time
                    // Neural Radiance Caching for Path Tracing", 2021, sec. 3.4):
                    // a(x1..xn) = (sum over i >= 2 of sqrt(|x(i-1) - xi|^2 /
                    // (p(wi) |cos(theta_i)|)))^2 against the primary footprint
                    // a0 = |x0 - x1|^2 / (4 pi |cos(theta_1)|); the path ends
                    // once a > c a0. A specular bounce (infinite pdf) adds nothing.
                    const float cosine = fmaxf(fabsf(dot(geometricNormal, rayDirection)), 1e-6f);
                    const float d2 = distance * distance;
                    float2 spread = bounce == 0u ? make_float2(d2 / (12.566370614f * cosine), 0.0f) : p.cache.spread[slot];
                    if (bounce > 0u && !previousWasDelta && at(previousBsdfPdf, 0) > 0.0f)
                        spread.y += sqrtf(d2 / (at(previousBsdfPdf, 0) * cosine));
                    p.cache.spread[slot] = spread;
                    terminate = terminate || spread.y * spread.y > p.cache.spreadFactor * spread.x;
                }
                if (training || terminate) {
                    const float3 qp = (hit - p.cache.sceneMin) * p.cache.sceneScale;
                    const float4 q0 = make_float4(qp.x, qp.y, qp.z, -rayDirection.x);
                    const float4 q1 = make_float4(-rayDirection.y, -rayDirection.z, normal.x, normal.y);
                    const float4 q2 = make_float4(normal.z, roughness.x, (spec.wavelength - 380.0f) / 400.0f, 0.0f);
                    if (training) {
                        if (bounce < kCacheMaxVertices) {
                            const uint32_t r = p.cache.trainIndex[slot] * kCacheMaxVertices + bounce;
                            float4* rec = reinterpret_cast<float4*>(p.cache.trainRecords) + r * 3u;
                            rec[0] = q0;
                            rec[1] = q1;
                            rec[2] = q2;
                            p.cache.trainState[r] = make_float2(throughput, radiance);
                            p.cache.trainVertices[p.cache.trainIndex[slot]] = bounce + 1u;
                        }
                    } else {
                        // The cache replaces everything from this vertex on.
                        const uint32_t j = appendIndex(p.cache.counters + 0);
                        float4* rec = reinterpret_cast<float4*>(p.cache.queries) + static_cast<size_t>(j) * 3u;
                        rec[0] = q0;
                        rec[1] = q1;
                        rec[2] = q2;
                        p.cache.querySlot[j] = slot;
                        storeLight();
                        record[kLaneThroughput + onlyLane] = at(throughput, 0);
                        mask = 0u;
                    }
                }
            }
            const float3 emissionRgb = surfaceEmissionRgb(s, primitive, surfaceUv);
            // No emission, no spectrum to build: the same zero.
            V emission = V(0.0f);
            if (!(emissionRgb.x <= 0.0f && emissionRgb.y <= 0.0f && emissionRgb.z <= 0.0f)) emission = illuminantSpectrum(emissionRgb, spec);
            V emissionMisWeight = V(1.0f);
            if (!previousWasDelta && (emissionRgb.x > 0.0f || emissionRgb.y > 0.0f || emissionRgb.z > 0.0f)) {
                const float emissionCosine = fabsf(dot(geometricNormal, -rayDirection));
                const float lightPdf = emissionCosine <= 0.0f
                                           ? 0.0f
                                           : __ldg(&s.emissive[primitive].y) * (distance * distance) / emissionCosine;
                emissionMisWeight = powerHeuristic(previousBsdfPdf, V(lightPdf));
            }
            radiance = radiance + throughput * emission * emissionMisWeight;

            const float transmission = kFull ? clampf(material->transmissionOpacityIor.x, 0.0f, 1.0f) : 0.0f;
            float3 transmissionColorRgb = xyz(material->transmissionColorThinWalled);
            if (transmission > 0.0f) {
                const float4 t = materialTexture<kFull>(lodBase, s, material->textureIndices1.z, surfaceUv, f4(transmissionColorRgb, 1.0f));
                transmissionColorRgb = f3(t.x, t.y, t.z);
            }
            const V transmissionColor = kFull ? weightedReflectance(transmission, transmissionColorRgb, spec) : V(0.0f);
            float subsurface = 0.0f;
            V diffuseColor = baseColor;
            float3 subsurfaceColorRgb = xyz(material->subsurfaceColor);
            float3 subsurfaceRadiusRgb = make_float3(gmax(material->subsurfaceRadius.x, 0.001f), gmax(material->subsurfaceRadius.y, 0.001f),
                                                     gmax(material->subsurfaceRadius.z, 0.001f));
            if (kFull && (material->subsurfaceWeightScale.x > 0.0f || material->textureIndices2.x != kMissingTexture)) {
                subsurface = clampf(materialTexture<kFull>(lodBase, s, material->textureIndices2.x, surfaceUv,
                                                          f4(material->subsurfaceWeightScale.x)).x, 0.0f, 1.0f);
                if (subsurface > 0.0f) {
                    const float4 c = materialTexture<kFull>(lodBase, s, material->textureIndices2.y, surfaceUv,
                                                           f4(xyz(material->subsurfaceColor), 1.0f));
                    subsurfaceColorRgb = f3(c.x, c.y, c.z);
                    const float4 r = materialTexture<kFull>(lodBase, s, material->textureIndices2.z, surfaceUv,
                                                           f4(xyz(material->subsurfaceRadius), 1.0f));
                    subsurfaceRadiusRgb = make_float3(gmax(r.x, 0.001f), gmax(r.y, 0.001f), gmax(r.z, 0.001f));
                    const V subsurfaceColor = reflectanceSpectrum(subsurfaceColorRgb, spec);
                    diffuseColor = mix(baseColor, subsurfaceColor, subsurface);
                }
            }
            const V ior = dispersedIor(gmax(material->transmissionOpacityIor.z, 1.0001f), material->transmissionMedium.z,
                                           material->transmissionMedium.w, spec.wavelength);
            const float specularWeight = clampf(
                materialTexture<kFull>(lodBase, s, material->textureIndices3.x, surfaceUv, f4(material->specularWeightColor.x)).x, 0.0f, 1.0f);
            const float4 specularColorSample = materialTexture<kFull>(
                lodBase, s, material->textureIndices3.y, surfaceUv,
                make_float4(material->specularWeightColor.y, material->specularWeightColor.z, material->specularWeightColor.w, 1.0f));
            const V specularColor =
                clampf(reconstructLikelyWhite(f3(specularColorSample.x, specularColorSample.y, specularColorSample.z), spec), 0.0f, 1.0f);
            V dielectricReflectance;
            if (material->transmissionMedium.z <= 0.0f || material->transmissionMedium.w <= 1.0f) {
                const float r = (at(ior, 0) - 1.0f) / (at(ior, 0) + 1.0f);  // no dispersion: one index for all lanes
                dielectricReflectance = V(r * r);
            } else {
                const V r = (ior - V(1.0f)) / (ior + V(1.0f));
                dielectricReflectance = r * r;
            }
            const V f0 = mix(clampf(dielectricReflectance * V(specularWeight) * specularColor, 0.0f, 1.0f), baseColor, metalness);
            float coat = 0.0f;
            float2 coatRoughness = make_float2(material->coatWeightRoughnessIor.y, material->subsurfaceRadius.w);
            V coatF0 = V(0.0f);
            if (kFull && (material->coatWeightRoughnessIor.x > 0.0f || material->textureIndices3.z != kMissingTexture)) {
                coat = clampf(materialTexture<kFull>(lodBase, s, material->textureIndices3.z, surfaceUv,
                                                    f4(material->coatWeightRoughnessIor.x)).x, 0.0f, 1.0f);
                if (coat > 0.0f) {
                    const float4 cc = materialTexture<kFull>(lodBase, s, material->textureIndices3.w, surfaceUv, f4(xyz(material->coatColor), 1.0f));
                    const V coatColor = reflectanceSpectrum(f3(cc.x, cc.y, cc.z), spec);
                    const float4 cr = materialTexture<kFull>(lodBase, s, material->textureIndices4.x, surfaceUv,
                                                            make_float4(coatRoughness.x, coatRoughness.y, 0.0f, 1.0f));
                    coatRoughness = make_float2(clampf(cr.x, 0.02f, 1.0f), clampf(cr.y, 0.02f, 1.0f));
                    const float coatIor = gmax(material->coatWeightRoughnessIor.z, 1.0001f);
                    float coatReflectance = (coatIor - 1.0f) / (coatIor + 1.0f);
                    coatReflectance = coatReflectance * coatReflectance;
                    coatF0 = clampf(V(coatReflectance) * coatColor, 0.0f, 1.0f);
                }
            }
            const float sheen =
                kFull ? clampf(materialTexture<kFull>(lodBase, s, material->textureIndices1.w, surfaceUv, f4(material->coatColor.w)).x, 0.0f, 1.0f)
                      : 0.0f;
            const float4 sheenColorSample = materialTexture<kFull>(lodBase, s, material->textureIndices2.w, surfaceUv,
                                                                  f4(xyz(material->sheenColorMode), 1.0f));
            const V sheenColor = kFull ? weightedReflectance(sheen, f3(sheenColorSample.x, sheenColorSample.y, sheenColorSample.z), spec) : V(0.0f);
            const float sheenRoughness = clampf(
                materialTexture<kFull>(lodBase, s, material->textureIndices4.y, surfaceUv, f4(material->transmissionScatter.w)).x, 0.01f, 1.0f);
            const bool sheenZeltner = material->sheenColorMode.w > 0.5f;
            const float translucentWeight = !kFull ? 0.0f : clampf(
                materialTexture<kFull>(lodBase, s, material->textureIndices5.x, surfaceUv, f4(material->translucentColorWeight.w)).x, 0.0f, 1.0f);
            const float4 translucentSample = materialTexture<kFull>(lodBase, s, material->textureIndices5.y, surfaceUv,
                                                                   f4(xyz(material->translucentColorWeight), 1.0f));
            const V translucentColor = kFull ? weightedReflectance(translucentWeight, f3(translucentSample.x, translucentSample.y, translucentSample.z), spec) : V(0.0f);

            const float3 viewDirection = normalize(-rayDirection);
            const float nDotView = gmax(dot(normal, viewDirection), 0.0f);
            // sheenAlbedo only ever appears multiplied by sheen; with sheen == 0
            // those products are exact zeros for any finite albedo.
            const float sheenAlbedo = sheen == 0.0f ? 0.0f
                                      : (sheenZeltner ? sheenZeltnerDirectionalAlbedo(nDotView, sheenRoughness)
                                                      : sheenDirectionalAlbedo(nDotView, sheenRoughness));
            const V sheenProbability = !kFull ? V(0.0f) : clampf(V(sheen * sheenAlbedo) * luminance1(sheenColor), 0.0f, 0.95f);
            const V coatContribution = coat > 0.0f ? V(coat) * fresnelSchlick(nDotView, coatF0) : V(0.0f);
            const V coatProbability = clampf(luminance1(coatContribution), 0.0f, 0.95f);
            const V baseFresnel = fresnelSchlick(nDotView, f0);
            const V specularContribution = baseFresnel;
            const V diffuseContribution = (V(1.0f) - baseFresnel) * V(diffuseWeight) * V(1.0f - translucentWeight) *
                                          V(1.0f - metalness) * diffuseColor;
            const V translucentContribution = !kFull ? V(0.0f) : (V(1.0f) - baseFresnel) * V(translucentWeight) * V(1.0f - metalness) * translucentColor;
            const V specularEnergy = luminance1(specularContribution);
            const V diffuseEnergy = luminance1(diffuseContribution);
            const V translucentEnergy = luminance1(translucentContribution);
            const V baseEnergy = diffuseEnergy + translucentEnergy;
            const V specularProbability = clampf(specularEnergy / gmax(specularEnergy + baseEnergy, V(1e-5f)), 0.05f, 0.95f);
            const V translucentProbability = !kFull ? V(0.0f) : whereMask(maskGreater(baseEnergy, V(1e-5f)), translucentEnergy / baseEnergy, V(0.0f));
            const uint32_t lightCount = kLit ? 1u : s.lightCount;
            const bool hasMeshLights = kLit ? false : s.hasMeshLights != 0u;

            const ShadingFrame frame = shadingFrame<kFull>(normal, tangent, viewDirection, nDotView, roughness, coatRoughness, coat);
            SurfaceParams<V> sp;
            sp.diffuseColor = diffuseColor;
            sp.transmission = transmission;
            sp.subsurface = subsurface;
            sp.diffuseWeight = diffuseWeight;
            sp.diffuseRoughness = diffuseRoughness;
            sp.diffuseModel = diffuseModel;
            sp.translucentWeight = translucentWeight;
            sp.translucentColor = translucentColor;
            sp.metalness = metalness;
            sp.roughness = roughness;
            sp.f0 = f0;
            sp.coat = coat;
            sp.coatRoughness = coatRoughness;
            sp.coatF0 = coatF0;
            sp.sheen = sheen;
            sp.sheenColor = sheenColor;
            sp.sheenRoughness = sheenRoughness;
            sp.sheenZeltner = sheenZeltner;

            // Light samples. Lanes that select different lights draw different
            // directions: one pass per light selected.
            const V directSpecularEnergy = specularEnergy + luminance1(coatContribution) + sheenProbability;
            V lightWeightTotal = V(0.0f), selectionPdf = V(0.0f);
            U picked, rngAfter;
            if (lightCount > 0u) {
                // :1469-1592 analytic light sample
                sampleAnalyticLight(s.lightCount, lights, lightAxes, hit, normal, diffuseEnergy, directSpecularEnergy, translucentEnergy,
                                    mask, rng, picked, selectionPdf, lightWeightTotal);
            }
            // Light-sample slot j: the value a visible sample adds, and its shadow ray.
            auto lightSample = [&](uint32_t j, uint32_t kind, uint32_t index, const GpuLight& record, float3 direction,
                                   float maximumDistance, uint32_t lanes, V a, V g1, V g2, V g3) {
                if (kReplay || lanes == 0u) return;
                const V value = combineShadow(kind, a, clampf(reconstructLikelyWhite(f3(1.0f), spec), 0.0f, 1.0f), g1, g2, g3);
                float traceDistance = maximumDistance;
                const bool needsRay = analyticNeedsRay(record, maximumDistance, traceDistance);
                // A blocked sample adds a * 0 * ..., zero unless a factor is not
                // finite, and then the visible value is not finite either.
                bool general = record.shadowColor.x != 0.0f || record.shadowColor.y != 0.0f || record.shadowColor.z != 0.0f ||
                               (record.shadow.y >= 0.0f && record.shadow.z > 0.0f);
#pragma unroll
                for (int k = 0; k < kLanes; ++k) {
                    if (!(lanes >> k & 1u)) continue;
                    general = general || !isfinite(at(value, k));
                }
                V& slotValue = j == 0u ? lightValue : (j == 1u ? secondValue : thirdValue);
                slotValue = whereMask(lanes, value, slotValue);
                if (!needsRay) return;
                if (general) {
#pragma unroll
                    for (int k = 0; k < kLanes; ++k)
                        if (lanes >> k & 1u)
                            p.shadowFactors[(first + k) * lightSlots + j] = make_float4(at(a, k), at(g1, k), at(g2, k), at(g3, k));
                }
                emitShadow(p, group, kLanes == 3 ? lanes : entry & 7u, kind | (j << 2) | (general ? kShadowGeneral : 0u) | (index << 8),
                           offsetSurfaceOrigin(hit, orientedGeometricNormal, direction), direction, traceDistance);
            };
            uint32_t open = mask;
#pragma unroll 1
            while (open != 0u) {
            uint32_t lanes = open;
            uint32_t lightRng = rng;
            if (lightCount > 0u) {
                const uint32_t lightIndex = at(picked, kLanes == 3 ? static_cast<int>(firstLane(open)) : 0);
#pragma unroll
                for (int k = 0; k < kLanes; ++k)
                    if (at(picked, k) != lightIndex) lanes &= ~(1u << k);
                const GpuLight& light = lights[lightIndex];
                float3 lightDirection = f3(0.0f, 1.0f, 0.0f);
                float3 lightRadiance = f3(0.0f);
                float inversePdf = 0.0f;
                float maximumShadowDistance = 10000.0f;
                float2 lightUv = make_float2(0.0f, 0.0f);  // dome: its texture coordinates of the direction
                const uint32_t type = light.textureInfo.z;
                if (type == 0u) {
                    float lightPdf = 0.0f;
                    sampleDomeLight(s, light, lightRng, lightDirection, lightPdf);
                    if (light.textureInfo.x != kMissingTexture || light.textureInfo.w != kMissingTexture) lightUv = domeUv(light, lightDirection);
                    lightRadiance = sampleDomeAt(s, light, lightUv);
                    inversePdf = lightPdf > 0.0f ? 1.0f / lightPdf : 0.0f;
                } else if (type == 5u) {
                    const float halfAngle = 0.5f * radians(clampf(light.geometry.z, 0.0f, 359.999f));
                    if (halfAngle <= 1e-6f) {
                        lightDirection = lightAxisOf(lights, lightAxes, lightIndex);
                        inversePdf = 1.0f;
                    } else {
                        const float cosineMaximum = gcos(halfAngle);
                        const float cosineTheta = mix(cosineMaximum, 1.0f, randomFloat(lightRng));
                        const float sineTheta = sqrtf(gmax(1.0f - cosineTheta * cosineTheta, 0.0f));
                        const float phi = kTwoPi * randomFloat(lightRng);
                        float sinePhi, cosinePhi;
                        gsincos(phi, sinePhi, cosinePhi);
                        lightDirection = normalize(xyz(light.basisX) * (cosinePhi * sineTheta) +
                                                   xyz(light.basisY) * (sinePhi * sineTheta) + xyz(light.basisZ) * cosineTheta);
                        inversePdf = 1.0f;
                    }
                    lightRadiance = xyz(light.colorIntensity) * light.colorIntensity.w;
                } else {
                    const float lu = randomFloat(lightRng);
                    const float lv = randomFloat(lightRng);
                    float3 lightPosition = xyz(light.position);
                    const float3 lightAxis = lightAxisOf(lights, lightAxes, lightIndex);
                    float3 lightNormal = -lightAxis;
                    if (type == 1u) {
                        lightPosition = lightPosition + ((lu - 0.5f) * xyz(light.axisU) + (lv - 0.5f) * xyz(light.axisV));
                    } else if (type == 2u) {
                        const float diskRadius = sqrtf(lu);
                        float sinePhi, cosinePhi;
                        gsincos(kTwoPi * lv, sinePhi, cosinePhi);
                        lightPosition = lightPosition + diskRadius * (cosinePhi * xyz(light.axisU) + sinePhi * xyz(light.axisV));
                    } else if (type == 3u) {
                        lightNormal = uniformSphere(lightRng);
                        lightPosition = lightPosition + light.geometry.x * lightNormal;
                    } else if (type == 4u) {
                        float sinePhi, cosinePhi;
                        gsincos(kTwoPi * lv, sinePhi, cosinePhi);
                        lightNormal = normalize(cosinePhi * xyz(light.basisY) + sinePhi * xyz(light.basisZ));
                        lightPosition = lightPosition + ((lu - 0.5f) * xyz(light.axisU) + light.geometry.x * lightNormal);
                    }
                    const float3 toLight = lightPosition - hit;
                    const float distanceSquared = dot(toLight, toLight);
                    const float lightDistance = sqrtf(gmax(distanceSquared, 1e-8f));
                    lightDirection = toLight / lightDistance;
                    const float emissionCosine = gmax(dot(lightNormal, -lightDirection), 0.0f);
                    if (emissionCosine > 0.0f && light.controls.w > 0.0f) {
                        const float shapingCosine = gmax(dot(lightAxis, lightDirection), 0.0f);
                        const float focus = gpow(shapingCosine, gmax(light.shaping.x, 0.0f));
                        const float3 focusColor = mix(xyz(light.focusTint), f3(1.0f), focus);
                        float3 textureValue = f3(1.0f);
                        if (!(type != 1u || light.textureInfo.x == kMissingTexture)) {
                            const float4 t = textureSample(s, light.textureInfo.x, make_float2(lu, lv));
                            textureValue = f3(t.x, t.y, t.z);
                        }
                        lightRadiance = xyz(light.colorIntensity) * light.colorIntensity.w * textureValue * focusColor *
                                        shapingConeFactor(light, shapingCosine);
                        inversePdf = light.controls.w * emissionCosine / gmax(distanceSquared, 1e-8f);
                        maximumShadowDistance = gmax(lightDistance - 0.003f, 0.001f);
                    }
                }
                if (inversePdf > 0.0f) {
                    const LobeTerms terms = lobeTerms(frame, lightDirection);
                    const V direct = evaluateDirectSurface<kFull>(frame, terms, lightDirection, sp, light.controls.x, light.controls.y);
                    const uint32_t lit = maskGreater(direct, V(0.0f)) & lanes;
                    if (lit != 0u) {
                        const V spectralLight = illuminantSpectrum(lightRadiance, spec);
                        V misWeight = V(1.0f);
                        if (type == 0u) {
                            misWeight = powerHeuristic(environmentLightPdf(s.textures, s.textureCount, s.lightCount, lights, lightDirection,
                                                                           diffuseEnergy, directSpecularEnergy, translucentEnergy,
                                                                           lightWeightTotal, lightIndex, lightUv),
                                                       surfaceReflectionPdf<kFull>(frame, terms, sheenProbability, coatProbability,
                                                                                   specularProbability, translucentProbability));
                        }
                        lightSample(0u, kShadowAnalytic, lightIndex, light, lightDirection, maximumShadowDistance, lit,
                                    throughput * direct * spectralLight, V(inversePdf), misWeight, gmax(selectionPdf, V(1e-8f)));
                    }
                }
            } else if (!kLit && !hasMeshLights) {
                // :1593-1668 fallback sun and sky
                const bool zUp = f.zUp != 0u;
                const float3 up = zUp ? f3(0.0f, 0.0f, 1.0f) : f3(0.0f, 1.0f, 0.0f);
                const float3 azimuth = zUp ? normalize(f3(1.0f, 1.0f, 0.0f)) : normalize(f3(1.0f, 0.0f, 1.0f));
                const float3 sunDirection = normalize(up * 0.9659258f + azimuth * 0.2588190f);
                const GpuLight& dummy = s.lights[0];
                const V direct = evaluateDirectSurface<kFull>(frame, lobeTerms(frame, sunDirection), sunDirection, sp, 1.0f, 1.0f);
                const V spectralSun = illuminantSpectrum(f3(3.45575f, 3.14159f, 2.82743f), spec);
                lightSample(0u, kShadowSun, 0u, dummy, sunDirection, 10000.0f, maskGreater(direct, V(0.0f)) & lanes,
                            throughput * direct * spectralSun, V(0.0f), V(0.0f), V(0.0f));
                const float3 skyDirection = cosineHemisphere(normal, lightRng);
                const V skyDirect = evaluateDirectSurface<kFull>(frame, lobeTerms(frame, skyDirection), skyDirection, sp, 1.0f, 0.0f);
                const V spectralSky = illuminantSpectrum(environment(s, f, skyDirection), spec);
                lightSample(1u, kShadowSky, 0u, dummy, skyDirection, 10000.0f, maskGreater(skyDirect, V(0.0f)) & lanes,
                            throughput * skyDirect * spectralSky, V(kPi / gmax(dot(normal, skyDirection), 1e-4f)), V(0.0f), V(0.0f));
                if (translucentWeight > 0.0f) {
                    const float3 backSkyDirection = cosineHemisphere(-normal, lightRng);
                    const V backSkyDirect = evaluateDirectSurface<kFull>(frame, lobeTerms(frame, backSkyDirection), backSkyDirection, sp, 1.0f, 0.0f);
                    const V spectralBack = illuminantSpectrum(environment(s, f, backSkyDirection), spec);
                    lightSample(2u, kShadowSky, 0u, dummy, backSkyDirection, 10000.0f, maskGreater(backSkyDirect, V(0.0f)) & lanes,
                                throughput * backSkyDirect * spectralBack,
                                V(kPi / gmax(dot(-normal, backSkyDirection), 1e-4f)), V(0.0f), V(0.0f));
                }
            }

            if (!kLit && hasMeshLights) {
                // :1670-1731 emissive-triangle sample
                const uint32_t primitiveCount = s.primitiveCount;
                const float target = randomFloat(lightRng);
                uint32_t low = 0u, high = primitiveCount - 1u;
                while (low < high) {
                    const uint32_t middle = low + (high - low) / 2u;
                    if (target <= __ldg(&s.emissive[middle].x)) high = middle;
                    else low = middle + 1u;
                }
                const uint32_t lightPrimitive = low;
                if (lightPrimitive != primitive && __ldg(&s.emissive[lightPrimitive].y) > 0.0f) {
                    const float root = sqrtf(randomFloat(lightRng));
                    const float second = randomFloat(lightRng);
                    const float w0 = 1.0f - root, w1 = root * (1.0f - second), w2 = root * second;
                    const float3 lightP0 = xyz(__ldg(s.vertices + __ldg(s.indices + lightPrimitive * 3u + 0u)));
                    const float3 lightP1 = xyz(__ldg(s.vertices + __ldg(s.indices + lightPrimitive * 3u + 1u)));
                    const float3 lightP2 = xyz(__ldg(s.vertices + __ldg(s.indices + lightPrimitive * 3u + 2u)));
                    const float3 lightPosition = lightP0 * w0 + lightP1 * w1 + lightP2 * w2;
                    const float3 lightNormal = normalize(cross(lightP1 - lightP0, lightP2 - lightP0));
                    const float3 toLight = lightPosition - hit;
                    const float distanceSquared = dot(toLight, toLight);
                    const float lightDistance = sqrtf(gmax(distanceSquared, 1e-8f));
                    const float3 lightDirection = toLight / lightDistance;
                    const float emissionCosine = fabsf(dot(lightNormal, -lightDirection));
                    const float lightPdf =
                        emissionCosine <= 0.0f ? 0.0f : __ldg(&s.emissive[lightPrimitive].y) * distanceSquared / emissionCosine;
                    if (lightPdf > 0.0f) {
                        const LobeTerms terms = lobeTerms(frame, lightDirection);
                        const V direct = evaluateDirectSurface<kFull>(frame, terms, lightDirection, sp, 1.0f, 1.0f);
                        const uint32_t lit = maskGreater(direct, V(0.0f)) & lanes;
                        if (lit != 0u && !kReplay) {
                            const float2 lightUv = surfaceTextureCoordinates(s, lightPrimitive, w1, w2);
                            float3 lightEmissionRgb = surfaceEmissionRgb(s, lightPrimitive, lightUv);
                            lightEmissionRgb = lightEmissionRgb * surfaceOpacity(s, lightPrimitive, w1, w2);
                            const V spectralLight = illuminantSpectrum(lightEmissionRgb, spec);
                            const V bsdfPdf = surfaceReflectionPdf<kFull>(frame, terms, sheenProbability, coatProbability,
                                                                          specularProbability, translucentProbability);
                            const V misWeight = powerHeuristic(V(lightPdf), bsdfPdf);
                            const V a = throughput * direct * spectralLight;
                            const float maxDistance = gmax(lightDistance - 0.003f, 0.001f);
                            const V value = a * (misWeight / V(lightPdf));
                            secondValue = whereMask(lit, value, secondValue);
                            if (!(maxDistance <= 0.001f)) {
                                emitShadow(p, group, kLanes == 3 ? lit : entry & 7u, kShadowMesh | (1u << 2),
                                           offsetSurfaceOrigin(hit, orientedGeometricNormal, lightDirection), lightDirection, maxDistance);
                            }
                        }
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < kLanes; ++k)
                if (lanes >> k & 1u) put(rngAfter, k, lightRng);
            open &= ~lanes;
            }

            storeLight();
            if (lastBounce) continue;  // the same for every thread
            __syncthreads();

            // The BSDF sample, one pass per part of lanes that decide alike.
            open = mask;
#pragma unroll 1
            while (open != 0u) {
            const int lead = kLanes == 3 ? static_cast<int>(firstLane(open)) : 0;
            uint32_t lanes = open;
            uint32_t state = at(rngAfter, lead);
#pragma unroll
            for (int k = 0; k < kLanes; ++k)
                if (at(rngAfter, k) != state) lanes &= ~(1u << k);
            V weight = throughput;
            float3 direction = rayDirection;
            float3 origin;
            uint32_t newFlags = insideMedium ? kFlagInsideMedium : 0u;
            V bsdfPdf = V(0.0f), lightPdf = previousEnvironmentLightPdf;
            bool sampled = false;  // a lobe of the surface: MIS pdfs and roulette follow
            bool coneKept = false;  // a smooth reflection or refraction keeps the cone
            bool walking = false;   // kWalkDefer: walkKernel finishes this bounce
            if (randomFloat(state) < transmission) {
                // :1735-1777
                const float iorLead = at(ior, lead);
#pragma unroll
                for (int k = 0; k < kLanes; ++k)
                    if (__float_as_uint(at(ior, k)) != __float_as_uint(iorLead)) lanes &= ~(1u << k);
                const float eta = frontFace ? 1.0f / iorLead : iorLead;
                const float cosTheta = gmin(dot(-rayDirection, normal), 1.0f);
                float r0 = (1.0f - iorLead) / (1.0f + iorLead);
                r0 = r0 * r0;
                const float fresnel = r0 + (1.0f - r0) * gpow5(1.0f - cosTheta);
                const float3 refracted = refract(rayDirection, normal, eta);
                const bool totalInternalReflection = dot(refracted, refracted) < 1e-8f;
                const bool thinWalled = material->transmissionColorThinWalled.w > 0.5f;
                bool refractedThroughBoundary = false;
                if (totalInternalReflection || randomFloat(state) < fresnel) {
                    direction = reflect(rayDirection, normal);
                } else {
                    direction = thinWalled ? rayDirection : normalize(refracted);
                    refractedThroughBoundary = !thinWalled;
                }
                const float transmissionDepth = gmax(material->transmissionMedium.x, 0.0f);
                weight = weight * (transmissionDepth > 0.0f ? V(1.0f) : transmissionColor);
                if (refractedThroughBoundary) {
                    if (frontFace) {
#pragma unroll
                        for (int k = 0; k < kLanes; ++k) {
                            if (!(lanes >> k & 1u)) continue;
                            const float spectralTransmission = gmax(at(transmissionColor, k), 0.001f);
                            put(mediumAbsorption, k, transmissionDepth > 0.0f ? -glog(spectralTransmission) / transmissionDepth : 0.0f);
                        }
                        const V spectralScatter = gmax(reconstructRgb(xyz(material->transmissionScatter), spec), V(0.0f));
                        const V scattering = transmissionDepth > 0.0f ? spectralScatter / V(transmissionDepth) : spectralScatter;
                        mediumScattering = whereMask(lanes, scattering, mediumScattering);
                        mediumAnisotropy = whereMask(lanes, V(material->transmissionMedium.y), mediumAnisotropy);
                        newFlags = kFlagInsideMedium;
                    } else {
                        newFlags = 0u;
                    }
                }
                origin = hit + direction * 0.002f;
                newFlags |= kFlagEnvironmentOnMiss | kFlagPreviousWasDelta;
                coneKept = true;
            } else {
                // :1779-1858 BSDF sampling chain: the lobe, then its
                // direction, then the weight of that direction.
                enum : int { kSheen, kCoat, kSpecular, kTranslucent, kDiffuse };
                int lobe;
                sampled = true;
                origin = hit + orientedGeometricNormal * 0.002f;
                if (decide<true>(sheenProbability, lead, lanes, state)) {
                    lobe = kSheen;
                } else {
                    weight = weight * (V(1.0f - sheen * sheenAlbedo) / gmax(V(1.0f) - sheenProbability, V(1e-4f)));
                    if (decide<true>(coatProbability, lead, lanes, state)) {
                        lobe = kCoat;
                    } else {
                        weight = weight * ((V(1.0f) - coatContribution) / gmax(V(1.0f) - coatProbability, V(1e-4f)));
                        if (decide<false>(specularProbability, lead, lanes, state)) {
                            lobe = kSpecular;
                        } else if (decide<true>(translucentProbability, lead, lanes, state)) {
                            lobe = kTranslucent;
                            weight = weight * (translucentContribution /
                                               gmax((V(1.0f) - specularProbability) * translucentProbability, V(1e-4f)));
                        } else {
                            lobe = kDiffuse;
                            weight = weight * (diffuseContribution /
                                               gmax((V(1.0f) - specularProbability) * (V(1.0f) - translucentProbability), V(1e-4f)));
                            if (subsurface > 0.0f && randomFloat(state) < subsurface) {
                                const V radius = gmax(reconstructRgb(subsurfaceRadiusRgb, spec) *
                                                          V(gmax(material->subsurfaceWeightScale.y, 0.0f)),
                                                      V(0.001f));
                                const V albedo = reflectanceSpectrum(subsurfaceColorRgb, spec);
                                if (kWalk == kWalkDefer) {
                                    // This bounce's extension queue has been traced: it holds the walks. Each lane
                                    // walks alone, from a start of its own.
                                    uint32_t* walks = (bounce & 1u) ? p.queue[1] : p.queue[0];
#pragma unroll
                                    for (int k = 0; k < kLanes; ++k) {
                                        if (!(lanes >> k & 1u)) continue;
                                        const uint32_t own = first + k;
                                        if (own != slot) {
                                            p.ray[2u * own] = ray0;
                                            p.ray[2u * own + 1u] = ray1;
                                            p.hit[own] = hitRec;
                                            if (lodOn) p.cone[own] = cone;
                                        }
                                        p.walkEntry[own] = make_float4(hit.x, hit.y, hit.z, at(radius, k));
                                        p.walkNormal[own] = make_float4(orientedGeometricNormal.x, orientedGeometricNormal.y,
                                                                        orientedGeometricNormal.z, at(albedo, k));
                                        p.walkState[own] = make_float4(material->subsurfaceWeightScale.z,
                                                                       __uint_as_float(state), at(weight, k), 0.0f);
                                        walks[appendIndex(p.counters + kCountWalks)] = own;
                                    }
                                    walking = true;
                                } else if (kWalk == kWalkReplay) {
                                    // The deferred walk failed; its RNG state after the walk.
                                    state = __float_as_uint(p.walkState[slot].y);
                                } else if constexpr (kLanes == 1) {
                                    float3 exitOrigin, exitDirection;
                                    float attenuation;
                                    if (randomWalkSubsurface(s, p, hit, orientedGeometricNormal, at(radius, 0), at(albedo, 0),
                                                             material->subsurfaceWeightScale.z, state, exitOrigin, exitDirection,
                                                             attenuation)) {
                                        weight = weight * V(attenuation);
                                        origin = exitOrigin;
                                        direction = exitDirection;
                                        newFlags |= kFlagEnvironmentOnMiss | kFlagPreviousWasDelta;
                                        sampled = false;
                                    }
                                }
                            }
                        }
                    }
                }
                if (sampled && !walking) {
                    const bool coatLobe = kFull && lobe == kCoat;
                    const float2 alpha = coatLobe ? frame.coatAlpha : frame.alpha;
                    if (coatLobe || lobe == kSpecular) {
                        direction = sampleGGXReflectionAnisotropic(rayDirection, frame, alpha, state);
                    } else {
                        direction = cosineHemisphere(kFull && lobe == kTranslucent ? -normal : normal, state);
                    }
                    const LobeTerms terms = lobeTerms(frame, direction);
                    bool environmentOnMiss = false;
                    if (coatLobe || lobe == kSpecular) {
                        const V ggx = ggxSampleWeightAnisotropic(frame, terms, direction, alpha, coatLobe ? frame.maskViewCoat : frame.maskView,
                                                                 coatLobe ? terms.dCoat : terms.d, whereMask(coatLobe ? 7u : 0u, coatF0, f0));
                        weight = weight * (coatLobe ? V(coat) * ggx / coatProbability : ggx / specularProbability);
                        environmentOnMiss = coatLobe ? gmax(coatRoughness.x, coatRoughness.y) < 0.2f : gmax(roughness.x, roughness.y) < 0.2f;
                    } else if (kFull && lobe == kSheen) {
                        const float response = sheenResponse(normal, viewDirection, direction, sheenRoughness, sheenZeltner);
                        weight = weight * (V(sheen) * sheenColor * V(response) / gmax(sheenProbability * V(terms.cosine), V(1e-6f)));
                        environmentOnMiss = true;
                    } else if (kFull && lobe == kTranslucent) {
                        origin = offsetSurfaceOrigin(hit, orientedGeometricNormal, direction);
                    } else {
                        V response = V(terms.nDotL <= 0.0f || nDotView <= 0.0f ? 0.0f : terms.cosine);
                        if (kFull && diffuseModel != 0u)
                            response = evaluateDiffuseReflection(normal, viewDirection, direction, diffuseColor, diffuseRoughness, diffuseModel);
                        weight = weight * ratioLikelyOne(response, V(gmax(terms.cosine, 1e-6f)));
                    }
                    if (lightCount > 0u || hasMeshLights) {
                        // :1859-1874
                        bsdfPdf = surfaceReflectionPdf<kFull>(frame, terms, sheenProbability, coatProbability, specularProbability,
                                                              translucentProbability);
                        newFlags |= kFlagEnvironmentOnMiss;
                        lightPdf = lightCount > 0u ? environmentLightPdf(s.textures, s.textureCount, s.lightCount, lights, direction,
                                                                         diffuseEnergy, directSpecularEnergy, translucentEnergy,
                                                                         lightWeightTotal, ~0u, make_float2(0.0f, 0.0f))
                                                   : V(0.0f);
                    } else {
                        // Neither pdf is set: both stay what they were.
                        bsdfPdf = previousBsdfPdf;
                        newFlags |= (environmentOnMiss ? kFlagEnvironmentOnMiss : 0u) | (previousWasDelta ? kFlagPreviousWasDelta : 0u);
                    }
                }
            }
            open &= ~lanes;
            uint32_t alive = walking ? 0u : lanes;
            if (sampled && !walking) {
                if (bounce >= 2u) {
                    // :1875-1879 Russian roulette
                    const V survival = clampf(weight, 0.1f, 0.95f);
                    alive &= ~maskGreater(V(randomFloat(state)), survival);
                    weight = weight / survival;
                }
            }
            if (alive != 0u) advance(alive, origin, direction, state, newFlags, coneKept, weight, bsdfPdf, lightPdf);
            }
    }
    if (!misses) return;
    // The bounce's misses, at the end of the launch rather than in one of their own.
    const uint32_t missCount = p.counters[kCountMisses];
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < missCount; i += gridDim.x * blockDim.x)
        shadeMiss(s, f, p, p.missQueue[i], lightSlots);
}

}  // namespace
}  // namespace hdcx
