// integrator.cu - wavefront form of the reference's spectral path tracer.
//
// The reference runs one megakernel invocation per pixel (GLSL main(),
// src/gpu/vulkan_path_tracer.cpp:1189-1891): for every sample and each of the
// three wavelength lanes it loops over bounces, tracing, shading, sampling
// lights and the BSDF. Here every (pixel, sample, lane) is a path slot of a
// wave, the lanes of a sample travel together while they share their path
// (device/paths.cuh), and each bounce is a few queue-driven kernels:
//   generate  - camera ray, RNG seed and wavelengths (:1191-1213);
//   trace     - closest-hit traversal of the extension queue (:1228-1243) and
//               any-hit visibility of the shadow queue of the bounce before
//               (:855-912), in one launch unless stages are timed;
//   shade     - miss/emission/medium/material/NEE/BSDF/roulette (:1245-1879),
//               appending surviving paths to the next extension queue and
//               light-sample rays to the shadow queue; one launch for entries
//               of several lanes and, where lanes part, one for single lanes;
//   walk      - deferred subsurface walks (scenes that have them);
// and one accumulate kernel per wave adds the lane radiances through the
// sensor (:1882-1884). A path's radiance gets its contributions in the
// megakernel's order: light-sample contributions of bounce b are stored per
// shadow slot and added, in slot order, before anything of bounce b+1.
// Queues are compacted with warp-aggregated atomics; kernels loop over the
// device-side queue length, so a frame needs no host round trip.
#include "integrator.h"
#include "nrc.h"
#include "nvtx_range.h"

#include <algorithm>
#include <stdexcept>
#include <string>
#include <vector>

#include "device/paths.cuh"
#include "device/shading.cuh"
#include "device/traverse.cuh"
#include "device/walk.cuh"
#include "shade.h"

namespace hdcx {
namespace {

#define CUDA_OK(expr)                                                                                  \
    do {                                                                                               \
        cudaError_t err__ = (expr);                                                                    \
        if (err__ != cudaSuccess) throw std::runtime_error(std::string("render: ") + #expr + ": " +     \
                                                           cudaGetErrorString(err__));                 \
    } while (0)

struct WaveDesc {
    uint32_t sampleBase;   // first sample offset of the wave (relative to the render)
    uint32_t samples;      // samples per pixel in the wave
    uint32_t pixelBase;    // first pixel
    uint32_t pixels;       // pixels in the wave
    uint32_t count;        // samples * pixels * 3
};

// Pixel number `index` of the order in which a wave takes the image: bands of
// four rows, in blocks of eight columns. The samples of a pixel are neighbours
// in a wave and the pixels of a block too, so a warp's camera rays and first
// hits lie close together.
HDCX_D uint32_t tiledPixel(const FrameConst& f, uint32_t index)
{
    const uint32_t band = index / (f.width * 4u);
    const uint32_t inBand = index - band * f.width * 4u;
    const uint32_t rows = min(4u, f.height - band * 4u);
    const uint32_t block = inBand / (8u * rows);
    const uint32_t inBlock = inBand - block * 8u * rows;
    const uint32_t columns = min(8u, f.width - block * 8u);
    const uint32_t row = inBlock / columns;
    return (band * 4u + row) * f.width + block * 8u + (inBlock - row * columns);
}

// ---------------------------------------------------------------------------
// generate: main() prologue (vulkan_path_tracer.cpp:1191-1223), one thread
// per group: the lanes of a sample share its seed, so its camera ray too.
// ---------------------------------------------------------------------------
__global__ void generateKernel(FrameConst f, WaveDesc w, PathBuffers p)
{
    const uint32_t group = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t groups = w.count / 3u;
    if (group == 0) {
        const unsigned long long lanes = static_cast<unsigned long long>(w.count) << 32;
        *reinterpret_cast<unsigned long long*>(p.counters + kCountQueue) = lanes | (p.split ? w.count : groups);
    }
    if (group >= groups) return;
    const uint32_t pixel = tiledPixel(f, w.pixelBase + group / w.samples);
    const uint32_t sampleNumber = f.sampleIndex + w.sampleBase + group % w.samples;
    const uint32_t px = pixel % f.width, py = pixel / f.width;
    const uint32_t index = pixel;
    uint32_t rng = hashState(index ^ (sampleNumber * 0x9e3779b9u) ^ 0xa511e9b3u);
    const float wavelengthShift = u2f(hashState(index ^ 0x68bc21ebu)) * (1.0f / 4294967296.0f);
    const float jx = randomFloat(rng);
    const float jy = randomFloat(rng);
    const float u = (u2f(px) + jx) / u2f(f.width);
    const float v = (u2f(py) + jy) / u2f(f.height);
    const float3 direction = normalize(f.lowerLeft + u * f.horizontal + v * f.vertical - f.origin);
    float wavelengths[3];
#pragma unroll
    for (uint32_t lane = 0; lane < 3u; ++lane) {
        wavelengths[lane] =
            380.0f + 400.0f * fract(wavelengthShift + (u2f(sampleNumber & 31u) + 0.5f) / 32.0f + u2f(lane) / 3.0f);
        const Spectrum s = makeSpectrum(wavelengths[lane]);
        p.laneSpectrum[4u * static_cast<size_t>(group) + lane] = make_float4(s.br, s.bg, s.bb, s.planck);
    }
    p.laneSpectrum[4u * static_cast<size_t>(group) + 3u] = make_float4(wavelengths[0], wavelengths[1], wavelengths[2], 0.0f);
    float4* light = reinterpret_cast<float4*>(lightRecord(p, group));
    light[0] = light[1] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    if (p.lightSlots > 1u) light[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    float4* record = reinterpret_cast<float4*>(laneRecord(p, group));
    record[0] = make_float4(1.0f, 1.0f, 1.0f, 0.0f);
    record[1] = record[2] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    for (uint32_t lane = 0; lane < 3u; ++lane) {
        const uint32_t slot = group * 3u + lane;
        uint32_t flags = kFlagEnvironmentOnMiss | kFlagPreviousWasDelta;
        if (p.cache.enabled) {
            // Training paths: a deterministic subset chosen by the path identity.
            const uint32_t key = hashState(pixel ^ hashState(sampleNumber * 0x9e3779b9u + lane * 0x85ebca6bu + 0x27d4eb2fu));
            if (key < p.cache.trainThreshold) {
                const uint32_t t = atomicAdd(p.cache.counters + 1, 1u);
                if (t < p.cache.trainCapacity) {
                    flags |= kFlagTraining;
                    p.cache.trainIndex[slot] = t;
                    p.cache.trainSlot[t] = slot;
                    p.cache.trainVertices[t] = 0u;
                    for (uint32_t b = 0; b < kCacheMaxVertices; ++b)
                        p.cache.trainState[t * kCacheMaxVertices + b] = make_float2(-1.0f, 0.0f);
                }
            }
        }
        if (lane == 0u || p.split) {
            p.ray[2u * slot] = make_float4(f.origin.x, f.origin.y, f.origin.z, __uint_as_float(rng));
            p.ray[2u * slot + 1u] = make_float4(direction.x, direction.y, direction.z, __uint_as_float(flags));
            if (p.cone != nullptr) p.cone[slot] = make_float2(0.0f, f.pixelSpread);
            if (p.split) p.queue[0][slot] = (group << 3) | (1u << lane);
        }
    }
    if (!p.split) p.queue[0][group] = (group << 3) | 7u;
}

// ---------------------------------------------------------------------------
// extend: closest hit of every queued ray (vulkan_path_tracer.cpp:1228-1243)
// ---------------------------------------------------------------------------
// Resident blocks of 128 threads per SM the traversal kernels are compiled
// for (8: 64 registers per thread).
#ifndef HDCX_TRACE_MIN_BLOCKS
#define HDCX_TRACE_MIN_BLOCKS 8
#endif

// kInst (traversal kernels): 0 single-level scenes, 1 scenes with instancers.
//
// One thread per entry traces the ray its lanes share: up to the first
// decision that parts them, one traversal serves three paths. Hits and misses
// go to separate queues, so that shading warps hold only hits; entries of
// several lanes and of one lane have shade kernels of their own, unless the
// scene keeps nearly all lanes together (PathBuffers::merged).
// ---------------------------------------------------------------------------
template <Accept kMode, bool kCount, int kInst>
HDCX_D void extendEntry(const DeviceScene& s, const PathBuffers& p, uint32_t entry, uint32_t& fault, uint2* work)
{
    const uint32_t slot = entryLeader(entry);
    const float4 o = p.ray[2u * slot];
    const float4 d = p.ray[2u * slot + 1u];
    HitRecord h;
    if (traceRay<kMode, false, kCount, kInst>(s, xyz(o), xyz(d), 0.001f, 10000.0f, __float_as_uint(o.w), h, fault, work)) {
        p.hit[slot] = make_float4(h.t, __uint_as_float(h.primitive), h.b1, h.b2);
        if (p.merged != 0u || __popc(entry & 7u) == 1) p.hitQueue[appendIndex(p.counters + kCountHits)] = entry;
        else p.groupQueue[appendIndex(p.counters + kCountGroups)] = entry;
    } else {
        p.missQueue[appendIndex(p.counters + kCountMisses)] = entry;
    }
}

// ---------------------------------------------------------------------------
// shadow: visibility of light samples (vulkan_path_tracer.cpp:855-912). The
// value of a visible sample is already in its light-sample slots; a blocked
// ray clears them, or (kShadowGeneral) recomputes them from the factors.
// ---------------------------------------------------------------------------
template <bool kOpaque, bool kCount, int kInst>
HDCX_D void shadowEntry(const DeviceScene& s, const PathBuffers& p, uint32_t i, uint32_t& fault, uint2* work)
{
    constexpr Accept kMode = kOpaque ? Accept::Opaque : Accept::Threshold;
    const float4 o = p.shadowRay[2u * i];
    const float4 d = p.shadowRay[2u * i + 1u];
    const uint32_t info = p.shadowInfo[i];
    const GpuLight& light = s.lights[info >> 8];
    const bool general = (info & kShadowGeneral) != 0u;
    const bool falloff = general && light.shadow.y >= 0.0f && light.shadow.z > 0.0f;
    HitRecord h;
    h.t = 0.0f;
    const bool blocked =
        falloff ? traceRay<kMode, false, kCount, kInst>(s, xyz(o), xyz(d), 0.001f, o.w, 0u, h, fault, work)
                : traceRay<kMode, true, kCount, kInst>(s, xyz(o), xyz(d), 0.001f, o.w, 0u, h, fault, work);
    if (!blocked) return;
    const uint32_t entry = __float_as_uint(d.w);
    const uint32_t j = (info >> 2) & 3u;
    float3 visibility = f3(0.0f);
    if (general) {
        float strength = 1.0f;
        if (falloff) {
            const float falloffDistance = gmin(light.shadow.z, gmax(light.shadow.y, 0.0f));
            strength = clampf((light.shadow.y - h.t) / gmax(falloffDistance, 1e-6f), 0.0f, 1.0f);
            strength = gpow(strength, gmax(light.shadow.w, 0.0f));
        }
        visibility = mix(f3(1.0f), xyz(light.shadowColor), strength);
    }
    for (uint32_t lane = 0; lane < 3u; ++lane) {
        if (!(entry >> lane & 1u)) continue;
        const uint32_t group = entry >> 3, slot = group * 3u + lane;
        float value = 0.0f;
        if (general) {
            const float4 fct = p.shadowFactors[slot * p.lightSlots + j];
            const float* spectra = spectrumRecord(p, group);
            const Spectrum spec = spectrumFromBasis(spectra[12u + lane], reinterpret_cast<const float4*>(spectra)[lane]);
            const float sv = reflectanceSpectrum(visibility, spec);
            const uint32_t kind = info & 3u;
            value = kind == kShadowAnalytic ? fct.x * sv * fct.y * fct.z / fct.w : (kind == kShadowSun ? fct.x * sv : fct.x * sv * fct.y);
        }
        lightRecord(p, group)[kLaneLight + 3u * j + lane] = value;
    }
}

// What one launch traces: the extension queue of a bounce, the shadow queue of
// the bounce before it, or both. The two are independent, and together their
// rays fill the tail that each launch ends in: when nothing asks for their
// separate times or counts they are traced in one launch.
struct TraceWork {
    const uint32_t* queue;                 // extension entries; null: none
    const unsigned long long* queueCount;
    const unsigned long long* shadowCount;  // null: no shadow rays
};

template <bool kOpaque, bool kCount, int kInst, bool kExtend, bool kShadow>
__global__ void __launch_bounds__(128, HDCX_TRACE_MIN_BLOCKS) traceKernel(DeviceScene s, PathBuffers p, TraceWork t)
{
    const unsigned long long extensions = kExtend ? *t.queueCount : 0ull;
    const unsigned long long shadows = kShadow ? *t.shadowCount : 0ull;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        if (kExtend) atomicAdd(p.stats + 0, extensions >> 32);
        if (kShadow) atomicAdd(p.stats + 1, shadows >> 32);
    }
    const uint32_t first = static_cast<uint32_t>(extensions);
    const uint32_t n = first + static_cast<uint32_t>(shadows);
    uint2 work = make_uint2(0u, 0u);
    uint32_t fault = 0u;  // traversal faults of this thread's rays
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        if (kExtend && (!kShadow || i < first)) {
            extendEntry<kOpaque ? Accept::Opaque : Accept::Stochastic, kCount, kInst>(s, p, t.queue[i], fault, &work);
        } else if (kShadow) {
            shadowEntry<kOpaque, kCount, kInst>(s, p, i - first, fault, &work);
        }
    }
    if (fault != 0u) atomicOr(reinterpret_cast<unsigned int*>(p.stats + 7), fault);
    if (kCount) {
        atomicAdd(p.stats + (kExtend ? 3 : 5), static_cast<unsigned long long>(work.x));
        atomicAdd(p.stats + (kExtend ? 4 : 6), static_cast<unsigned long long>(work.y));
    }
}

// ---------------------------------------------------------------------------
// walk: the deferred subsurface random walks of one bounce (:1153-1186), a
// traversal kernel of its own instead of up to eight traversals nested in the
// full shade kernel. A walk that exits finishes the bounce as the inline form
// does (the exit ray is the path's next ray; no MIS bookkeeping, no roulette);
// a walk whose boundary ray escapes stores its RNG state and queues the path
// for shadeKernel<..., kWalkReplay>, which finishes the bounce the inline way.
// ---------------------------------------------------------------------------
//
// A thread steps one walk at a time and takes the next when its walk ends, so
// every iteration of a warp traces a boundary ray per thread: walks end after
// one to eight rays, and a thread per walk left most of a warp waiting for its
// longest one.
template <int kInst>
__global__ void __launch_bounds__(128, HDCX_TRACE_MIN_BLOCKS)
    walkKernel(DeviceScene s, PathBuffers p, const uint32_t* walks, uint32_t* nextQueue, unsigned long long* nextCount,
               uint32_t* replayQueue)
{
    const uint32_t n = p.counters[kCountWalks];
    uint32_t rays = 0u, fault = 0u;
    uint32_t slot = 0u;
    bool walking = false;
    SubsurfaceWalk w;
    for (;;) {
        if (!walking) {
            const uint32_t i = appendIndex(p.counters + kCountWalkNext);
            if (i >= n) break;
            slot = walks[i];
            const float4 entry = p.walkEntry[slot];
            const float4 outward = p.walkNormal[slot];
            const float4 state = p.walkState[slot];
            w = beginWalk(xyz(entry), xyz(outward), entry.w, outward.w, state.x, __float_as_uint(state.y));
            walking = true;
        }
        ++rays;
        const int result = stepWalk<kInst>(s, w, fault);
        if (result == kWalkContinues) continue;
        walking = false;
        const float4 state = p.walkState[slot];
        const uint32_t lane = 1u << (slot % 3u);
        if (result == kWalkExits) {
            const uint32_t flags = kFlagEnvironmentOnMiss | kFlagPreviousWasDelta |
                                   (__float_as_uint(p.ray[2u * slot + 1u].w) & (kFlagInsideMedium | kFlagTraining));
            laneRecord(p, slot / 3u)[kLaneThroughput + slot % 3u] = state.z * w.attenuation;
            laneRecord(p, slot / 3u)[kLaneBsdfPdf + slot % 3u] = 0.0f;
            p.ray[2u * slot] = make_float4(w.origin.x, w.origin.y, w.origin.z, __uint_as_float(w.rng));
            p.ray[2u * slot + 1u] = make_float4(w.direction.x, w.direction.y, w.direction.z, __uint_as_float(flags));
            if (p.cone != nullptr) p.cone[slot] = make_float2(0.0f, -1.0f);
            nextQueue[appendEntry(nextCount, lane)] = ((slot / 3u) << 3) | lane;
        } else {
            p.walkState[slot] = make_float4(state.x, __uint_as_float(w.rng), state.z, 0.0f);
            replayQueue[appendIndex(p.counters + kCountReplays)] = ((slot / 3u) << 3) | lane;
        }
    }
    if (rays != 0u) atomicAdd(p.stats + 2, static_cast<unsigned long long>(rays));
    if (fault != 0u) atomicOr(reinterpret_cast<unsigned int*>(p.stats + 7), fault);
}

// ---------------------------------------------------------------------------
// accumulate: sensor and per-pixel batch sums (vulkan_path_tracer.cpp:1882-1884),
// and the running mean once a pixel's last wave has been added
// ---------------------------------------------------------------------------
//
// A pixel's samples add up in order, but what each adds (seven exponentials per
// wavelength) does not depend on the others: a thread per sample computes it,
// then a thread per pixel adds the block's values. Bound by instruction issue:
// eight samples at 1920x1080 took 1.6 ms with the sensor's RGB and XYZ each
// evaluating the exponentials and these branching, 0.69 ms with neither.
constexpr uint32_t kAccumulateThreads = 256;

// What sample `group` adds: sensor RGB (a third of the lanes' sum) and XYZ.
HDCX_D void sampleValue(const PathBuffers& p, uint32_t group, float3& rgb, double xyz[3])
{
    const float4* light = reinterpret_cast<const float4*>(lightRecord(p, group));
    const float4 la = light[0], lb = light[1], wl = p.laneSpectrum[4u * static_cast<size_t>(group) + 3u];
    float radiances[3] = {la.x + la.w, la.y + lb.x, la.z + lb.y};
    if (p.lightSlots > 1u) {
        const float4 lc = light[2];
        radiances[0] = radiances[0] + lb.z + lc.y;
        radiances[1] = radiances[1] + lb.w + lc.z;
        radiances[2] = radiances[2] + lc.x + lc.w;
    }
    const float wavelengths[3] = {wl.x, wl.y, wl.z};
    float3 spectral = f3(0.0f);
    double sx = 0.0, sy = 0.0, sz = 0.0;
#pragma unroll
    for (uint32_t lane = 0; lane < 3u; ++lane) {
        const float radiance = radiances[lane];
        const float3 x = sensorXyz(wavelengths[lane]);
        spectral = spectral + spectralSensor(x) * radiance;
        sx = __dadd_rn(sx, __dmul_rn(static_cast<double>(x.x), static_cast<double>(radiance)));
        sy = __dadd_rn(sy, __dmul_rn(static_cast<double>(x.y), static_cast<double>(radiance)));
        sz = __dadd_rn(sz, __dmul_rn(static_cast<double>(x.z), static_cast<double>(radiance)));
    }
    rgb = f3(spectral.x / 3.0f, spectral.y / 3.0f, spectral.z / 3.0f);
    xyz[0] = __ddiv_rn(sx, 3.0);
    xyz[1] = __ddiv_rn(sy, 3.0);
    xyz[2] = __ddiv_rn(sz, 3.0);
}

__global__ void __launch_bounds__(kAccumulateThreads) accumulateKernel(FrameConst f, WaveDesc w, PathBuffers p, FrameBuffers fb)
{
    __shared__ float3 rgbs[kAccumulateThreads];
    __shared__ double xyzs[3][kAccumulateThreads];
    // Pixels per block, and samples per pass (a pixel with more than the block
    // has threads takes several).
    const uint32_t step = min(w.samples, kAccumulateThreads);
    const uint32_t pixels = kAccumulateThreads / step;
    const uint32_t firstLocal = blockIdx.x * pixels;
    const uint32_t local = firstLocal + threadIdx.x;
    const bool adds = threadIdx.x < pixels && local < w.pixels;
    const uint32_t pixel = adds ? tiledPixel(f, w.pixelBase + local) : 0u;
    float4 b = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
    double bx = 0.0, by = 0.0, bz = 0.0;
    if (adds && w.sampleBase != 0u) {
        b = fb.batch[pixel];
        bx = fb.batchXyz[3 * pixel + 0], by = fb.batchXyz[3 * pixel + 1], bz = fb.batchXyz[3 * pixel + 2];
    }
    for (uint32_t base = 0; base < w.samples; base += step) {
        const uint32_t mine = threadIdx.x / step, sample = base + threadIdx.x % step;
        if (mine < pixels && firstLocal + mine < w.pixels && sample < w.samples) {
            double xyz[3];
            sampleValue(p, (firstLocal + mine) * w.samples + sample, rgbs[threadIdx.x], xyz);
            for (int k = 0; k < 3; ++k) xyzs[k][threadIdx.x] = xyz[k];
        }
        __syncthreads();
        if (adds) {
            for (uint32_t s = 0; s < min(step, w.samples - base); ++s) {
                const uint32_t t = threadIdx.x * step + s;
                const float3 rgb = rgbs[t];
                b = make_float4(b.x + rgb.x, b.y + rgb.y, b.z + rgb.z, 0.0f);
                bx = __dadd_rn(bx, xyzs[0][t]);
                by = __dadd_rn(by, xyzs[1][t]);
                bz = __dadd_rn(bz, xyzs[2][t]);
            }
        }
        __syncthreads();
    }
    if (!adds) return;
    if (w.sampleBase + w.samples < f.sampleCount) {
        fb.batch[pixel] = b;
        fb.batchXyz[3 * pixel + 0] = bx;
        fb.batchXyz[3 * pixel + 1] = by;
        fb.batchXyz[3 * pixel + 2] = bz;
        return;
    }
    // The pixel's last wave: pixels[index] = vec4((previous * previousWeight +
    // batchRadiance) / totalWeight, 1.0) (vulkan_path_tracer.cpp:1886-1890); the
    // FP64 XYZ sums add the batch. A restart (sampleIndex 0) gives the previous
    // mean weight 0; it is not read, so whatever the output buffer held (NaN
    // included) cannot leak in.
    const float4 prev = f.sampleIndex == 0 ? make_float4(0.0f, 0.0f, 0.0f, 0.0f) : fb.rgba[pixel];
    const float previousWeight = u2f(f.sampleIndex);
    const float totalWeight = previousWeight + u2f(f.sampleCount);
    fb.rgba[pixel] = make_float4((prev.x * previousWeight + b.x) / totalWeight, (prev.y * previousWeight + b.y) / totalWeight,
                                 (prev.z * previousWeight + b.z) / totalWeight, 1.0f);
    const double sums[3] = {bx, by, bz};
    for (int k = 0; k < 3; ++k) {
        const double base = f.sampleIndex == 0 ? 0.0 : fb.xyz[3 * pixel + k];
        fb.xyz[3 * pixel + k] = __dadd_rn(base, sums[k]);
    }
}


__global__ void primaryKernel(DeviceScene s, FrameConst f, uint32_t sampleNumber, uint32_t* primitives, float* distances)
{
    const uint32_t pixel = blockIdx.x * blockDim.x + threadIdx.x;
    if (pixel >= f.width * f.height) return;
    const uint32_t px = pixel % f.width, py = pixel / f.width;
    uint32_t rng = hashState(pixel ^ (sampleNumber * 0x9e3779b9u) ^ 0xa511e9b3u);
    const float jx = randomFloat(rng);
    const float jy = randomFloat(rng);
    const float u = (u2f(px) + jx) / u2f(f.width);
    const float v = (u2f(py) + jy) / u2f(f.height);
    const float3 direction = normalize(f.lowerLeft + u * f.horizontal + v * f.vertical - f.origin);
    HitRecord h;
    uint32_t fault = 0u;  // primary hits of hdcx_trace_primary and the AOVs: a fault leaves the pixel a miss
    const bool found = s.opaque ? traceRay<Accept::Opaque, false>(s, f.origin, direction, 0.001f, 10000.0f, rng, h, fault)
                                : traceRay<Accept::Stochastic, false>(s, f.origin, direction, 0.001f, 10000.0f, rng, h, fault);
    primitives[pixel] = found ? h.primitive : kInvalidPrimitive;
    distances[pixel] = found ? h.t : 0.0f;
}

// ---------------------------------------------------------------------------
// radiance-cache mode: predictions into the terminated paths, suffix targets
// of the training paths
// ---------------------------------------------------------------------------
__global__ void cacheApplyKernel(PathBuffers p)
{
    const uint32_t n = p.cache.counters[0];
    for (uint32_t j = blockIdx.x * blockDim.x + threadIdx.x; j < n; j += gridDim.x * blockDim.x) {
        const uint32_t slot = p.cache.querySlot[j];
        lightRecord(p, slot / 3u)[kLaneRadiance + slot % 3u] += laneRecord(p, slot / 3u)[kLaneThroughput + slot % 3u] * fmaxf(p.cache.predictions[j], 0.0f);
    }
}

__global__ void cacheTargetsKernel(PathBuffers p)
{
    const uint32_t n = min(p.cache.counters[1], p.cache.trainCapacity);
    for (uint32_t t = blockIdx.x * blockDim.x + threadIdx.x; t < n; t += gridDim.x * blockDim.x) {
        const uint32_t slot = p.cache.trainSlot[t];
        const float* light = lightRecord(p, slot / 3u) + slot % 3u;
        float total = light[kLaneRadiance] + light[kLaneLight];
        for (uint32_t j = 1; j < p.lightSlots; ++j) total += light[kLaneLight + 3u * j];
        const uint32_t vertices = min(p.cache.trainVertices[t], kCacheMaxVertices);
        for (uint32_t b = 0; b < vertices; ++b) {
            const uint32_t r = t * kCacheMaxVertices + b;
            const float2 st = p.cache.trainState[r];
            if (!(st.x > 0.0f)) continue;
            const float target = (total - st.y) / st.x;
            if (!(target >= 0.0f && target < 3.0e38f)) continue;
            const uint32_t j = atomicAdd(p.cache.counters + 2, 1u);
            const float4* src = reinterpret_cast<const float4*>(p.cache.trainRecords) + r * 3u;
            float4* dst = reinterpret_cast<float4*>(p.cache.sampleQueries) + static_cast<size_t>(j) * 3u;
            dst[0] = src[0];
            dst[1] = src[1];
            dst[2] = src[2];
            p.cache.sampleTargets[j] = target;
        }
    }
}

int gridFor(uint32_t maxItems, int perSm)
{
    int device = 0, sms = 148;
    cudaGetDevice(&device);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
    const int blocks = static_cast<int>((static_cast<uint64_t>(maxItems) + 127u) / 128u);
    return std::max(1, std::min(blocks, sms * perSm));
}

std::vector<WaveDesc> planWaves(uint32_t pixels, uint32_t samples, uint64_t capacity)
{
    std::vector<WaveDesc> waves;
    const uint64_t perSample = static_cast<uint64_t>(pixels) * 3u;
    if (perSample <= capacity) {
        const uint32_t k = static_cast<uint32_t>(std::max<uint64_t>(1u, std::min<uint64_t>(samples, capacity / perSample)));
        for (uint32_t s0 = 0; s0 < samples; s0 += k) {
            const uint32_t ks = std::min(k, samples - s0);
            waves.push_back({s0, ks, 0u, pixels, static_cast<uint32_t>(ks * perSample)});
        }
    } else {
        const uint32_t chunk = static_cast<uint32_t>(capacity / 3u);
        for (uint32_t s0 = 0; s0 < samples; ++s0) {
            for (uint32_t p0 = 0; p0 < pixels; p0 += chunk) {
                const uint32_t np = std::min(chunk, pixels - p0);
                waves.push_back({s0, 1u, p0, np, np * 3u});
            }
        }
    }
    return waves;
}

struct EventPair {
    cudaEvent_t start, stop;
    int stage;
};

}  // namespace

// ---------------------------------------------------------------------------
// hit sort: the hit queue in material order, so that a shading warp's lanes
// run the same material's code (scenes whose materials take very different
// paths: glass, subsurface walks, cut-out leaves). A counting sort over
// material bins: per-block shared histograms, one global reservation per bin
// and block iteration. Order within a bin is arbitrary; every path's result
// is independent of queue order.
// ---------------------------------------------------------------------------
__device__ __forceinline__ uint32_t hitMaterialBin(const DeviceScene& s, const PathBuffers& p, uint32_t entry)
{
    const uint32_t primitive = __float_as_uint(p.hit[entryLeader(entry)].y);
    return __ldg(s.triangleMaterials + primitive) % kHitBins;
}

__global__ void __launch_bounds__(256) countHitBinsKernel(DeviceScene s, PathBuffers p, const uint32_t* hits, const uint32_t* count)
{
    __shared__ uint32_t histogram[kHitBins];
    for (uint32_t b = threadIdx.x; b < kHitBins; b += blockDim.x) histogram[b] = 0u;
    __syncthreads();
    const uint32_t n = *count;
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x)
        atomicAdd(&histogram[hitMaterialBin(s, p, hits[i])], 1u);
    __syncthreads();
    for (uint32_t b = threadIdx.x; b < kHitBins; b += blockDim.x)
        if (histogram[b] != 0u) atomicAdd(p.hitBins + b, histogram[b]);
}

// Exclusive prefix sum of the bin counts into the cursors (one warp).
__global__ void scanHitBinsKernel(PathBuffers p)
{
    constexpr uint32_t kPerLane = kHitBins / 32u;
    const uint32_t lane = threadIdx.x;
    uint32_t counts[kPerLane];
    uint32_t local = 0u;
    for (uint32_t k = 0; k < kPerLane; ++k) {
        counts[k] = p.hitBins[lane * kPerLane + k];
        local += counts[k];
    }
    uint32_t inclusive = local;
    for (uint32_t d = 1; d < 32u; d <<= 1) {
        const uint32_t v = __shfl_up_sync(0xffffffffu, inclusive, d);
        if (lane >= d) inclusive += v;
    }
    uint32_t offset = inclusive - local;
    for (uint32_t k = 0; k < kPerLane; ++k) {
        p.hitBins[kHitBins + lane * kPerLane + k] = offset;
        offset += counts[k];
    }
}

__global__ void __launch_bounds__(256) scatterHitsKernel(DeviceScene s, PathBuffers p, const uint32_t* hits, const uint32_t* count)
{
    __shared__ uint32_t histogram[kHitBins];
    __shared__ uint32_t start[kHitBins];
    const uint32_t n = *count;
    // The loop bound is the same for every thread of the block (base is
    // per block), so the barriers inside are reached by all of them.
    for (uint32_t base = blockIdx.x * blockDim.x; base < n; base += gridDim.x * blockDim.x) {
        for (uint32_t b = threadIdx.x; b < kHitBins; b += blockDim.x) histogram[b] = 0u;
        __syncthreads();
        const uint32_t i = base + threadIdx.x;
        const bool valid = i < n;
        const uint32_t entry = valid ? hits[i] : 0u;
        const uint32_t bin = valid ? hitMaterialBin(s, p, entry) : 0u;
        const uint32_t rank = valid ? atomicAdd(&histogram[bin], 1u) : 0u;
        __syncthreads();
        for (uint32_t b = threadIdx.x; b < kHitBins; b += blockDim.x)
            if (histogram[b] != 0u) start[b] = atomicAdd(p.hitBins + kHitBins + b, histogram[b]);
        __syncthreads();
        if (valid) p.sortedHits[start[bin] + rank] = entry;
        __syncthreads();
    }
}

// ---------------------------------------------------------------------------
// ray sort (tuning knob sort_rays): secondary extension rays are reordered
// within chunks of kRayChunk queue entries by a direction cell, so that a
// warp traces rays of similar direction. The queue's own order already keeps
// rays of nearby pixels, and so of nearby origins, close together: sorting
// within a chunk keeps that and adds directional coherence, with no global
// pass. Order within a cell is arbitrary; every path's result is independent
// of queue order.
// ---------------------------------------------------------------------------
constexpr uint32_t kRayChunk = 1024;  // queue entries per block iteration (256 threads x 4)
constexpr uint32_t kRayCells = 128;   // 6 cube faces x 4 x 4 cells (96 used)

__device__ __forceinline__ uint32_t directionCell(float4 d)
{
    const float ax = fabsf(d.x), ay = fabsf(d.y), az = fabsf(d.z);
    uint32_t face;
    float u, v, m;
    if (ax >= ay && ax >= az) {
        face = d.x < 0.0f ? 1u : 0u;
        u = d.y;
        v = d.z;
        m = ax;
    } else if (ay >= az) {
        face = d.y < 0.0f ? 3u : 2u;
        u = d.x;
        v = d.z;
        m = ay;
    } else {
        face = d.z < 0.0f ? 5u : 4u;
        u = d.x;
        v = d.y;
        m = az;
    }
    const float inv = m > 0.0f ? 2.0f / m : 0.0f;  // (u/m + 1) * 2 in [0, 4]
    const uint32_t cu = min(static_cast<uint32_t>(fmaxf(fmaf(u, inv, 2.0f), 0.0f)), 3u);
    const uint32_t cv = min(static_cast<uint32_t>(fmaxf(fmaf(v, inv, 2.0f), 0.0f)), 3u);
    return face * 16u + cu * 4u + cv;
}

__global__ void __launch_bounds__(256) sortRaysKernel(PathBuffers p, uint32_t* queue, const unsigned long long* count)
{
    __shared__ uint32_t cursor[kRayCells];
    __shared__ uint32_t sorted[kRayChunk];
    const uint32_t n = static_cast<uint32_t>(*count);
    constexpr uint32_t kPer = kRayChunk / 256u;
    // The loop bound is the same for every thread of the block, so the
    // barriers inside are reached by all of them.
    for (uint32_t base = blockIdx.x * kRayChunk; base < n; base += gridDim.x * kRayChunk) {
        if (threadIdx.x < kRayCells) cursor[threadIdx.x] = 0u;
        __syncthreads();
        uint32_t entry[kPer], cell[kPer], rank[kPer];
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t i = base + k * 256u + threadIdx.x;
            entry[k] = i < n ? queue[i] : 0u;
            cell[k] = i < n ? directionCell(p.ray[2u * entryLeader(entry[k]) + 1u]) : 0u;
            rank[k] = i < n ? atomicAdd(&cursor[cell[k]], 1u) : 0u;
        }
        __syncthreads();
        if (threadIdx.x < 32u) {
            // Exclusive prefix sum of the cell counts, four cells per lane.
            const uint32_t lane = threadIdx.x;
            uint32_t c[4], local = 0u;
#pragma unroll
            for (uint32_t k = 0; k < 4u; ++k) {
                c[k] = cursor[lane * 4u + k];
                local += c[k];
            }
            uint32_t inclusive = local;
#pragma unroll
            for (uint32_t d = 1; d < 32u; d <<= 1) {
                const uint32_t v = __shfl_up_sync(0xffffffffu, inclusive, d);
                if (lane >= d) inclusive += v;
            }
            uint32_t offset = inclusive - local;
#pragma unroll
            for (uint32_t k = 0; k < 4u; ++k) {
                cursor[lane * 4u + k] = offset;
                offset += c[k];
            }
        }
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            if (base + k * 256u + threadIdx.x < n) sorted[cursor[cell[k]] + rank[k]] = entry[k];
        }
        __syncthreads();
#pragma unroll
        for (uint32_t k = 0; k < kPer; ++k) {
            const uint32_t i = base + k * 256u + threadIdx.x;
            if (i < n) queue[i] = sorted[k * 256u + threadIdx.x];
        }
        __syncthreads();
    }
}

template <bool kCount, int kInst>
void launchTraceOf(const DeviceScene& scene, const PathBuffers& paths, const TraceWork& t, int grid, cudaStream_t stream)
{
    const bool extend = t.queueCount != nullptr, shadow = t.shadowCount != nullptr;
    if (scene.opaque) {
        if (extend && shadow) {
            if constexpr (!kCount) traceKernel<true, false, kInst, true, true><<<grid, 128, 0, stream>>>(scene, paths, t);
        } else if (extend) traceKernel<true, kCount, kInst, true, false><<<grid, 128, 0, stream>>>(scene, paths, t);
        else traceKernel<true, kCount, kInst, false, true><<<grid, 128, 0, stream>>>(scene, paths, t);
    } else {
        if (extend && shadow) {
            if constexpr (!kCount) traceKernel<false, false, kInst, true, true><<<grid, 128, 0, stream>>>(scene, paths, t);
        } else if (extend) traceKernel<false, kCount, kInst, true, false><<<grid, 128, 0, stream>>>(scene, paths, t);
        else traceKernel<false, kCount, kInst, false, true><<<grid, 128, 0, stream>>>(scene, paths, t);
    }
    CUDA_OK(cudaGetLastError());
}

// Both queues at once are for renders that do not count (see TraceWork).
void launchTrace(const DeviceScene& scene, const PathBuffers& paths, const TraceWork& t, bool count, int grid, cudaStream_t stream)
{
    if (count) {
        if (scene.instances) launchTraceOf<true, 1>(scene, paths, t, grid, stream);
        else launchTraceOf<true, 0>(scene, paths, t, grid, stream);
    } else {
        if (scene.instances) launchTraceOf<false, 1>(scene, paths, t, grid, stream);
        else launchTraceOf<false, 0>(scene, paths, t, grid, stream);
    }
}

// Whether the full shade kernels defer subsurface walks to walkKernel: path
// buffers with walk buffers (plain and radiance-cache mode alike).
bool deferWalks(const PathBuffers& paths)
{
    return paths.walkEntry != nullptr && paths.walkNormal != nullptr && paths.walkState != nullptr;
}

void launchShadeGroups(const ShadeVariant& v, const ShadeLaunch& l)
{
    if (v.full) shadeFullGroups(v.lit, l);
    else shadePlainGroups(v.lit, l);
}

void launchShadeSingles(const ShadeVariant& v, const ShadeLaunch& l)
{
    if (!v.full) shadePlainSingles(v.lit, v.cache, l);
    else if (v.lit) shadeFullSinglesLit(v.cache, v.defer, l);
    else shadeFullSinglesUnlit(v.cache, v.defer, l);
}

void launchShadeReplays(const ShadeVariant& v, const ShadeLaunch& l)
{
    if (v.lit) shadeFullReplaysLit(v.cache, l);
    else shadeFullReplaysUnlit(v.cache, l);
}

void renderFrame(const DeviceScene& scene, const FrameConst& frame, const PathBuffers& buffers, FrameBuffers& fb,
                 cudaStream_t stream, StageTimes* timing, bool countTraversal, uint64_t* launches, CacheRun* cacheRun)
{
    PathBuffers paths = buffers;  // what this call's launches get: its counters move from bounce to bounce
    const bool cacheMode = cacheRun != nullptr && cacheRun->cache != nullptr && paths.cache.enabled != 0u;
    if (!cacheMode) paths.cache.enabled = 0u;
    uint64_t launched = 0;
    const uint32_t pixels = frame.width * frame.height;
    const uint64_t wavePaths = paths.wavePaths ? std::min(paths.wavePaths, paths.capacity) : paths.capacity;
    const std::vector<WaveDesc> waves = planWaves(pixels, std::max(frame.sampleCount, 1u), wavePaths);
    const int traceGrid = gridFor(static_cast<uint32_t>(wavePaths), static_cast<int>(std::max(paths.traceBlocksPerSm, 1u)));
    const int shadeGrid = gridFor(static_cast<uint32_t>(wavePaths), static_cast<int>(std::max(paths.shadeBlocksPerSm, 1u)));
    const int replayGrid = gridFor(static_cast<uint32_t>(wavePaths), 8);
    const bool sortHits = paths.sortHits != 0u && paths.sortedHits != nullptr && paths.hitBins != nullptr;
    const bool sortRays = paths.sortRays != 0u;
    // Subsurface walks in walkKernel (scenes that can take them).
    const bool walks = scene.fullShading && scene.hasSubsurface && deferWalks(paths);
    const int sortGrid = std::max(1, gridFor(static_cast<uint32_t>(wavePaths), 8) / 2);  // 256-thread blocks
    std::vector<EventPair> events;
    auto timed = [&](int stage, auto&& launch) {
        if (!timing) {
            launch();
            return;
        }
        EventPair e{};
        e.stage = stage;
        CUDA_OK(cudaEventCreate(&e.start));
        CUDA_OK(cudaEventCreate(&e.stop));
        CUDA_OK(cudaEventRecord(e.start, stream));
        launch();
        CUDA_OK(cudaEventRecord(e.stop, stream));
        events.push_back(e);
    };
    const bool lit = scene.lightCount > 0u && !scene.hasMeshLights;
    paths.lightSlots = lit ? 1u : (scene.hasMeshLights ? 2u : 3u);
    // Lanes travel alone in radiance-cache mode (training paths and queries
    // are per lane) and where walks run inside the shade kernel.
    paths.split = cacheMode || (scene.fullShading && !deferWalks(paths)) ? 1u : 0u;
    // Scenes whose lanes part seldom shade every entry in one launch: entries of
    // one lane are too few for a kernel of their own to pay for its latency
    // (40 us a bounce, a warp's walk through cold instructions).
    paths.merged = !paths.split && scene.partsLanes == 0u ? 1u : 0u;
    // Stage times and traversal counts are those of separate launches.
    const bool fused = timing == nullptr && !countTraversal;
    const ShadeVariant variant{scene.fullShading != 0u, lit, cacheMode, deferWalks(paths)};
    uint32_t* const allCounters = paths.counters;
    auto counter64 = [](uint32_t* set, uint32_t word) { return reinterpret_cast<unsigned long long*>(set + word); };
    // Material order of a hit queue (tuning sort_hits).
    auto sortedByMaterial = [&](const uint32_t* hits, const uint32_t* count) {
        if (!sortHits) return hits;
        CUDA_OK(cudaMemsetAsync(paths.hitBins, 0, 2 * kHitBins * sizeof(uint32_t), stream));
        countHitBinsKernel<<<sortGrid, 256, 0, stream>>>(scene, paths, hits, count);
        scanHitBinsKernel<<<1, 32, 0, stream>>>(paths);
        scatterHitsKernel<<<sortGrid, 256, 0, stream>>>(scene, paths, hits, count);
        launched += 3;
        return static_cast<const uint32_t*>(paths.sortedHits);
    };
    for (const WaveDesc& w : waves) {
        NvtxRange waveRange("hdcx wave");
        if (cacheMode) CUDA_OK(cudaMemsetAsync(paths.cache.counters, 0, 3 * sizeof(uint32_t), stream));
        // (A clear before every bounce was a launch in each: 2 us of its latency.)
        paths.counters = allCounters;
        CUDA_OK(cudaMemsetAsync(allCounters, 0, kCountEnd * sizeof(uint32_t), stream));
        generateKernel<<<(w.count / 3u + 127u) / 128u, 128, 0, stream>>>(frame, w, paths);
        CUDA_OK(cudaGetLastError());
        for (uint32_t bounce = 0; bounce < frame.maxBounces; ++bounce) {
            uint32_t* inQueue = paths.queue[bounce & 1u];
            uint32_t* outQueue = paths.queue[(bounce + 1u) & 1u];
            uint32_t* counters = allCounters + bounce * kCountWords;
            paths.counters = counters;
            unsigned long long* inCount = counter64(counters, kCountQueue);
            unsigned long long* outCount = counter64(counters + kCountWords, kCountQueue);
            const unsigned long long* previousShadows = bounce > 0u ? counter64(counters - kCountWords, kCountShadow) : nullptr;
            if (sortRays && bounce > 0u) {
                sortRaysKernel<<<sortGrid, 256, 0, stream>>>(paths, inQueue, inCount);
                launched += 1;
            }
            timed(0, [&] {
                launchTrace(scene, paths, TraceWork{inQueue, inCount, fused ? previousShadows : nullptr}, countTraversal, traceGrid, stream);
            });
            timed(1, [&] {
                ShadeLaunch launch{scene, frame, paths, bounce, nullptr, nullptr, outQueue, outCount, true, shadeGrid, stream};
                if (!paths.split) {
                    launch.count = counters + (paths.merged ? kCountHits : kCountGroups);
                    launch.queue = sortedByMaterial(paths.merged ? paths.hitQueue : paths.groupQueue, launch.count);
                    launchShadeGroups(variant, launch);
                    launch.misses = false;
                    launched += 1;
                }
                if (!paths.merged) {
                    launch.count = counters + kCountHits;
                    launch.queue = sortedByMaterial(paths.hitQueue, launch.count);
                    launchShadeSingles(variant, launch);
                    launched += 1;
                }
                if (walks) {
                    // The deferred walks (in this bounce's traced extension
                    // queue), then the failed ones re-shaded (queued in the
                    // hit queue, which has been shaded).
                    if (scene.instances) walkKernel<1><<<traceGrid, 128, 0, stream>>>(scene, paths, inQueue, outQueue, outCount, paths.hitQueue);
                    else walkKernel<0><<<traceGrid, 128, 0, stream>>>(scene, paths, inQueue, outQueue, outCount, paths.hitQueue);
                    launch.queue = paths.hitQueue;
                    launch.count = counters + kCountReplays;
                    launch.misses = false;
                    launch.grid = replayGrid;
                    launchShadeReplays(variant, launch);
                    launched += 2;
                }
            });
            CUDA_OK(cudaGetLastError());
            launched += 1;
            if (!fused || bounce + 1u == frame.maxBounces) {
                timed(2, [&] {
                    launchTrace(scene, paths, TraceWork{nullptr, nullptr, counter64(counters, kCountShadow)}, countTraversal, traceGrid, stream);
                });
                launched += 1;
            }
        }
        if (cacheMode) {
            // Predictions for the terminated paths, then one training round on
            // this wave's suffix samples (the next wave sees the update).
            uint32_t counts[3] = {0, 0, 0};
            CUDA_OK(cudaMemcpyAsync(counts, paths.cache.counters, sizeof counts, cudaMemcpyDeviceToHost, stream));
            CUDA_OK(cudaStreamSynchronize(stream));
            nrc::query(cacheRun->cache, paths.cache.queries, counts[0], paths.cache.predictions, stream);
            cacheApplyKernel<<<gridFor(std::max(counts[0], 1u), 8), 128, 0, stream>>>(paths);
            cacheTargetsKernel<<<gridFor(std::max(std::min(counts[1], paths.cache.trainCapacity), 1u), 8), 128, 0, stream>>>(paths);
            CUDA_OK(cudaGetLastError());
            CUDA_OK(cudaMemcpyAsync(counts, paths.cache.counters, sizeof counts, cudaMemcpyDeviceToHost, stream));
            CUDA_OK(cudaStreamSynchronize(stream));
            cacheRun->queries += counts[0];
            cacheRun->samples += counts[2];
            if (counts[2] > 0u) {
                cacheRun->lastLoss = nrc::train(cacheRun->cache, paths.cache.sampleQueries, paths.cache.sampleTargets, counts[2],
                                                cacheRun->trainSteps, stream);
            }
            launched += 2;
        }
        launched += 2;
        const uint32_t blockPixels = kAccumulateThreads / std::min(w.samples, kAccumulateThreads);
        accumulateKernel<<<(w.pixels + blockPixels - 1u) / blockPixels, kAccumulateThreads, 0, stream>>>(frame, w, paths, fb);
        CUDA_OK(cudaGetLastError());
    }
    if (launches) *launches = launched;
    if (timing) {
        CUDA_OK(cudaStreamSynchronize(stream));
        timing->waves = static_cast<uint32_t>(waves.size());
        for (EventPair& e : events) {
            float ms = 0.0f;
            CUDA_OK(cudaEventElapsedTime(&ms, e.start, e.stop));
            if (e.stage == 0) {
                timing->extendMs += ms;
                timing->extendLaunches++;
            } else if (e.stage == 1) {
                timing->shadeMs += ms;
            } else {
                timing->shadowMs += ms;
            }
            cudaEventDestroy(e.start);
            cudaEventDestroy(e.stop);
        }
    }
}

__global__ void upscaleNearestKernel(const float4* src, uint32_t srcWidth, uint32_t srcHeight, float4* dst,
                                     uint32_t width, uint32_t height)
{
    const uint64_t pixel = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (pixel >= uint64_t(width) * height) return;
    const uint32_t x = static_cast<uint32_t>(pixel % width), y = static_cast<uint32_t>(pixel / width);
    // render_pass.cpp:55-60: source = min(size - 1, destination * size / destinationSize).
    const uint32_t sy = static_cast<uint32_t>(min(uint64_t(srcHeight - 1u), uint64_t(y) * srcHeight / height));
    const uint32_t sx = static_cast<uint32_t>(min(uint64_t(srcWidth - 1u), uint64_t(x) * srcWidth / width));
    dst[pixel] = src[uint64_t(sy) * srcWidth + sx];
}

void launchUpscaleNearest(const float4* src, uint32_t srcWidth, uint32_t srcHeight, float4* dst, uint32_t width,
                          uint32_t height, cudaStream_t stream)
{
    const uint64_t pixels = uint64_t(width) * height;
    if (pixels == 0 || srcWidth == 0 || srcHeight == 0) return;
    upscaleNearestKernel<<<static_cast<unsigned>((pixels + 255u) / 256u), 256, 0, stream>>>(src, srcWidth, srcHeight, dst,
                                                                                          width, height);
    CUDA_OK(cudaGetLastError());
}

// One level of a texture's mip pyramid: each texel the mean of the 2x2
// texels below it (the last row / column reused for odd sizes), level 0
// decoded to linear RGBA (sRGB through the sampler's table).
__global__ void mipLevelKernel(TexDesc t, const float4* below, uint32_t bw, uint32_t bh, float4* out, uint32_t w, uint32_t h)
{
    const uint64_t i = uint64_t(blockIdx.x) * blockDim.x + threadIdx.x;
    if (i >= uint64_t(w) * h) return;
    const uint32_t x = static_cast<uint32_t>(i % w), y = static_cast<uint32_t>(i / w);
    const uint32_t x0 = min(2u * x, bw - 1u), x1 = min(2u * x + 1u, bw - 1u);
    const uint32_t y0 = min(2u * y, bh - 1u), y1 = min(2u * y + 1u, bh - 1u);
    float4 a, b, c, d;
    if (below == nullptr) {
        a = texelFetch(t, static_cast<int>(x0), static_cast<int>(y0));
        b = texelFetch(t, static_cast<int>(x1), static_cast<int>(y0));
        c = texelFetch(t, static_cast<int>(x0), static_cast<int>(y1));
        d = texelFetch(t, static_cast<int>(x1), static_cast<int>(y1));
    } else {
        a = below[size_t(y0) * bw + x0];
        b = below[size_t(y0) * bw + x1];
        c = below[size_t(y1) * bw + x0];
        d = below[size_t(y1) * bw + x1];
    }
    out[i] = make_float4(((a.x + b.x) + (c.x + d.x)) * 0.25f, ((a.y + b.y) + (c.y + d.y)) * 0.25f,
                         ((a.z + b.z) + (c.z + d.z)) * 0.25f, ((a.w + b.w) + (c.w + d.w)) * 0.25f);
}

uint64_t mipTexels(uint32_t width, uint32_t height, uint32_t& levels)
{
    uint64_t total = 0;
    levels = 1;
    uint32_t w = width, h = height;
    while (w > 1u || h > 1u) {
        w = std::max(1u, w >> 1);
        h = std::max(1u, h >> 1);
        total += uint64_t(w) * h;
        ++levels;
    }
    return total;
}

void buildMips(TexDesc& desc, float4* mips, cudaStream_t stream)
{
    uint32_t levels = 1;
    mipTexels(desc.width, desc.height, levels);
    uint32_t bw = desc.width, bh = desc.height;
    const float4* below = nullptr;
    float4* out = mips;
    for (uint32_t k = 1; k < levels; ++k) {
        const uint32_t w = std::max(1u, bw >> 1), h = std::max(1u, bh >> 1);
        const uint64_t n = uint64_t(w) * h;
        mipLevelKernel<<<static_cast<unsigned>((n + 255u) / 256u), 256, 0, stream>>>(desc, below, bw, bh, out, w, h);
        CUDA_OK(cudaGetLastError());
        below = out;
        out += n;
        bw = w;
        bh = h;
    }
    desc.mips = mips;
    desc.levels = levels;
}

void tracePrimary(const DeviceScene& scene, const FrameConst& frame, uint32_t sampleNumber, uint32_t* primitives,
                  float* distances, cudaStream_t stream)
{
    const uint32_t pixels = frame.width * frame.height;
    primaryKernel<<<(pixels + 127u) / 128u, 128, 0, stream>>>(scene, frame, sampleNumber, primitives, distances);
    CUDA_OK(cudaGetLastError());
}

}  // namespace hdcx
