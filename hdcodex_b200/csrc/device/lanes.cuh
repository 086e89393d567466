// lanes.cuh - one value per wavelength lane of a sample.
//
// The three wavelength lanes of a sample start from the same seed, so they
// meet the same hits and draw the same directions until a decision that
// depends on a lane's own value (a lobe probability, roulette, a dispersed
// refraction) parts them. Lanes that are still together are shaded by one
// thread: what does not depend on the wavelength is one float, what does is a
// Lanes3. Shading functions are templates over that type (V): float for a
// single lane, Lanes3 for three. Every operator is the binary32 operation of
// the scalar code per component, in the same order, so both forms give the
// same bits.
#pragma once

#include "common.cuh"

namespace hdcx {

struct Lanes3 {
    float x, y, z;
    Lanes3() = default;
    HDCX_D Lanes3(float s) : x(s), y(s), z(s) {}
    HDCX_D Lanes3(float a, float b, float c) : x(a), y(b), z(c) {}
};

HDCX_D Lanes3 operator+(Lanes3 a, Lanes3 b) { return Lanes3(a.x + b.x, a.y + b.y, a.z + b.z); }
HDCX_D Lanes3 operator-(Lanes3 a, Lanes3 b) { return Lanes3(a.x - b.x, a.y - b.y, a.z - b.z); }
HDCX_D Lanes3 operator*(Lanes3 a, Lanes3 b) { return Lanes3(a.x * b.x, a.y * b.y, a.z * b.z); }
HDCX_D Lanes3 operator/(Lanes3 a, Lanes3 b) { return Lanes3(a.x / b.x, a.y / b.y, a.z / b.z); }
HDCX_D Lanes3 gmin(Lanes3 a, Lanes3 b) { return Lanes3(gmin(a.x, b.x), gmin(a.y, b.y), gmin(a.z, b.z)); }
HDCX_D Lanes3 gmax(Lanes3 a, Lanes3 b) { return Lanes3(gmax(a.x, b.x), gmax(a.y, b.y), gmax(a.z, b.z)); }
HDCX_D Lanes3 clampf(Lanes3 v, float lo, float hi) { return gmin(gmax(v, Lanes3(lo)), Lanes3(hi)); }
HDCX_D Lanes3 mix(Lanes3 x, Lanes3 y, float a) { return x * Lanes3(1.0f - a) + y * Lanes3(a); }
HDCX_D Lanes3 mix(Lanes3 x, Lanes3 y, Lanes3 a) { return x * (Lanes3(1.0f) - a) + y * a; }
HDCX_D Lanes3 luminance1(Lanes3 s) { return Lanes3(luminance1(s.x), luminance1(s.y), luminance1(s.z)); }

// Number of lanes of V, and the matching unsigned type.
template <class V>
struct LaneTraits;
template <>
struct LaneTraits<float> {
    static constexpr int kCount = 1;
    using U = uint32_t;
};
template <>
struct LaneTraits<Lanes3> {
    static constexpr int kCount = 3;
    using U = uint3;
};

// Component k; a constant k (unrolled loops) keeps the value in registers, a
// variable one selects.
HDCX_D float at(float v, int) { return v; }
HDCX_D float at(const Lanes3& v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }
HDCX_D uint32_t at(uint32_t v, int) { return v; }
HDCX_D uint32_t at(const uint3& v, int k) { return k == 0 ? v.x : (k == 1 ? v.y : v.z); }
HDCX_D void put(float& v, int, float s) { v = s; }
HDCX_D void put(Lanes3& v, int k, float s)
{
    if (k == 0) v.x = s;
    else if (k == 1) v.y = s;
    else v.z = s;
}
HDCX_D void put(uint32_t& v, int, uint32_t s) { v = s; }
HDCX_D void put(uint3& v, int k, uint32_t s)
{
    if (k == 0) v.x = s;
    else if (k == 1) v.y = s;
    else v.z = s;
}

// Bit k set where component k satisfies the comparison.
HDCX_D uint32_t maskGreater(float a, float b) { return a > b ? 1u : 0u; }
HDCX_D uint32_t maskGreater(Lanes3 a, Lanes3 b) { return (a.x > b.x ? 1u : 0u) | (a.y > b.y ? 2u : 0u) | (a.z > b.z ? 4u : 0u); }
HDCX_D uint32_t maskLess(float a, float b) { return a < b ? 1u : 0u; }
HDCX_D uint32_t maskLess(Lanes3 a, Lanes3 b) { return maskGreater(b, a); }
HDCX_D bool allZero(float v) { return v == 0.0f; }
HDCX_D bool allZero(Lanes3 v) { return v.x == 0.0f && v.y == 0.0f && v.z == 0.0f; }
HDCX_D float whereMask(uint32_t m, float a, float b) { return (m & 1u) ? a : b; }
HDCX_D Lanes3 whereMask(uint32_t m, Lanes3 a, Lanes3 b)
{
    return Lanes3((m & 1u) ? a.x : b.x, (m & 2u) ? a.y : b.y, (m & 4u) ? a.z : b.z);
}

// a / b where both are often equal (finite and positive, so the quotient is
// exactly one): the comparison spares most warps the divisions.
HDCX_D bool exactlyOne(float a, float b) { return a == b && a > 0.0f && a < INFINITY; }
HDCX_D float ratioLikelyOne(float a, float b) { return exactlyOne(a, b) ? 1.0f : a / b; }
HDCX_D Lanes3 ratioLikelyOne(Lanes3 a, Lanes3 b)
{
    if (exactlyOne(a.x, b.x) && exactlyOne(a.y, b.y) && exactlyOne(a.z, b.z)) return Lanes3(1.0f);
    return a / b;
}
// a / b where b is often one.
HDCX_D float overLikelyOne(float a, float b) { return b == 1.0f ? a : a / b; }
HDCX_D Lanes3 overLikelyOne(Lanes3 a, Lanes3 b)
{
    if (b.x == 1.0f && b.y == 1.0f && b.z == 1.0f) return a;
    return a / b;
}

// x * (1 - a) + y * a of a wavelength-independent pair by a lane value.
HDCX_D float mixBy(float x, float y, float a) { return mix(x, y, a); }
HDCX_D Lanes3 mixBy(float x, float y, Lanes3 a) { return mix(Lanes3(x), Lanes3(y), a); }

HDCX_D float dispersed(float iorAtD, float b, float a, float scale, float wavelength)
{
    const float cauchyIor = a + b / (wavelength * wavelength);
    return mix(iorAtD, cauchyIor, clampf(scale, 0.0f, 1.0f));
}
HDCX_D Lanes3 dispersed(float iorAtD, float b, float a, float scale, Lanes3 w)
{
    return Lanes3(dispersed(iorAtD, b, a, scale, w.x), dispersed(iorAtD, b, a, scale, w.y), dispersed(iorAtD, b, a, scale, w.z));
}

}  // namespace hdcx
