// Unit tests of hdcx::boundedWave (hdcodex_b200/csrc/wave_plan.h): an
// automatic wave and the device memory that is free. Prints one line per
// failed check and exits non-zero if any failed.
#include "wave_plan.h"

#include <cstdio>

int main()
{
    using namespace hdcx;
    int failures = 0;
    auto expect = [&](bool ok, const char* what, uint64_t a, uint64_t b) {
        if (ok) return;
        std::printf("FAILED %s: free %llu held %llu\n", what, static_cast<unsigned long long>(a), static_cast<unsigned long long>(b));
        ++failures;
    };
    constexpr uint64_t kWave = 12ull << 20;
    for (uint64_t mib = 0; mib <= 16384; mib += 37) {
        for (uint64_t held : {0ull, 5ull, 70000ull, 1000000ull, 12ull << 20, 48ull << 20}) {
            const uint64_t freeBytes = mib << 20;
            const uint64_t wave = boundedWave(kWave, freeBytes, held);
            const uint64_t bound = (freeBytes + held * kPathStateBytes) / 4 * 3;
            expect(wave <= kWave, "at most the wave asked for", freeBytes, held);
            expect(wave >= kMinimumAutomaticWave, "at least the smallest wave", freeBytes, held);
            // Three quarters of free and held memory, unless the smallest wave or the held buffers are more.
            if (wave > kMinimumAutomaticWave && wave > held) expect(wave * kPathStateBytes <= bound, "memory of the wave", freeBytes, held);
            // And no less than fits: one path more would not, or was not asked for.
            if (wave < kWave) expect((wave + 1) * kPathStateBytes > bound, "memory left over", freeBytes, held);
            if (held >= kWave) expect(wave == kWave, "held buffers serve as they are", freeBytes, held);
        }
    }
    if (boundedWave(3, 0, 0) != 3) expect(false, "a wave below the smallest is kept", 0, 0);
    if (failures == 0) std::printf("all wave plan checks passed\n");
    return failures != 0;
}
