// dev::Split (csrc/arap_device.cuh) on the host: differences of doubles formed
// in FP32 against the rounded FP64 difference.
#include <cstdio>
#include <limits>
#include <random>
#include <vector>

#include "device_on_host.h"

#include "arap_device.cuh"

using namespace arapgpu;

namespace {

int failures = 0;
// NaN where an operand is outside [2^-76, 2^128) and not zero, else the
// difference within `ulps` units of 2^-24
void check(double a, double b, double ulps) {
    const float got = dev::Split(a) - dev::Split(b);
    const double want = a - b;
    const auto outside = [](double x) { return !(std::fabs(x) < 0x1p128) || (std::fabs(x) < 0x1p-76 && std::fabs(x) >= 0x1p-1022); };
    const bool ok = outside(a) || outside(b) ? got != got
                                             : std::fabs((double)got - want) <= ulps * 0x1p-24 * std::fabs(want);
    if (!ok && ++failures < 20) std::printf("%a - %a: %a, not %a\n", a, b, (double)got, want);
}

}  // namespace

int main() {
    // half a unit of the result, and what the roundings of the lower parts leave
    constexpr double ulps = 1.001;
    const double inf = std::numeric_limits<double>::infinity();
    const std::vector<double> special = {0.0, 1.0, 0x1.fffffffffffffp0, 0x1p-76, 0x1.fffffffffffffp-77, 0x1p-1022, 0x1p127,
                                         0x1.fffffffffffffp126, 0x1p128, 1e40, 1e300, inf,
                                         std::numeric_limits<double>::quiet_NaN(), -1.0, -0x1p-80, -1e40, -inf};
    for (const double a : special)
        for (const double b : special)
            if (!(std::fabs(a - b) >= 0x1p127 && std::fabs(a - b) < inf)) check(a, b, ulps);
    std::mt19937_64 rng(5);
    auto unit = [&] { return (double)(rng() >> 11) * 0x1p-53; };
    for (int i = 0; i < 2000000; ++i) {
        // coordinates of any magnitudes, and neighbours at any distance
        const double a = (unit() - 0.5) * std::pow(2.0, (int)(rng() % 40) - 20);
        const double b = i % 2 ? (unit() - 0.5) * std::pow(2.0, (int)(rng() % 40) - 20)
                               : a + (unit() - 0.5) * std::pow(10.0, -(double)(rng() % 9));
        check(a, b, ulps);
    }
    for (int i = 0; i < 2000000; ++i) {  // on both sides of a power of two, and of zero
        const double c = std::pow(2.0, (int)(rng() % 9) - 4), s = std::pow(2.0, -(double)(rng() % 50));
        check(c * (1.0 + s * unit()), c * (1.0 - s * unit()), ulps);
        check(c * s * unit(), -c * s * unit(), ulps);
    }
    std::printf(failures ? "failed\n" : "ok\n");
    return failures ? 1 : 0;
}
