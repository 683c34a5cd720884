// The conversions on the integer pipe (csrc/arap_device.cuh) on the host,
// against the conversions of the language: the same value for every class of
// argument, bit for bit but for a NaN's payload.
#include <cstdio>
#include <limits>
#include <random>
#include <vector>

#include "device_on_host.h"

#include "arap_device.cuh"

using namespace arapgpu;

namespace {

int failures = 0;
template <typename T> void same(const char *what, double x, T got, T want) {
    const bool ok = want != want ? got != got : std::memcmp(&got, &want, sizeof got) == 0;
    if (!ok && ++failures < 20) std::printf("%s of %a: %a, not %a\n", what, x, (double)got, (double)want);
}

}  // namespace

int main() {
    constexpr float inf = std::numeric_limits<float>::infinity();
    std::vector<float> f = {0.f, 1.f, 1.5f, 0x1.fffffep127f, 0x1p-126f, 0x1.fffffcp-127f, 0x1p-149f, 0x1.8p-130f, inf,
                            std::numeric_limits<float>::quiet_NaN(), 0x1.fffffep-1f, 0x1p-125f};
    std::mt19937_64 rng(3);
    for (int i = 0; i < 200000; ++i) f.push_back(bits_as<float>((uint32_t)rng() & 0x7fffffffu));
    for (const float x : f)
        for (const float s : {x, -x}) {
            same("to_double", s, dev::to_double(s), (double)s);
            if (std::fabs(s) < inf) same("to_double_finite", s, dev::to_double_finite(s), std::fabs(s) < 0x1p-126f ? 0.0 * (double)s : (double)s);
        }
    std::vector<double> d = {0x1.ffffffp127, 0x1.fffffefp127, 0x1.fffffffp127, 0x1p128, 1e300, 0x1.ffffffp-127, 0x1p-126,
                             0x1p-150, 0x1p-1074, 1.0, 0x1.000001p0, 0x1.000003p0, 0x1.0000010000001p0, 0.0, (double)inf,
                             std::numeric_limits<double>::quiet_NaN()};
    for (int i = 0; i < 200000; ++i) d.push_back(bits_as<double>(rng() & 0x7fffffffffffffffull));
    for (int i = 0; i < 200000; ++i) d.push_back((double)bits_as<float>((uint32_t)rng() & 0x7f7fffffu) * (1.0 + 0x1p-40 * (double)(rng() >> 40)));
    for (const double x : d)
        for (const double s : {x, -x}) same("to_float_rn", s, dev::to_float_rn(s), (float)s);
    std::printf(failures ? "failed\n" : "ok\n");
    return failures ? 1 : 0;
}
