// The device intrinsics csrc/arap_device.cuh calls, for a host compiler. Include
// before it. Warp shuffles are there to compile only.
#pragma once

#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstdint>
#include <cstring>

template <typename To, typename From> inline To bits_as(From x) {
    static_assert(sizeof(To) == sizeof(From), "same size");
    To y;
    std::memcpy(&y, &x, sizeof y);
    return y;
}
inline int __double2hiint(double x) { return (int)(bits_as<uint64_t>(x) >> 32); }
inline int __double2loint(double x) { return (int)bits_as<uint64_t>(x); }
inline double __hiloint2double(int h, int l) { return bits_as<double>((uint64_t)(uint32_t)h << 32 | (uint32_t)l); }
inline long long __double_as_longlong(double x) { return bits_as<long long>(x); }
inline float __uint_as_float(unsigned x) { return bits_as<float>(x); }
inline unsigned __float_as_uint(float x) { return bits_as<unsigned>(x); }
inline float rsqrtf(float x) { return 1.0f / std::sqrt(x); }
inline float __fdividef(float a, float b) { return a / b; }
template <typename T> inline T __shfl_sync(unsigned, T x, int) { return x; }
template <typename T> inline T __shfl_xor_sync(unsigned, T x, int) { return x; }
using std::fabs;
using std::max;
using std::sqrt;
