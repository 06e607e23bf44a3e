// What a kernel of warp operations needs to run on the host: the 32 lanes of a
// warp are threads, and each warp operation is a meeting of all of them. One
// warp at a time; __shared__ is static.
#pragma once

#include <stdint.h>

#include <algorithm>
#include <barrier>
#include <cmath>
#include <cstring>
#include <thread>
#include <vector>

struct float4 {
    float x, y, z, w;
};
struct uint4 {
    uint32_t x, y, z, w;
};
struct Dim {
    uint32_t x;
};
inline float4 make_float4(float x, float y, float z, float w) { return {x, y, z, w}; }
inline uint4 make_uint4(uint32_t x, uint32_t y, uint32_t z, uint32_t w) { return {x, y, z, w}; }

inline thread_local Dim threadIdx{0}, blockIdx{0};
inline std::barrier<> warp_meet(32);
inline uint64_t warp_slot[32];

#define __global__ static
#define __device__
#define __host__
#define __shared__ static
#define __forceinline__ inline
#define __noinline__
#define __launch_bounds__(...)

using std::max;
using std::min;

template <class T>
T __ldg(const T* p) {
    return *p;
}
inline uint32_t __float_as_uint(float f) {
    uint32_t u;
    std::memcpy(&u, &f, 4);
    return u;
}
inline float __uint_as_float(uint32_t u) {
    float f;
    std::memcpy(&f, &u, 4);
    return f;
}
inline int __popc(uint32_t x) { return __builtin_popcount(x); }
inline int __ffs(uint32_t x) { return __builtin_ffs((int)x); }

// f(slots) of every lane's value, the same in all lanes.
template <class T, class F>
auto warp_all(T v, const F& f) {
    uint64_t word = 0;
    std::memcpy(&word, &v, sizeof v);
    warp_slot[threadIdx.x & 31u] = word;
    warp_meet.arrive_and_wait();
    T all[32];
    for (int k = 0; k < 32; k++) std::memcpy(&all[k], &warp_slot[k], sizeof v);
    const auto r = f(all);
    warp_meet.arrive_and_wait();
    return r;
}
inline void __syncwarp() { warp_meet.arrive_and_wait(); }
inline uint32_t __ballot_sync(uint32_t, bool p) {
    return warp_all(p, [](const bool* a) {
        uint32_t m = 0;
        for (int k = 0; k < 32; k++) m |= (a[k] ? 1u : 0u) << k;
        return m;
    });
}
inline uint32_t __reduce_min_sync(uint32_t, uint32_t v) {
    return warp_all(v, [](const uint32_t* a) { return *std::min_element(a, a + 32); });
}
inline uint32_t __reduce_max_sync(uint32_t, uint32_t v) {
    return warp_all(v, [](const uint32_t* a) { return *std::max_element(a, a + 32); });
}
template <class T>
T __shfl_sync(uint32_t, T v, int from) {
    return warp_all(v, [&](const T* a) { return a[from & 31]; });
}
template <class T>
T __shfl_xor_sync(uint32_t, T v, int with) {
    return warp_all(v, [&](const T* a) { return a[(threadIdx.x ^ (uint32_t)with) & 31u]; });
}
inline uint32_t atomicMax(uint32_t* p, uint32_t v) {
    const uint32_t old = *p;
    *p = std::max(old, v);
    return old;
}

// kernel() run by the 32 lanes of one warp.
template <class F>
void run_warp(const F& kernel) {
    std::vector<std::thread> lanes;
    for (uint32_t l = 0; l < 32; l++)
        lanes.emplace_back([&, l] {
            threadIdx.x = l;
            kernel();
        });
    for (auto& t : lanes) t.join();
}
