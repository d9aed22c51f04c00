// The CUDA names that the advection tiles use, as host C++: a block runs as one
// std::thread per CUDA thread (host_tile.cpp). Only what the headers need.
#pragma once
#include <algorithm>
#include <atomic>
#include <barrier>
#include <cmath>
#include <cstdint>
#include <cstring>

#define __device__
#define __global__
#define __shared__
#define __grid_constant__
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))
#define __launch_bounds__(...)

using std::max;
using std::min;

struct dim3 { unsigned x = 1, y = 1, z = 1; };
inline thread_local dim3 threadIdx;

// One block's barriers. Every barrier in the source is a site of its own (the instantiations of a template are
// different sites): CUDA lets the threads of a block meet only at the same one.
struct HostBlock {
    std::barrier<> all;
    std::atomic<const void *> site{nullptr};
    std::atomic<int> mixed{0};
    struct Warp {
        std::barrier<> lanes{32};
        std::atomic<unsigned> votes{0};
    } *warps;
    HostBlock(int threads) : all(threads), warps(new Warp[threads / 32]) {}
    ~HostBlock() { delete[] warps; }
};
inline thread_local HostBlock *host_block = nullptr;

inline void host_syncthreads(const void *site) {
    const void *none = nullptr;
    if (!host_block->site.compare_exchange_strong(none, site) && none != site) host_block->mixed = 1;
    host_block->all.arrive_and_wait();
    host_block->site = nullptr;
    host_block->all.arrive_and_wait();
}
#define __syncthreads() do { static const char site = 0; host_syncthreads(&site); } while (0)

inline int __any_sync(unsigned, bool p) {
    HostBlock::Warp &w = host_block->warps[threadIdx.y];
    if (p) w.votes |= 1u;
    w.lanes.arrive_and_wait();
    const int r = w.votes != 0;
    w.lanes.arrive_and_wait();
    w.votes = 0;
    w.lanes.arrive_and_wait();
    return r;
}

template <class T> inline T __ldg(const T *p) { return *p; }
inline long long __double_as_longlong(double d) { long long x; std::memcpy(&x, &d, 8); return x; }
inline double __longlong_as_double(long long x) { double d; std::memcpy(&d, &x, 8); return d; }
inline int __double2hiint(double d) { return (int)(__double_as_longlong(d) >> 32); }
inline int __double2loint(double d) { return (int)__double_as_longlong(d); }
inline double __hiloint2double(int hi, int lo) { return __longlong_as_double(((long long)hi << 32) | (unsigned)lo); }
inline double __dadd_rn(double a, double b) { return a + b; }
inline double __dmul_rn(double a, double b) { return a * b; }
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
inline int __clzll(long long x) { return x == 0 ? 64 : __builtin_clzll((unsigned long long)x); }
inline long long __mul64hi(long long a, long long b) { return (long long)(((__int128)a * b) >> 64); }
inline int __vimax3_s32(int a, int b, int c) { return max(max(a, b), c); }

using cudaError_t = int;
using cudaStream_t = void *;
constexpr int cudaSuccess = 0, cudaDevAttrMultiProcessorCount = 0, cudaFuncAttributeMaxDynamicSharedMemorySize = 0;
inline int cudaGetDevice(int *device) { return *device = 0; }
inline int cudaDeviceGetAttribute(int *value, int, int) { return *value = 152, cudaSuccess; }
inline int cudaFuncSetAttribute(const void *, int, int) { return cudaSuccess; }
