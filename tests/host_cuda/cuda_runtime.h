// Host stand-in for <cuda_runtime.h>: what the device headers of pyclaw_b200/csrc
// use, so that tests compile them with a C++ compiler and run them without a GPU.
//
// emu::run_cta runs one CTA, a host thread per CUDA thread.  Barriers are
// pthread barriers and shuffles go through a slot per lane between two of them,
// so a thread sanitizer sees the order that the device code asks for, and reports
// accesses to shared memory that nothing orders.
#pragma once

#include <pthread.h>

#include <algorithm>
#include <atomic>
#include <cmath>
#include <cstdint>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <string>
#include <thread>
#include <vector>

#define __CUDACC__ 1
#define __host__
#define __device__
#define __global__
#define __shared__ static
#define __forceinline__ inline
#define __noinline__ __attribute__((noinline))      // after the standard headers, which use the name

using std::copysign; using std::fabs; using std::fmax; using std::fmin; using std::isfinite; using std::max; using std::min;
using std::sqrt;

struct uint3 { unsigned x, y, z; };
struct double2 { double x, y; };
inline double2 make_double2(double x, double y) { return double2{x, y}; }

inline thread_local uint3 threadIdx, blockIdx, blockDim, gridDim;

namespace emu {

struct Warp { pthread_barrier_t bar; uint64_t slot[32]; };
struct Cta { pthread_barrier_t bar; std::vector<Warp> warps; std::atomic<int> any; };
inline thread_local Cta* cta = nullptr;

inline void warp_sync() { pthread_barrier_wait(&cta->warps[threadIdx.x / 32].bar); }
inline uint64_t from_lane(uint64_t v, int lane)
{
    Warp& w = cta->warps[threadIdx.x / 32];
    w.slot[threadIdx.x & 31] = v;
    warp_sync();
    const uint64_t r = lane >= 0 && lane < 32 ? w.slot[lane] : v;
    warp_sync();
    return r;
}
inline int cta_any(bool p)
{
    pthread_barrier_wait(&cta->bar);
    if (p) cta->any = 1;
    pthread_barrier_wait(&cta->bar);
    const int r = cta->any;
    pthread_barrier_wait(&cta->bar);
    cta->any = 0;
    return r;
}

template <class F> void run_cta(int threads, F body)
{
    Cta c;
    c.any = 0;
    c.warps = std::vector<Warp>(threads / 32);
    pthread_barrier_init(&c.bar, nullptr, threads);
    for (Warp& w : c.warps) pthread_barrier_init(&w.bar, nullptr, 32);
    std::vector<std::thread> ts;
    for (int t = 0; t < threads; t++)
        ts.emplace_back([&, t] {
            cta = &c;
            threadIdx = uint3{(unsigned)t, 0, 0};
            blockDim = uint3{(unsigned)threads, 1, 1};
            gridDim = uint3{1, 1, 1};
            body();
        });
    for (std::thread& t : ts) t.join();
}

// Errors of the hardware's approximations of 1/y and 1/sqrt(x): they have 20 bits
// behind the binary point; `seed_error` moves them further off (relative).
inline double seed_error = 0.0;
inline double high_word(double r)
{
    uint64_t b;
    std::memcpy(&b, &r, 8);
    b &= 0xffffffff00000000ULL;
    std::memcpy(&r, &b, 8);
    return r;
}
inline double rcp_seed(double y) { return high_word(1.0 / y * (1.0 + seed_error)); }
inline double rsqrt_seed(double x) { return high_word(1.0 / std::sqrt(x) * (1.0 + seed_error)); }

}  // namespace emu

inline long long __double_as_longlong(double v) { long long b; std::memcpy(&b, &v, 8); return b; }
inline double __longlong_as_double(long long b) { double v; std::memcpy(&v, &b, 8); return v; }
inline int __double2hiint(double v) { return (int)(__double_as_longlong(v) >> 32); }
inline int __double2loint(double v) { return (int)__double_as_longlong(v); }
inline double __hiloint2double(int hi, int lo) { return __longlong_as_double(((long long)hi << 32) | (unsigned)lo); }
inline double __fma_rn(double a, double b, double c) { return std::fma(a, b, c); }
template <class T> inline T __ldg(const T* p) { return *p; }
inline long long clock64() { return 0; }
inline unsigned __cvta_generic_to_shared(const void*) { return 0; }

inline void __syncwarp() { emu::warp_sync(); }
inline void __syncthreads() { pthread_barrier_wait(&emu::cta->bar); }
inline int __syncthreads_or(int p) { return emu::cta_any(p != 0); }
inline int __syncthreads_and(int p) { return !emu::cta_any(p == 0); }
inline void __threadfence() { std::atomic_thread_fence(std::memory_order_seq_cst); }
template <class T> inline T emu_shfl(T v, int lane)
{
    uint64_t b = 0;
    std::memcpy(&b, &v, sizeof v);
    b = emu::from_lane(b, lane);
    std::memcpy(&v, &b, sizeof v);
    return v;
}
template <class T> inline T __shfl_sync(unsigned, T v, int lane) { return emu_shfl(v, lane); }
template <class T> inline T __shfl_up_sync(unsigned, T v, int d) { return emu_shfl(v, (int)(threadIdx.x & 31) - d); }
template <class T> inline T __shfl_down_sync(unsigned, T v, int d) { return emu_shfl(v, (int)(threadIdx.x & 31) + d); }
template <class T> inline T __shfl_xor_sync(unsigned, T v, int m) { return emu_shfl(v, (int)(threadIdx.x & 31) ^ m); }
inline int __any_sync(unsigned, int p)
{
    emu::Warp& w = emu::cta->warps[threadIdx.x / 32];
    w.slot[threadIdx.x & 31] = p != 0;
    emu::warp_sync();
    int r = 0;
    for (uint64_t s : w.slot) r |= (int)s;
    emu::warp_sync();
    return r;
}
inline int __all_sync(unsigned m, int p) { return !__any_sync(m, p == 0); }
template <class T> inline T atomicAdd(T* p, T v) { return __atomic_fetch_add(p, v, __ATOMIC_SEQ_CST); }
template <class T> inline T atomicExch(T* p, T v) { return __atomic_exchange_n(p, v, __ATOMIC_SEQ_CST); }
template <class T> inline T atomicMax(T* p, T v)
{
    T old = __atomic_load_n(p, __ATOMIC_SEQ_CST);
    while (old < v && !__atomic_compare_exchange_n(p, &old, v, false, __ATOMIC_SEQ_CST, __ATOMIC_SEQ_CST)) {}
    return old;
}
