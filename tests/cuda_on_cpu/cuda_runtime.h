// Enough of the CUDA language to compile a kernel's source with g++ and run
// one CTA of it on host threads, a thread for each CUDA thread: the warp votes
// and shuffles of full warps and __syncthreads are barriers.  With it a test
// can give a kernel buffers that end at an unreadable page, so that an access
// out of range is seen on the CPU.
#pragma once

#include <stddef.h>
#include <stdint.h>

#include <barrier>
#include <memory>
#include <thread>
#include <vector>

#define __device__
#define __host__
#define __global__
#define __forceinline__ inline
#define __launch_bounds__(...)
#define __restrict__
#define __shared__ static   // one CTA at a time

using cudaStream_t = void *;
using cudaError_t = int;

struct Dim3 {
    unsigned x = 0, y = 0, z = 0;
};
inline thread_local Dim3 threadIdx;
inline Dim3 blockIdx, blockDim, gridDim;

struct CpuWarp {
    std::barrier<> bar{32};
    uint32_t word[32] = {};
};
inline std::vector<std::unique_ptr<CpuWarp>> cpu_warps;
inline std::unique_ptr<std::barrier<>> cpu_cta;

inline void __syncthreads() { cpu_cta->arrive_and_wait(); }

inline uint32_t __shfl_sync(uint32_t, uint32_t v, int src) {
    CpuWarp &w = *cpu_warps[threadIdx.x / 32];
    w.word[threadIdx.x % 32] = v;
    w.bar.arrive_and_wait();
    const uint32_t r = w.word[src & 31];
    w.bar.arrive_and_wait();
    return r;
}
inline uint32_t __ballot_sync(uint32_t, bool p) {
    CpuWarp &w = *cpu_warps[threadIdx.x / 32];
    w.word[threadIdx.x % 32] = p;
    w.bar.arrive_and_wait();
    uint32_t r = 0;
    for (int i = 0; i < 32; ++i) r |= w.word[i] << i;
    w.bar.arrive_and_wait();
    return r;
}
inline int __ffs(uint32_t x) { return __builtin_ffs((int)x); }

// CTA `block` of `grid` CTAs of `threads` (a multiple of 32).
template <class F>
void run_cta(unsigned block, unsigned grid, unsigned threads, F kernel) {
    blockIdx.x = block;
    gridDim.x = grid;
    blockDim.x = threads;
    cpu_warps.clear();
    for (unsigned w = 0; w < threads / 32; ++w) cpu_warps.push_back(std::make_unique<CpuWarp>());
    cpu_cta = std::make_unique<std::barrier<>>(threads);
    std::vector<std::thread> t;
    for (unsigned i = 0; i < threads; ++i)
        t.emplace_back([i, &kernel] {
            threadIdx.x = i;
            kernel();
        });
    for (auto &x : t) x.join();
}
